// Units of any other channel count and short last columns, with A's values.
#define CA_ANY_CHANNELS 1
#define CA_FWD_VALUES 1
#include "fwd_sweep.cuh"
