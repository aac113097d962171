// Units of exactly 8, 16, 32 or 64 real channels, with A's values.
#define CA_ANY_CHANNELS 0
#define CA_FWD_VALUES 1
#include "fwd_sweep.cuh"
