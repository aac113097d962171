// Units of any other channel count up to 64.
#define CA_ANY_CHANNELS 1
#include "emit_sweep.cuh"
