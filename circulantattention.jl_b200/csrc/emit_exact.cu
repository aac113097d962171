// Units of exactly 8, 16, 32 or 64 real channels.
#define CA_ANY_CHANNELS 0
#include "emit_sweep.cuh"
