// The FP64 mover for calls with few particles: eight lanes per particle.
#define GPAT_FP64_TEAM 8
#include "mover_fp64.cu"
