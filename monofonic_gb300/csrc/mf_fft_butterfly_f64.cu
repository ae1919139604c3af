// Instantiation unit: forward N-grid passes with FP64 butterflies.
#define MF_T double
#define MF_PART_BUTTERFLY
#include "mf_launch_impl.cuh"
