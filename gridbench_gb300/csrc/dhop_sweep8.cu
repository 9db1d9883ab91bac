// The sweep form of the FP32 hopping kernel for rows (or tiles) of 8 slices.
#define SWEEP_TE 8
#include "dhop_sweep.inl"
