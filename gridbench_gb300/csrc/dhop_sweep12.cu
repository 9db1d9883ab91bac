// The sweep form of the FP32 hopping kernel for rows (or tiles) of 12 slices.
#define SWEEP_TE 12
#include "dhop_sweep.inl"
