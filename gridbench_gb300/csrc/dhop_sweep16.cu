// The sweep form of the FP32 hopping kernel for rows (or tiles) of 16 slices.
#define SWEEP_TE 16
#include "dhop_sweep.inl"
