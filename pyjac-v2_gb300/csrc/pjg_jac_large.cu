// The thread-per-state Jacobian kernel: the form for large mechanisms.
#include "pjg_wave.cuh"

PJG_WAVE_INSTANCE(KIND_JAC, pjg::kLargeBlocks)
