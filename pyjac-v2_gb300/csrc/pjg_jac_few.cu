// The thread-per-state Jacobian kernel: the form for few blocks.
#include "pjg_wave.cuh"

PJG_WAVE_INSTANCE(KIND_JAC, pjg::kFewBlocks)
