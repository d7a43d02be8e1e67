// The thread-per-state Jacobian kernel: the form for whole waves.
#include "pjg_wave.cuh"

PJG_WAVE_INSTANCE(KIND_JAC, PJG_JAC_MINB)
