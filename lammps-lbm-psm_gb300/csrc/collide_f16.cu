// collide_f16.cu -- the FP32-collision path on FP16 storage.
#include "collide_lowp.cuh"

LBMPSM_LOWP_PATH(f16, __half)
