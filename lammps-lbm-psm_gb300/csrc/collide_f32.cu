// collide_f32.cu -- the FP32-collision path on FP32 storage.
#include "collide_lowp.cuh"

LBMPSM_LOWP_PATH(f32, float)
