// collide_bf16.cu -- the FP32-collision path on BF16 storage.
#include "collide_lowp.cuh"

LBMPSM_LOWP_PATH(bf16, __nv_bfloat16)
