// Instantiations of the decode kernel for two resident blocks per SM, __nv_bfloat16 message storage.
#include "relaybp_decode.cuh"

RBPK_DEFINE_PICK2(pick2_bf16, __nv_bfloat16)
