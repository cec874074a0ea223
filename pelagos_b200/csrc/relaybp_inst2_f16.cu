// Instantiations of the decode kernel for two resident blocks per SM, __half message storage.
#include "relaybp_decode.cuh"

RBPK_DEFINE_PICK2(pick2_f16, __half)
