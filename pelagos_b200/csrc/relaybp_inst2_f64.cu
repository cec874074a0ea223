// Instantiations of the decode kernel for two resident blocks per SM, double message storage.
#include "relaybp_decode.cuh"

RBPK_DEFINE_PICK2(pick2_f64, double)
