#include "kls_lu_pipe.cuh"

LUP_DEFINE(256, 8, 4, ((const void*)lu_pipe_kernel<8, 2>))
