#include "kls_lu_pipe.cuh"

LUP_DEFINE(192, 6, 4, ((const void*)lu_pipe_kernel<6, 2>))
