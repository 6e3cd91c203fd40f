#include "kls_lu_pipe.cuh"

LUP_DEFINE(224, 7, 5, ((const void*)lu_pipe_kernel<7, 2>))
