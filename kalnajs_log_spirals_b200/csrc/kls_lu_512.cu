#include "kls_lu_pipe.cuh"

LUP_DEFINE(512, 16, 4, nullptr)
