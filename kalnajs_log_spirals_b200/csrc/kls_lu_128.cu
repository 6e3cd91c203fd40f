#include "kls_lu_pipe.cuh"

LUP_DEFINE(128, 4, 3, nullptr)
