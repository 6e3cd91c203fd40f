#include "kls_lu_pipe.cuh"

LUP_DEFINE(64, 2, 2, nullptr)
