#include "kls_lu_pipe.cuh"

LUP_DEFINE(320, 10, 4, nullptr)
