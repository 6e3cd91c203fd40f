#include "kls_lu_pipe.cuh"

LUP_DEFINE(416, 13, 4, nullptr)
