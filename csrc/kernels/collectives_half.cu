#include "collectives_typed.cuh"

HCCL_COLLECTIVES_OF(__half);
HCCL_COLLECTIVES_OF(__nv_bfloat16);
