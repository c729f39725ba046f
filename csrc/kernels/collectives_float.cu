#include "collectives_typed.cuh"

HCCL_COLLECTIVES_OF(float);
HCCL_COLLECTIVES_OF(double);
