#include "collectives_typed.cuh"

HCCL_COLLECTIVES_OF(int32_t);
HCCL_COLLECTIVES_OF(uint32_t);
