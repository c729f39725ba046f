#include "collectives_typed.cuh"

HCCL_COLLECTIVES_OF(int8_t);
HCCL_COLLECTIVES_OF(uint8_t);
