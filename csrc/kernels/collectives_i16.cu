#include "collectives_typed.cuh"

HCCL_COLLECTIVES_OF(int16_t);
HCCL_COLLECTIVES_OF(uint16_t);
