#include "collectives_typed.cuh"

HCCL_COLLECTIVES_OF(long long);
HCCL_COLLECTIVES_OF(unsigned long long);
