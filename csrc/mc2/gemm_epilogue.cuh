// Epilogue of the GEMM kernels for results in local memory: tensor memory -> registers -> a 128-byte-swizzled staging tile ->
// TMA store. The stores leave shared memory asynchronously and write whole 128-byte row segments whatever the result type, so the
// epilogue warps only read tensor memory, convert and store to shared memory (two staging tiles in turn where they fit), and the
// ragged right and lower edges are clipped by the tensor map. One B200 against per-thread 16-byte stores from the staging tile: 1000 x 6144 x 4096
// 54.5 -> 53.3 us, 64 x 128256 x 4096 with fp32 results (which left registers 16 bytes per row) 229.7 -> 226.4 us, large products the same.
#pragma once
#include "sm100_ptx.cuh"
#include <cuda_bf16.h>

namespace hccl {
namespace mc2 {

using namespace sm100;

constexpr int kStageTileBytes = 128 * 128;      // 128 rows x 128 bytes: 64 bf16 or 32 fp32 columns

template <int N> __device__ __forceinline__ void TmaStoreWaitRead() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ uint4 PackBf16x8(const uint32_t *v)
{
    uint4 o;
    __nv_bfloat162 t0 = __floats2bfloat162_rn(__uint_as_float(v[0]), __uint_as_float(v[1]));
    __nv_bfloat162 t1 = __floats2bfloat162_rn(__uint_as_float(v[2]), __uint_as_float(v[3]));
    __nv_bfloat162 t2 = __floats2bfloat162_rn(__uint_as_float(v[4]), __uint_as_float(v[5]));
    __nv_bfloat162 t3 = __floats2bfloat162_rn(__uint_as_float(v[6]), __uint_as_float(v[7]));
    o.x = *(uint32_t *)&t0; o.y = *(uint32_t *)&t1; o.z = *(uint32_t *)&t2; o.w = *(uint32_t *)&t3;
    return o;
}

// Stores the 128 x BN accumulator tile at tensor-memory address `tmem` (this warp's lane quarter, first column) to rows row0 ... and
// columns col0 ... of C. Called by the 128 epilogue threads (et = 0 ... 127, lane quarter = et / 32) together; thread 0 issues the
// stores, waits for its staging tile to be free again, and has to TmaStoreWaitAll() before the CTA ends. `tiles` counts the staging
// tiles used so far. released() is called once by every thread when the accumulator has been read.
template <int BN, int BUFS, class Released>
__device__ __forceinline__ void StoreTileTma(const CUtensorMap *tmapC, bool fp32, uint32_t N, uint32_t tmem, uint8_t *staging, uint32_t et, uint32_t row0, uint32_t col0,
                                             uint32_t &tiles, Released released)
{
    static_assert(BN % 32 == 0 && BN >= 64, "whole staging tiles");
    const uint32_t swz = et & 7;
    const uint32_t passes = fp32 ? BN / 32 : (BN + 63) / 64;
#pragma unroll 1
    for (uint32_t pass = 0; pass < passes; ++pass) {
        uint32_t off = pass * (fp32 ? 32u : 64u);
        if (BN % 64 && off > BN - (fp32 ? 32u : 64u)) off = BN - 64;         // BN = 224: the last tile stores 32 columns a second time
        const uint32_t col = col0 + off;
        uint8_t *tile = staging + (BUFS > 1 ? tiles % BUFS : 0) * kStageTileBytes;
        uint4 *mine = (uint4 *)(tile + et * 128);
        if (et == 0) TmaStoreWaitRead<BUFS - 1>();
        uint32_t v[64];
        TmemLd32x32(tmem + off, *(uint32_t(*)[32])&v[0]);
        if (!fp32) TmemLd32x32(tmem + off + 32, *(uint32_t(*)[32])&v[32]);
        TmemLdWait();
        asm volatile("bar.sync 1, 128;" ::: "memory");       // the staging tile is free
        if (fp32) {
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) mine[q ^ swz] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        } else {
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) mine[q ^ swz] = PackBf16x8(&v[8 * q]);
        }
        if (pass + 1 == passes) released();
        FenceProxyAsyncShared();
        asm volatile("bar.sync 1, 128;" ::: "memory");       // the staging tile is complete
        if (et == 0) {
            if (col < N) TmaStore2D(tmapC, tile, (int32_t)col, (int32_t)row0);
            TmaStoreCommit();
        }
        ++tiles;
    }
}

}  // namespace mc2
}  // namespace hccl
