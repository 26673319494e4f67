// Moves a [128 x 128] FP32 state between global memory and its transposed place in tensor memory (lane = value column e,
// column = key channel d) for the state kernels, 256 threads: thread (half, e) owns lane e and half of the columns.
#pragma once

#include "kda_common.cuh"
#include "kda_tc.cuh"

namespace kda {
namespace tc {

// Layouts in global memory: ROWS = [e][d] (v-first states), COLS = [d][e] (k-first states and the segment buffers).
// COLS is coalesced as it is (consecutive lanes, consecutive e).  ROWS would touch 32 lines per warp access, 8 us for the
// 64 KB with scalar loads; it goes through shared memory (`stage`, 64 KB, chunks of 16 bytes XOR-swizzled by the row)
// where the caller has the room, and by 16-byte accesses otherwise.
__device__ __forceinline__ int stage_idx(int e, int chunk) { return e * 128 + ((chunk ^ (e & 7)) << 2); }

// src NULL: zero state.  With `stage` all 256 threads call (named barrier 1).
__device__ __forceinline__ void state_fill(uint32_t tmem_acc, const float* src, bool rows, float* stage, int tid, int e, int half) {
    const bool staged = src && rows && stage;
    if (staged) {
#pragma unroll 4
        for (int i = 0; i < 16; ++i) {
            const int q = tid + 256 * i, r = q >> 5, c = q & 31;
            cp_async16_z(stage + stage_idx(r, c), src + r * 128 + 4 * c, true);
        }
        cp_async_commit();
        cp_async_wait<0>();
        bar_sync(1, 256);
    }
    for (int d0 = 64 * half; d0 < 64 * half + 64; d0 += 16) {
        uint32_t r[16];
        if (!src) {
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = 0u;
        } else if (rows) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c = (d0 >> 2) + j;
                const uint4 x = *reinterpret_cast<const uint4*>(staged ? stage + stage_idx(e, c) : src + (size_t)e * 128 + 4 * c);
                r[4 * j] = x.x; r[4 * j + 1] = x.y; r[4 * j + 2] = x.z; r[4 * j + 3] = x.w;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(src[(size_t)(d0 + j) * 128 + e]);
        }
        tmem_st16(tmem_acc + d0, r);
    }
    tmem_wait_st();
    if (staged) {  // the caller reuses the space for bulk copies
        fence_async_smem();
        bar_sync(1, 256);
    }
}

__device__ __forceinline__ void state_drain(uint32_t tmem_acc, float* dst, bool rows, float* stage, int tid, int e, int half) {
    const bool staged = rows && stage;
    for (int d0 = 64 * half; d0 < 64 * half + 64; d0 += 16) {
        uint32_t r[16];
        tmem_ld16(tmem_acc + d0, r);
        tmem_wait_ld();
        if (rows) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c = (d0 >> 2) + j;
                *reinterpret_cast<uint4*>(staged ? stage + stage_idx(e, c) : dst + (size_t)e * 128 + 4 * c) =
                    make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) dst[(size_t)(d0 + j) * 128 + e] = __uint_as_float(r[j]);
        }
    }
    if (staged) {
        bar_sync(1, 256);
#pragma unroll 4
        for (int i = 0; i < 16; ++i) {
            const int q = tid + 256 * i, r = q >> 5, c = q & 31;
            *reinterpret_cast<uint4*>(dst + r * 128 + 4 * c) = *reinterpret_cast<const uint4*>(stage + stage_idx(r, c));
        }
    }
}

// where sequence n, head h has its state in a caller's [N][H][..][..] tensor (NULL stays NULL)
__device__ __forceinline__ const float* state_of(const float* base, const KdaParams& p, int n, int h) {
    return base ? base + ((size_t)n * p.H + h) * p.dk * p.dv : nullptr;
}

}  // namespace tc
}  // namespace kda
