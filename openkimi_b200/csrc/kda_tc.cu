// Tensor-core (tcgen05 / TMEM) stages of the KDA op for BF16 operands.
#include "kda_common.cuh"
#include "kda_state.cuh"
#include "kda_tc.cuh"
#include "kda_tmap.cuh"

namespace kda {

using namespace tc;

// ---------------------------------------------------------------------------------------
// Self-test of the MMA building block: D[128 x N] = A[128 x K] * B[K x N] with one CTA,
// operands converted to BF16 and laid out by the kernel in the core-matrix layout.  The
// host chooses the operand views and passes the descriptor strides, so the layout rules
// of kda_tc.cuh are checked against a plain matrix product.
//   a_mode 0: shared, K-major (stored CM rows=m, cols=k)   1: shared, MN-major (CM rows=k, cols=m)
//          2: tensor memory (lane = m, two BF16 per 32-bit column)
//   b_mode 0: shared, K-major (stored CM rows=n, cols=k)   1: shared, MN-major (CM rows=k, cols=n)
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 1)
mma_selftest_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ D, int N, int K,
                    int a_mode, int b_mode, int lbo_a, int sbo_a, int step_a, int lbo_b, int sbo_b, int step_b,
                    int neg_a, int m_rows, int* status) {
    extern __shared__ __align__(128) unsigned char dyn[];
    __nv_bfloat16* sA = reinterpret_cast<__nv_bfloat16*>(dyn);
    __nv_bfloat16* sB = sA + 128 * 128;
    __shared__ uint64_t bar;
    __shared__ uint32_t tmem_base_s;
    const int tid = threadIdx.x, warp = tid >> 5;
    if (warp == 0) {
        tmem_alloc(&tmem_base_s, 256);
        tmem_relinquish();
    }
    if (tid == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    for (int idx = tid; idx < 128 * K; idx += 128) {
        int m = idx / K, k = idx % K;
        __nv_bfloat16 v = __float2bfloat16_rn(A[idx]);
        if (a_mode == 0) sA[cm_idx(m, k, K)] = v;
        else if (a_mode == 1) sA[cm_idx(k, m, 128)] = v;
    }
    for (int idx = tid; idx < K * N; idx += 128) {
        int k = idx / N, n = idx % N;
        __nv_bfloat16 v = __float2bfloat16_rn(B[idx]);
        if (b_mode == 0) sB[cm_idx(n, k, K)] = v;
        else sB[cm_idx(k, n, N)] = v;
    }
    fence_async_smem();
    const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
    if (m_rows != 128) {  // clear the accumulator so that untouched lanes read as zero
        uint32_t z[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) z[j] = 0u;
        for (int c0 = 0; c0 < N; c0 += 16) tmem_st16(tmem + lane_off + c0, z);
        tmem_wait_st();
    }
    if (a_mode == 2) {
        for (int c0 = 0; c0 < K / 2; c0 += 16) {
            uint32_t r[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = pack_bf16(A[tid * K + 2 * (c0 + j)], A[tid * K + 2 * (c0 + j) + 1]);
            tmem_st16(tmem + lane_off + 128 + c0, r);
        }
        tmem_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
        tc_fence_after();
        const uint32_t idesc = make_idesc(m_rows, N, a_mode == 1, b_mode == 1, neg_a != 0);
        for (int s = 0; s < K / 16; ++s) {
            uint64_t bd = make_desc(smem_u32(sB) + s * step_b, lbo_b, sbo_b);
            if (a_mode == 2) mma_ts(tmem, tmem + 128 + s * 8, bd, idesc, s > 0);
            else mma_ss(tmem, make_desc(smem_u32(sA) + s * step_a, lbo_a, sbo_a), bd, idesc, s > 0);
        }
        mma_commit(&bar);
    }
    const bool ok = mbar_wait(&bar, 0, status, 1);
    tc_fence_after();
    if (ok) {
        for (int c0 = 0; c0 < N; c0 += 16) {
            uint32_t r[16];
            tmem_ld16(tmem + lane_off + c0, r);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) D[tid * N + c0 + j] = __uint_as_float(r[j]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 256);
}

// ---------------------------------------------------------------------------------------
// Self-test of the bounded wait: one CTA allocates tensor memory, arms an mbarrier for
// 2 * bytes, issues ONE bulk copy of `bytes`, and polls at most `poll_limit` times.  The
// wait must run out: the kernel records `code` in the status word, accounts for the bytes that
// were never sent so that the barrier completes as soon as the copy that IS in flight has
// landed, waits for that (bounded), frees its tensor memory and returns.  Nothing hangs.
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 1) wait_selftest_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                               uint32_t poll_limit, int code, int* status) {
    __shared__ __align__(128) float buf[64];
    __shared__ uint64_t bar;
    __shared__ uint32_t tmem_base_s;
    const int tid = threadIdx.x, warp = tid >> 5;
    constexpr uint32_t BYTES = 64 * sizeof(float);
    if (warp == 0) {
        tmem_alloc(&tmem_base_s, 32);
        tmem_relinquish();
    }
    if (tid == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (tid == 0) {
        mbar_expect_tx(&bar, 2 * BYTES);  // twice what the copy below delivers
        tma_load_1d(buf, src, BYTES, &bar);
    }
    bool ok = mbar_wait(&bar, 0, status, code, poll_limit);
    ok = __syncthreads_and(ok);
    if (!ok) {
        if (tid == 0) mbar_complete_tx(&bar, BYTES);
        const bool landed = mbar_wait(&bar, 0, status, code << 8);  // the copy in flight, default limit
        if (__syncthreads_and(landed) && tid < 64) dst[tid] = buf[tid];
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base_s, 32);
}

// ---------------------------------------------------------------------------------------
// fwd_state on tensor cores.  One CTA per (sequence, head), or per segment of the chunk numbering and head; value column e
// is TMEM lane e.  The state is kept TRANSPOSED in tensor memory for the whole walk: Sacc[e][d] (FP32, 128 columns).
// Per chunk:
//   A  read Sacc -> BF16 copy Sbf (MMA operand, also the chunk-entry checkpoint), decay Sacc
//   1  WSacc = Sbf * W^T        (V'^T = U^T - WSacc)        Oacc  = Sbf * Qt^T
//   B  V'^T -> BF16 Vbf (MMA operand) and the V' record
//   2  Sacc += Vbf * Kh         Oacc += Vbf * Aqk^T
// Bound by the chain A, W S, B, K V: two MMA round trips and two conversions per chunk.  Everything else is kept off that
// chain by giving it to other warps: a producer warp requests the records (linear bulk copies into a two-stage ring), four
// warps turn finished Oacc tiles into output rows while the next chunk runs, records that leave the chip (checkpoint, V')
// are stored after the MMA issue they used to precede.  One thread issues all products of one accumulator, so only the
// products the chain needs are waited for; it is an elected lane of a warp-uniform branch, whose descriptors stay in uniform
// registers (a lane of a divergent branch spends 50 ns per MMA on moving them there).
// 96 chains of 32 chunks: 82 -> 73 us; 8 chunks of one sequence: 21.1 -> 17.0 us.
// Measured and not kept: a third stage with a half-size output tile (76 us), checkpoint and V' read back from tensor memory
// by more warps (87 us: their loads queue with the chain's), output rows stored straight from registers (+1 us a chunk).
// ---------------------------------------------------------------------------------------
namespace fs {
constexpr int D = 128, MAIN = 256, OUTT = 128, NTHR = MAIN + OUTT + 32;
constexpr uint32_t WT = 0, QT = 16384, KH = 32768, UT = 49152, AQ = 65536, GAM = 73728, STAGE = 74240;
constexpr uint32_t OUT = 2 * STAGE, TOTAL = OUT + 16384;  // output tile bf16 [64][128] behind the two stages
constexpr uint32_t SACC = 0, SBF = 128, WSACC = 192, OACC = 256, VBF = 320, TMEM_COLS = 512;
}  // namespace fs

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float2 t = __bfloat1622float2(h[i]);
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
    }
}

// Phase A of both state kernels: this thread's 64 columns of the accumulator, all loads in flight at once.  pk receives
// the BF16 copy (pairs), which also goes to `bf`; the accumulator is decayed by gam.
__device__ __forceinline__ void state_convert(uint32_t acc, uint32_t bf, int c0, const float* gam, uint32_t (&pk)[4][8]) {
    uint32_t r[4][16];
#pragma unroll
    for (int g = 0; g < 4; ++g) tmem_ld16(acc + c0 + 16 * g, r[g]);
    tmem_wait_ld();
#pragma unroll
    for (int g = 0; g < 4; ++g) {
#pragma unroll
        for (int j = 0; j < 8; ++j) pk[g][j] = pack_bf16(__uint_as_float(r[g][2 * j]), __uint_as_float(r[g][2 * j + 1]));
        tmem_st8(bf + (c0 + 16 * g) / 2, pk[g]);
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
            const float4 gm = *reinterpret_cast<const float4*>(gam + c0 + 16 * g + j);
            r[g][j] = __float_as_uint(__uint_as_float(r[g][j]) * gm.x);
            r[g][j + 1] = __float_as_uint(__uint_as_float(r[g][j + 1]) * gm.y);
            r[g][j + 2] = __float_as_uint(__uint_as_float(r[g][j + 2]) * gm.z);
            r[g][j + 3] = __float_as_uint(__uint_as_float(r[g][j + 3]) * gm.w);
        }
        tmem_st16(acc + c0 + 16 * g, r[g]);
    }
    tmem_wait_st();
}
// 16 BF16 values (columns c0 .. c0 + 15 of row e) into a core-matrix record of `cols` columns
__device__ __forceinline__ void store_record16(__nv_bfloat16* dst, int e, int c0, int cols, const uint32_t (&pk)[8]) {
    *reinterpret_cast<uint4*>(dst + cm_idx(e, c0, cols)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
    *reinterpret_cast<uint4*>(dst + cm_idx(e, c0 + 8, cols)) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
}

__global__ void __launch_bounds__(fs::NTHR, 1)
kda_fwd_state_tc(const KdaParams p, const __grid_constant__ RowMaps maps, const StateSegs segs) {
    using namespace fs;
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ uint64_t full[2], empty[2], wsbar, sbar, obar, ofree;
    __shared__ uint32_t tmem_s;
    // main threads (half, e) = (tid / 128, tid % 128): TMEM lane e (value column e), and half of the accumulator
    // columns in every conversion phase (two warps share a lane quadrant); then the output threads, lane e each; then
    // the producer warp
    const int tid = threadIdx.x, warp = tid >> 5, e = tid & 127, half = tid >> 7;
    const int h = blockIdx.x;
    if (warp == 0) {
        tmem_alloc(&tmem_s, TMEM_COLS);
        tmem_relinquish();
    }
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(&wsbar, 1);
        mbar_init(&sbar, 1);
        mbar_init(&obar, 1);
        mbar_init(&ofree, OUTT / 32);
        mbar_fence_init();
    }
    pdl_wait();
    // the chunks of this CTA: one sequence, or one segment of the chunk numbering
    SeqCursor sq;
    int cb, ce;
    if (segs.len > 0) {
        cb = blockIdx.y * segs.len;
        ce = min(cb + segs.len, p.NT);
        sq.load_of_chunk(p, cb);
    } else {
        sq.load(p, blockIdx.y);
        cb = sq.c_begin;
        ce = sq.c_end;
    }
    const WsLayout L = ws_layout(p.NT, p.H, p.dk, p.dv, p.dtype);
    char* ws = (char*)p.workspace;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_s + ((uint32_t)((warp & 3) * 32) << 16);  // this warp's lane quadrant
    const uint32_t tmem0 = tmem_s;
    const bool save = !(p.flags & KDA_FLAG_NO_SAVE);     // forward-only calls write no checkpoint and no V' record
    const bool with_o = !(p.flags & KDA_FLAG_NO_OUTPUT);  // a walk for the records only leaves the output products out
    const bool vfirst = p.flags & KDA_FLAG_STATE_V_FIRST;
    float* stage_space = reinterpret_cast<float*>(dyn);  // before the first and after the last chunk's copies
    if (tid < MAIN) {
        // state entering the segment (what the previous one ended with), or a sequence (h0 or zero)
        if (cb > sq.c_begin)
            state_fill(tmem + SACC, segs.E + (((size_t)blockIdx.y - 1) * p.H + h) * D * D, false, nullptr, tid, e, half);
        else
            state_fill(tmem + SACC, state_of(p.h0, p, sq.n, h), vfirst, stage_space, tid, e, half);
    }
    __syncthreads();

    bool ok = true;
    if (tid < MAIN) {
        KDA_PHASE_BEGIN();
        const int wu = __shfl_sync(0xffffffffu, warp, 0);  // warp 0: WSacc and Sacc, warp 1: Oacc
        for (int c = cb; c < ce; ++c) {
            const int i = c - cb, stage = i & 1;
            unsigned char* b = dyn + stage * STAGE;
            const uint32_t sb = smem_u32(b);
            const size_t rec = (size_t)c * p.H + h;
            if (c == sq.c_end) {  // (segments only) the walk enters the next sequence
                sq.load_of_chunk(p, c);
                state_fill(tmem + SACC, state_of(p.h0, p, sq.n, h), vfirst, nullptr, tid, e, half);
            }
            ok = mbar_wait(&full[stage], (i >> 1) & 1, p, 2) && ok;
            KDA_PHASE(0);
            // ---- A: BF16 copy of the entering state, decay
            uint32_t pk[4][8];
            state_convert(tmem + SACC, tmem + SBF, 64 * half, reinterpret_cast<const float*>(b + GAM), pk);
            KDA_PHASE(1);
            tc_fence_before();
            ok = bar_and(1, MAIN, ok);
            if (!ok) break;
            if (wu < 2 && elect_one()) {
                tc_fence_after();
                constexpr uint32_t id_mn = make_idesc(128, 64, false, true);
                constexpr uint32_t id_k = make_idesc(128, 64, false, false);
                if (wu == 0) {
#pragma unroll
                    for (int s = 0; s < 8; ++s)  // WSacc = Sbf (K = d) * W^T record, MN-major B
                        mma_ts(tmem0 + WSACC, tmem0 + SBF + s * 8, make_desc(sb + WT + s * 2048, 1024, 128), id_mn, s > 0);
                    mma_commit(&wsbar);
                } else if (with_o) {
                    if (i > 0) ok = mbar_wait(&ofree, (i - 1) & 1, p, 4);  // the previous chunk's output has left Oacc
                    tc_fence_after();
                    if (ok) {
#pragma unroll
                        for (int s = 0; s < 8; ++s)  // Oacc = Sbf * Qt^T, K-major B (rows = i)
                            mma_ts(tmem0 + OACC, tmem0 + SBF + s * 8, make_desc(sb + QT + s * 256, 128, 2048), id_k, s > 0);
                    }
                }
            }
            __syncwarp();
            if (save) {
                __nv_bfloat16* gS0 = (__nv_bfloat16*)(ws + L.S0) + rec * D * D;
#pragma unroll
                for (int g = 0; g < 4; ++g) store_record16(gS0, e, 64 * half + 16 * g, D, pk[g]);
            }
            // ---- B: V'^T = U^T - (W S)^T
            const __nv_bfloat16* sU = reinterpret_cast<const __nv_bfloat16*>(b + UT);
            float u[2][16];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                float t8[8];
                unpack8(*reinterpret_cast<const uint4*>(sU + cm_idx(e, 32 * half + 8 * g, C)), t8);
#pragma unroll
                for (int j = 0; j < 8; ++j) u[g >> 1][8 * (g & 1) + j] = t8[j];
            }
            ok = mbar_wait(&wsbar, i & 1, p, 4) && ok;
            tc_fence_after();
            KDA_PHASE(2);
            uint32_t vk[2][8];
            {
                uint32_t r[2][16];
                tmem_ld16(tmem + WSACC + 32 * half, r[0]);
                tmem_ld16(tmem + WSACC + 32 * half + 16, r[1]);
                tmem_wait_ld();
#pragma unroll
                for (int g = 0; g < 2; ++g) {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        vk[g][j] = pack_bf16(u[g][2 * j] - __uint_as_float(r[g][2 * j]), u[g][2 * j + 1] - __uint_as_float(r[g][2 * j + 1]));
                    tmem_st8(tmem + VBF + (32 * half + 16 * g) / 2, vk[g]);
                }
                tmem_wait_st();
            }
            KDA_PHASE(3);
            tc_fence_before();
            ok = bar_and(1, MAIN, ok);
            if (!ok) break;
            if (wu < 2 && elect_one()) {
                tc_fence_after();
                constexpr uint32_t id_k = make_idesc(128, 64, false, false);
                constexpr uint32_t id_s = make_idesc(128, 128, false, true);
                if (wu == 0) {
#pragma unroll
                    for (int s = 0; s < 4; ++s)  // Sacc += Vbf (K = i) * Kh, MN-major B
                        mma_ts(tmem0 + SACC, tmem0 + VBF + s * 8, make_desc(sb + KH + s * 4096, 2048, 128), id_s, true);
                    mma_commit(&sbar);
                } else if (with_o) {
#pragma unroll
                    for (int s = 0; s < 4; ++s)  // Oacc += Vbf (K = j) * Aqk^T, K-major B (rows = i)
                        mma_ts(tmem0 + OACC, tmem0 + VBF + s * 8, make_desc(sb + AQ + s * 256, 128, 1024), id_k, true);
                    mma_commit(&obar);
                }
            }
            __syncwarp();
            if (save) {
                __nv_bfloat16* gV = (__nv_bfloat16*)(ws + L.U) + rec * C * D;
#pragma unroll
                for (int g = 0; g < 2; ++g) store_record16(gV, e, 32 * half + 16 * g, C, vk[g]);
            }
            // (both: the next chunk overwrites the operands of the output products too)
            ok = mbar_wait(&sbar, i & 1, p, 4) && (!with_o || mbar_wait(&obar, i & 1, p, 4)) && ok;
            tc_fence_after();
            if (tid == 0) mbar_arrive(&empty[stage]);
            KDA_PHASE(4);
            if (c + 1 == sq.c_end && c + 1 < ce && p.ht && ok)
                state_drain(tmem + SACC, const_cast<float*>(state_of(p.ht, p, sq.n, h)), vfirst, nullptr, tid, e, half);
        }
        ok = bar_and(1, MAIN, ok);
        // the sequence that ends with the last chunk (one without tokens hands its initial state on)
        if (ok && ce == sq.c_end && p.ht)
            state_drain(tmem + SACC, const_cast<float*>(state_of(p.ht, p, sq.n, h)), vfirst, stage_space, tid, e, half);
    } else if (tid < MAIN + OUTT) {
        // ---- output rows.  The accumulator holds O^T (lane = channel): the tile is transposed through shared memory and
        //      goes out with one bulk-tensor store (row by row for a partial chunk)
        const int ot = tid - MAIN;
        __nv_bfloat16* o = (__nv_bfloat16*)p.o;
        __nv_bfloat16* sO = reinterpret_cast<__nv_bfloat16*>(dyn + OUT);
        for (int c = cb; c < ce && with_o; ++c) {
            sq.move_to(p, c);
            ok = mbar_wait(&obar, (c - cb) & 1, p, 4);
            ok = bar_and(2, OUTT, ok);
            if (!ok) break;
            tc_fence_after();
            uint32_t r[4][16];
#pragma unroll
            for (int g = 0; g < 4; ++g) tmem_ld16(tmem + OACC + 16 * g, r[g]);
            tmem_wait_ld();
            tc_fence_before();
            __syncwarp();
            if ((tid & 31) == 0) mbar_arrive(&ofree);
            tma_store_wait_read();  // the previous chunk's rows have left the staging tile
            bar_sync(2, OUTT);
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
                for (int j = 0; j < 16; ++j) sO[(16 * g + j) * D + e] = __float2bfloat16_rn(__uint_as_float(r[g][j]));
            fence_async_smem();
            bar_sync(2, OUTT);
            const long long tok0 = sq.tok(c);
            const int len = sq.rows(c);
            if (maps.ok && len == C) {  // the whole tile with one bulk-tensor store
                if (ot == 0) {
                    tma_store_tile(&maps.m[0], h * D, (int)tok0, sO);
                    tma_store_commit();
                }
            } else if (ot < len) {
                tma_store_1d(o + ((size_t)(tok0 + ot) * p.H + h) * D, sO + ot * D, D * 2);
                tma_store_commit();
            }
        }
        tma_store_wait_all();
    } else if ((tid & 31) == 0) {
        // ---- the six records of every chunk, one chunk ahead of their use
        int i = 0;
        for (; i < ce - cb; ++i) {
            const int stage = i & 1;
            if (i >= 2 && !mbar_wait(&empty[stage], ((i >> 1) - 1) & 1, p, 2)) break;
            const size_t rec = (size_t)(cb + i) * p.H + h;
            unsigned char* b = dyn + stage * STAGE;
            mbar_expect_tx(&full[stage], with_o ? STAGE : STAGE - 16384 - 8192);
            tma_load_1d(b + GAM, (const float*)(ws + L.gamC) + rec * D, 512, &full[stage]);
            tma_load_1d(b + WT, (const __nv_bfloat16*)(ws + L.W) + rec * C * D, 16384, &full[stage]);
            tma_load_1d(b + UT, (const __nv_bfloat16*)(ws + L.U) + rec * C * D, 16384, &full[stage]);
            tma_load_1d(b + KH, (const __nv_bfloat16*)(ws + L.Kh) + rec * C * D, 16384, &full[stage]);
            if (!with_o) continue;
            tma_load_1d(b + QT, (const __nv_bfloat16*)(ws + L.Qt) + rec * C * D, 16384, &full[stage]);
            tma_load_1d(b + AQ, (const __nv_bfloat16*)(ws + L.Aqk) + rec * C * C, 8192, &full[stage]);
        }
        // (whatever became of the walk, no copy is in flight when the CTA leaves)
        for (int j = i > 2 ? i - 2 : 0; j < i; ++j) mbar_wait(&full[j & 1], (j >> 1) & 1, p, 2);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem0, TMEM_COLS);
}

// ---------------------------------------------------------------------------------------
// bwd_state on tensor cores: same organisation, reverse chunk order, dS^T resident in TMEM.
//   0  dVacc = dO^T * Aqk (before the conversion: it needs the chunk's records only)
//   A  dSacc -> BF16 dSbf (operand + checkpoint of the dS entering the chunk), decay dSacc
//   1  dVacc += dSbf * Kh^T         dSacc += dO^T * Qt
//   B  dV'^T -> BF16 dVbf and the dV' record
//   2  dSacc -= dVbf * W
// Four producer warps fetch the records (bulk copies) and the dO tile (16-byte asynchronous copies into the core-matrix
// layout) into a three-stage ring.  96 chains of 32 chunks: 92 -> 67 us.
// ---------------------------------------------------------------------------------------
namespace bs {
constexpr int D = 128, MAIN = 256, PROD = 128, NTHR = MAIN + PROD;
constexpr uint32_t WT = 0, QT = 16384, KH = 32768, DO = 49152, AQ = 65536, GAM = 73728, STAGE = 74240;
constexpr uint32_t TMA_BYTES = 16384 * 3 + 8192 + 512;
constexpr uint32_t SACC = 0, SBF = 128, VACC = 192, VBF = 256, TMEM_COLS = 512;
}  // namespace bs

// PARTIAL (segments only): the contribution of the segment's own dO to the dS at its start, from a zero dS at its end where
// the sequence goes on behind it; nothing else is stored.
template <bool PARTIAL>
__global__ void __launch_bounds__(bs::NTHR, 1) kda_bwd_state_tc(const KdaParams p, const StateSegs segs) {
    using namespace bs;
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ uint64_t full[3], empty[3], vbar, sbar;
    __shared__ uint32_t tmem_s;
    // main threads (half, e) = (tid / 128, tid % 128): TMEM lane e, and half of the columns of every conversion phase
    const int tid = threadIdx.x, warp = tid >> 5, e = tid & 127, half = tid >> 7;
    const int h = blockIdx.x;
    pdl_wait();
    // the chunks of this CTA, walked from the last to the first: one sequence, or one segment of the chunk numbering
    SeqCursor sq;  // sequence of the current chunk
    int cb, ce;
    if (segs.len > 0) {
        cb = blockIdx.y * segs.len;
        ce = min(cb + segs.len, p.NT);
        if (PARTIAL) {  // only the sequence that the segment's first chunk continues has anyone to hand its dS to
            sq.load_of_chunk(p, cb);
            if (sq.c_begin == cb) return;
            ce = min(ce, sq.c_end);
        } else {
            sq.load_of_chunk(p, ce - 1);
        }
    } else {
        sq.load(p, blockIdx.y);
        cb = sq.c_begin;
        ce = sq.c_end;
    }
    const int nc = ce - cb;
    const WsLayout L = ws_layout(p.NT, p.H, p.dk, p.dv, p.dtype);
    const char* ws = (const char*)p.workspace;
    char* sc = (char*)p.bwd_scratch;
    const __nv_bfloat16* dO = (const __nv_bfloat16*)p.grad_o;
    if (warp == 0) {
        tmem_alloc(&tmem_s, TMEM_COLS);
        tmem_relinquish();
    }
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            mbar_init(&full[i], 1 + PROD / 32);  // the bulk copies, and the dO rows of every producer warp
            mbar_init(&empty[i], 1);
        }
        mbar_init(&vbar, 1);
        mbar_init(&sbar, 1);
        mbar_fence_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_s + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t tmem0 = tmem_s;
    const bool vfirst = p.flags & KDA_FLAG_STATE_V_FIRST;
    float* stage_space = reinterpret_cast<float*>(dyn);  // before the first and after the last chunk's copies
    if (tid < MAIN) {
        // dS at the end of the segment (what the next one found at its start), or of a sequence (grad_ht or zero)
        if (ce < sq.c_end)
            state_fill(tmem + SACC, PARTIAL ? nullptr : segs.E + (((size_t)blockIdx.y + 1) * p.H + h) * D * D, false, nullptr, tid, e, half);
        else
            state_fill(tmem + SACC, state_of(p.grad_ht, p, sq.n, h), vfirst, stage_space, tid, e, half);
    }
    __syncthreads();

    bool ok = true;
    // step k = 0..nc-1 processes chunk ce-1-k
    if (tid < MAIN) {
        const int wu = __shfl_sync(0xffffffffu, warp, 0);  // warp 0: dVacc, warp 1: dSacc
        int stage = 0;
        uint32_t ring_phase = 0;  // parity of full[stage]: flips every time the ring wraps
        for (int k = 0; k < nc; ++k) {
            const int c = ce - 1 - k;
            unsigned char* b = dyn + stage * STAGE;
            const uint32_t sb = smem_u32(b);
            const size_t rec = (size_t)c * p.H + h;
            if (c < sq.c_begin) {  // (segments only) the walk enters the previous sequence
                sq.load_of_chunk(p, c);
                state_fill(tmem + SACC, state_of(p.grad_ht, p, sq.n, h), vfirst, nullptr, tid, e, half);
            }
            ok = mbar_wait(&full[stage], ring_phase, p, 2) && ok;
            if (wu == 0 && elect_one() && ok) {
                constexpr uint32_t id_v1 = make_idesc(128, 64, true, true);  // dO^T (MN-major A) * Aqk (MN-major B)
                tc_fence_after();
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    mma_ss(tmem0 + VACC, make_desc(sb + DO + s * 4096, 2048, 128), make_desc(sb + AQ + s * 2048, 1024, 128), id_v1,
                           s > 0);
            }
            __syncwarp();
            uint32_t pk[4][8];
            state_convert(tmem + SACC, tmem + SBF, 64 * half, reinterpret_cast<const float*>(b + GAM), pk);
            tc_fence_before();
            ok = bar_and(1, MAIN, ok);
            if (!ok) break;
            if (wu < 2 && elect_one()) {
                tc_fence_after();
                constexpr uint32_t id_v2 = make_idesc(128, 64, false, false);  // dSbf (TMEM) * Kh^T (K-major B)
                constexpr uint32_t id_s1 = make_idesc(128, 128, true, true);   // dO^T * Qt (MN-major B)
                if (wu == 0) {
#pragma unroll
                    for (int s = 0; s < 8; ++s)
                        mma_ts(tmem0 + VACC, tmem0 + SBF + s * 8, make_desc(sb + KH + s * 256, 128, 2048), id_v2, true);
                    mma_commit(&vbar);
                } else {
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                        mma_ss(tmem0 + SACC, make_desc(sb + DO + s * 4096, 2048, 128), make_desc(sb + QT + s * 4096, 2048, 128), id_s1,
                               true);
                }
            }
            __syncwarp();
            if (!PARTIAL) {
                __nv_bfloat16* gdS = (__nv_bfloat16*)(sc + L.dS) + rec * D * D;
#pragma unroll
                for (int g = 0; g < 4; ++g) store_record16(gdS, e, 64 * half + 16 * g, D, pk[g]);
            }
            ok = mbar_wait(&vbar, k & 1, p, 4) && ok;
            tc_fence_after();
            uint32_t vk[2][8];
            {
                uint32_t r[2][16];
                tmem_ld16(tmem + VACC + 32 * half, r[0]);
                tmem_ld16(tmem + VACC + 32 * half + 16, r[1]);
                tmem_wait_ld();
#pragma unroll
                for (int g = 0; g < 2; ++g) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) vk[g][j] = pack_bf16(__uint_as_float(r[g][2 * j]), __uint_as_float(r[g][2 * j + 1]));
                    tmem_st8(tmem + VBF + (32 * half + 16 * g) / 2, vk[g]);
                }
                tmem_wait_st();
            }
            tc_fence_before();
            ok = bar_and(1, MAIN, ok);
            if (!ok) break;
            if (wu == 1 && elect_one()) {
                tc_fence_after();
                constexpr uint32_t id_w = make_idesc(128, 128, false, false, true);  // -dVbf (TMEM) * W (K-major B, rows = d)
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    mma_ts(tmem0 + SACC, tmem0 + VBF + s * 8, make_desc(sb + WT + s * 256, 128, 1024), id_w, true);
                mma_commit(&sbar);
            }
            __syncwarp();
            if (!PARTIAL) {
                __nv_bfloat16* gdV = (__nv_bfloat16*)(sc + L.dVn) + rec * C * D;
#pragma unroll
                for (int g = 0; g < 2; ++g) store_record16(gdV, e, 32 * half + 16 * g, C, vk[g]);
            }
            ok = mbar_wait(&sbar, k & 1, p, 4) && ok;
            tc_fence_after();
            if (tid == 0) mbar_arrive(&empty[stage]);
            if (!PARTIAL && c == sq.c_begin && c > cb && p.grad_h0 && ok)
                state_drain(tmem + SACC, const_cast<float*>(state_of(p.grad_h0, p, sq.n, h)), vfirst, nullptr, tid, e, half);
            if (++stage == 3) {
                stage = 0;
                ring_phase ^= 1;
            }
        }
        ok = bar_and(1, MAIN, ok);
        if (PARTIAL) {
            if (ok) state_drain(tmem + SACC, segs.E + ((size_t)blockIdx.y * p.H + h) * D * D, false, nullptr, tid, e, half);
        } else if (ok && cb == sq.c_begin && p.grad_h0) {  // (a sequence without tokens hands grad_ht on)
            state_drain(tmem + SACC, const_cast<float*>(state_of(p.grad_h0, p, sq.n, h)), vfirst, stage_space, tid, e, half);
        }
    } else {
        const int pt = tid - MAIN, pw = pt >> 5;
        auto landed = [&](int k) {  // the dO rows of step k are in place: hand them to the tensor cores' proxy
            fence_async_smem();
            __syncwarp();
            if ((pt & 31) == 0) mbar_arrive(&full[k % 3]);
        };
        int k = 0;
        for (; k < nc; ++k) {
            const int stage = k % 3, c = ce - 1 - k;
            if (k >= 3 && !bar_and(2, PROD, mbar_wait(&empty[stage], (k / 3 - 1) & 1, p, 2))) break;
            const size_t rec = (size_t)c * p.H + h;
            unsigned char* b = dyn + stage * STAGE;
            if ((pt & 31) == 0) {
                if (pw == 0) {
                    mbar_expect_tx(&full[stage], TMA_BYTES);
                    tma_load_1d(b + AQ, (const __nv_bfloat16*)(ws + L.Aqk) + rec * C * C, 8192, &full[stage]);
                    tma_load_1d(b + GAM, (const float*)(ws + L.gamC) + rec * D, 512, &full[stage]);
                } else if (pw == 1) {
                    tma_load_1d(b + KH, (const __nv_bfloat16*)(ws + L.Kh) + rec * C * D, 16384, &full[stage]);
                } else if (pw == 2) {
                    tma_load_1d(b + QT, (const __nv_bfloat16*)(ws + L.Qt) + rec * C * D, 16384, &full[stage]);
                } else {
                    tma_load_1d(b + WT, (const __nv_bfloat16*)(ws + L.W) + rec * C * D, 16384, &full[stage]);
                }
            }
            __syncwarp();
            // dO tile -> core-matrix layout cm(i, e; 128), 16-byte chunks, zero rows past the end
            sq.move_to(p, c);
            const long long tok0 = sq.tok(c);
            const int len = sq.rows(c);
            __nv_bfloat16* sdo = reinterpret_cast<__nv_bfloat16*>(b + DO);
#pragma unroll
            for (int u = 0; u < C * (D / 8) / PROD; ++u) {
                const int q = pt + PROD * u, i = q >> 4, e8 = (q & 15) * 8;
                const bool valid = i < len;
                const size_t row = (size_t)(tok0 + (valid ? i : 0)) * p.H + h;
                cp_async16_z(sdo + cm_idx(i, e8, D), dO + row * D + e8, valid);
            }
            cp_async_commit();
            if (k >= 1) {
                cp_async_wait<1>();
                landed(k - 1);
            }
        }
        cp_async_wait<0>();
        if (k == nc && nc > 0) landed(nc - 1);
        // (whatever became of the walk, no copy is in flight when the CTA leaves)
        if (k < nc) {
            if (k > 0) landed(k - 1);
            for (int j = k > 3 ? k - 3 : 0; j < k; ++j) mbar_wait(&full[j % 3], (j / 3) & 1, p, 2);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem0, TMEM_COLS);
}

cudaError_t simt_stage(const KdaParams& p, int stage, cudaStream_t s);
cudaError_t launch_fwd_intra_tc(const KdaParams& p, cudaStream_t s);
cudaError_t launch_bwd_intra(const KdaParams& p, cudaStream_t s);
cudaError_t launch_bwd_wy_tc(const KdaParams& p, cudaStream_t s);
StateSegs state_segs(const KdaParams& p, bool bwd);
cudaError_t launch_fwd_segments(const KdaParams& p, const StateSegs& segs, cudaStream_t s);
cudaError_t launch_seg_combine(const KdaParams& p, const StateSegs& segs, bool bwd, cudaStream_t s);
void prof_mark(cudaStream_t s);

enum { ST_FWD_INTRA = 0, ST_FWD_STATE = 1, ST_BWD_STATE = 2, ST_BWD_CHUNK = 3, ST_PARAM_REDUCE = 4 };

bool tc_supported(const KdaParams& p) { return p.dtype == KDA_DTYPE_BF16 && p.dk == 128 && p.dv == 128; }

static bool stage_simt(const KdaParams& p, int stage) { return (p.flags >> (5 + stage)) & 1; }

cudaError_t tc_fwd(const KdaParams& p, cudaStream_t s) {
    cudaError_t e;
    if ((e = stage_simt(p, ST_FWD_INTRA) ? simt_stage(p, ST_FWD_INTRA, s) : launch_fwd_intra_tc(p, s)) != cudaSuccess) return e;
    prof_mark(s);
    if (stage_simt(p, ST_FWD_STATE)) {
        if ((e = simt_stage(p, ST_FWD_STATE, s)) != cudaSuccess) return e;
    } else {
        const StateSegs segs = state_segs(p, false);
        if (segs.len > 0 && !(p.flags & KDA_FLAG_BORDERS_READY) && (e = launch_fwd_segments(p, segs, s)) != cudaSuccess) return e;
        constexpr int smem = fs::TOTAL;
        if ((e = allow_smem(kda_fwd_state_tc, smem)) != cudaSuccess)
            return e;
        RowMaps maps = {};
        maps.ok = !(p.flags & KDA_FLAG_ROW_COPIES) && make_row_map(&maps.m[0], p.o, (long long)p.B * p.T, p.H, C);
        if ((e = launch_dependent(kda_fwd_state_tc, dim3(p.H, segs.len > 0 ? segs.count : p.N), fs::NTHR, smem, s, p, maps, segs)) != cudaSuccess)
            return e;
    }
    prof_mark(s);
    return cudaGetLastError();
}

cudaError_t tc_bwd(const KdaParams& p, cudaStream_t s) {
    cudaError_t e;
    if (stage_simt(p, ST_BWD_STATE)) {
        if ((e = simt_stage(p, ST_BWD_STATE, s)) != cudaSuccess) return e;
    } else {
        constexpr int smem = 3 * bs::STAGE;
        if ((e = allow_smem(kda_bwd_state_tc<false>, smem)) != cudaSuccess)
            return e;
        const StateSegs segs = state_segs(p, true);
        if (segs.len > 0) {
            if ((e = allow_smem(kda_bwd_state_tc<true>, smem)) != cudaSuccess)
                return e;
            if ((e = launch_dependent(kda_bwd_state_tc<true>, dim3(p.H, segs.count), bs::NTHR, smem, s, p, segs)) != cudaSuccess) return e;
            if ((e = launch_seg_combine(p, segs, true, s)) != cudaSuccess) return e;
        }
        if ((e = launch_dependent(kda_bwd_state_tc<false>, dim3(p.H, segs.len > 0 ? segs.count : p.N), bs::NTHR, smem, s, p, segs)) != cudaSuccess)
            return e;
    }
    prof_mark(s);
    if (stage_simt(p, ST_BWD_CHUNK)) {  // fused FP32-math kernel
        if ((e = simt_stage(p, ST_BWD_CHUNK, s)) != cudaSuccess) return e;
        prof_mark(s);
    } else {  // chunk-level adjoints, then the guarded intra kernel
        if ((e = stage_simt(p, 4) ? simt_stage(p, 5, s) : launch_bwd_wy_tc(p, s)) != cudaSuccess) return e;
        prof_mark(s);
        if ((e = launch_bwd_intra(p, s)) != cudaSuccess) return e;
        prof_mark(s);
    }
    if (p.flags & KDA_FLAG_GATE) {
        if ((e = simt_stage(p, ST_PARAM_REDUCE, s)) != cudaSuccess) return e;
    }
    prof_mark(s);
    return cudaGetLastError();
}

}  // namespace kda

extern "C" int kda_selftest_mma(const float* A, const float* B, float* D, int N, int K, int a_mode, int b_mode, int lbo_a,
                                int sbo_a, int step_a, int lbo_b, int sbo_b, int step_b, int neg_a, int m_rows,
                                int* status, void* stream) {
    if (!A || !B || !D || !status) return KDA_ERR_NULL;
    if (N < 16 || N > 128 || N % 16 || K < 16 || K > 128 || K % 16 || (m_rows != 64 && m_rows != 128)) return KDA_ERR_SHAPE;
    // the strides must keep every operand read inside the tile the kernel wrote
    if (lbo_a < 16 || sbo_a < 16 || lbo_b < 16 || sbo_b < 16 || lbo_a > 4096 || sbo_a > 4096 || lbo_b > 4096 || sbo_b > 4096)
        return KDA_ERR_SHAPE;
    size_t smem = 2 * 128 * 128 * sizeof(__nv_bfloat16);
    cudaError_t e = cudaFuncSetAttribute(kda::mma_selftest_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return KDA_ERR_LAUNCH;
    kda::mma_selftest_kernel<<<1, 128, smem, (cudaStream_t)stream>>>(A, B, D, N, K, a_mode, b_mode, lbo_a, sbo_a, step_a,
                                                                     lbo_b, sbo_b, step_b, neg_a, m_rows, status);
    return cudaGetLastError() == cudaSuccess ? KDA_OK : KDA_ERR_LAUNCH;
}

extern "C" int kda_selftest_wait(const float* src, float* dst, int poll_limit, int code, int* status, void* stream) {
    if (!src || !dst || !status) return KDA_ERR_NULL;
    if (poll_limit < 1 || poll_limit > 4096 || code < 1 || code > 255) return KDA_ERR_SHAPE;
    if (((uintptr_t)src & 15) != 0) return KDA_ERR_ALIGN;
    kda::wait_selftest_kernel<<<1, 128, 0, (cudaStream_t)stream>>>(src, dst, (uint32_t)poll_limit, code, status);
    return cudaGetLastError() == cudaSuccess ? KDA_OK : KDA_ERR_LAUNCH;
}

KDA_PHASE_EXPORT(kda_debug_phases_state)
