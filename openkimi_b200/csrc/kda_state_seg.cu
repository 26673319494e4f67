// The state recurrence of long sequences in parallel segments (BF16 path, d = 128).
//
// kda_fwd_state_tc / kda_bwd_state_tc walk the chunks of a sequence one after the other: a chain of dependent MMA
// round trips (about 2 us per chunk) on ONE SM per (sequence, head), while a batch of few or unevenly long sequences
// leaves most of the 148 SMs idle.  A chunk maps its entering state linearly,
//     S1^T = S0^T M + (U^T Kh),        M = diag(gamma) - W^T Kh,
// so the chunks are cut into segments of equal length (in the global chunk numbering, across sequence borders):
//   1  every segment runs the recurrence from a zero state -> its own contribution E, and, if it lies inside one
//      sequence, from the identity -> its transition X = M_1 M_2 ... (both at once, two halves of one CTA)
//   2  the states at the segment borders follow one after the other, S = S X + E, in FP32 on the CUDA cores
//      (the rows of S^T are independent: 16 CTAs per chain, eight rows each)
//   3  every segment runs as before, from its true entering state
// X carries the same BF16 operands and FP32 accumulators as the state itself; step 2 rounds nothing.  The backward
// walks the other way with X^T.  Work doubles (and X costs as much again, on warps that would idle), the chain shrinks
// from n chunks to 2 len + n / len short steps.
//
// Measured (six heads, the launches of the stage together): one sequence of 256 chunks, forward: 503 -> 95 us, of which
// some 30 for step 1 and 35 for step 3 (at 148 busy SMs the walks are bound by the records' traffic, 5.5 TB/s); 16 documents of
// 65536 tokens, both directions: 905 -> 514 us; 4 sequences of 64 chunks, both directions: 339 -> 183 us.
#include <math.h>

#include <algorithm>

#include "kda_common.cuh"
#include "kda_state.cuh"
#include "kda_tc.cuh"

namespace kda {

using namespace tc;

namespace sg {
constexpr int D = 128, NTHR = 512;
constexpr uint32_t WT = 0, UT = 16384, KH = 32768, GAM = 49152, STAGE = 49664, TOTAL = 2 * STAGE;
// tensor memory of one half: state, BF16 copy (V' takes its place once the first product has read it), first product
constexpr uint32_t SACC = 0, SBF = 128, WSACC = 192, HALF_COLS = 256, TMEM_COLS = 512;
}  // namespace sg

// X is kept as X^T, chunks of row r swizzled by r: consecutive lanes write it coalesced (lane = row of X), and it can be
// read from a linear copy in shared memory without bank conflicts both along rows (backward) and by threads that own
// one row each (forward)
__device__ __forceinline__ int xt_idx(int r, int c) { return r * 128 + ((((c >> 2) ^ (r & 31)) << 2) | (c & 3)); }

__global__ void __launch_bounds__(sg::NTHR, 1) kda_fwd_segment_tc(const KdaParams p, const StateSegs segs) {
    using namespace sg;
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ uint64_t full[2], mmabar;
    __shared__ uint32_t tmem_s;
    // part 0 carries the state, part 1 the transition; inside a part as in kda_fwd_state_tc
    const int tid = threadIdx.x, warp = tid >> 5, e = tid & 127, half = (tid >> 7) & 1, part = tid >> 8;
    const int h = blockIdx.x, seg = blockIdx.y;
    pdl_wait();
    int cb = seg * segs.len;
    const int ce = min(cb + segs.len, p.NT);
    SeqCursor sq;
    sq.load_of_chunk(p, ce - 1);
    if (sq.c_end == ce) return;                // nobody needs the state at the end of this segment
    const bool inside = sq.c_begin < cb;       // the sequence came in from the previous segment
    cb = max(cb, sq.c_begin);
    const WsLayout L = ws_layout(p.NT, p.H, p.dk, p.dv, p.dtype);
    const char* ws = (const char*)p.workspace;
    if (warp == 0) {
        tmem_alloc(&tmem_s, TMEM_COLS);
        tmem_relinquish();
    }
    if (tid == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        mbar_init(&mmabar, inside ? 2 : 1);
        mbar_fence_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem0 = tmem_s + part * HALF_COLS;
    const uint32_t tmem = tmem0 + ((uint32_t)((warp & 3) * 32) << 16);
    const bool on = part == 0 || inside;
    if (part == 1) {  // identity
        for (int d0 = 64 * half; d0 < 64 * half + 64; d0 += 16) {
            uint32_t r[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = d0 + j == e ? __float_as_uint(1.f) : 0u;
            tmem_st16(tmem + SACC + d0, r);
        }
        tmem_wait_st();
    } else {
        state_fill(tmem + SACC, inside ? nullptr : state_of(p.h0, p, sq.n, h), p.flags & KDA_FLAG_STATE_V_FIRST, nullptr, tid, e, half);
    }
    auto issue_loads = [&](int c, int stage) {
        if ((tid & 31) != 0 || warp >= 4) return;
        const size_t rec = (size_t)c * p.H + h;
        unsigned char* b = dyn + stage * STAGE;
        if (warp == 0) {
            mbar_expect_tx(&full[stage], STAGE);
            tma_load_1d(b + WT, (const __nv_bfloat16*)(ws + L.W) + rec * C * D, 16384, &full[stage]);
        } else if (warp == 1) {
            tma_load_1d(b + UT, (const __nv_bfloat16*)(ws + L.U) + rec * C * D, 16384, &full[stage]);
        } else if (warp == 2) {
            tma_load_1d(b + KH, (const __nv_bfloat16*)(ws + L.Kh) + rec * C * D, 16384, &full[stage]);
        } else {
            tma_load_1d(b + GAM, (const float*)(ws + L.gamC) + rec * D, 512, &full[stage]);
        }
    };
    issue_loads(cb, 0);
    uint32_t phase = 0;
    bool ok = true;
    for (int c = cb; c < ce; ++c) {
        const int stage = (c - cb) & 1;
        unsigned char* b = dyn + stage * STAGE;
        if (c + 1 < ce) issue_loads(c + 1, stage ^ 1);
        ok = mbar_wait(&full[stage], ((c - cb) >> 1) & 1, p, 2);
        if (!__syncthreads_and(ok)) { ok = false; break; }
        if (on) {  // BF16 copy of the entering state, decay
            const float* gam = reinterpret_cast<const float*>(b + GAM);
            for (int d0 = 64 * half; d0 < 64 * half + 64; d0 += 16) {
                uint32_t r[16], pk[8];
                tmem_ld16(tmem + SACC + d0, r);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 8; ++j) pk[j] = pack_bf16(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
                tmem_st8(tmem + SBF + d0 / 2, pk);
#pragma unroll
                for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * gam[d0 + j]);
                tmem_st16(tmem + SACC + d0, r);
            }
            tmem_wait_st();
        }
        tc_fence_before();
        __syncthreads();
        const uint32_t sb = smem_u32(b);
        if ((tid & 255) == 0 && on) {
            tc_fence_after();
            constexpr uint32_t id_mn = make_idesc(128, 64, false, true);
#pragma unroll
            for (int s = 0; s < 8; ++s)  // (W S)^T = Sbf (K = d) * W^T record
                mma_ts(tmem0 + WSACC, tmem0 + SBF + s * 8, make_desc(sb + WT + s * 2048, 1024, 128), id_mn, s > 0);
            mma_commit(&mmabar);
        }
        ok = mbar_wait(&mmabar, phase, p, 4);
        phase ^= 1;
        tc_fence_after();
        if (!__syncthreads_and(ok)) { ok = false; break; }
        if (on) {  // V'^T = U^T - (W S)^T; the transition has no U
            const __nv_bfloat16* sU = reinterpret_cast<const __nv_bfloat16*>(b + UT);
            for (int i0 = 32 * half; i0 < 32 * half + 32; i0 += 16) {
                uint32_t r[16], pk[8];
                float u[16];
                tmem_ld16(tmem + WSACC + i0, r);
                tmem_wait_ld();
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    float t8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                    if (part == 0) bf16x8_to_f32(*reinterpret_cast<const uint4*>(sU + cm_idx(e, i0 + 8 * g, C)), t8);
#pragma unroll
                    for (int j = 0; j < 8; ++j) u[8 * g + j] = t8[j];
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    pk[j] = pack_bf16(u[2 * j] - __uint_as_float(r[2 * j]), u[2 * j + 1] - __uint_as_float(r[2 * j + 1]));
                tmem_st8(tmem + SBF + i0 / 2, pk);
            }
            tmem_wait_st();
        }
        tc_fence_before();
        __syncthreads();
        if ((tid & 255) == 0 && on) {
            tc_fence_after();
            constexpr uint32_t id_s = make_idesc(128, 128, false, true);
#pragma unroll
            for (int s = 0; s < 4; ++s)  // Sacc += V'^T (K = i) * Kh
                mma_ts(tmem0 + SACC, tmem0 + SBF + s * 8, make_desc(sb + KH + s * 4096, 2048, 128), id_s, true);
            mma_commit(&mmabar);
        }
        ok = mbar_wait(&mmabar, phase, p, 4);
        phase ^= 1;
        tc_fence_after();
        if (!__syncthreads_and(ok)) { ok = false; break; }
    }
    if (ok && on) {
        const size_t base = ((size_t)seg * p.H + h) * D * D;
        if (part == 0) {
            state_drain(tmem + SACC, segs.E + base, false, nullptr, tid, e, half);
        } else {
            for (int d0 = 64 * half; d0 < 64 * half + 64; d0 += 16) {
                uint32_t r[16];
                tmem_ld16(tmem + SACC + d0, r);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 16; ++j) segs.X[base + xt_idx(d0 + j, e)] = __uint_as_float(r[j]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_s, TMEM_COLS);
}

// Step 2.  One CTA per (sequence, head, eight rows of S^T): E of every segment that a sequence leaves becomes the true
// state there.  Thread = two columns x a quarter of the inner index, in packed FP32 pairs; X arrives by bulk copies (64 KB
// per step and CTA from L2, as long as the arithmetic); 1.3 us a step, twice that with sixteen rows per CTA and no less
// with 512 threads.  Latency bound: with STAGES = 2 a CTA has the next segment's X in
// flight, with STAGES = 1 two CTAs share an SM (more chains than one CTA per SM covers).
namespace sc {
constexpr int D = 128, ROWS = 8, NTHR = 256, GROUPS = NTHR / 64, OWN = D * ROWS / NTHR;
constexpr uint32_t XBYTES = D * D * 4, SBYTES = D * ROWS * 4;
constexpr uint32_t total(int stages) { return stages * XBYTES + SBYTES + GROUPS * SBYTES; }
}  // namespace sc

template <bool BWD, int STAGES>
__global__ void __launch_bounds__(sc::NTHR, 3 - STAGES) kda_seg_combine(const KdaParams p, const StateSegs segs) {
    using namespace sc;
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ uint64_t full[2];
    const int tid = threadIdx.x, h = blockIdx.y, n = blockIdx.z, e0 = blockIdx.x * ROWS;
    pdl_wait();
    int c0, nc;
    seq_chunks(p, n, c0, nc);
    if (nc == 0) {  // no chunk of this sequence is visited by any segment: its state passes through here
        const float* src = BWD ? p.grad_ht : p.h0;
        float* dst = BWD ? p.grad_h0 : p.ht;
        if (dst)
            for (int i = tid; i < ROWS * D; i += NTHR) {
                const size_t at = ((size_t)n * p.H + h) * D * D + state_idx(p, i & (D - 1), e0 + i / D);
                dst[at] = src ? src[at] : 0.f;
            }
        return;
    }
    const int sa = c0 / segs.len, sz = (c0 + nc - 1) / segs.len;  // first and last segment of the sequence
    const int steps = sz - sa - 1;                                // transitions to apply
    if (steps <= 0) return;
    if (tid == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        mbar_fence_init();
    }
    __syncthreads();
    auto mat = [&](int k) { return ((size_t)(BWD ? sz - k : sa + k) * p.H + h) * D * D; };  // k-th segment from the known end
    auto issue = [&](int k) {
        if (tid == 0) {
            const int st = STAGES == 2 ? k & 1 : 0;
            mbar_expect_tx(&full[st], XBYTES);
            tma_load_1d(dyn + st * XBYTES, segs.X + mat(k), XBYTES, &full[st]);
        }
    };
    float* S = reinterpret_cast<float*>(dyn + STAGES * XBYTES);  // [d][row]
    float* part = S + D * ROWS;                                   // [group][column][row]
    issue(1);
    if (STAGES == 2 && steps > 1) issue(2);
    // thread's share of the rows: OWN of one column d
    const int md = tid / (ROWS / OWN), mr = OWN * (tid & (ROWS / OWN - 1));
    static_assert(OWN == 4, "one 16-byte word");
    *reinterpret_cast<float4*>(S + md * ROWS + mr) = *reinterpret_cast<const float4*>(segs.E + mat(0) + (size_t)md * D + e0 + mr);
    const int lane64 = tid & 63, group = tid >> 6;
    for (int k = 1; k <= steps; ++k) {
        float4* E = reinterpret_cast<float4*>(segs.E + mat(k) + (size_t)md * D + e0 + mr);
        const float4 own = *E;
        const bool ok = STAGES == 2 ? mbar_wait(&full[k & 1], ((k - 1) >> 1) & 1, p, 2) : mbar_wait(&full[0], (k - 1) & 1, p, 2);
        if (!__syncthreads_and(ok)) {
            if (STAGES == 2 && k < steps) mbar_wait(&full[(k + 1) & 1], (k >> 1) & 1, p, 2);  // the other copy in flight
            return;
        }
        const float* x = reinterpret_cast<const float*>(dyn + (STAGES == 2 ? k & 1 : 0) * XBYTES);
        float2 acc[2][ROWS / 2];  // two columns, pairs of rows
#pragma unroll
        for (int r = 0; r < ROWS / 2; ++r) acc[0][r] = acc[1][r] = make_float2(0.f, 0.f);
        const int colA = BWD ? 2 * lane64 : lane64, colB = BWD ? 2 * lane64 + 1 : lane64 + 64;
#pragma unroll 4
        for (int d = group * (D / GROUPS); d < (group + 1) * (D / GROUPS); d += 4) {
            float xa[4], xb[4];
            if (BWD) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 v = *reinterpret_cast<const float2*>(x + xt_idx(d + j, colA));
                    xa[j] = v.x; xb[j] = v.y;
                }
            } else {
                const float4 va = *reinterpret_cast<const float4*>(x + xt_idx(colA, d)), vb = *reinterpret_cast<const float4*>(x + xt_idx(colB, d));
                xa[0] = va.x; xa[1] = va.y; xa[2] = va.z; xa[3] = va.w;
                xb[0] = vb.x; xb[1] = vb.y; xb[2] = vb.z; xb[3] = vb.w;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float2 sv[ROWS / 2];
#pragma unroll
                for (int r = 0; r < ROWS / 4; ++r) {
                    const float4 t = *reinterpret_cast<const float4*>(S + (d + j) * ROWS + 4 * r);
                    sv[2 * r] = make_float2(t.x, t.y);
                    sv[2 * r + 1] = make_float2(t.z, t.w);
                }
                const float2 a2 = make_float2(xa[j], xa[j]), b2 = make_float2(xb[j], xb[j]);
#pragma unroll
                for (int r = 0; r < ROWS / 2; ++r) {
                    acc[0][r] = __ffma2_rn(sv[r], a2, acc[0][r]);
                    acc[1][r] = __ffma2_rn(sv[r], b2, acc[1][r]);
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            float* dst = part + (group * D + (c ? colB : colA)) * ROWS;
#pragma unroll
            for (int r = 0; r < ROWS / 4; ++r)
                *reinterpret_cast<float4*>(dst + 4 * r) = make_float4(acc[c][2 * r].x, acc[c][2 * r].y, acc[c][2 * r + 1].x, acc[c][2 * r + 1].y);
        }
        __syncthreads();
        if (k + STAGES <= steps) issue(k + STAGES);
        float4 v = own;
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            const float4 t = *reinterpret_cast<const float4*>(part + (g * D + md) * ROWS + mr);
            v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
        }
        *E = v;
        *reinterpret_cast<float4*>(S + md * ROWS + mr) = v;
        __syncthreads();
    }
}

// CTAs of step 2, counting one chain per sequence and head
static long long combine_ctas(const KdaParams& p) { return (long long)p.N * p.H * (sc::D / sc::ROWS); }

// Segment length, 0 for whole sequences, from the times measured on a B200 (us): a walk takes 6 plus 2.1 per chunk of the
// longest sequence (the dependent chain) or 2.4 per chunk and SM (the records' traffic); both passes over segments of
// `len` take 18 (three launches) plus 4.5 len plus 1.4 per segment border and wave of step 2.  len is what one wave of
// the chip needs, but no shorter than what balances the border steps.
static int segment_length(const KdaParams& p) {
    if (p.NT < 8) return 0;
    const double sms = sm_count();
    const double longest = p.max_chunks > 0 ? p.max_chunks : (double)p.NT / p.N;
    const double per_sm = p.NT * (double)p.H / sms;
    const double border = 1.4 * ceil(combine_ctas(p) / (2.0 * sms));
    const int len = (int)ceil(std::max(per_sm, sqrt(longest * border / 4.5)));
    const double whole = 6.0 + std::max(2.1 * longest, 2.4 * per_sm);
    const double split = 18.0 + 4.5 * len + border * longest / len;
    return split < 0.9 * whole ? len : 0;
}

int segment_count(const KdaParams& p) {
    if (p.dtype != KDA_DTYPE_BF16 || p.dk != 128 || p.dv != 128 || p.NT <= 0 || p.N <= 0) return 0;
    if (p.flags & (KDA_FLAG_FORCE_SIMT | (3 << 6))) return 0;  // a state stage in FP32 arithmetic
    const int len = segment_length(p);
    return len > 0 ? (p.NT + len - 1) / len : 0;
}

StateSegs state_segs(const KdaParams& p, bool bwd) {
    StateSegs r = {};
    r.count = segment_count(p);
    if (r.count == 0) return r;
    r.len = segment_length(p);
    const size_t m = seg_matrix_floats(r.count, p.H, p.dk);
    const WsLayout L = ws_layout(p.NT, p.H, p.dk, p.dv, p.dtype);
    const bool nosave = p.flags & KDA_FLAG_NO_SAVE;
    float* f = p.borders ? p.borders : (float*)((char*)p.workspace + (nosave ? L.total_nosave : p.conv_q ? L.total_conv : L.total));
    r.E = f;
    r.X = f + m;
    if (bwd) r.E = (float*)((char*)p.bwd_scratch + (p.conv_q ? L.bwd_total_conv : L.bwd_total));
    return r;
}

cudaError_t launch_seg_combine(const KdaParams& p, const StateSegs& segs, bool bwd, cudaStream_t s) {
    const bool two = combine_ctas(p) > sm_count();  // two CTAs per SM
    auto kern = bwd ? (two ? kda_seg_combine<true, 1> : kda_seg_combine<true, 2>)
                    : (two ? kda_seg_combine<false, 1> : kda_seg_combine<false, 2>);
    const int smem = (int)sc::total(two ? 1 : 2);
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    return launch_dependent(kern, dim3(sc::D / sc::ROWS, p.H, p.N), sc::NTHR, smem, s, p, segs);
}

cudaError_t launch_fwd_segments(const KdaParams& p, const StateSegs& segs, cudaStream_t s) {
    cudaError_t e = allow_smem(kda_fwd_segment_tc, (int)sg::TOTAL);
    if (e != cudaSuccess) return e;
    if ((e = launch_dependent(kda_fwd_segment_tc, dim3(p.H, segs.count), sg::NTHR, sg::TOTAL, s, p, segs)) != cudaSuccess) return e;
    return launch_seg_combine(p, segs, false, s);
}

}  // namespace kda
