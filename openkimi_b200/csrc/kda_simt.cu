// KDA chunkwise forward and backward with FP32 CUDA-core arithmetic.
//
// This is the "FP32-operand validation mode" of the library: every contraction is an FP32
// FMA loop, every pairwise decay 2^(G_i - G_j) is evaluated exactly (no factorisation, so
// no span guard is needed), and the state is FP32.  The same four stages, with the same
// workspace records, are what the tensor-core kernels implement:
//
//   fwd_intra  (one CTA per chunk x head)   prologue, Aqk, L, T=(I+diag(beta)L)^-1, W, U
//   fwd_state  (one CTA per seq x head x dv-panel, sequential over chunks)  V', O, S
//   bwd_state  (same grid, reverse order)   dV', dS
//   bwd_chunk  (one CTA per chunk x head)   everything else, down to the raw-input grads
//
// The math follows the recurrence of k3mini/model.py:115-129 rewritten per 64-token chunk.
// (the SPLIT instantiation of kda_bwd_chunk returns early by design: no "unreachable loop" remarks)
#pragma nv_diag_suppress 128
#include "kda_common.cuh"
#include "kda_tc.cuh"

namespace kda {

void prof_mark(cudaStream_t s);
cudaError_t simt_state(const KdaParams& p, bool bwd, cudaStream_t s);  // kda_simt_state.cu

constexpr int NTHREADS = 256;
constexpr int KS = 16;  // k-slice of the tile product
template <int D>
__host__ __device__ constexpr int row_stride() { return D + 4; }  // rows of q, k, G, v in shared memory: no bank conflict down a column
constexpr int CP = C + 4;  // row stride of the [64][64] matrices in shared memory: rows start on 16-byte boundaries

// thread (ty, tx) = (tid / 16, tid % 16) owns rows 4 ty + r and columns col(tx, c) of a tile product
__device__ __forceinline__ int tile_col(int tx, int c) { return 4 * tx + (c & 3) + 64 * (c >> 2); }

// ---------------------------------------------------------------------------------------
// acc[4][N/16] += A[64 x K] * B[K x N], operands fetched through functors la(m,k), lb(k,n)
// (from global or shared memory, any element type) and staged through shared memory in
// slices of KS.  A thread's 4 x 4 (4 x 8) tile costs two (three) 16-byte shared loads per k;
// the next slice is fetched into registers while the current one is worked on, and the two
// staging buffers alternate, so that a slice costs one barrier and no exposed memory latency.
// a_kfast / b_kfast say which index is contiguous in the operand's memory, so that the
// staging loads coalesce.
// ---------------------------------------------------------------------------------------
template <int N>
constexpr int st_floats() { return 2 * KS * (C + 4 + N + 4); }

template <int M, int N, class LA, class LB>
__device__ __forceinline__ void mm_tile(float (&acc)[4][N / 16], int K, LA la, LB lb, float* st, bool a_kfast, bool b_kfast) {
    static_assert(M == C, "64 output rows");
    constexpr int SA = M + 4, SB = N + 4, BUF = KS * (SA + SB), NA = M * KS / NTHREADS, NB = N * KS / NTHREADS;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    float ra[NA], rb[NB];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int u = 0; u < NA; ++u) {
            const int idx = tid + NTHREADS * u;
            ra[u] = a_kfast ? la(idx / KS, k0 + idx % KS) : la(idx % M, k0 + idx / M);
        }
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            const int idx = tid + NTHREADS * u;
            rb[u] = b_kfast ? lb(k0 + idx % KS, idx / KS) : lb(k0 + idx / N, idx % N);
        }
    };
    __syncthreads();  // operands in shared memory are complete
    fetch(0);
    for (int k0 = 0, buf = 0; k0 < K; k0 += KS, buf ^= 1) {
        float *stA = st + buf * BUF, *stB = stA + KS * SA;
#pragma unroll
        for (int u = 0; u < NA; ++u) {
            const int idx = tid + NTHREADS * u;
            stA[a_kfast ? (idx % KS) * SA + idx / KS : (idx / M) * SA + idx % M] = ra[u];
        }
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            const int idx = tid + NTHREADS * u;
            stB[b_kfast ? (idx % KS) * SB + idx / KS : (idx / N) * SB + idx % N] = rb[u];
        }
        __syncthreads();
        if (k0 + KS < K) fetch(k0 + KS);
#pragma unroll 4
        for (int k = 0; k < KS; ++k) {  // (not unrolled further: a CTA runs the code of every product once)
            float a[4], b[N / 16];
            const float4 av = *reinterpret_cast<const float4*>(stA + k * SA + 4 * ty);
            a[0] = av.x; a[1] = av.y; a[2] = av.z; a[3] = av.w;
#pragma unroll
            for (int g = 0; g < N / 64; ++g) {
                const float4 bv = *reinterpret_cast<const float4*>(stB + k * SB + 64 * g + 4 * tx);
                b[4 * g] = bv.x; b[4 * g + 1] = bv.y; b[4 * g + 2] = bv.z; b[4 * g + 3] = bv.w;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < N / 16; ++c) acc[r][c] = fmaf(a[r], b[c], acc[r][c]);
        }
    }
    __syncthreads();
}

template <int M, int N>
__device__ __forceinline__ void zero_acc(float (&acc)[M][N]) {
#pragma unroll
    for (int r = 0; r < M; ++r)
#pragma unroll
        for (int c = 0; c < N; ++c) acc[r][c] = 0.f;
}

// sum over the 16 lanes that share a row (tx = 0..15 within a half warp)
__device__ __forceinline__ float row16_sum(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------------------------------
// Prologue of one chunk x head into shared memory:
//   sq, sk  normalised q, k (x / max(||x||, 1e-6), k3mini/model.py:218-219) or raw
//   sG      inclusive cumulative log2-decay of the chunk (rows >= len repeat the last value)
//   sv      v (optional)          sbeta  beta after the optional sigmoid (0 on padding rows)
//   srq,srk 1 / max(||x||, eps) per row (1 when the norm is not applied); scratch: 4 D floats
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ float4 load_quad(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load_quad(const __nv_bfloat16* p) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16),
                       __uint_as_float(r.y & 0xffff0000u));
}

template <typename T, int D>
__device__ __forceinline__ void load_prologue(const KdaParams& p, const ChunkInfo& ci, int h, float* sq, float* sk,
                                              float* sG, float* sv, float* sbeta, float* srq, float* srk, float* scratch) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool l2 = p.flags & KDA_FLAG_QK_L2NORM, gate = p.flags & KDA_FLAG_GATE, sig = p.flags & KDA_FLAG_BETA_SIGMOID;
    const float negA = gate ? -expf(p.A_log[h]) : 0.f;
    // the rows of the chunk, four elements per access and all of a thread's accesses to a tensor in flight at once
    constexpr int QN = C * D / 4 / NTHREADS;
    auto rows_in = [&](const T* src, float* dst, bool is_gate) {
        float4 x[QN];
#pragma unroll
        for (int u = 0; u < QN; ++u) {
            const int idx = tid + NTHREADS * u, r = idx / (D / 4), d = idx % (D / 4) * 4;
            x[u] = r < ci.len ? load_quad(src + ((size_t)(ci.tok0 + r) * p.H + h) * D + d) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < QN; ++u) {
            const int idx = tid + NTHREADS * u, r = idx / (D / 4), d = idx % (D / 4) * 4;
            float4 y = x[u];
            if (is_gate) {
                float v[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (gate) v[j] = negA * softplus_f(v[j] + (p.dt_bias ? p.dt_bias[h * D + d + j] : 0.f));
                    v[j] = r < ci.len ? v[j] * LOG2E : 0.f;
                }
                y = make_float4(v[0], v[1], v[2], v[3]);
            }
            *reinterpret_cast<float4*>(dst + r * row_stride<D>() + d) = y;
        }
    };
    rows_in((const T*)p.q, sq, false);
    rows_in((const T*)p.k, sk, false);
    rows_in((const T*)p.g, sG, true);
    if (sv) rows_in((const T*)p.v, sv, false);
    if (tid < C) {
        float b = 0.f;
        if (tid < ci.len) {
            b = ldf((const T*)p.beta + (size_t)(ci.tok0 + tid) * p.H + h);
            if (sig) b = sigmoid_f(b);
        }
        sbeta[tid] = b;
    }
    __syncthreads();
    // cumulative gate: 16-row groups summed on their own, then the totals of the groups before are added
    for (int it = tid; it < D * 4; it += NTHREADS) {
        const int d = it % D, grp = it / D;
        float run = 0.f;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            run += sG[(16 * grp + r) * row_stride<D>() + d];
            sG[(16 * grp + r) * row_stride<D>() + d] = run;
        }
        scratch[it] = run;
    }
#pragma unroll 4
    for (int r = warp; r < C; r += NTHREADS / 32) {
        float rq = 1.f, rk = 1.f;
        if (l2) {
            float ssq = 0.f, ssk = 0.f;
#pragma unroll
            for (int m = 0; m < D / 32; ++m) {
                const float a = sq[r * row_stride<D>() + lane + 32 * m], b = sk[r * row_stride<D>() + lane + 32 * m];
                ssq += a * a;
                ssk += b * b;
            }
            ssq = warp_sum(ssq);
            ssk = warp_sum(ssk);
            rq = 1.f / fmaxf(sqrtf(ssq), 1e-6f);
            rk = 1.f / fmaxf(sqrtf(ssk), 1e-6f);
#pragma unroll
            for (int m = 0; m < D / 32; ++m) {
                sq[r * row_stride<D>() + lane + 32 * m] *= rq;
                sk[r * row_stride<D>() + lane + 32 * m] *= rk;
            }
        }
        if (lane == 0) {
            srq[r] = rq;
            srk[r] = rk;
        }
    }
    __syncthreads();
    for (int it = tid; it < D * 4; it += NTHREADS) {
        const int d = it % D, grp = it / D;
        if (grp == 0) continue;
        float before = 0.f;
        for (int g = 0; g < grp; ++g) before += scratch[g * D + d];
#pragma unroll
        for (int r = 0; r < 16; ++r) sG[(16 * grp + r) * row_stride<D>() + d] += before;
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------------------
// fwd_intra
// ---------------------------------------------------------------------------------------
template <typename T, int D>
__global__ void __launch_bounds__(NTHREADS, 1) kda_fwd_intra_simt(const KdaParams p) {
    extern __shared__ __align__(16) float smem[];
    float* sq = smem;
    float* sk = sq + C * row_stride<D>();
    float* sG = sk + C * row_stride<D>();
    float* sv = sG + C * row_stride<D>();
    float* sA = sv + C * row_stride<D>();       // [64][CP]
    float* sL = sA + C * CP;
    float* sT = sL + C * CP;
    float* sbeta = sT + C * CP;
    float* srq = sbeta + C;
    float* srk = srq + C;
    float* st = srk + C;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ty = tid >> 4, tx = tid & 15;
    const int c = blockIdx.x / p.H, h = blockIdx.x % p.H;
    pdl_wait();
    const ChunkInfo ci = chunk_info(p, c);
    const WsLayout L = ws_layout(p.NT, p.H, p.dk, p.dv, p.dtype);
    char* ws = (char*)p.workspace;
    const size_t rec = (size_t)c * p.H + h;
    T* gW = (T*)(ws + L.W) + rec * C * D;
    T* gU = (T*)(ws + L.U) + rec * C * D;
    T* gA = (T*)(ws + L.Aqk) + rec * C * C;
    T* gQt = (T*)(ws + L.Qt) + rec * C * D;
    T* gKh = (T*)(ws + L.Kh) + rec * C * D;
    T* gT = (T*)(ws + L.Tm) + rec * C * C;
    float* gGam = (float*)(ws + L.gamC) + rec * D;

    load_prologue<T, D>(p, ci, h, sq, sk, sG, sv, sbeta, srq, srk, st);
    const bool save = !(p.flags & KDA_FLAG_NO_SAVE);  // forward-only calls keep nothing for a backward
    if (save) {  // prologue results kept for the backward
        float* gGc = (float*)(ws + L.Gc) + rec * C * D;
        T* gQn = (T*)(ws + L.Qn) + rec * C * D;
        T* gKn = (T*)(ws + L.Kn) + rec * C * D;
        float* gaux = (float*)(ws + L.aux) + rec * 3 * C;
        for (int idx = tid; idx < C * D; idx += NTHREADS) {
            // d = 128: the chunk-swizzled row layout the tensor-core backward reads (swz_f32 / swz_bf16)
            const int r = idx / D, dd = idx % D;
            gGc[D == 128 ? tc::swz_f32(r, dd) : idx] = sG[r * row_stride<D>() + dd];
            stf(gQn + (D == 128 ? (sizeof(T) == 2 ? tc::swz_bf16(r, dd) : tc::swz_f32(r, dd)) : idx), sq[r * row_stride<D>() + dd]);
            stf(gKn + (D == 128 ? (sizeof(T) == 2 ? tc::swz_bf16(r, dd) : tc::swz_f32(r, dd)) : idx), sk[r * row_stride<D>() + dd]);
        }
        if (tid < C) {
            gaux[tid] = srq[tid];
            gaux[C + tid] = srk[tid];
            gaux[2 * C + tid] = sbeta[tid];
        }
    }

    // exact pairwise products.  A warp takes the rows i and 63 - i (65 pairs together, the same for every warp); its
    // lanes are eight keys x four quarters of the channels, so that a pair costs two shuffles per product instead of five
    {
        constexpr int DQ = D / 4;
        const int jl = lane >> 2, dq0 = (lane & 3) * 4;  // quarter: channels 4 (lane & 3) + 16 m + {0..3}
        for (int it = warp; it < C; it += NTHREADS / 32) {
            const int i = it < C / 2 ? it : C - 1 - (it - C / 2);
            float4 qi[DQ / 4], ki[DQ / 4], gi[DQ / 4];
#pragma unroll
            for (int m = 0; m < DQ / 4; ++m) {
                qi[m] = *reinterpret_cast<const float4*>(sq + i * row_stride<D>() + dq0 + 16 * m);
                ki[m] = *reinterpret_cast<const float4*>(sk + i * row_stride<D>() + dq0 + 16 * m);
                gi[m] = *reinterpret_cast<const float4*>(sG + i * row_stride<D>() + dq0 + 16 * m);
            }
            for (int j0 = 0; j0 < C; j0 += 8) {
                const int j = j0 + jl, jr = j < i ? j : i;  // (lanes past the diagonal repeat it)
                float a = 0.f, l = 0.f;
                if (j0 <= i) {
#pragma unroll
                    for (int m = 0; m < DQ / 4; ++m) {
                        const float4 kj = *reinterpret_cast<const float4*>(sk + jr * row_stride<D>() + dq0 + 16 * m);
                        const float4 gj = *reinterpret_cast<const float4*>(sG + jr * row_stride<D>() + dq0 + 16 * m);
                        float kd = kj.x * exp2f(gi[m].x - gj.x);
                        a = fmaf(qi[m].x, kd, a);
                        l = fmaf(ki[m].x, kd, l);
                        kd = kj.y * exp2f(gi[m].y - gj.y);
                        a = fmaf(qi[m].y, kd, a);
                        l = fmaf(ki[m].y, kd, l);
                        kd = kj.z * exp2f(gi[m].z - gj.z);
                        a = fmaf(qi[m].z, kd, a);
                        l = fmaf(ki[m].z, kd, l);
                        kd = kj.w * exp2f(gi[m].w - gj.w);
                        a = fmaf(qi[m].w, kd, a);
                        l = fmaf(ki[m].w, kd, l);
                    }
#pragma unroll
                    for (int o = 1; o <= 2; o <<= 1) {
                        a += __shfl_xor_sync(0xffffffffu, a, o);
                        l += __shfl_xor_sync(0xffffffffu, l, o);
                    }
                }
                if ((lane & 3) == 0) {
                    sA[i * CP + j] = (j <= i) ? a * p.scale : 0.f;
                    sL[i * CP + j] = (j < i) ? l : 0.f;
                }
            }
        }
    }
    __syncthreads();

    // T = (I + diag(beta) L)^-1 by forward substitution, 16 rows at a time: four lanes of a warp own a column, first sum
    // what the rows before the block contribute, then solve the block in registers.  No barrier between dependent rows.
    {
        const int col = tid >> 2, part = tid & 3;
        for (int b = 0; b < C; b += 16) {
            float s[16], t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int r = 0; r < 16; ++r) s[r] = 0.f;
            for (int j = part; j < b; j += 4) {
                const float tj = sT[j * CP + col];
#pragma unroll
                for (int r = 0; r < 16; ++r) s[r] = fmaf(sL[(b + r) * CP + j], tj, s[r]);
            }
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                float x = s[r];
#pragma unroll
                for (int m = 0; 4 * m < r; ++m) x = fmaf(sL[(b + r) * CP + b + 4 * m + part], t[m], x);  // (unknown entries are 0)
                x += __shfl_xor_sync(0xffffffffu, x, 1);
                x += __shfl_xor_sync(0xffffffffu, x, 2);
                const float v = col <= b + r ? (b + r == col ? 1.f : 0.f) - sbeta[b + r] * x : 0.f;
                if (part == (r & 3)) {
                    t[r >> 2] = v;
                    sT[(b + r) * CP + col] = v;
                }
            }
            __syncwarp();
        }
    }
    __syncthreads();

    // records that depend only on the prologue
    for (int idx = tid; idx < C * C; idx += NTHREADS) {
        int i = idx / C, j = idx % C;
        stf(gA + tc::cm_idx(i, j, C), sA[i * CP + j]);
        if (save) stf(gT + tc::cm_idx(i, j, C), sT[i * CP + j]);
    }
    for (int idx = tid; idx < C * D; idx += NTHREADS) {
        const int i = idx / D, d = idx % D, at = i * row_stride<D>() + d;
        const float G = sG[at], gl = sG[(C - 1) * row_stride<D>() + d], gam = exp2f(G);
        stf(gQt + tc::cm_idx(i, d, D), p.scale * sq[at] * gam);
        stf(gKh + tc::cm_idx(i, d, D), sk[at] * exp2f(gl - G));
        if (i == C - 1) gGam[d] = gam;
        // operands of the WY products, in place: beta * k * 2^G and beta * v
        sq[at] = sbeta[i] * sk[at] * gam;
        sv[at] = sbeta[i] * sv[at];
    }
    {
        float acc[4][D / 16];
        zero_acc(acc);
        mm_tile<C, D>(acc, C, [&](int m, int k) { return sT[m * CP + k]; }, [&](int k, int n) { return sq[k * row_stride<D>() + n]; },
                      st, true, false);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int cc = 0; cc < D / 16; ++cc) stf(gW + tc::cm_idx(tile_col(tx, cc), 4 * ty + r, C), acc[r][cc]);
        zero_acc(acc);
        mm_tile<C, D>(acc, C, [&](int m, int k) { return sT[m * CP + k]; }, [&](int k, int n) { return sv[k * row_stride<D>() + n]; },
                      st, true, false);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int cc = 0; cc < D / 16; ++cc) stf(gU + tc::cm_idx(tile_col(tx, cc), 4 * ty + r, C), acc[r][cc]);
    }
}

// ---------------------------------------------------------------------------------------
// bwd_chunk: all chunk-local adjoints, the exact pairwise intra step, the reverse cumulative
// sum of the gate gradient and the chain rule through gate / L2 norm / sigmoid.
// ---------------------------------------------------------------------------------------
// SPLIT = true stops after the chunk-level adjoints and leaves them in the scratch buffer for
// the separate intra kernel of the BF16 path (used to validate the two halves independently).
// one entry of the hand-over matrices dAqk / dM in the layout bwd_intra reads: three BF16 tiles
// cm(i, j; 64) whose sum is x
__device__ __forceinline__ void store_split3(__nv_bfloat16* base, int i, int j, float x) {
    uint32_t p0, p1, p2;
    split3_bf16(x, 0.f, p0, p1, p2);
    unsigned short* b = reinterpret_cast<unsigned short*>(base) + tc::cm_idx(i, j, C);
    b[0] = (unsigned short)(p0 & 0xffffu);
    b[C * C] = (unsigned short)(p1 & 0xffffu);
    b[2 * C * C] = (unsigned short)(p2 & 0xffffu);
}

template <typename T, int D, bool SPLIT = false>
__global__ void __launch_bounds__(NTHREADS, 1) kda_bwd_chunk_simt(const KdaParams p) {
    extern __shared__ __align__(16) float smem[];
    float* sq = smem;
    float* sk = sq + C * row_stride<D>();
    float* sG = sk + C * row_stride<D>();
    float* sW = sG + C * row_stride<D>();        // dW, later scratch
    float* sT = sW + C * row_stride<D>();        // [64][CP]
    float* sdA = sT + C * CP;
    float* sdM = sdA + C * CP;     // first holds dT
    float* sY = sdM + C * CP;
    float* sbeta = sY + C * CP;
    float* srq = sbeta + C;
    float* srk = srq + C;
    float* sdb = srk + C;          // dbeta accumulator
    float* scol = sdb + C;         // [D] last-row term of dG
    float* sred = scol + D;        // [8] block reduction
    float* st = sred + 8;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ty = tid >> 4, tx = tid & 15;
    const int c = blockIdx.x / p.H, h = blockIdx.x % p.H;
    pdl_wait();
    const ChunkInfo ci = chunk_info(p, c);
    const WsLayout L = ws_layout(p.NT, p.H, p.dk, p.dv, p.dtype);
    const char* ws = (const char*)p.workspace;
    char* sc = (char*)p.bwd_scratch;
    const size_t rec = (size_t)c * p.H + h;
    const T* gVn = (const T*)(ws + L.U) + rec * C * D;
    const T* gT = (const T*)(ws + L.Tm) + rec * C * C;
    const T* gS0 = (const T*)(ws + L.S0) + rec * D * D;
    const float* gGam = (const float*)(ws + L.gamC) + rec * D;
    const T* gdS = (const T*)(sc + L.dS) + rec * D * D;
    const T* gdV = (const T*)(sc + L.dVn) + rec * C * D;
    const T* dO = (const T*)p.grad_o;
    const T* v = (const T*)p.v;
    const float scale = p.scale;

    load_prologue<T, D>(p, ci, h, sq, sk, sG, nullptr, sbeta, srq, srk, st);
    for (int idx = tid; idx < C * C; idx += NTHREADS) sT[(idx / C) * CP + idx % C] = ldf(gT + tc::cm_idx(idx / C, idx % C, C));
    if (tid < C) sdb[tid] = 0.f;

    auto ldo = [&](int i, int e) { return i < ci.len ? ldf(dO + ((size_t)(ci.tok0 + i) * p.H + h) * D + e) : 0.f; };
    auto ldv = [&](int i, int e) { return i < ci.len ? ldf(v + ((size_t)(ci.tok0 + i) * p.H + h) * D + e) : 0.f; };

    float dq_a[4][D / 16], dk_a[4][D / 16], dG_a[4][D / 16];
    float db_r[4] = {0.f, 0.f, 0.f, 0.f};
    zero_acc(dq_a);
    zero_acc(dk_a);
    zero_acc(dG_a);

    // 1. dAqk = tril(dO V'^T)
    {
        float acc[4][4];
        zero_acc(acc);
        mm_tile<C, C>(acc, D, [&](int m, int k) { return ldo(m, k); }, [&](int k, int n) { return ldf(gVn + tc::cm_idx(k, n, C)); }, st,
                      true, true);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                int i = 4 * ty + r, j = tile_col(tx, cc);
                sdA[i * CP + j] = (i >= j) ? acc[r][cc] : 0.f;
                if constexpr (SPLIT) {
                    store_split3((__nv_bfloat16*)(sc + L.dAM) + rec * 6 * C * C, i, j, i > j ? sdA[i * CP + j] : 0.f);
                    if (i == j) ((float*)(sc + L.dAd))[rec * C + i] = sdA[i * CP + j];
                }
            }
    }
    // 2. dW = -dV' S0^T
    {
        float acc[4][D / 16];
        zero_acc(acc);
        mm_tile<C, D>(acc, D, [&](int m, int k) { return ldf(gdV + tc::cm_idx(k, m, C)); },
                      [&](int k, int n) { return ldf(gS0 + tc::cm_idx(k, n, D)); }, st, true, true);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int cc = 0; cc < D / 16; ++cc) sW[(4 * ty + r) * row_stride<D>() + tile_col(tx, cc)] = -acc[r][cc];
    }
    // 3. dT = tril(dW (beta K~)^T + dV' (beta V)^T)   -> sdM
    {
        float acc[4][4];
        zero_acc(acc);
        mm_tile<C, C>(acc, D, [&](int m, int k) { return sW[m * row_stride<D>() + k]; },
                      [&](int k, int n) { return sbeta[n] * sk[n * row_stride<D>() + k] * exp2f(sG[n * row_stride<D>() + k]); }, st, true, true);
        mm_tile<C, C>(acc, D, [&](int m, int k) { return ldf(gdV + tc::cm_idx(k, m, C)); },
                      [&](int k, int n) { return sbeta[n] * ldv(n, k); }, st, true, true);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                int i = 4 * ty + r, j = tile_col(tx, cc);
                sdM[i * CP + j] = (i >= j) ? acc[r][cc] : 0.f;
            }
    }
    // 4. dM = -T^T dT T^T (strictly lower part is what the intra step uses)
    {
        float acc[4][4];
        zero_acc(acc);
        mm_tile<C, C>(acc, C, [&](int m, int k) { return sdM[m * CP + k]; }, [&](int k, int n) { return sT[n * CP + k]; }, st,
                      true, true);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) sY[(4 * ty + r) * CP + tile_col(tx, cc)] = acc[r][cc];
        zero_acc(acc);
        mm_tile<C, C>(acc, C, [&](int m, int k) { return sT[k * CP + m]; }, [&](int k, int n) { return sY[k * CP + n]; }, st,
                      false, false);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                int i = 4 * ty + r, j = tile_col(tx, cc);
                sdM[i * CP + j] = (i > j) ? -acc[r][cc] : 0.f;
                if constexpr (SPLIT)
                    store_split3((__nv_bfloat16*)(sc + L.dAM) + rec * 6 * C * C + 3 * C * C, i, j, sdM[i * CP + j]);
            }
    }
    // 5. d(beta K~) = T^T dW
    {
        float acc[4][D / 16];
        zero_acc(acc);
        mm_tile<C, D>(acc, C, [&](int m, int k) { return sT[k * CP + m]; }, [&](int k, int n) { return sW[k * row_stride<D>() + n]; }, st,
                      false, false);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int cc = 0; cc < D / 16; ++cc) {
                int i = 4 * ty + r, d = tile_col(tx, cc);
                if constexpr (SPLIT) {
                    stf((T*)(sc + L.dKb) + rec * C * D + handover_idx(i, d), acc[r][cc]);
                    continue;
                }
                float gam = exp2f(sG[i * row_stride<D>() + d]);
                float kt = sk[i * row_stride<D>() + d] * gam;
                float dkt = sbeta[i] * acc[r][cc];
                dk_a[r][cc] += dkt * gam;
                dG_a[r][cc] += dkt * kt;
                db_r[r] += acc[r][cc] * kt;
            }
    }
    // 6. d(beta V) = T^T dV'  -> dv
    {
        float acc[4][D / 16];
        zero_acc(acc);
        mm_tile<C, D>(acc, C, [&](int m, int k) { return sT[k * CP + m]; }, [&](int k, int n) { return ldf(gdV + tc::cm_idx(n, k, C)); },
                      st, false, false);
        T* dv = (T*)p.grad_v;
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int cc = 0; cc < D / 16; ++cc) {
                int i = 4 * ty + r, e = tile_col(tx, cc);
                if (i < ci.len) {
                    stf(dv + ((size_t)(ci.tok0 + i) * p.H + h) * D + e, sbeta[i] * acc[r][cc]);
                    db_r[r] += acc[r][cc] * ldv(i, e);
                }
            }
    }
    // 7. dQt = dO S0^T
    {
        float acc[4][D / 16];
        zero_acc(acc);
        mm_tile<C, D>(acc, D, [&](int m, int k) { return ldo(m, k); }, [&](int k, int n) { return ldf(gS0 + tc::cm_idx(k, n, D)); }, st,
                      true, true);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int cc = 0; cc < D / 16; ++cc) {
                int i = 4 * ty + r, d = tile_col(tx, cc);
                if constexpr (SPLIT) {
                    stf((T*)(sc + L.dQt) + rec * C * D + handover_idx(i, d), acc[r][cc]);
                    continue;
                }
                float gam = exp2f(sG[i * row_stride<D>() + d]);
                dq_a[r][cc] += scale * acc[r][cc] * gam;
                dG_a[r][cc] += acc[r][cc] * scale * sq[i * row_stride<D>() + d] * gam;
            }
    }
    // 8. dKh = V' dS^T ; its column sums feed the last row of dG
    {
        float acc[4][D / 16];
        zero_acc(acc);
        mm_tile<C, D>(acc, D, [&](int m, int k) { return ldf(gVn + tc::cm_idx(k, m, C)); },
                      [&](int k, int n) { return ldf(gdS + tc::cm_idx(k, n, D)); }, st, true, true);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int cc = 0; cc < D / 16; ++cc) {
                int i = 4 * ty + r, d = tile_col(tx, cc);
                if constexpr (SPLIT) {
                    stf((T*)(sc + L.dKh) + rec * C * D + handover_idx(i, d), acc[r][cc]);
                    sW[i * row_stride<D>() + d] = 0.f;
                    continue;
                }
                float dec = exp2f(sG[(C - 1) * row_stride<D>() + d] - sG[i * row_stride<D>() + d]);
                float kh = sk[i * row_stride<D>() + d] * dec;
                dk_a[r][cc] += acc[r][cc] * dec;
                dG_a[r][cc] -= acc[r][cc] * kh;
                sW[i * row_stride<D>() + d] = acc[r][cc] * kh;
            }
    }
    __syncthreads();
    for (int it = tid; it < 4 * D; it += NTHREADS) {
        float t = 0.f;
#pragma unroll
        for (int r = 0; r < 16; ++r) t += sW[(16 * (it / D) + r) * row_stride<D>() + it % D];
        st[it] = t;
    }
    __syncthreads();
    for (int d = tid; d < D; d += NTHREADS) scol[d] = (st[d] + st[D + d]) + (st[2 * D + d] + st[3 * D + d]);
    __syncthreads();
    // 9. d(gamC)[d] = sum_e dS[d][e] S0[d][e]
    for (int d = warp; d < D; d += NTHREADS / 32) {
        float s = 0.f;
        for (int e = lane; e < D; e += 32) s = fmaf(ldf(gdS + tc::cm_idx(e, d, D)), ldf(gS0 + tc::cm_idx(e, d, D)), s);
        s = warp_sum(s);
        if (lane == 0) scol[d] += s * gGam[d];
    }
    if constexpr (SPLIT) {  // hand over: beta gradient so far and dGamma_C * Gamma_C
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float s = row16_sum(db_r[r]);
            if (tx == 0) ((float*)(sc + L.dbp))[rec * C + 4 * ty + r] = s;
        }
        __syncthreads();
        for (int d = tid; d < D; d += NTHREADS) ((float*)(sc + L.gC))[rec * D + d] = scol[d];
        return;
    }
    // 10. intra step with exact pairwise decays.  A thread's tile is four rows i x four channels d (twice that for
    //     d = 128): walking the keys j in front of the tile it needs k_j, G_j and column j of dA and dM for its rows,
    //     walking the queries behind it q, k, G and row entries of dA and dM, four 16-byte loads per 16 pairs each way.
    //     dA^T and beta dM^T go where T and Y were.
    __syncthreads();
    for (int idx = tid; idx < C * C; idx += NTHREADS) {
        const int i = idx & 63, j = idx >> 6;
        sT[j * CP + i] = sdA[i * CP + j];
        sY[j * CP + i] = sdM[i * CP + j];
    }
    __syncthreads();
#pragma unroll
    for (int g = 0; g < D / 64; ++g) {
        const int d0 = tile_col(tx, 4 * g), i0 = 4 * ty;
        float gi[4][4], a1[4][4], a2[4][4], c1[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float4 v = *reinterpret_cast<const float4*>(sG + (i0 + r) * row_stride<D>() + d0);
            gi[r][0] = v.x; gi[r][1] = v.y; gi[r][2] = v.z; gi[r][3] = v.w;
#pragma unroll
            for (int c = 0; c < 4; ++c) a1[r][c] = a2[r][c] = c1[r][c] = 0.f;
        }
        // `inside`: pairs of the tile's own rows, where only j < i counts (the diagonal pair has decay 1 and contributes
        // equal and opposite amounts to dG, so it is kept out of dG exactly)
        auto keys = [&](int j, bool inside) {
            const float4 kv = *reinterpret_cast<const float4*>(sk + j * row_stride<D>() + d0), gv = *reinterpret_cast<const float4*>(sG + j * row_stride<D>() + d0);
            const float4 av = *reinterpret_cast<const float4*>(sT + j * CP + i0), mv = *reinterpret_cast<const float4*>(sY + j * CP + i0);
            const float kj[4] = {kv.x, kv.y, kv.z, kv.w}, gj[4] = {gv.x, gv.y, gv.z, gv.w};
            const float da[4] = {av.x, av.y, av.z, av.w}, dm[4] = {mv.x, mv.y, mv.z, mv.w};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (inside && i0 + r <= j) continue;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float kd = kj[c] * exp2f(gi[r][c] - gj[c]);
                    a1[r][c] = fmaf(da[r], kd, a1[r][c]);
                    a2[r][c] = fmaf(dm[r], kd, a2[r][c]);
                }
            }
        };
        auto queries = [&](int ii, bool inside) {
            const float4 qv = *reinterpret_cast<const float4*>(sq + ii * row_stride<D>() + d0), kv = *reinterpret_cast<const float4*>(sk + ii * row_stride<D>() + d0);
            const float4 gv = *reinterpret_cast<const float4*>(sG + ii * row_stride<D>() + d0);
            const float4 av = *reinterpret_cast<const float4*>(sdA + ii * CP + i0), mv = *reinterpret_cast<const float4*>(sdM + ii * CP + i0);
            const float q4[4] = {qv.x, qv.y, qv.z, qv.w}, k4[4] = {kv.x, kv.y, kv.z, kv.w}, g4[4] = {gv.x, gv.y, gv.z, gv.w};
            const float b = sbeta[ii];
            const float da[4] = {scale * av.x, scale * av.y, scale * av.z, scale * av.w}, dm[4] = {b * mv.x, b * mv.y, b * mv.z, b * mv.w};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (inside && ii <= i0 + r) continue;
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    c1[r][c] = fmaf(fmaf(da[r], q4[c], dm[r] * k4[c]), exp2f(g4[c] - gi[r][c]), c1[r][c]);
            }
        };
#pragma unroll 2
        for (int j = 0; j < i0; ++j) keys(j, false);
#pragma unroll
        for (int j = 0; j < 3; ++j) keys(i0 + j, true);
#pragma unroll
        for (int j = 1; j < 4; ++j) queries(i0 + j, true);
#pragma unroll 2
        for (int ii = i0 + 4; ii < C; ++ii) queries(ii, false);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = i0 + r;
            const float diag = scale * sdA[i * CP + i], b = sbeta[i];
            const float4 qv = *reinterpret_cast<const float4*>(sq + i * row_stride<D>() + d0), kv = *reinterpret_cast<const float4*>(sk + i * row_stride<D>() + d0);
            const float qi[4] = {qv.x, qv.y, qv.z, qv.w}, ki[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float dq_in = scale * a1[r][c], dk_row = b * a2[r][c];
                db_r[r] += ki[c] * a2[r][c];
                dq_a[r][4 * g + c] += dq_in + diag * ki[c];
                dk_a[r][4 * g + c] += dk_row + c1[r][c] + diag * qi[c];
                dG_a[r][4 * g + c] += qi[c] * dq_in + ki[c] * dk_row - ki[c] * c1[r][c];
            }
        }
    }
    // 11. dbeta rows
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        float s = row16_sum(db_r[r]);
        if (tx == 0) sdb[4 * ty + r] = s;
    }
    // 12. reverse cumulative sum of dG and the gate chain
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int cc = 0; cc < D / 16; ++cc) sW[(4 * ty + r) * row_stride<D>() + tile_col(tx, cc)] = dG_a[r][cc];
    __syncthreads();
    // thread = (channel, 16-row group): group totals first, then the sums from the last row up
    for (int it = tid; it < 4 * D; it += NTHREADS) {
        const int d = it % D, grp = it / D;
        float t = 0.f;
#pragma unroll
        for (int r = 0; r < 16; ++r) t += sW[(16 * grp + r) * row_stride<D>() + d];
        st[it] = t;
    }
    __syncthreads();
    {
        const bool gate = p.flags & KDA_FLAG_GATE;
        const float negA = gate ? -expf(p.A_log[h]) : 0.f;
        const T* g = (const T*)p.g;
        T* dg = (T*)p.grad_g;
        float dA = 0.f, dbias[4 * D / NTHREADS];
#pragma unroll
        for (int u = 0; u < 4 * D / NTHREADS; ++u) {
            const int it = tid + NTHREADS * u, d = it % D, grp = it / D;
            float run = scol[d];
            for (int gg = 3; gg > grp; --gg) run += st[gg * D + d];
            float db = 0.f;
#pragma unroll 8
            for (int r = 15; r >= 0; --r) {
                const int i = 16 * grp + r;
                run += sW[i * row_stride<D>() + d];
                if (i < ci.len) {
                    const size_t off = ((size_t)(ci.tok0 + i) * p.H + h) * D + d;
                    if (gate) {
                        float z = ldf(g + off);
                        if (p.dt_bias) z += p.dt_bias[h * D + d];
                        dA = fmaf(run, negA * softplus_f(z), dA);
                        const float dx = run * negA * sigmoid_f(z);
                        db += dx;
                        stf(dg + off, dx);
                    } else {
                        stf(dg + off, run);
                    }
                }
            }
            dbias[u] = db;
        }
        __syncthreads();  // the group totals have been read
        if (gate) {
#pragma unroll
            for (int u = 0; u < 4 * D / NTHREADS; ++u) st[tid + NTHREADS * u] = dbias[u];
            dA = warp_sum(dA);
            if (lane == 0) sred[warp] = dA;
            __syncthreads();
            for (int d = tid; d < D; d += NTHREADS)
                ((float*)(sc + L.dbias_part))[rec * D + d] = (st[3 * D + d] + st[2 * D + d]) + (st[D + d] + st[d]);
            if (tid == 0) {
                float s = 0.f;
                for (int w = 0; w < NTHREADS / 32; ++w) s += sred[w];
                ((float*)(sc + L.dA_part))[rec] = s;
            }
        }
    }
    // 13. chain through the L2 norm, 14. through the sigmoid
    {
        const bool l2 = p.flags & KDA_FLAG_QK_L2NORM;
        T* dq = (T*)p.grad_q;
        T* dk = (T*)p.grad_k;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = 4 * ty + r;
            float dotq = 0.f, dotk = 0.f;
            if (l2) {
#pragma unroll
                for (int cc = 0; cc < D / 16; ++cc) {
                    dotq += sq[i * row_stride<D>() + tile_col(tx, cc)] * dq_a[r][cc];
                    dotk += sk[i * row_stride<D>() + tile_col(tx, cc)] * dk_a[r][cc];
                }
                dotq = row16_sum(dotq);
                dotk = row16_sum(dotk);
            }
            if (i < ci.len) {
#pragma unroll
                for (int cc = 0; cc < D / 16; ++cc) {
                    int d = tile_col(tx, cc);
                    size_t off = ((size_t)(ci.tok0 + i) * p.H + h) * D + d;
                    float a = dq_a[r][cc], b = dk_a[r][cc];
                    if (l2) {
                        a = (a - sq[i * row_stride<D>() + d] * dotq) * srq[i];
                        b = (b - sk[i * row_stride<D>() + d] * dotk) * srk[i];
                    }
                    stf(dq + off, a);
                    stf(dk + off, b);
                }
            }
        }
        if (tid < ci.len) {
            float b = sbeta[tid], db = sdb[tid];
            if (p.flags & KDA_FLAG_BETA_SIGMOID) db *= b * (1.f - b);
            stf((T*)p.grad_beta + (size_t)(ci.tok0 + tid) * p.H + h, db);
        }
    }
}

// deterministic reduction of the per-chunk partial parameter gradients: one block per head and 32 channels; 32 groups of
// 32 threads each sum every 32nd chunk in order, then the group sums are added in a fixed order
__global__ void __launch_bounds__(1024) kda_param_reduce(const KdaParams p) {
    __shared__ float sb[32][33];
    __shared__ float sa[32];
    pdl_wait();
    const WsLayout L = ws_layout(p.NT, p.H, p.dk, p.dv, p.dtype);
    const char* sc = (const char*)p.bwd_scratch;
    const int h = blockIdx.x, lane = threadIdx.x & 31, d = 32 * blockIdx.y + lane, grp = threadIdx.x >> 5;
    const float* pb = (const float*)(sc + L.dbias_part);
    const float* pa = (const float*)(sc + L.dA_part);
    // (sixteen loads in flight per thread, added in chunk order: the loop is a chain of round trips otherwise)
    float s = 0.f;
    for (int c0 = grp; c0 < p.NT; c0 += 32 * 16) {
        float v[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            const int c = c0 + 32 * u;
            v[u] = c < p.NT ? pb[((size_t)c * p.H + h) * p.dk + d] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 16; ++u) s += v[u];
    }
    sb[grp][lane] = s;
    if (blockIdx.y == 0) {  // dA_log: thread t takes every 1024th chunk
        float a = 0.f;
        for (int c = threadIdx.x; c < p.NT; c += 1024) a += pa[(size_t)c * p.H + h];
        a = warp_sum(a);
        if (lane == 0) sa[grp] = a;
    }
    __syncthreads();
    if (grp == 0) {
        if (p.grad_dt_bias) {
            float t = 0.f;
#pragma unroll
            for (int g = 0; g < 32; ++g) t += sb[g][lane];
            p.grad_dt_bias[h * p.dk + d] = t;
        }
        if (blockIdx.y == 0 && lane == 0 && p.grad_A_log) {
            float t = 0.f;
            for (int g = 0; g < 32; ++g) t += sa[g];
            p.grad_A_log[h] = t;
        }
    }
}

// ---------------------------------------------------------------------------------------
// host-side launchers
// ---------------------------------------------------------------------------------------
template <int D>
constexpr size_t smem_intra() { return (size_t)(4 * C * row_stride<D>() + 3 * C * CP + 3 * C + st_floats<D>()) * 4; }
template <int D>
constexpr size_t smem_bwd_chunk() {
    return (size_t)(4 * C * row_stride<D>() + 4 * C * CP + 4 * C + D + 8 + st_floats<D>()) * 4;
}

template <typename K>
static cudaError_t set_smem(K kernel, size_t bytes) {
    return allow_smem(kernel, (int)bytes);
}

template <typename T, int D>
static cudaError_t launch_stage(const KdaParams& p, int stage, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    switch (stage) {
        case 0:
            if ((e = set_smem(kda_fwd_intra_simt<T, D>, smem_intra<D>())) != cudaSuccess) return e;
            return launch_dependent(kda_fwd_intra_simt<T, D>, p.NT * p.H, NTHREADS, smem_intra<D>(), s, p);
        case 1: return simt_state(p, false, s);
        case 2: return simt_state(p, true, s);
        case 3:
            if ((e = set_smem(kda_bwd_chunk_simt<T, D>, smem_bwd_chunk<D>())) != cudaSuccess) return e;
            return launch_dependent(kda_bwd_chunk_simt<T, D, false>, p.NT * p.H, NTHREADS, smem_bwd_chunk<D>(), s, p);
        case 5:
            if ((e = set_smem(kda_bwd_chunk_simt<T, D, true>, smem_bwd_chunk<D>())) != cudaSuccess) return e;
            return launch_dependent(kda_bwd_chunk_simt<T, D, true>, p.NT * p.H, NTHREADS, smem_bwd_chunk<D>(), s, p);
        default:
            return launch_dependent(kda_param_reduce, dim3(p.H, p.dk / 32), 1024, 0, s, p);
    }
}

// stage: 0 fwd_intra, 1 fwd_state, 2 bwd_state, 3 bwd_chunk, 4 param_reduce, 5 bwd_chunk stopped after the adjoints
cudaError_t simt_stage(const KdaParams& p, int stage, cudaStream_t s) {
    if (p.dtype == KDA_DTYPE_F32)
        return p.dk == 64 ? launch_stage<float, 64>(p, stage, s) : launch_stage<float, 128>(p, stage, s);
    return p.dk == 64 ? launch_stage<__nv_bfloat16, 64>(p, stage, s) : launch_stage<__nv_bfloat16, 128>(p, stage, s);
}

cudaError_t simt_fwd(const KdaParams& p, cudaStream_t s) {
    cudaError_t e;
    for (int st = 0; st < 2; ++st) {
        if ((e = simt_stage(p, st, s)) != cudaSuccess) return e;
        prof_mark(s);
    }
    return cudaSuccess;
}

cudaError_t simt_bwd(const KdaParams& p, cudaStream_t s) {
    cudaError_t e;
    for (int st = 2; st < 5; ++st) {
        if (st == 4 && !(p.flags & KDA_FLAG_GATE)) break;
        if ((e = simt_stage(p, st, s)) != cudaSuccess) return e;
        prof_mark(s);
    }
    return cudaSuccess;
}

}  // namespace kda
