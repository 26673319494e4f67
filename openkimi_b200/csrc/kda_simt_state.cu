// The two state kernels of the FP32 CUDA-core mode: sequential over the chunks of one sequence, for one head and one
// panel of BV state columns (the columns are independent).
//
//   forward   V' = U - W S      O = Qt S + Aqk V'      S <- diag(gamC) S + Kh^T V'
//   backward  dV' = Aqk^T dO + Kh dS                   dS <- diag(gamC) dS + Qt^T dO - W^T dV'
//
// Bound by the dependent chain of one chunk.  The chunk's records arrive as linear 16-byte asynchronous copies, each
// requested as soon as the previous chunk's product has consumed the same record, so that no product waits for memory;
// every product reads its operands where they are.  The copies turn the records' 8 x 8 core matrices (cm_idx) into padded
// rows, read four elements at a time along the second index.  Products whose second index is the output row give a thread
// four rows x two columns (`rows4`); products whose second index is the inner one give a thread one row x eight columns
// and walk the inner index by fours (`dots`); both split the inner index over thread groups.
#include "kda_common.cuh"
#include "kda_tc.cuh"

namespace kda {

namespace ss {
constexpr int NT = 256;

__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
    const float4 r = *reinterpret_cast<const float4*>(p);
    v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
}
__device__ __forceinline__ void load4(const __nv_bfloat16* p, float (&v)[4]) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(r.x << 16); v[1] = __uint_as_float(r.x & 0xffff0000u);
    v[2] = __uint_as_float(r.y << 16); v[3] = __uint_as_float(r.y & 0xffff0000u);
}

// Row stride of a record in shared memory: 16 bytes more than a row, so that neither a walk along a row nor eight rows
// at the same column meet in a bank
template <typename T>
constexpr int stride(int cols) { return cols + 16 / (int)sizeof(T); }

// asynchronous copy of a record cm(row, col; COLS) of R rows into plain rows, by the whole CTA
template <int R, int COLS, typename T>
__device__ __forceinline__ void copy_record(T* dst, const T* src) {
    constexpr int E = 16 / sizeof(T);  // elements of a chunk: a half row (FP32) or a row (BF16) of a core matrix
#pragma unroll
    for (int q = threadIdx.x; q < R * COLS / E; q += NT) {
        const int at = q * E, blk = at >> 6, r = blk / (COLS / 8) * 8 + ((at >> 3) & 7), c = blk % (COLS / 8) * 8 + (at & 7);
        tc::cp_async16_z(dst + r * stride<T>(COLS) + c, src + at, true);
    }
}
__device__ __forceinline__ void copy_floats(float* dst, const float* src, int n) {
    for (int o = threadIdx.x * 4; o < n; o += NT * 4) tc::cp_async16_z(dst + o, src + o, true);
}

// acc[4][2] = sum over k of A(k, 4 rq + r) * B[k][2 ep + c] for this thread group's share of k.
// A: record of K rows (k) and COLS columns (output row); B: float [K][BV]; R = number of output rows
template <int R, int COLS, int K, int BV, typename T>
__device__ __forceinline__ void rows4(float (&acc)[4][2], const T* A, const float* B) {
    constexpr int RQ = R / 4, SPLIT = NT / (RQ * (BV / 2));
    static_assert(SPLIT >= 1 && K % SPLIT == 0, "thread groups");
    const int rq = threadIdx.x % RQ, ep = (threadIdx.x / RQ) % (BV / 2), ks = threadIdx.x / (RQ * (BV / 2));
#pragma unroll 8
    for (int k = ks * (K / SPLIT); k < (ks + 1) * (K / SPLIT); ++k) {
        float a[4];
        load4(A + k * stride<T>(COLS) + 4 * rq, a);
        const float2 b = *reinterpret_cast<const float2*>(B + k * BV + 2 * ep);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            acc[r][0] = fmaf(a[r], b.x, acc[r][0]);
            acc[r][1] = fmaf(a[r], b.y, acc[r][1]);
        }
    }
}
// leaves a rows4 result in part[group][R][BV]
template <int R, int BV>
constexpr int rows4_groups() { return NT / (R / 4 * (BV / 2)); }
template <int R, int BV>
__device__ __forceinline__ void rows4_store(const float (&acc)[4][2], float* part) {
    constexpr int RQ = R / 4;
    const int rq = threadIdx.x % RQ, ep = (threadIdx.x / RQ) % (BV / 2), ks = threadIdx.x / (RQ * (BV / 2));
#pragma unroll
    for (int r = 0; r < 4; ++r)
        *reinterpret_cast<float2*>(part + (ks * R + 4 * rq + r) * BV + 2 * ep) = make_float2(acc[r][0], acc[r][1]);
}
// sum of the partial results of one element
template <int R, int BV, int GROUPS>
__device__ __forceinline__ float part_sum(const float* part, int at) {
    float s = 0.f;
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) s += part[g * R * BV + at];
    return s;
}

// acc[8] += sum over this thread's share of k of A(row, k) * B[k][8 cg + c]: thread = one of R rows x eight columns x a
// part of the inner index.  A: record of rows (output row) and K columns (k)
template <int R, int BV>
constexpr int dots_groups() { return NT / (R * (BV / 8)); }
template <int R, int K, int BV, typename T>
__device__ __forceinline__ void dots(float (&acc)[8], const T* A, const float* B) {
    constexpr int KN = K / dots_groups<R, BV>();
    const int row = threadIdx.x % R, cg = (threadIdx.x / R) % (BV / 8), ks = threadIdx.x / (R * (BV / 8));
#pragma unroll 2
    for (int k = ks * KN; k < (ks + 1) * KN; k += 4) {
        float a[4];
        load4(A + row * stride<T>(K) + k, a);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 b0 = *reinterpret_cast<const float4*>(B + (k + j) * BV + 8 * cg), b1 = *reinterpret_cast<const float4*>(B + (k + j) * BV + 8 * cg + 4);
            acc[0] = fmaf(a[j], b0.x, acc[0]); acc[1] = fmaf(a[j], b0.y, acc[1]);
            acc[2] = fmaf(a[j], b0.z, acc[2]); acc[3] = fmaf(a[j], b0.w, acc[3]);
            acc[4] = fmaf(a[j], b1.x, acc[4]); acc[5] = fmaf(a[j], b1.y, acc[5]);
            acc[6] = fmaf(a[j], b1.z, acc[6]); acc[7] = fmaf(a[j], b1.w, acc[7]);
        }
    }
}
template <int R, int BV>
__device__ __forceinline__ void dots_store(const float (&acc)[8], float* part) {
    const int row = threadIdx.x % R, cg = (threadIdx.x / R) % (BV / 8), ks = threadIdx.x / (R * (BV / 8));
    float4* dst = reinterpret_cast<float4*>(part + (ks * R + row) * BV + 8 * cg);
    dst[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    dst[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
}

// shared memory: the records W, Qt, Kh, Aqk, then S [D][BV], V' [64][BV], a second [64][BV] (U panel / dO), partial sums
template <typename T, int D, int BV>
struct Smem {
    static constexpr int WREC = D * stride<T>(C) * (int)sizeof(T), REC = C * stride<T>(D) * (int)sizeof(T);
    static constexpr int W = 0, QT = WREC, KH = QT + REC, AQ = KH + REC, S = AQ + C * stride<T>(C) * (int)sizeof(T), VN = S + D * BV * 4, X = VN + C * BV * 4;
    static constexpr int GAM = X + C * BV * 4, PART = GAM + D * 4;
    // partial sums of rows4 and of dots (the numbers of floats do not depend on R)
    static constexpr int P4 = rows4_groups<C, BV>() * C * BV, P8 = dots_groups<C, BV>() * C * BV;
    static constexpr int TOTAL = PART + (P4 + P8) * 4;
};
}  // namespace ss

template <typename T, int D, int BV>
__global__ void __launch_bounds__(ss::NT, 1) kda_fwd_state_simt(const KdaParams p) {
    using namespace ss;
    using M = Smem<T, D, BV>;
    extern __shared__ __align__(16) unsigned char dyn[];
    T *sW = (T*)(dyn + M::W), *sQt = (T*)(dyn + M::QT), *sKh = (T*)(dyn + M::KH), *sA = (T*)(dyn + M::AQ);
    float *sS = (float*)(dyn + M::S), *sVn = (float*)(dyn + M::VN), *sGam = (float*)(dyn + M::GAM), *part = (float*)(dyn + M::PART);
    const int tid = threadIdx.x;
    const int e0 = blockIdx.x * BV, h = blockIdx.y, n = blockIdx.z;
    const WsLayout L = ws_layout(p.NT, p.H, p.dk, p.dv, p.dtype);
    char* ws = (char*)p.workspace;
    const bool save = !(p.flags & KDA_FLAG_NO_SAVE), with_o = !(p.flags & KDA_FLAG_NO_OUTPUT);
    pdl_wait();
    SeqCursor sq;
    sq.load(p, n);
    const size_t sbase = ((size_t)n * p.H + h) * D * D;
    auto rec_of = [&](int c) { return (size_t)c * p.H + h; };
    const int ui = tid & 63, uc = (tid >> 6) * (BV / 4);  // this thread's row and first column of [64][BV] results
    T* gUbase = (T*)(ws + L.U);
    auto load_u = [&](int c, float (&u)[BV / 4]) {
#pragma unroll
        for (int j = 0; j < BV / 4; ++j) u[j] = ldf(gUbase + rec_of(c) * C * D + tc::cm_idx(e0 + uc + j, ui, C));
    };
    for (int idx = tid; idx < D * BV; idx += NT) {
        const int d = idx / BV, e = idx % BV;
        sS[idx] = p.h0 ? p.h0[sbase + state_idx(p, d, e0 + e)] : 0.f;
    }
    float u[BV / 4];
    // copy groups in the order of use: W (with gamC), Qt and Aqk, Kh
    auto get_w = [&](int c) {
        copy_record<D, C>(sW, (const T*)(ws + L.W) + rec_of(c) * C * D);
        tc::cp_async_commit();
    };
    auto get_q = [&](int c) {
        copy_record<C, D>(sQt, (const T*)(ws + L.Qt) + rec_of(c) * C * D);
        copy_record<C, C>(sA, (const T*)(ws + L.Aqk) + rec_of(c) * C * C);
        tc::cp_async_commit();
    };
    auto get_k = [&](int c) {
        copy_record<C, D>(sKh, (const T*)(ws + L.Kh) + rec_of(c) * C * D);
        copy_floats(sGam, (const float*)(ws + L.gamC) + rec_of(c) * D, D);
        tc::cp_async_commit();
    };
    if (sq.c_begin < sq.c_end) {
        get_w(sq.c_begin);
        get_q(sq.c_begin);
        get_k(sq.c_begin);
        load_u(sq.c_begin, u);
    }
    for (int c = sq.c_begin; c < sq.c_end; ++c) {
        const bool more = c + 1 < sq.c_end;
        tc::cp_async_wait<2>();
        __syncthreads();
        if (save) {
            T* gS0 = (T*)(ws + L.S0) + rec_of(c) * D * D;
            for (int idx = tid; idx < D * BV; idx += NT) stf(gS0 + tc::cm_idx(e0 + idx / D, idx % D, D), sS[(idx % D) * BV + idx / D]);
        }
        {  // V' = U - W S
            float acc[4][2] = {};
            rows4<C, C, D, BV>(acc, sW, sS);
            rows4_store<C, BV>(acc, part);
            __syncthreads();
            if (more) get_w(c + 1);
            else tc::cp_async_commit();
#pragma unroll
            for (int j = 0; j < BV / 4; ++j) {
                const float vn = u[j] - part_sum<C, BV, rows4_groups<C, BV>()>(part, ui * BV + uc + j);
                sVn[ui * BV + uc + j] = vn;
                if (save) stf(gUbase + rec_of(c) * C * D + tc::cm_idx(e0 + uc + j, ui, C), vn);
            }
            if (more) load_u(c + 1, u);
        }
        tc::cp_async_wait<1>();  // Qt, Aqk and Kh of this chunk have landed
        __syncthreads();
        {
            if (with_o) {
                float acc[8] = {};  // O = Qt S + Aqk V'
                dots<C, D, BV>(acc, sQt, sS);
                dots<C, C, BV>(acc, sA, sVn);
                dots_store<C, BV>(acc, part + M::P4);
            }
            float kacc[4][2] = {};  // Kh^T V'
            rows4<D, D, C, BV>(kacc, sKh, sVn);
            rows4_store<D, BV>(kacc, part);
        }
        __syncthreads();
        if (more) get_q(c + 1);
        else tc::cp_async_commit();
        if (with_o && ui < sq.rows(c)) {
            T* o = (T*)p.o + ((size_t)(sq.tok(c) + ui) * p.H + h) * D + e0 + uc;
#pragma unroll
            for (int j = 0; j < BV / 4; ++j) stf(o + j, part_sum<C, BV, dots_groups<C, BV>()>(part + M::P4, ui * BV + uc + j));
        }
        for (int idx = tid; idx < D * BV; idx += NT)
            sS[idx] = sGam[idx / BV] * sS[idx] + part_sum<D, BV, rows4_groups<D, BV>()>(part, idx);
        __syncthreads();
        if (more) get_k(c + 1);
        else tc::cp_async_commit();
    }
    if (p.ht) {
        __syncthreads();
        for (int idx = tid; idx < D * BV; idx += NT) p.ht[sbase + state_idx(p, idx / BV, e0 + idx % BV)] = sS[idx];
    }
    tc::cp_async_wait<0>();
}

// Stores the dS entering each chunk (from the right) and dV'.
template <typename T, int D, int BV>
__global__ void __launch_bounds__(ss::NT, 1) kda_bwd_state_simt(const KdaParams p) {
    using namespace ss;
    using M = Smem<T, D, BV>;
    extern __shared__ __align__(16) unsigned char dyn[];
    T *sW = (T*)(dyn + M::W), *sQt = (T*)(dyn + M::QT), *sKh = (T*)(dyn + M::KH), *sA = (T*)(dyn + M::AQ);
    float *sS = (float*)(dyn + M::S), *sVn = (float*)(dyn + M::VN), *sdO = (float*)(dyn + M::X), *sGam = (float*)(dyn + M::GAM),
          *part = (float*)(dyn + M::PART);
    const int tid = threadIdx.x;
    const int e0 = blockIdx.x * BV, h = blockIdx.y, n = blockIdx.z;
    const WsLayout L = ws_layout(p.NT, p.H, p.dk, p.dv, p.dtype);
    const char* ws = (const char*)p.workspace;
    char* sc = (char*)p.bwd_scratch;
    pdl_wait();
    SeqCursor sq;
    sq.load(p, n);
    const size_t sbase = ((size_t)n * p.H + h) * D * D;
    auto rec_of = [&](int c) { return (size_t)c * p.H + h; };
    const int ui = tid & 63, uc = (tid >> 6) * (BV / 4);  // this thread's row and first column of [64][BV] arrays
    auto load_do = [&](int c, float (&x)[BV / 4]) {
        const bool valid = ui < sq.rows(c);
        const T* src = (const T*)p.grad_o + ((size_t)(sq.tok(c) + (valid ? ui : 0)) * p.H + h) * D + e0 + uc;
#pragma unroll
        for (int j = 0; j < BV / 4; ++j) x[j] = valid ? ldf(src + j) : 0.f;
    };
    for (int idx = tid; idx < D * BV; idx += NT) {
        const int d = idx / BV, e = idx % BV;
        sS[idx] = p.grad_ht ? p.grad_ht[sbase + state_idx(p, d, e0 + e)] : 0.f;
    }
    // copy groups in the order of use: Aqk and Kh, Qt and W (with gamC)
    auto get_a = [&](int c) {
        copy_record<C, C>(sA, (const T*)(ws + L.Aqk) + rec_of(c) * C * C);
        copy_record<C, D>(sKh, (const T*)(ws + L.Kh) + rec_of(c) * C * D);
        tc::cp_async_commit();
    };
    auto get_w = [&](int c) {
        copy_record<C, D>(sQt, (const T*)(ws + L.Qt) + rec_of(c) * C * D);
        copy_record<D, C>(sW, (const T*)(ws + L.W) + rec_of(c) * C * D);
        copy_floats(sGam, (const float*)(ws + L.gamC) + rec_of(c) * D, D);
        tc::cp_async_commit();
    };
    float x[BV / 4];
    if (sq.c_begin < sq.c_end) {
        get_a(sq.c_end - 1);
        get_w(sq.c_end - 1);
        load_do(sq.c_end - 1, x);
    }
    for (int c = sq.c_end - 1; c >= sq.c_begin; --c) {
        const bool more = c > sq.c_begin;
#pragma unroll
        for (int j = 0; j < BV / 4; ++j) sdO[ui * BV + uc + j] = x[j];
        tc::cp_async_wait<1>();
        __syncthreads();
        if (more) load_do(c - 1, x);
        T* gdS = (T*)(sc + L.dS) + rec_of(c) * D * D;
        for (int idx = tid; idx < D * BV; idx += NT) stf(gdS + tc::cm_idx(e0 + idx / D, idx % D, D), sS[(idx % D) * BV + idx / D]);
        {  // dV' = Aqk^T dO + Kh dS
            float acc[4][2] = {}, own[8] = {};
            rows4<C, C, C, BV>(acc, sA, sdO);
            rows4_store<C, BV>(acc, part);
            dots<C, D, BV>(own, sKh, sS);
            dots_store<C, BV>(own, part + M::P4);
            __syncthreads();
            if (more) get_a(c - 1);
            else tc::cp_async_commit();
            T* gdV = (T*)(sc + L.dVn) + rec_of(c) * C * D;
#pragma unroll
            for (int j = 0; j < BV / 4; ++j) {
                const int at = ui * BV + uc + j;
                const float s = part_sum<C, BV, rows4_groups<C, BV>()>(part, at) + part_sum<C, BV, dots_groups<C, BV>()>(part + M::P4, at);
                sVn[at] = s;
                stf(gdV + tc::cm_idx(e0 + uc + j, ui, C), s);
            }
        }
        tc::cp_async_wait<1>();
        __syncthreads();
        {  // dS <- diag(gamC) dS + Qt^T dO - W^T dV'
            float acc[4][2] = {}, own[8] = {};
            rows4<D, D, C, BV>(acc, sQt, sdO);
            rows4_store<D, BV>(acc, part);
            dots<D, C, BV>(own, sW, sVn);
            dots_store<D, BV>(own, part + M::P4);
            __syncthreads();
            for (int idx = tid; idx < D * BV; idx += NT)
                sS[idx] = sGam[idx / BV] * sS[idx] + part_sum<D, BV, rows4_groups<D, BV>()>(part, idx) -
                          part_sum<D, BV, dots_groups<D, BV>()>(part + M::P4, idx);
        }
        __syncthreads();
        if (more) get_w(c - 1);
        else tc::cp_async_commit();
    }
    if (p.grad_h0) {
        __syncthreads();
        for (int idx = tid; idx < D * BV; idx += NT) p.grad_h0[sbase + state_idx(p, idx / BV, e0 + idx % BV)] = sS[idx];
    }
    tc::cp_async_wait<0>();
}

template <typename T, int D, int BV>
static cudaError_t launch_state(const KdaParams& p, bool bwd, cudaStream_t s) {
    auto kern = bwd ? kda_bwd_state_simt<T, D, BV> : kda_fwd_state_simt<T, D, BV>;
    constexpr int smem = ss::Smem<T, D, BV>::TOTAL;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    return launch_dependent(kern, dim3(D / BV, p.H, p.N), ss::NT, smem, s, p);
}

// Panels of eight columns while all of them are resident at once (the chunk step is a chain of latencies); wider ones
// beyond that (each panel reads all records of the chunk): what 256 threads cover with four rows x two columns each.
template <typename T, int D>
static cudaError_t launch_panels(const KdaParams& p, bool bwd, cudaStream_t s) {
    constexpr int WIDE = 2048 / D;
    const long long narrow = (long long)p.N * p.H * (D / 8), resident = (long long)sm_count() * (232448 / (ss::Smem<T, D, 8>::TOTAL + 1024));
    return narrow <= resident ? launch_state<T, D, 8>(p, bwd, s) : launch_state<T, D, WIDE>(p, bwd, s);
}

cudaError_t simt_state(const KdaParams& p, bool bwd, cudaStream_t s) {
    if (p.dtype == KDA_DTYPE_F32) return p.dk == 64 ? launch_panels<float, 64>(p, bwd, s) : launch_panels<float, 128>(p, bwd, s);
    return p.dk == 64 ? launch_panels<__nv_bfloat16, 64>(p, bwd, s) : launch_panels<__nv_bfloat16, 128>(p, bwd, s);
}

}  // namespace kda
