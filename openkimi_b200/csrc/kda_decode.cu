// Recurrent KDA for decoding: the reference recurrence (k3mini/model.py:121-128) over a few tokens per
// (sequence, head), FP32 state in and out.
//
//   S~ = diag(alpha) S          pred = k^T S~          S' = S~ + k (beta (v - pred))^T          o = scale S'^T q
//
// What bounds it: for many (sequence, head) units the HBM traffic of the dk x dv FP32 state (2 x 64 KB per unit at
// d = 128, read once and written once however many tokens the call has); for few units latency.
//
// Value columns are independent of one another, so a WARP owns R of them with all their key channels and keeps that
// part of the state in registers over all tokens of the call: no shared-memory round trip of the state, no barrier
// between the warps inside a token.  Both inner products a token needs are taken from the OLD state,
//     pred = sum_d (k_d alpha_d) S_d       o = sum_d (scale q_d alpha_d) S_d + (scale q.k) (beta (v - pred)),
// so one reduction across the lanes serves both and the update of the state is off the critical path.
//   * [dv][dk] states: a lane holds four consecutive key channels of every column (a row is one 512-byte line);
//   * [dk][dv] states: a lane holds four consecutive value columns at every (128 / lanes)th key channel.
// The tokens' prologue (L2 norm, gate, sigmoid) is evaluated once per CTA, a warp per token, into shared memory.
//
// 1536 units, one token: 48.2 us with the state in shared memory -> 36.1 us, 5.6 TB/s; one sequence of six heads:
// 6.6 -> 3.6 us; eight tokens of four sequences: eight launches of 7 us -> 7.0 us.
#include "kda_common.cuh"

namespace kda {

namespace dec {
constexpr int NW = 4;     // warps per CTA
constexpr int TB = 16;    // tokens whose prologue is in shared memory at a time
// floats of one token's prologue: k alpha, scale q alpha, alpha, k (4 x D), v (D), beta, scale q.k, padding
__host__ __device__ constexpr int tok_floats(int D) { return 5 * D + 4; }
}  // namespace dec

template <typename T, int N>
__device__ __forceinline__ void load_n(const T* p, float (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = ldf(p + i);
}
template <>
__device__ __forceinline__ void load_n<__nv_bfloat16, 4>(const __nv_bfloat16* p, float (&v)[4]) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(r.x << 16); v[1] = __uint_as_float(r.x & 0xffff0000u);
    v[2] = __uint_as_float(r.y << 16); v[3] = __uint_as_float(r.y & 0xffff0000u);
}
template <>
__device__ __forceinline__ void load_n<float, 4>(const float* p, float (&v)[4]) {
    const float4 r = *reinterpret_cast<const float4*>(p);
    v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
}

// vec: the caller's rows start on a four-element boundary
template <typename T, int N>
__device__ __forceinline__ void load_row(const T* p, float (&v)[N], int vec) {
    if (vec) {
        load_n(p, v);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = ldf(p + i);
    }
}

// Sums val[0..M) over the LD lanes that differ in the given lane bits (bit0, 2 bit0, ..., LD / 2 * bit0), halving the
// number of values a lane carries at every level: afterwards val[0] of a lane is the total of value `which`
// (the lane bits read from the lowest level up as the most significant bit of the index first).
template <int M, int LD, int BIT0>
struct TransposeSum {
    static __device__ __forceinline__ void run(float (&val)[M], int lane, int& which) {
        if constexpr (LD > 1) {
            const bool up = lane & BIT0;
            if constexpr (M > 1) {
                float half[M / 2];
#pragma unroll
                for (int i = 0; i < M / 2; ++i) {
                    const float keep = up ? val[M / 2 + i] : val[i], send = up ? val[i] : val[M / 2 + i];
                    half[i] = keep + __shfl_xor_sync(0xffffffffu, send, BIT0);
                }
                which = 2 * which + (up ? 1 : 0);
                TransposeSum<M / 2, LD / 2, 2 * BIT0>::run(half, lane, which);
                val[0] = half[0];
            } else {
                val[0] += __shfl_xor_sync(0xffffffffu, val[0], BIT0);
                TransposeSum<1, LD / 2, 2 * BIT0>::run(val, lane, which);
            }
        }
    }
};

// T: element type; D: channels; VF: [dv][dk] state; R: value columns per warp
template <typename T, int D, bool VF, int R>
__global__ void __launch_bounds__(32 * dec::NW) kda_recurrent_kernel(
    const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, const T* __restrict__ g,
    const T* __restrict__ beta, const float* __restrict__ A_log, const float* __restrict__ dt_bias,
    const float* state_in, float* state_out, T* __restrict__ o, int H, int Tlen, int flags, float scale, int vec) {
    using namespace dec;
    constexpr int LD = VF ? D / 4 : 128 / R;          // lanes along the key channels of one column
    constexpr int LE = 32 / LD;                       // lane groups along the value columns
    constexpr int NE = R / LE, ND = D / LD;           // columns and key channels a lane holds
    constexpr int BIT0 = VF ? 1 : LE;                 // lowest lane bit of the key-channel index
    static_assert(VF ? ND == 4 : NE == 4, "one 16-byte word per access");
    extern __shared__ __align__(16) float sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NP = D / (R * NW);                  // CTAs per (sequence, head)
    const int nh = blockIdx.x / NP, h = nh % H, n = nh / H;
    const int ld = VF ? lane & (LD - 1) : lane / LE, le = VF ? lane / LD : lane & (LE - 1);
    const int e0 = (blockIdx.x % NP * NW + warp) * R;     // first column of this warp
    // column i of this lane, key channel j of this lane
    auto col = [&](int i) { return VF ? e0 + le + LE * i : e0 + 4 * le + i; };
    auto chn = [&](int j) { return VF ? 4 * ld + j : ld + LD * j; };
    const bool l2 = flags & KDA_FLAG_QK_L2NORM, gate = flags & KDA_FLAG_GATE, sig = flags & KDA_FLAG_BETA_SIGMOID;
    const size_t sbase = (size_t)nh * D * D;
    pdl_wait();

    // the state is requested first; it arrives behind the prologue
    float S[NE][ND];
    if (state_in) {
        if constexpr (VF) {
#pragma unroll
            for (int i = 0; i < NE; ++i) {
                const float4 x = __ldcs(reinterpret_cast<const float4*>(state_in + sbase + (size_t)col(i) * D + 4 * ld));
                S[i][0] = x.x; S[i][1] = x.y; S[i][2] = x.z; S[i][3] = x.w;
            }
        } else {
#pragma unroll
            for (int j = 0; j < ND; ++j) {
                const float4 x = __ldcs(reinterpret_cast<const float4*>(state_in + sbase + (size_t)chn(j) * D + e0 + 4 * le));
                S[0][j] = x.x; S[1][j] = x.y; S[2][j] = x.z; S[3][j] = x.w;
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < NE; ++i)
#pragma unroll
            for (int j = 0; j < ND; ++j) S[i][j] = 0.f;
    }
    constexpr int PC = D / 32;                        // prologue: consecutive channels per lane
    float negA = 0.f, bias[PC];
#pragma unroll
    for (int i = 0; i < PC; ++i) bias[i] = 0.f;
    if (gate) {
        negA = -expf(A_log[h]);
        if (dt_bias)
#pragma unroll
            for (int i = 0; i < PC; ++i) bias[i] = dt_bias[h * D + PC * lane + i];
    }
    for (int t0 = 0; t0 < Tlen; t0 += TB) {
        const int nt = min(TB, Tlen - t0);
        if (t0) __syncthreads();                      // the previous tokens' prologue has been consumed
        for (int t = warp; t < nt; t += NW) {         // prologue of a token (k3mini/model.py:217-223)
            const size_t row = ((size_t)n * Tlen + t0 + t) * H + h;
            float qv[PC], kv[PC], gv[PC], vv[PC];
            load_row(q + row * D + PC * lane, qv, vec);
            load_row(k + row * D + PC * lane, kv, vec);
            load_row(g + row * D + PC * lane, gv, vec);
            load_row(v + row * D + PC * lane, vv, vec);
            float b = ldf(beta + row);
            if (l2) {
                float sq = 0.f, sk = 0.f;
#pragma unroll
                for (int i = 0; i < PC; ++i) {
                    sq = fmaf(qv[i], qv[i], sq);
                    sk = fmaf(kv[i], kv[i], sk);
                }
                const float iq = 1.f / fmaxf(sqrtf(warp_sum(sq)), 1e-6f), ik = 1.f / fmaxf(sqrtf(warp_sum(sk)), 1e-6f);
#pragma unroll
                for (int i = 0; i < PC; ++i) {
                    qv[i] *= iq;
                    kv[i] *= ik;
                    if (sizeof(T) == 2) {  // BF16 activations: the reference rounds the normalised rows back (model.py:218-219)
                        qv[i] = __bfloat162float(__float2bfloat16_rn(qv[i]));
                        kv[i] = __bfloat162float(__float2bfloat16_rn(kv[i]));
                    }
                }
            }
            float* s = sm + t * tok_floats(D);
            float qk = 0.f;
#pragma unroll
            for (int i = 0; i < PC; ++i) {
                if (gate) gv[i] = negA * softplus_f(gv[i] + bias[i]);
                const float al = expf(gv[i]), qs = scale * qv[i];
                qk = fmaf(qs, kv[i], qk);
                const int d = PC * lane + i;
                s[d] = kv[i] * al;
                s[D + d] = qs * al;
                s[2 * D + d] = al;
                s[3 * D + d] = kv[i];
                s[4 * D + d] = vv[i];
            }
            qk = warp_sum(qk);
            if (sig) b = sigmoid_f(b);
            if (lane == 0) {
                s[5 * D] = b;
                s[5 * D + 1] = qk;
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int t = 0; t < nt; ++t) {
            const float* s = sm + t * tok_floats(D);
            float dot[2 * NE], al[ND], kk[ND];
#pragma unroll
            for (int i = 0; i < 2 * NE; ++i) dot[i] = 0.f;
            if constexpr (VF) {
                float ka[4], qa[4];
                load_n(s + 4 * ld, ka);
                load_n(s + D + 4 * ld, qa);
                load_n(s + 2 * D + 4 * ld, al);
                load_n(s + 3 * D + 4 * ld, kk);
#pragma unroll
                for (int i = 0; i < NE; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        dot[i] = fmaf(ka[j], S[i][j], dot[i]);
                        dot[NE + i] = fmaf(qa[j], S[i][j], dot[NE + i]);
                    }
            } else {
#pragma unroll
                for (int j = 0; j < ND; ++j) {
                    const float ka = s[chn(j)], qa = s[D + chn(j)];
                    al[j] = s[2 * D + chn(j)];
                    kk[j] = s[3 * D + chn(j)];
#pragma unroll
                    for (int i = 0; i < NE; ++i) {
                        dot[i] = fmaf(ka, S[i][j], dot[i]);
                        dot[NE + i] = fmaf(qa, S[i][j], dot[NE + i]);
                    }
                }
            }
            int which = 0;
            TransposeSum<2 * NE, LD, BIT0>::run(dot, lane, which);
            // `which` = NE * (0: prediction, 1: output) + column; the lane bit BIT0 tells the two kinds apart
            static_assert(2 * NE <= LD, "every lane ends with exactly one value");
            const bool is_out = lane & BIT0;
            const int mine = col(which & (NE - 1));
            const float err = s[5 * D] * (s[4 * D + mine] - dot[0]);
            const float pair = __shfl_xor_sync(0xffffffffu, err, BIT0);
            if (is_out) {
                // the first 2 NE reduction lanes hold all values, the others copies
                if (ld < 2 * NE) stf(o + (((size_t)n * Tlen + t0 + t) * H + h) * D + mine, fmaf(s[5 * D + 1], pair, dot[0]));
            }
#pragma unroll
            for (int i = 0; i < NE; ++i) {
                // lane that holds the prediction of this lane's column i: reduction bits = column index, lowest bit last
                int src = 0;
#pragma unroll
                for (int m = NE / 2, b = 2; m >= 1; m >>= 1, b <<= 1) src |= (i & m) ? b * BIT0 : 0;
                src |= VF ? lane & ~(LD - 1) : lane & (LE - 1);
                const float ei = __shfl_sync(0xffffffffu, err, src);
#pragma unroll
                for (int j = 0; j < ND; ++j) S[i][j] = fmaf(al[j], S[i][j], kk[j] * ei);
            }
        }
    }
    if (!state_out) return;
    if constexpr (VF) {
#pragma unroll
        for (int i = 0; i < NE; ++i)
            __stcs(reinterpret_cast<float4*>(state_out + sbase + (size_t)col(i) * D + 4 * ld),
                   make_float4(S[i][0], S[i][1], S[i][2], S[i][3]));
    } else {
#pragma unroll
        for (int j = 0; j < ND; ++j)
            __stcs(reinterpret_cast<float4*>(state_out + sbase + (size_t)chn(j) * D + e0 + 4 * le),
                   make_float4(S[0][j], S[1][j], S[2][j], S[3][j]));
    }
}

struct RecurrentArgs {
    const void *q, *k, *v, *g, *beta;
    const float *A_log, *dt_bias, *state_in;
    float* state_out;
    void* o;
    int N, T, H, flags;
    float scale;
    int vec;
};

template <typename T, int D, bool VF, int R>
static cudaError_t launch_recurrent(const RecurrentArgs& a, cudaStream_t s) {
    const int tb = a.T < dec::TB ? a.T : dec::TB;
    const size_t smem = (size_t)tb * dec::tok_floats(D) * sizeof(float);
    return launch_dependent(kda_recurrent_kernel<T, D, VF, R>, a.N * a.H * (D / (R * dec::NW)), 32 * dec::NW, smem, s,
                            (const T*)a.q, (const T*)a.k, (const T*)a.v, (const T*)a.g, (const T*)a.beta, a.A_log, a.dt_bias,
                            a.state_in, a.state_out, (T*)a.o, a.H, a.T, a.flags, a.scale, a.vec);
}

// Columns per warp: eight give short dependent chains per token, sixteen half as many CTAs that evaluate the same token's
// prologue, more loads in flight per warp and, for [dk][dv] states, 64 instead of 32 consecutive bytes per access.  So eight
// until every SM has 64 KB of [dv][dk] states, or 16 KB of [dk][dv] states, to move.  Eight against sixteen (us; d = 128 unless
// said, BF16, launches back to back):
//   units                      6            48           148           222           592          1536
//   [dv][dk], 1 token      3.0 : 3.5    3.6 : 3.7     4.9 : 5.0     7.5 : 5.8    14.2 : 13.4   35.8 : 36.0
//   [dv][dk], 16 tokens   11.3 : 13.6  13.6 : 14.0   19.0 : 18.2   32.2 : 22.4   69.7 : 58.7    171 : 152
//   [dk][dv], 1 token      3.5 : 3.7    4.4 : 3.8     5.9 : 4.9     9.5 : 6.0    19.4 : 12.8   48.1 : 36.3
//   [dk][dv], 16 tokens   11.4 : 13.2  14.1 : 13.6   20.1 : 17.7   34.1 : 22.0   76.2 : 53.8    184 : 137
//   d = 64, [dv][dk], 1    2.6 : 2.7    2.7 : 2.8     2.9 : 2.9     3.2 : 3.4     4.3 : 4.5     9.2 : 8.4
//   d = 64, [dk][dv], 1    2.7 : 2.7    2.8 : 2.8     3.3 : 3.0     3.7 : 3.5     5.3 : 4.5    12.8 : 9.9
template <typename T, int D>
static cudaError_t launch_columns(const RecurrentArgs& a, cudaStream_t s) {
    const bool vf = a.flags & KDA_FLAG_STATE_V_FIRST;
    if ((long long)a.N * a.H * D * D < (vf ? 16384LL : 4096LL) * sm_count())
        return vf ? launch_recurrent<T, D, true, 8>(a, s) : launch_recurrent<T, D, false, 8>(a, s);
    return vf ? launch_recurrent<T, D, true, 16>(a, s) : launch_recurrent<T, D, false, 16>(a, s);
}

}  // namespace kda

extern "C" int kda_recurrent_fwd(const void* q, const void* k, const void* v, const void* g, const void* beta,
                                 const float* A_log, const float* dt_bias, const float* state_in, float* state_out, void* o,
                                 int32_t N, int32_t T, int32_t H, int32_t dk, int32_t dv, int32_t dtype, int32_t flags,
                                 float scale, void* stream) {
    using namespace kda;
    if (!q || !k || !v || !g || !beta || !o) return KDA_ERR_NULL;
    if ((flags & KDA_FLAG_GATE) && !A_log) return KDA_ERR_NULL;
    if (N <= 0 || H <= 0 || T <= 0 || dk != dv || (dk != 64 && dk != 128)) return KDA_ERR_SHAPE;
    if ((long long)N * H > 0x7fffffffLL / 8) return KDA_ERR_SHAPE;  // (at most four CTAs per unit)
    if (dtype != KDA_DTYPE_F32 && dtype != KDA_DTYPE_BF16) return KDA_ERR_DTYPE;
    if (((uintptr_t)state_in | (uintptr_t)state_out) & 15) return KDA_ERR_ALIGN;
    const int vec = (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)g) & (dtype == KDA_DTYPE_F32 ? 15 : 7)) == 0;
    const RecurrentArgs a = {q, k, v, g, beta, A_log, dt_bias, state_in, state_out, o, N, T, H, flags, scale, vec};
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e;
    if (dtype == KDA_DTYPE_F32)
        e = dk == 64 ? launch_columns<float, 64>(a, s) : launch_columns<float, 128>(a, s);
    else
        e = dk == 64 ? launch_columns<__nv_bfloat16, 64>(a, s) : launch_columns<__nv_bfloat16, 128>(a, s);
    return e == cudaSuccess ? KDA_OK : fail_cuda(e);
}

// `status` stays for callers of the earlier kernel, which waited for a bulk copy; nothing here waits.
extern "C" int kda_recurrent_step(const void* q, const void* k, const void* v, const void* g, const void* beta,
                                  const float* A_log, const float* dt_bias, const float* state_in, float* state_out, void* o,
                                  int32_t N, int32_t H, int32_t dk, int32_t dv, int32_t dtype, int32_t flags, float scale,
                                  int32_t* status, void* stream) {
    (void)status;
    if (!state_in || !state_out) return KDA_ERR_NULL;
    return kda_recurrent_fwd(q, k, v, g, beta, A_log, dt_bias, state_in, state_out, o, N, 1, H, dk, dv, dtype, flags, scale,
                             stream);
}
