// fwd_intra (BF16 operands, d = 128): everything of a chunk that does not need the state.  Two CTAs of 256 threads per SM walk
// the (chunk, head) units (UnitWalk); each requests the inputs of its next unit as soon as their place is free.
//
//   1  rows: q, k, v, gate tiles arrive as bulk-tensor tile copies.  L2 norm of the q and k rows, sigmoid, beta*v.  The
//      CONV instantiation reads the pre-convolution projections instead (three halo rows before the chunk included) and applies
//      the causal depthwise filter + SiLU of k3mini/model.py:76-88,181-185 before anything else sees the rows
//   2  gate channel-wise: activation, within-chunk cumulative sum G (log2), span guard
//   3  Aqk and L: warp = (16-row block I, 64 channels).  The diagonal block in FP32 multiply-adds: with the midpoint m of its rows as
//      reference, x_i 2^(G_i - m) against k_j 2^(m - G_j), where the block passes the guard; else pair by pair, one exp2 each.
//      Earlier blocks on mma.sync with operands made in registers, one BF16 pass: x_i 2^(G_i - r_I) against k_j 2^(r_I - G_j),
//      r_I = G at the first row of block I, every exponent <= 0.  The two channel halves meet in shared memory.  The Qt and
//      Kh records
//   4  Aqk record; T = (I + diag(beta) L)^-1; the operand beta*k*2^G
//   5  T record; W^T = (beta k 2^G)^T T^T and U^T = (beta v)^T T^T as tcgen05 MMAs (M = 128 channels); W, U records
//
// What bounds it: one unit is a chain of short dependent stages (a dozen barriers).  Two CTAs share an SM so that one unit's waits are
// the other's issue slots.  A unit lives in 110 KB for that: the off-diagonal products' operands never touch shared memory, the
// diagonal blocks' scaled rows lie where the partial sums go afterwards, L turns into T in place, beta v and beta k 2^G are MMA
// operands where the tile copies left v and q, and the next unit's rows are requested as their places fall free.  Operand tiles in
// shared memory took one CTA of 512 threads (3072 units 304 -> 231 us, twice 1536 units of wide spans 353 -> 271; with
// the convolution 12288 units 1443 -> 1131).  The diagonal blocks as TF32 products of operands split in two are faster (3072
// units by 22 us) and three times as far from 64-bit sums: the share of their BF16 records that come out rounded the other way is
// 3e-4 against 1e-4.  So are the inverse's products (5 us): 2.3e-3 against 1.4e-3 of T where keys are alike.
#include "kda_common.cuh"
#include "kda_conv_bwd.cuh"
#include "kda_tc.cuh"
#include "kda_tmap.cuh"

namespace kda {

using namespace tc;

namespace fi {
constexpr int D = 128, NTHR = 256;
constexpr int LDR = 68, LDA = 20;            // row strides in floats: L / T, partial diagonal blocks of Aqk
constexpr uint32_t SQ = 0;                   // q rows, then q^ bf16 [64][128] (swz_bf16); later beta k^ 2^G
constexpr uint32_t SK = SQ + 16384;          // k rows, then k^
constexpr uint32_t SV = SK + 16384;          // v rows, then beta v (swz_bf16)
constexpr uint32_t SG = SV + 16384;          // G f32 [64][128] (swz_f32)
constexpr uint32_t SM = SG + 32768;          // gate rows bf16 [64][128] as they arrive; the diagonal blocks' scaled rows; then
                                             // f32 [64][LDR]: L, T; partial blocks of Aqk above the diagonal
constexpr uint32_t SU = SM + 64 * LDR * 4;   // 8 KB: gate totals of the four 16-row groups f32 [4][128] | the rest of the
                                             // scaled rows | partial diagonal blocks of Aqk | inner products of the inverse | T bf16 cm(i, j; 64)
constexpr uint32_t TAPS = SG;                // when G is dead: the filter taps of the next unit, f32 [3][8][16][4]
constexpr uint32_t SMID = SU + 8192;         // f32 [4][128] midpoint of every (16-row block, channel)
constexpr uint32_t SBETA = SMID + 2048;      // f32 [3][64]: 1/|q|, 1/|k|, beta (the aux record)
constexpr uint32_t SPASS = SBETA + 768;      // int [4][2]: guard decision of every block, per 64 channels
constexpr uint32_t SBAR = SPASS + 32;        // four mbarriers, the tensor-memory base
constexpr uint32_t HALO = SBAR + 48;         // fused convolution: rows -3 .. -1 of q, k, v, bf16 [3][3][128]
constexpr uint32_t TOTAL = HALO, TOTAL_CONV = HALO + 9 * 256;
static_assert(TOTAL_CONV <= 115712, "two CTAs per SM");
constexpr uint32_t T_W = 0, T_U = 64, TMEM_COLS = 128;
constexpr int LDS = 20;                      // row stride in floats of a warp's scaled rows: [2][16][LDS], over SM and SU
static_assert(8 * 2 * 16 * LDS * 4 <= SMID - SM, "scaled rows of eight warps");
}  // namespace fi
using fi::LDR;

// T = (I + diag(beta) L)^-1 by blocks, in place: M holds L (strictly lower) and receives T on and below the diagonal blocks; rows
// of LDR floats.  The four 16 x 16 diagonal blocks are inverted by forward substitution in FP32, one warp each (a dependent
// chain of 16 rows, lane = column); everything below them is products, T_ba = -T_bb (beta L)_ba T_aa for the block pairs (0, 1)
// and (2, 3), then the same with 32 x 32 halves, in FP32 multiply-adds.  sY (32 rows of LDY floats) takes the inner products.
constexpr int LDY = 36;

__device__ __forceinline__ void invert_diagonal(float* M, const float* sbeta, int blk, int lane) {
    const int col = lane & 15;
    float t[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const float* lrow = M + (16 * blk + r) * LDR + 16 * blk;
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int j = 0; j < r; j += 4) {
            const float4 l = *reinterpret_cast<const float4*>(lrow + j);
            s0 = fmaf(l.x, t[j], s0);
            if (j + 1 < r) s1 = fmaf(l.y, t[j + 1], s1);
            if (j + 2 < r) s0 = fmaf(l.z, t[j + 2], s0);
            if (j + 3 < r) s1 = fmaf(l.w, t[j + 3], s1);
        }
        t[r] = (r == col ? 1.f : 0.f) - sbeta[16 * blk + r] * (s0 + s1);
        if (r < col) t[r] = 0.f;
    }
    __syncwarp();
    if (lane < 16) {
#pragma unroll
        for (int r = 0; r < 16; ++r) M[(16 * blk + r) * LDR + 16 * blk + col] = t[r];
    }
}

// mma.sync fragments (lane = 4 g + t).  The contracted index may be dealt out in any order that both operands share: of sixteen
// channels a lane holds 4 t .. 4 t + 3, one 16-byte word of G and one 8-byte word of q^ and k^, for one step.  Row (and key) number g of a tile stands for row bit_reverse(g): with the row swizzle of the tiles (swz_f32,
// swz_bf16) the loads of a quarter warp then fall into different banks.
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void exp2_diff(const float4& a, const float4& b, float (&f)[4]) {  // 2^(a - b)
    f[0] = ex2_approx(a.x - b.x); f[1] = ex2_approx(a.y - b.y); f[2] = ex2_approx(a.z - b.z); f[3] = ex2_approx(a.w - b.w);
}
__device__ __forceinline__ void unpack4(const uint2& u, float (&f)[4]) {
    f[0] = __uint_as_float(u.x << 16); f[1] = __uint_as_float(u.x & 0xffff0000u);
    f[2] = __uint_as_float(u.y << 16); f[3] = __uint_as_float(u.y & 0xffff0000u);
}

// a 2 x 2 tile over `K4` groups of four inner elements: rows of A (float4 along k), rows k of B (two columns)
template <int K4>
__device__ __forceinline__ void tile22(float2 (&acc)[2], const float* A, const float* B, int ldb, int kstep) {
#pragma unroll 2
    for (int m = 0; m < K4; ++m) {
        const float4 a0 = *reinterpret_cast<const float4*>(A + m * kstep), a1 = *reinterpret_cast<const float4*>(A + LDR + m * kstep);
        const float x0[4] = {a0.x, a0.y, a0.z, a0.w}, x1[4] = {a1.x, a1.y, a1.z, a1.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 b = *reinterpret_cast<const float2*>(B + (m * kstep + j) * ldb);
            acc[0] = __ffma2_rn(make_float2(x0[j], x0[j]), b, acc[0]);
            acc[1] = __ffma2_rn(make_float2(x1[j], x1[j]), b, acc[1]);
        }
    }
}
// row i of a tile whose inner index was split over lanes i = 0, 1
__device__ __forceinline__ float2 sum_row(const float2 (&acc)[2], int i) {
    const float2 give = i ? acc[0] : acc[1], own = i ? acc[1] : acc[0];
    return make_float2(own.x + __shfl_xor_sync(0xffffffffu, give.x, 1), own.y + __shfl_xor_sync(0xffffffffu, give.y, 1));
}
__device__ __forceinline__ void invert_products(float* M, const float* sbeta, float* sY, int warp, int lane) {
    float2 acc[2] = {};
    {   // pairs of 16 x 16 blocks: four warps each, inner index over two lanes (alternating groups of four)
        const int pr = warp >> 2, a = 32 * pr, b = a + 16, i = lane & 1;
        const int r0 = 4 * (warp & 3) + 2 * (lane >> 4), c0 = 2 * ((lane >> 1) & 7), k0 = 4 * i;
        tile22<2>(acc, M + (b + r0) * LDR + a + k0, M + (a + k0) * LDR + a + c0, LDR, 8);
        const float2 y = sum_row(acc, i);
        const float be = sbeta[b + r0 + i];
        *reinterpret_cast<float2*>(sY + (16 * pr + r0 + i) * LDY + c0) = make_float2(be * y.x, be * y.y);
        bar_sync(1 + pr, 128);  // the pair's warps have read L_ba
        acc[0] = acc[1] = make_float2(0.f, 0.f);
        tile22<2>(acc, M + (b + r0) * LDR + b + k0, sY + (16 * pr + k0) * LDY + c0, LDY, 8);
        const float2 x = sum_row(acc, i);
        *reinterpret_cast<float2*>(M + (b + r0 + i) * LDR + a + c0) = make_float2(-x.x, -x.y);
    }
    __syncthreads();
    // the 32 x 32 halves: a warp has eight rows and sixteen columns.  (Blocks above the diagonal hold other things: their products
    // are left out.)
    const int r0 = 8 * (warp >> 1) + 2 * (lane >> 3), c16 = 16 * (warp & 1), c0 = c16 + 2 * (lane & 7);
    acc[0] = acc[1] = make_float2(0.f, 0.f);
    if (c16) tile22<4>(acc, M + (32 + r0) * LDR + 16, M + 16 * LDR + c0, LDR, 4);
    else tile22<8>(acc, M + (32 + r0) * LDR, M + c0, LDR, 4);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float be = sbeta[32 + r0 + i];
        *reinterpret_cast<float2*>(sY + (r0 + i) * LDY + c0) = make_float2(be * acc[i].x, be * acc[i].y);
    }
    __syncthreads();
    acc[0] = acc[1] = make_float2(0.f, 0.f);
    if (warp < 4) tile22<4>(acc, M + (32 + r0) * LDR + 32, sY + c0, LDY, 4);
    else tile22<8>(acc, M + (32 + r0) * LDR + 32, sY + c0, LDY, 4);
#pragma unroll
    for (int i = 0; i < 2; ++i) *reinterpret_cast<float2*>(M + (32 + r0 + i) * LDR + c0) = make_float2(-acc[i].x, -acc[i].y);
}

template <bool CONV>
__global__ void __launch_bounds__(fi::NTHR, 2) kda_fwd_intra_tc(const KdaParams p, const __grid_constant__ RowMaps maps, const WsLayout L) {
    using namespace fi;
    extern __shared__ __align__(1024) unsigned char dyn[];
    __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(dyn + SQ);
    __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(dyn + SK);
    float* sG = reinterpret_cast<float*>(dyn + SG);
    __nv_bfloat16* sV = reinterpret_cast<__nv_bfloat16*>(dyn + SV);
    __nv_bfloat16* sRG = reinterpret_cast<__nv_bfloat16*>(dyn + SM);
    float* sM = reinterpret_cast<float*>(dyn + SM);
    float* stot = reinterpret_cast<float*>(dyn + SU);
    float* sAd = reinterpret_cast<float*>(dyn + SU);
    float* sY = reinterpret_cast<float*>(dyn + SU);
    __nv_bfloat16* sTB = reinterpret_cast<__nv_bfloat16*>(dyn + SU);
    float4* sW = reinterpret_cast<float4*>(dyn + TAPS);
    float* smid = reinterpret_cast<float*>(dyn + SMID);
    float* saux = reinterpret_cast<float*>(dyn + SBETA);
    float* sbeta = saux + 2 * C;
    int* spass = reinterpret_cast<int*>(dyn + SPASS);
    uint64_t* kbar = reinterpret_cast<uint64_t*>(dyn + SBAR);  // k (and every halo row)
    uint64_t* qbar = kbar + 1;  // q, v
    uint64_t* gbar = kbar + 2;  // gate
    uint64_t* wbar = kbar + 3;  // W and U products
    uint32_t* tmem_s = reinterpret_cast<uint32_t*>(kbar + 4);
    __nv_bfloat16* sHalo = reinterpret_cast<__nv_bfloat16*>(dyn + HALO);

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (warp-uniform: roles and MMA issue)
    char* ws = (char*)p.workspace;
    const __nv_bfloat16* q = (const __nv_bfloat16*)p.q;
    const __nv_bfloat16* k = (const __nv_bfloat16*)p.k;
    const __nv_bfloat16* v = (const __nv_bfloat16*)p.v;
    const __nv_bfloat16* g = (const __nv_bfloat16*)p.g;
    const __nv_bfloat16* beta = (const __nv_bfloat16*)p.beta;
    const bool l2 = p.flags & KDA_FLAG_QK_L2NORM, gate = p.flags & KDA_FLAG_GATE, sig = p.flags & KDA_FLAG_BETA_SIGMOID;
    const bool save = !(p.flags & KDA_FLAG_NO_SAVE);  // forward-only calls keep nothing for a backward

    KDA_PHASE_BEGIN();
    if (warp == 0) {
        tmem_alloc(tmem_s, TMEM_COLS);
        tmem_relinquish();
    }
    if (tid >= 64 && tid < 68) prefetch_map(&maps.m[tid - 64]);
    if (tid == 32) {
        mbar_init(kbar, 1);
        mbar_init(gbar, 1);
        mbar_init(qbar, 2);  // (the threads that issue q and v)
        mbar_init(wbar, 2);  // two issuing threads commit the W and U products
        mbar_fence_init();
    }
    pdl_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem0 = *tmem_s;

    // thread roles of the element-wise stages
    const int hw = tid >> 4, c8r = (tid & 15) * 8;               // rows: a half warp has the rows 4 hw .. 4 hw + 3, a lane 8 channels
    const int qt = warp >> 1, gh = warp & 1, gd = 64 * gh + 2 * lane;  // gate: 16-row group, half, the first of two channels
    const bool tiles = maps.ok != 0;  // whole tiles with bulk-tensor copies; rows past the end of the sequence are masked when read
    auto row_src = [&](const __nv_bfloat16* base, const ChunkInfo& ci, int h, int i) { return base + ((size_t)(ci.tok0 + i) * p.H + h) * D; };
    // (a thread is held up by every copy it issues: each tile has its own)
    auto load_rows = [&](uint32_t dst, const CUtensorMap* m, const ChunkInfo& ci, int h, uint64_t* bar, uint32_t more) {
        mbar_expect_tx(bar, C * D * 2 + more);
        tma_load_tile(dyn + dst, m, h * D, (int)ci.tok0, bar);
        tma_load_tile(dyn + dst + 8192, m, h * D + 64, (int)ci.tok0, bar);
    };
    auto request_g = [&](const ChunkInfo& ci, int h) {
        if (tiles && tid == 0) {
            mbar_expect_tx(gbar, C * D * 2);
            tma_load_tile(sRG, &maps.m[3], h * D, (int)ci.tok0, gbar);
        }
    };
    auto request_k = [&](const ChunkInfo& ci, int h) {
        if (!tiles) return;
        const bool halo = CONV && ci.lc > 0;
        if (tid == 32) load_rows(SK, &maps.m[1], ci, h, kbar, halo ? 9 * 256u : 0u);
        if constexpr (CONV) {  // three rows before the chunk, unless it starts its sequence
            if (halo) {
                if (warp == 2 && lane < 9)
                    tma_load_1d(sHalo + lane * D, row_src(lane < 3 ? q : lane < 6 ? k : v, ci, h, lane % 3 - 3), 256, kbar);
            } else if (tid < 9 * 16) {
                reinterpret_cast<uint4*>(sHalo)[tid] = make_uint4(0, 0, 0, 0);
            }
        }
    };
    auto request_qv = [&](const ChunkInfo& ci, int h) {
        if (!tiles) return;
        if (tid == 64) load_rows(SQ, &maps.m[0], ci, h, qbar, 0);
        if (tid == 96) load_rows(SV, &maps.m[2], ci, h, qbar, 0);
    };
    const uint4 zero4 = make_uint4(0, 0, 0, 0);
    auto copy_rows = [&](const ChunkInfo& ci, int h) {  // no tensor maps: the same tiles with plain loads, at the start of the unit
#pragma unroll 1
        for (int x = tid; x < 4 * C * 16; x += NTHR) {
            const int t4 = x >> 10, i = (x >> 4) & 63, c8 = (x & 15) * 8;
            const uint4 u = i < ci.len ? *reinterpret_cast<const uint4*>(row_src(t4 == 0 ? q : t4 == 1 ? k : t4 == 2 ? v : g, ci, h, i) + c8) : zero4;
            *reinterpret_cast<uint4*>(t4 == 3 ? sRG + i * D + c8 : reinterpret_cast<__nv_bfloat16*>(dyn + SQ) + t4 * C * D + swz_bf16(i, c8)) = u;
        }
        if (CONV && tid < 9 * 16) {
            const int r = tid >> 4;
            reinterpret_cast<uint4*>(sHalo)[tid] =
                ci.lc > 0 ? *reinterpret_cast<const uint4*>(row_src(r < 3 ? q : r < 6 ? k : v, ci, h, r % 3 - 3) + 8 * (tid & 15)) : zero4;
        }
        __syncthreads();
    };
    // rows past the end of a partial chunk (the tile copies brought what follows in memory): q, k, v zero, no decay
    auto clear_tail = [&](int len) {
#pragma unroll 1
        for (int x = tid; x < 4 * C * 16; x += NTHR) {
            const int t4 = x >> 10, i = (x >> 4) & 63, c8 = (x & 15) * 8;
            const uint32_t w = t4 == 3 && gate ? 0xff80ff80u : 0u;  // softplus(-inf) = 0
            if (i >= len)
                *reinterpret_cast<uint4*>(t4 == 3 ? sRG + i * D + c8 : reinterpret_cast<__nv_bfloat16*>(dyn + SQ) + t4 * C * D + swz_bf16(i, c8)) =
                    make_uint4(w, w, w, w);
        }
        __syncthreads();
    };
    struct Scalars {  // (beta stays in its storage type: a conversion here would wait for the load)
        float a_log;
        float2 bias;
        __nv_bfloat16 rb;
    };
    auto request_scalars = [&](const ChunkInfo& ci, int h, Scalars& sc) {
        sc.a_log = gate ? p.A_log[h] : 0.f;
        sc.bias = make_float2(0.f, 0.f);
        if (gate && p.dt_bias) sc.bias = make_float2(p.dt_bias[h * D + gd], p.dt_bias[h * D + gd + 1]);
        const int i = 4 * hw + (lane & 3);
        sc.rb = beta[(size_t)(ci.tok0 + (i < ci.len ? i : 0)) * p.H + h];
    };
    // filter taps of a head, padded to four: entry (tensor, channel) at [tensor][channel % 8][channel / 8], so that the sixteen
    // lanes of a half warp read consecutive 16-byte words
    auto request_taps = [&](int h) {
        if constexpr (CONV) {
#pragma unroll 1
            for (int e = tid; e < 3 * D; e += NTHR)
                stage_taps(sW + (e & ~(D - 1)) + (e & 7) * 16 + ((e & (D - 1)) >> 3), e < D ? p.conv_q : e < 2 * D ? p.conv_k : p.conv_v, h, e & (D - 1), p.conv_ksize);
            cp_async_commit();
        }
    };
    auto load_g8 = [&](int i, int c8, float (&x)[8]) {
        const float4 a = *reinterpret_cast<const float4*>(sG + swz_f32(i, c8));
        const float4 b = *reinterpret_cast<const float4*>(sG + swz_f32(i, c8 + 4));
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    };
    const int n_units = p.NT * p.H;
    Scalars nx;
    // unit u = (chunk u / H, head (u + chunk) % H): the head is skewed by the chunk index so that the units a
    // CTA visits (stride gridDim.x) cycle through ALL heads even when the stride shares a factor with H
    // (heads differ in cost: the ones whose tiles fail the span guard take the exact path)
    UnitWalk uw;
    uw.init(blockIdx.x, gridDim.x, p.H);
    ChunkInfo ci = chunk_info(p, blockIdx.x / p.H);
    request_g(ci, uw.head());
    request_k(ci, uw.head());
    request_qv(ci, uw.head());
    request_scalars(ci, uw.head(), nx);
    request_taps(uw.head());
    cp_async_wait<0>();
    if (CONV) __syncthreads();
    uint32_t it = 0;
    bool ok = true, more = false;
    for (; uw.unit < n_units; ++it) {
    const int c = uw.c, h = uw.head();
    const size_t rec = (size_t)c * p.H + h;
    const float a_log_h = nx.a_log;
    const float2 bias = nx.bias;
    if (!tiles) copy_rows(ci, h);
    const int bi = 4 * hw + (lane & 3);
    const float be = bi < ci.len ? (sig ? sigmoid_f(__bfloat162float(nx.rb)) : __bfloat162float(nx.rb)) : 0.f;  // beta of row bi
    if ((lane & 15) < 4) sbeta[bi] = be;
    if (tiles) ok = mbar_wait(gbar, it & 1, p, 8);
    if (CONV || ci.len < C) {
        if (tiles) ok = mbar_wait(kbar, it & 1, p, 8) && mbar_wait(qbar, it & 1, p, 8) && ok;
        if (ci.len < C) clear_tail(ci.len);
    }
    KDA_PHASE(0);
    // ---- L2 norm of the q and k rows, in place, two rows at a time.  The four sums of squares of a half warp (row m, tensor t) are
    //      reduced by a transposing exchange, after which four lanes have each and turn it into 1 / norm: one square root and one
    //      division, long instruction sequences, instead of four
    auto normalise2 = [&](int i0, uint4 (&x4)[4]) {  // x4: row i0 q, k, row i0 + 1 q, k
        if (l2) {
            float s4[4], s2[2];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                float x[8];
                float2 a = make_float2(0.f, 0.f);
                bf16x8_to_f32(x4[m], x);
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    const float2 x2 = make_float2(x[j], x[j + 1]);
                    a = __ffma2_rn(x2, x2, a);  // explicit: both instantiations must round alike
                }
                s4[m] = a.x + a.y;
            }
            const bool b8 = lane & 8, b4 = lane & 4;
#pragma unroll
            for (int j = 0; j < 2; ++j) s2[j] = (b8 ? s4[2 + j] : s4[j]) + __shfl_xor_sync(0xffffffffu, b8 ? s4[j] : s4[2 + j], 8);
            float s1 = (b4 ? s2[1] : s2[0]) + __shfl_xor_sync(0xffffffffu, b4 ? s2[0] : s2[1], 4);
            s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
            s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
            const float rn = 1.f / fmaxf(sqrtf(s1), 1e-6f);
            if ((lane & 3) == 0) saux[(b4 ? C : 0) + i0 + (b8 ? 1 : 0)] = rn;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const float n = __shfl_sync(0xffffffffu, rn, (lane & 16) + 4 * m);
                float x[8];
                bf16x8_to_f32(x4[m], x);
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] *= n;
                x4[m] = f32_to_bf16x8(x);
            }
        } else if ((lane & 3) == 0) {
            saux[(lane & 4 ? C : 0) + i0 + (lane & 8 ? 1 : 0)] = 1.f;
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) *reinterpret_cast<uint4*>((m & 1 ? sK : sQ) + swz_bf16(i0 + (m >> 1), c8r)) = x4[m];
    };
    auto store_v = [&](int m, const uint4& v4) {  // beta v of row 4 hw + m, the operand of the U product
        const float b = __shfl_sync(0xffffffffu, be, (lane & 16) + m);
        float x[8];
        bf16x8_to_f32(v4, x);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] *= b;
        *reinterpret_cast<uint4*>(sV + swz_bf16(4 * hw + m, c8r)) = f32_to_bf16x8(x);
    };
    if constexpr (CONV) {
        // ---- 1: y[i] = silu(sum_j tap[j] x[i - 3 + j]) for the thread's four rows, rounded to BF16 like the stand-alone
        //      convolution; everything after sees only y
        auto conv_rows = [&](uint4(&out)[4], int tensor) {
            uint4 win[7];
#pragma unroll
            for (int r = 0; r < 7; ++r) {
                const int x = 4 * hw - 3 + r;
                win[r] = *reinterpret_cast<const uint4*>(x < 0 ? sHalo + (3 * tensor + x + 3) * D + c8r
                                                               : reinterpret_cast<__nv_bfloat16*>(dyn + SQ) + tensor * C * D + swz_bf16(x, c8r));
            }
            auto pick = [](const uint4& u, int j2) { return j2 == 0 ? u.x : j2 == 1 ? u.y : j2 == 2 ? u.z : u.w; };
            uint32_t o[4][4];
#pragma unroll
            for (int j2 = 0; j2 < 4; ++j2) {  // two channels in packed FMAs (the order of conv_pre)
                const int j = 2 * j2;
                const float4 wa = sW[tensor * D + j * 16 + (tid & 15)], wb = sW[tensor * D + (j + 1) * 16 + (tid & 15)];
                auto x2 = [&](int r) {
                    const uint32_t w = pick(win[r], j2);
                    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
                };
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const float2 pre = __ffma2_rn(make_float2(wa.w, wb.w), x2(m + 3),
                                                  __ffma2_rn(make_float2(wa.z, wb.z), x2(m + 2),
                                                             __ffma2_rn(make_float2(wa.y, wb.y), x2(m + 1), __fmul2_rn(make_float2(wa.x, wb.x), x2(m)))));
                    o[m][j2] = pack_bf16(silu_f(pre.x), silu_f(pre.y));
                }
            }
#pragma unroll
            for (int m = 0; m < 4; ++m) out[m] = 4 * hw + m < ci.len ? make_uint4(o[m][0], o[m][1], o[m][2], o[m][3]) : zero4;
        };
        uint4 rq4[4], rk4[4], rv4[4];
        conv_rows(rv4, 2);
        if (save) {
            __nv_bfloat16* gVc = (__nv_bfloat16*)(ws + L.Vc) + rec * C * D;
#pragma unroll
            for (int m = 0; m < 4; ++m) *reinterpret_cast<uint4*>(gVc + (4 * hw + m) * D + c8r) = rv4[m];
        }
        conv_rows(rq4, 0);
        conv_rows(rk4, 1);
        __syncthreads();  // every row has been read
#pragma unroll
        for (int m = 0; m < 4; ++m) store_v(m, rv4[m]);
#pragma unroll
        for (int m = 0; m < 4; m += 2) {
            uint4 x4[4] = {rq4[m], rk4[m], rq4[m + 1], rk4[m + 1]};
            normalise2(4 * hw + m, x4);
        }
    }
    KDA_PHASE(1);
    // ---- 2: gate.  Thread = (16-row group, two channels): running sums of the group, whose totals are passed on
    {
        const float negA = gate ? -expf(a_log_h) : 0.f;
        const uint32_t* raw = reinterpret_cast<const uint32_t*>(sRG + 16 * qt * D + gd);
        float2 run = make_float2(0.f, 0.f), Gr[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const uint32_t w = raw[r * (D / 2)];
            float2 gl = make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
            if (gate) gl = __fmul2_rn(make_float2(negA, negA), softplus_fast(__fadd2_rn(gl, bias)));
            run = __ffma2_rn(gl, make_float2(LOG2E, LOG2E), run);  // explicit: both instantiations must round alike
            Gr[r] = run;
        }
        *reinterpret_cast<float2*>(stot + qt * D + gd) = run;
        KDA_PHASE(2);
        if constexpr (!CONV) {  // (q is requested last and arrives last)
            if (tiles && ci.len == C) ok = mbar_wait(kbar, it & 1, p, 8) && mbar_wait(qbar, it & 1, p, 8) && ok;
#pragma unroll
            for (int m = 0; m < 4; m += 2) {
                const int i = 4 * hw + m;
                uint4 x4[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) x4[x] = *reinterpret_cast<const uint4*>((x & 1 ? sK : sQ) + swz_bf16(i + (x >> 1), c8r));
                store_v(m, *reinterpret_cast<const uint4*>(sV + swz_bf16(i, c8r)));
                store_v(m + 1, *reinterpret_cast<const uint4*>(sV + swz_bf16(i + 1, c8r)));
                normalise2(i, x4);
            }
        }
        __syncthreads();  // the totals of the groups are there
        float2 base = make_float2(0.f, 0.f);
        for (int b = 0; b < qt; ++b) base = __fadd2_rn(base, *reinterpret_cast<const float2*>(stot + b * D + gd));
        // Span guard, after k3mini/backends.py:17-19, of the block's 16 rows: every channel monotone non-increasing and finite (then its
        // span is first - last row), the largest span within the limit.  A block goes pair by pair unless both its halves pass
        // (a negative limit: every block).
        bool good = true;
        float2 first, prev = make_float2(INFINITY, INFINITY);
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            float2* at = reinterpret_cast<float2*>(sG + swz_f32(16 * qt + r, gd));
            const float2 x = __fadd2_rn(Gr[r], base);
            *at = x;
            good = good && x.x <= prev.x && x.y <= prev.y;
            prev = x;
            if (r == 0) first = x;
        }
        *reinterpret_cast<float2*>(smid + qt * D + gd) = make_float2(0.5f * (first.x + prev.x), 0.5f * (first.y + prev.y));
        good = good && isfinite(first.x) && isfinite(first.y) && isfinite(prev.x) && isfinite(prev.y) &&
               fmaxf(first.x - prev.x, first.y - prev.y) <= p.guard_span;
        good = __all_sync(0xffffffffu, good);
        if (lane == 0) spass[2 * qt + gh] = good;
    }
    fence_async_smem();
    __syncthreads();
    KDA_PHASE(3);
    if (save && lane == 0 && warp < 3) {  // prologue results for the backward: bulk stores straight from shared memory
        if (warp == 0) tma_store_1d((float*)(ws + L.Gc) + rec * C * D, sG, C * D * 4);
        if (warp == 1) tma_store_1d((__nv_bfloat16*)(ws + L.Qn) + rec * C * D, sQ, C * D * 2);
        if (warp == 2) {
            tma_store_1d((__nv_bfloat16*)(ws + L.Kn) + rec * C * D, sK, C * D * 2);
            tma_store_1d((float*)(ws + L.aux) + rec * 3 * C, saux, 3 * C * 4);
        }
        tma_store_commit();
    }
    uw.next();  // from here on the next unit of this CTA
    more = uw.unit < n_units;
    if (more) ci = chunk_info(p, uw.c);  // (dependent loads: issued well ahead of the requests that need them)
    // ---- 3: Aqk and L.  Warp = (block I, channel half hf)
    const int gq = lane >> 2, t = lane & 3;
    const int I = warp < 4 ? warp : 7 - warp, hf = warp >> 2;  // (a scheduler's two warps share the work of one to four block pairs)
    const int pr = ((gq & 1) << 2) | (gq & 2) | (gq >> 2), kt = (t >> 1) | ((t & 1) << 1);  // row g; keys 2t and 2t + 1 are kt, kt + 4
    float keep[4][8];  // the matrix this warp finishes, Aqk (half 0) or L (half 1): [J][4 n-tile + fragment], keep[3] the diagonal block
    {
        // The diagonal block, in FP32: rows pr, pr + 8 against keys kt + 4 n.  With the midpoint m of its rows as reference: row factors
        // 2^(G_i - m) and scaled key rows k_j 2^(m - G_j) (within 2^(+-116)) of sixteen channels at a time, made once each and kept in the
        // warp's part of SM / SU; or pair by pair, one exponential each.  Pairs j > i are computed too but never used; whatever they
        // overflow to is dropped.  Sums as chains of eight that meet in a tree.
        float dq[2][4] = {}, dl[2][4] = {}, hq[2][4], hl[2][4];
        const bool pass = spass[2 * I] & spass[2 * I + 1];
        float* sF = reinterpret_cast<float*>(dyn + SM) + warp * (2 * 16 * LDS);
        float* sKY = sF + 16 * LDS;
#pragma unroll 1
        for (int s = 0; s < 4; ++s) {
            float2 av[2][4] = {}, lv[2][4] = {};
            if (pass) {
                const int ch = 64 * hf + 16 * s + 4 * t;
                const float4 mid = *reinterpret_cast<const float4*>(smid + I * D + ch);
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const int row = 16 * I + pr + 8 * m;
                    const float4 G4 = *reinterpret_cast<const float4*>(sG + swz_f32(row, ch));
                    float f[4], y[4], kf[4];
                    unpack4(*reinterpret_cast<const uint2*>(sK + swz_bf16(row, ch)), kf);
                    exp2_diff(G4, mid, f);
                    exp2_diff(mid, G4, y);
                    *reinterpret_cast<float4*>(sF + (pr + 8 * m) * LDS + 4 * t) = make_float4(f[0], f[1], f[2], f[3]);
                    *reinterpret_cast<float4*>(sKY + (pr + 8 * m) * LDS + 4 * t) = make_float4(kf[0] * y[0], kf[1] * y[1], kf[2] * y[2], kf[3] * y[3]);
                }
                __syncwarp();
#pragma unroll 2
                for (int u = 0; u < 4; ++u) {
                    float2 qf[2][2], kf[2][2];
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        const float4 f = *reinterpret_cast<const float4*>(sF + (pr + 8 * m) * LDS + 4 * u);
                        const int at = swz_bf16(16 * I + pr + 8 * m, 64 * hf + 16 * s + 4 * u);
                        float a[4], b[4];
                        unpack4(*reinterpret_cast<const uint2*>(sQ + at), a);
                        unpack4(*reinterpret_cast<const uint2*>(sK + at), b);
                        qf[m][0] = __fmul2_rn(make_float2(a[0], a[1]), make_float2(f.x, f.y));
                        qf[m][1] = __fmul2_rn(make_float2(a[2], a[3]), make_float2(f.z, f.w));
                        kf[m][0] = __fmul2_rn(make_float2(b[0], b[1]), make_float2(f.x, f.y));
                        kf[m][1] = __fmul2_rn(make_float2(b[2], b[3]), make_float2(f.z, f.w));
                    }
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        const float4 y = *reinterpret_cast<const float4*>(sKY + (kt + 4 * n) * LDS + 4 * u);
#pragma unroll
                        for (int m = n >> 1; m < 2; ++m) {  // (keys 8 .. 15 have no pairs with rows 0 .. 7)
                            av[m][n] = __ffma2_rn(qf[m][0], make_float2(y.x, y.y), __ffma2_rn(qf[m][1], make_float2(y.z, y.w), av[m][n]));
                            lv[m][n] = __ffma2_rn(kf[m][0], make_float2(y.x, y.y), __ffma2_rn(kf[m][1], make_float2(y.z, y.w), lv[m][n]));
                        }
                    }
                }
                __syncwarp();
            } else {
#pragma unroll 1
                for (int u = 0; u < 4; ++u) {
                    const int ch = 64 * hf + 16 * s + 4 * u;
                    float4 Gr[2];
                    float qf[2][4], kf[2][4];
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        const int row = 16 * I + pr + 8 * m;
                        Gr[m] = *reinterpret_cast<const float4*>(sG + swz_f32(row, ch));
                        unpack4(*reinterpret_cast<const uint2*>(sQ + swz_bf16(row, ch)), qf[m]);
                        unpack4(*reinterpret_cast<const uint2*>(sK + swz_bf16(row, ch)), kf[m]);
                    }
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        const int key = 16 * I + kt + 4 * n;
                        const float4 Gk = *reinterpret_cast<const float4*>(sG + swz_f32(key, ch));
                        float kk[4];
                        unpack4(*reinterpret_cast<const uint2*>(sK + swz_bf16(key, ch)), kk);
#pragma unroll
                        for (int m = n >> 1; m < 2; ++m) {
                            float e[4];
                            exp2_diff(Gr[m], Gk, e);
                            const float2 y0 = __fmul2_rn(make_float2(kk[0], kk[1]), make_float2(e[0], e[1])), y1 = __fmul2_rn(make_float2(kk[2], kk[3]), make_float2(e[2], e[3]));
                            av[m][n] = __ffma2_rn(make_float2(qf[m][0], qf[m][1]), y0, __ffma2_rn(make_float2(qf[m][2], qf[m][3]), y1, av[m][n]));
                            lv[m][n] = __ffma2_rn(make_float2(kf[m][0], kf[m][1]), y0, __ffma2_rn(make_float2(kf[m][2], kf[m][3]), y1, lv[m][n]));
                        }
                    }
                }
            }
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int m = n >> 1; m < 2; ++m) {
                    float &a = dq[n >> 1][2 * m + (n & 1)], &l = dl[n >> 1][2 * m + (n & 1)], &ha = hq[n >> 1][2 * m + (n & 1)], &hb = hl[n >> 1][2 * m + (n & 1)];
                    const float a16 = av[m][n].x + av[m][n].y, l16 = lv[m][n].x + lv[m][n].y;
                    if (s & 1) a += ha + a16, l += hb + l16;
                    else ha = a16, hb = l16;
                }
        }
        __syncthreads();  // the scaled rows are dead: their place takes the partial sums
        float oq[3][2][4] = {}, ol[3][2][4] = {};
#pragma unroll 1
        for (int s = 0; s < 4; ++s) {
            // (every row of this loop is pr mod 8: one swizzled offset for all, a row is a constant away from row pr)
            const int ch = 64 * hf + 16 * s + 4 * t;
            const float* pG = sG + swz_f32(pr, ch);
            const __nv_bfloat16 *pK = sK + swz_bf16(pr, ch), *pQI = pK + (16 * I * 64 - 8192), *pKI = pK + 16 * I * 64;
            const float4 G0 = *reinterpret_cast<const float4*>(pG + 16 * I * D), G1 = *reinterpret_cast<const float4*>(pG + 16 * I * D + 8 * D);
            float q0[4], q1[4], k0[4], k1[4];
            unpack4(*reinterpret_cast<const uint2*>(pQI), q0);
            unpack4(*reinterpret_cast<const uint2*>(pQI + 8 * 64), q1);
            unpack4(*reinterpret_cast<const uint2*>(pKI), k0);
            unpack4(*reinterpret_cast<const uint2*>(pKI + 8 * 64), k1);
            if (I > 0) {  // earlier blocks: reference r_I (row 16 I, which the swizzle leaves as it is)
                const float4 rf = *reinterpret_cast<const float4*>(sG + 16 * I * D + ch);
                float f0[4], f1[4];
                exp2_diff(G0, rf, f0);
                exp2_diff(G1, rf, f1);
                uint32_t aq[4], ak[4];
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    aq[2 * x] = pack_bf16(q0[2 * x] * f0[2 * x], q0[2 * x + 1] * f0[2 * x + 1]);
                    aq[2 * x + 1] = pack_bf16(q1[2 * x] * f1[2 * x], q1[2 * x + 1] * f1[2 * x + 1]);
                    ak[2 * x] = pack_bf16(k0[2 * x] * f0[2 * x], k0[2 * x + 1] * f0[2 * x + 1]);
                    ak[2 * x + 1] = pack_bf16(k1[2 * x] * f1[2 * x], k1[2 * x + 1] * f1[2 * x + 1]);
                }
#pragma unroll
                for (int J = 0; J < 3; ++J)
                    if (J < I) {
#pragma unroll
                        for (int n = 0; n < 2; ++n) {
                            float kf[4], f[4];
                            unpack4(*reinterpret_cast<const uint2*>(pK + (16 * J + 8 * n) * 64), kf);
                            exp2_diff(rf, *reinterpret_cast<const float4*>(pG + (16 * J + 8 * n) * D), f);
                            const uint32_t b0 = pack_bf16(kf[0] * f[0], kf[1] * f[1]), b1 = pack_bf16(kf[2] * f[2], kf[3] * f[3]);
                            mma_bf16(oq[J][n], aq, b0, b1);
                            mma_bf16(ol[J][n], ak, b0, b1);
                        }
                    }
            }
        }
        // each half gives the other the partial sums of the matrix that one finishes: L to its place, Aqk to the
        // mirrored place above the diagonal blocks
        auto hand_over = [&](int J, const float (&give)[2][4], const float (&own)[2][4], float (&mine)[8]) {
            float* dst = hf == 0 ? sM + (16 * I + pr) * LDR + 16 * J + kt
                       : J < I   ? sM + (16 * J + pr) * LDR + 16 * I + kt
                                 : sAd + (16 * I + pr) * LDA + kt;
            const int ld = hf && J == I ? LDA : LDR;
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    dst[(x >> 1) * 8 * ld + 8 * n + 4 * (x & 1)] = give[n][x];
                    mine[4 * n + x] = own[n][x];
                }
        };
        if (hf) {
            hand_over(I, dq, dl, keep[3]);
#pragma unroll
            for (int J = 0; J < 3; ++J)
                if (J < I) hand_over(J, oq[J], ol[J], keep[J]);
        } else {
            hand_over(I, dl, dq, keep[3]);
#pragma unroll
            for (int J = 0; J < 3; ++J)
                if (J < I) hand_over(J, ol[J], oq[J], keep[J]);
        }
    }
    KDA_PHASE(4);
    // ---- the Qt, Kh and gamC records.  A warp takes eight rows x four channel chunks at a time (eight lanes = the rows of one core
    //      matrix: no bank conflicts, whole 128-byte lines); the later its block, the more products it had, the fewer it takes
    {
        __nv_bfloat16* gQt = (__nv_bfloat16*)(ws + L.Qt) + rec * C * D;
        __nv_bfloat16* gKh = (__nv_bfloat16*)(ws + L.Kh) + rec * C * D;
        const int beg = 16 * hf + (I == 0 ? 0 : I == 1 ? 8 : I == 2 ? 13 : 16), end = 16 * hf + (I == 0 ? 8 : I == 1 ? 13 : 16);
#pragma unroll 1
        for (int x = beg; x < end; ++x) {
            const int i = 8 * (x >> 2) + (lane & 7), c8 = 8 * (4 * (x & 3) + (lane >> 3));
            float G8[8], x8[8], o8[8], gl[8];
            load_g8(i, c8, G8);
            load_g8(C - 1, c8, gl);
            bf16x8_to_f32(*reinterpret_cast<const uint4*>(sQ + swz_bf16(i, c8)), x8);
#pragma unroll
            for (int j = 0; j < 8; ++j) o8[j] = p.scale * x8[j] * ex2_approx(G8[j]);
            *reinterpret_cast<uint4*>(gQt + cm_idx(i, c8, D)) = f32_to_bf16x8(o8);
            bf16x8_to_f32(*reinterpret_cast<const uint4*>(sK + swz_bf16(i, c8)), x8);
#pragma unroll
            for (int j = 0; j < 8; ++j) o8[j] = x8[j] * ex2_approx(gl[j] - G8[j]);
            *reinterpret_cast<uint4*>(gKh + cm_idx(i, c8, D)) = f32_to_bf16x8(o8);
        }
    }
    KDA_PHASE(5);
    if (save && lane == 0 && warp < 3) tma_store_wait_read();  // the bulk stores have read q^, k^, G
    __syncthreads();
    KDA_PHASE(6);
    // ---- 4: the halves' sums: Aqk record (half 0), L and the inverse of its diagonal block (half 1)
    auto other = [&](int J) { return hf ? sM + (16 * I + pr) * LDR + 16 * J + kt : J < I ? sM + (16 * J + pr) * LDR + 16 * I + kt : sAd + (16 * I + pr) * LDA + kt; };
    if (hf) {
#pragma unroll
        for (int J = 0; J < 4; ++J)
            if (J < I || J == 3) {
                float* dst = other(J == 3 ? I : J);
#pragma unroll
                for (int x = 0; x < 8; ++x) {
                    const int m8 = ((x >> 1) & 1) * 8, n8 = 8 * (x >> 2) + 4 * (x & 1);
                    dst[m8 * LDR + n8] += keep[J][x];
                }
            }
        __syncwarp();
        invert_diagonal(sM, sbeta, I, lane);
    } else {
        __nv_bfloat16* gA = (__nv_bfloat16*)(ws + L.Aqk) + rec * C * C;
#pragma unroll
        for (int J = 0; J < 4; ++J)
            if (J < I || J == 3) {
                const int Jb = J == 3 ? I : J;
                const float* src = other(Jb);
                const int ld = J == 3 ? LDA : LDR;
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        float a[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const float* s = src + m * 8 * ld + 8 * n + 4 * e;
                            a[e] = (keep[J][4 * n + 2 * m + e] + *s) * p.scale;
                            if (J == 3 && kt + 4 * e + 8 * n > pr + 8 * m) a[e] = 0.f;
                        }
                        // adjacent keys meet in a lane pair: lanes 0, 1 take keys (0, 1), (2, 3), lanes 2, 3 keys (4, 5), (6, 7)
                        const float got = __shfl_xor_sync(0xffffffffu, t < 2 ? a[1] : a[0], 2);
                        *reinterpret_cast<uint32_t*>(gA + cm_idx(16 * I + pr + 8 * m, 16 * Jb + 8 * n, C) + 2 * t) =
                            t < 2 ? pack_bf16(a[0], got) : pack_bf16(got, a[1]);
                    }
            }
        for (int J = I + 1; J < 4; ++J)
            *reinterpret_cast<uint4*>(gA + cm_idx(16 * I + (lane & 15), 16 * J + 8 * (lane >> 4), C)) = zero4;
    }
    KDA_PHASE(7);
    if (tid < D) ((float*)(ws + L.gamC))[rec * D + tid] = ex2_approx(sG[swz_f32(C - 1, tid)]);
    // ---- beta k^ 2^G, the operand of the W product, in place of q^
#pragma unroll 1
    for (int x = 0; x < 4; ++x) {
        const int i = 8 * warp + (lane & 7), c8 = 8 * (4 * x + (lane >> 3));
        float G8[8], kf[8];
        load_g8(i, c8, G8);
        bf16x8_to_f32(*reinterpret_cast<const uint4*>(sK + swz_bf16(i, c8)), kf);
        const float b = sbeta[i];
#pragma unroll
        for (int j = 0; j < 8; ++j) kf[j] = b * kf[j] * ex2_approx(G8[j]);
        *reinterpret_cast<uint4*>(sQ + swz_bf16(i, c8)) = f32_to_bf16x8(kf);
    }
    fence_async_smem();
    __syncthreads();
    KDA_PHASE(12);
    if (more) {  // k^ is dead
        request_k(ci, uw.head());
        request_scalars(ci, uw.head(), nx);
        request_taps(uw.head());
    }
    invert_products(sM, sbeta, sY, warp, lane);
    __syncthreads();
    KDA_PHASE(8);
    // ---- 5: T record; T as the B operand of the WY products (zero above the diagonal blocks, where other things were)
#pragma unroll 1
    for (int m = 0; m < 2; ++m) {
        // eight lanes = eight adjacent rows of one 8-column group: one core matrix of the records, 32 distinct banks
        const int x = tid + NTHR * m, i = (x & 7) | ((x >> 6) << 3), j8 = ((x >> 3) & 7) * 8;
        uint4 tb = zero4;
        if ((j8 >> 4) <= (i >> 4)) {
            float t8[8];
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
                const float4 t4 = *reinterpret_cast<const float4*>(sM + i * LDR + j8 + j);
                t8[j] = t4.x, t8[j + 1] = t4.y, t8[j + 2] = t4.z, t8[j + 3] = t4.w;
            }
            tb = f32_to_bf16x8(t8);
        }
        if (save) *reinterpret_cast<uint4*>((__nv_bfloat16*)(ws + L.Tm) + rec * C * C + cm_idx(i, j8, C)) = tb;
        *reinterpret_cast<uint4*>(sTB + cm_idx(i, j8, C)) = tb;
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (more) request_g(ci, uw.head());  // T is dead
    if (warp < 2 && elect_one()) {  // W^T and U^T (one issuing thread each)
        tc_fence_after();
        const uint32_t sb = smem_u32(dyn);
        constexpr uint32_t id = make_idesc(128, 64, true, false);
        const uint32_t acc = warp == 0 ? T_W : T_U, a_tile = warp == 0 ? SQ : SV;
#pragma unroll
        for (int s = 0; s < 4; ++s)
            mma_ss(tmem0 + acc, make_desc_sw128(sb + a_tile + s * 2048, 8192, 1024), make_desc(sb + SU + s * 256, 128, 1024), id, s > 0);
        mma_commit(wbar);
    }
    __syncwarp();
    KDA_PHASE(9);
    ok = mbar_wait(wbar, it & 1, p, 8) && ok;
    tc_fence_after();
    if (more) request_qv(ci, uw.head());
    KDA_PHASE(10);
    // W and U records: warps 0 .. 3 the four quadrants of W, warps 4 .. 7 of U
    if (ok) {
        const int qd = warp & 3, dd = 32 * qd + lane;
        __nv_bfloat16* dst = (__nv_bfloat16*)(ws + (warp < 4 ? L.W : L.U)) + rec * C * D;
        const uint32_t src = tmem0 + ((uint32_t)(32 * qd) << 16) + (warp < 4 ? T_W : T_U);
#pragma unroll
        for (int i0 = 0; i0 < C; i0 += 16) {
            uint32_t r[16];
            tmem_ld16(src + i0, r);
            tmem_wait_ld();
            *reinterpret_cast<uint4*>(dst + cm_idx(dd, i0, C)) =
                make_uint4(pack_bf16(__uint_as_float(r[0]), __uint_as_float(r[1])), pack_bf16(__uint_as_float(r[2]), __uint_as_float(r[3])),
                           pack_bf16(__uint_as_float(r[4]), __uint_as_float(r[5])), pack_bf16(__uint_as_float(r[6]), __uint_as_float(r[7])));
            *reinterpret_cast<uint4*>(dst + cm_idx(dd, i0 + 8, C)) =
                make_uint4(pack_bf16(__uint_as_float(r[8]), __uint_as_float(r[9])), pack_bf16(__uint_as_float(r[10]), __uint_as_float(r[11])),
                           pack_bf16(__uint_as_float(r[12]), __uint_as_float(r[13])), pack_bf16(__uint_as_float(r[14]), __uint_as_float(r[15])));
        }
    }
    if constexpr (CONV) cp_async_wait<0>();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    KDA_PHASE(11);
    if (!ok) break;  // a wait gave up (recorded in the status word): no further unit is started
    }
    if (!ok && more && tiles) {  // the next unit's copies are in flight: they must have landed before the CTA leaves
        mbar_wait(kbar, (it + 1) & 1, p, 8);
        mbar_wait(gbar, (it + 1) & 1, p, 8);
        mbar_wait(qbar, (it + 1) & 1, p, 8);
    }
    if (lane == 0 && warp < 3) tma_store_wait_all();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem0, TMEM_COLS);
}

cudaError_t launch_fwd_intra_tc(const KdaParams& p, cudaStream_t s) {
    auto kern = p.conv_q ? kda_fwd_intra_tc<true> : kda_fwd_intra_tc<false>;
    const uint32_t smem = p.conv_q ? fi::TOTAL_CONV : fi::TOTAL;
    const cudaError_t e = allow_smem(kern, (int)smem, true);
    if (e != cudaSuccess) return e;
    const int units = p.NT * p.H, ctas = 2 * sm_count();
    RowMaps maps = {};
    const long long tokens = (long long)p.B * p.T;
    maps.ok = !(p.flags & KDA_FLAG_ROW_COPIES) && make_row_map(&maps.m[0], p.q, tokens, p.H, C, true) && make_row_map(&maps.m[1], p.k, tokens, p.H, C, true) &&
              make_row_map(&maps.m[2], p.v, tokens, p.H, C, true) && make_row_map(&maps.m[3], p.g, tokens, p.H, C);
    return launch_dependent(kern, units < ctas ? units : ctas, fi::NTHR, smem, s, p, maps, ws_layout(p.NT, p.H, p.dk, p.dv, p.dtype));
}

}  // namespace kda

KDA_PHASE_EXPORT(kda_debug_phases_fwd_intra)
