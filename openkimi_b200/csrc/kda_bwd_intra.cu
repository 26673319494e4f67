// bwd_intra (BF16 path, d = 128): the guarded intra-chunk backward on tensor cores, the reverse
// cumulative sum of the gate gradient and the chain rule through gate / L2 norm / sigmoid.
// One CTA per SM walks the (chunk, head) units (UnitWalk).
//
// With D_ij = 2^(G_i - G_j) per channel (i >= j inside the chunk), dA = dAqk (strictly lower; its
// diagonal is handled apart), dM the gradient of I + diag(beta) L (strictly lower):
//   row side   a1_i = sum_{j<i} dA_ij k_j D_ij          a2_i = sum_{j<i} dM_ij k_j D_ij
//   col side   c1_j = sum_{i>j} (scale dA_ij q_i + beta_i dM_ij k_i) D_ij
// The chunk is cut into four 16-row blocks; every [16 rows x 32 channels] tile is one guard tile
// of the reference (experiments/kda_sm90/patch_fla_guarded_intra.py:35-63): per-channel monotone
// non-increasing, finite, max-over-channels span <= the runtime limit.  A block X whose tile
// passes gets the per-channel midpoint m_X = (max + min) / 2 as the reference of all its rows:
//   keys      KN_j = k_j 2^(m_X - G_j)          queries   QP_i = scale q_i 2^(G_i - m_X),
//                                                          KP_i = beta_i k_i 2^(G_i - m_X)
// (every factor within 2^(+-116) at the 232 limit).  Per channel these are contractions over the
// token index, so they run as tcgen05 MMAs with M = 128 channels:
//   accR_J[d, i] = sum_{j in J} dA_ij KN_j[d]   (i >= 16 J;  same with dM)       K = 16
//   accC_I[d, j] = sum_{i in I} dA_ij QP_i[d] + dM_ij KP_i[d]   (j < 16 (I+1))    K = 32
// and the read-back applies the remaining factor, one exp2 per (row, block):
//   a1_i = sum_{J <= I(i)} 2^(G_i - m_J) accR_J[d, i]        c1_j = sum_{I >= J(j)} 2^(m_I - G_j) accC_I[d, j]
// (exponents <= 0 for J < I; inside the diagonal block the pair of factors is the midpoint
// factorisation).  Precision: the gate gradient is a difference of large terms, plain TF32 products
// fail it by percents; every operand is therefore split three ways into BF16 (x = p0 + p1 + p2, 24
// bits) and each product runs as six BF16 passes (p0q0 + p0q1 + p1q0 + p1q1 + p0q2 + p2q0), which
// is at least the "tf32x3" class of the reference's contract.  dA / dM arrive already split from
// bwd_wy (three cm(i, j; 64) tiles each) and are used as they are.
// A tile that fails the guard (or a negative limit = exact mode) has no usable midpoint.  Its rows
// then take first-row references instead, which need no guard because every factor is <= 1:
// keys use r = G at the first row of the NEXT block (KN_j = k_j 2^(r - G_j), read-back 2^(G_i - r) for
// the rows of later blocks), queries use r' = G at the first row of their OWN block (QP_i = scale q_i
// 2^(G_i - r'), read-back 2^(r' - G_j) for the columns of earlier blocks).  So every off-diagonal block
// pair runs on the tensor cores whatever the guard says, and only the pairs INSIDE a rejected tile
// are evaluated on the CUDA cores in FP32 with one exp2 per pair.  Rejected tiles therefore see the
// same instructions with the guard on or off, hence the same bits.
#include <type_traits>

#include "kda_common.cuh"
#include "kda_conv_bwd.cuh"
#include "kda_tc.cuh"
#include "kda_tmap.cuh"

namespace kda {

using namespace tc;

namespace bi {
constexpr int D = 128, NTHR = 512, B = 16;
constexpr uint32_t SG = 0;                   // G f32 [64][128], chunk-swizzled rows (swz_f32) as the forward keeps it
constexpr uint32_t SQ = SG + 32768;          // q^ bf16 [64][128], chunk-swizzled rows (swz_bf16)
constexpr uint32_t SK = SQ + 16384;          // k^ bf16 [64][128], chunk-swizzled rows
constexpr uint32_t SB = SK + 16384;          // dAqk p0 p1 p2, dM p0 p1 p2: six cm(i, j; 64) bf16 tiles
constexpr uint32_t XB = SB + 49152;          // operand buffer X: three parts of cm(d, t; 64) bf16 [128][64]
constexpr uint32_t YB = XB + 49152;          // operand buffer Y
constexpr uint32_t SAUX = YB + 49152;        // f32 [64] 1/|q|, [64] 1/|k|, [64] beta
constexpr uint32_t SDB = SAUX + 768;         // f32 [64] beta gradient so far
constexpr uint32_t SDIAG = SDB + 256;        // f32 [64] diagonal of dAqk
constexpr uint32_t SMID = SDIAG + 256;       // f32 [2][4][128] key / query reference of every block and channel
constexpr uint32_t STOT = SMID + 4096;       // f32 [4][128] block totals of dG
constexpr uint32_t SSCR = STOT + 2048;       // f32 [4][128]
constexpr uint32_t SRED = SSCR + 2048;       // f32 [16]
constexpr uint32_t SREJ = SRED + 64;         // int [4][4]: tile (block, channel group) rejected
constexpr uint32_t FD = SREJ + 64;           // f32 [2][4][16][16] diagonal blocks of dAqk, dM rebuilt for rejected tiles, transposed
constexpr uint32_t SAUX2 = FD + 8192;        // the aux record of every other unit (requests ahead, CONVB)
constexpr uint32_t TOTAL = SAUX2 + 768;
static_assert(TOTAL <= 232448, "shared memory of a CTA");
// later uses of the dead operand space
constexpr uint32_t PF = YB;                  // bf16 [3][64][128]: dQt, dKh, dKb (after the MMAs that read Y)
constexpr uint32_t DG = YB;                  // bf16 [64][128]: the gate's gradient on its way out (after the assembly; not with CONVB)
constexpr uint32_t STG = SB;                 // f32 [3][64][128] staging of dq, dk, dbeta terms over SB and X (after all MMAs)
// fused short-convolution backward (CONVB): once their first users are done, Y holds the pre-convolution q and
// k rows -3 .. 63 (bf16 [67][128] each), and the staging area dq and dk of the convolved rows (bf16, every row in the
// first half of the FP32 row it was made from) and the four blocks' filter-gradient shares
constexpr uint32_t CXQ = YB, CXK = YB + 67 * 256, CTAPS = CXK + 67 * 256;  // CTAPS: f32 [2][128][4] padded filter taps
constexpr uint32_t CDYQ = STG, CDYK = STG + 64 * 128 * 4, CDW = STG + 2 * 64 * 128 * 4;
constexpr int CDS = 256;                     // row stride of dq, dk in elements
static_assert(CTAPS + 2 * 128 * 16 <= YB + 49152, "the projection rows and the taps share the Y buffer");
constexpr uint32_t TMEM_COLS = 512;
// The midpoint factors reach 2^(+-span/2) and the third BF16 part of an operand sits 2^-16 below its
// value, so the whole FP32 exponent range is used up at span ~205: tiles pass on to the tensor cores
// only up to TC_SPAN (the rest of the guard's range, up to 232, is evaluated exactly, which is the
// stricter choice), and every operand is scaled by 2^SHIFT (undone in the read-back factor) to centre
// the range: largest operand 2^(100+6), smallest third part ~2^(-100+6-7-16) > 2^-126.
constexpr float TC_SPAN = 200.f, SHIFT = 6.f;
__host__ __device__ constexpr uint32_t rcol(int J) { return 16u * J * (9 - J); }         // accR_J: 2 (64 - 16 J) columns
__host__ __device__ constexpr uint32_t ccol(int I) { return 320u + 8u * I * (I + 1); }  // accC_I: 16 (I + 1) columns
}  // namespace bi

// Two neighbouring rows of a channel in packed arithmetic: the kernel is bound by instruction issue and the latencies between its
// barriers, and the rows lie side by side in the registers of accumulators, hand-over words and G (with four-wide coefficients for
// rejected tiles and the gate's gradient leaving by tile copy 57 500 -> 43 000 warp instructions a unit; 3072 units 337 -> 302 us,
// 1536 units with three quarters of the tiles rejected 235 -> 206).
__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 ex2_2(float2 x) { return make_float2(ex2_approx(x.x), ex2_approx(x.y)); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, both(-1.f), a); }
__device__ __forceinline__ float2 bf2(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }

// eight operand values of one channel -> three BF16 parts, one 16-byte row of a core matrix each
__device__ __forceinline__ void store_parts(unsigned char* buf, int d, int t0, const float2 (&v)[4]) {
    uint32_t p[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float2 x = v[j];
#pragma unroll
        for (int part = 0; part < 3; ++part) {
            p[part][j] = pack_bf16(x.x, x.y);
            if (part < 2) x = sub2(x, bf2(p[part][j]));
        }
    }
    const uint32_t off = (uint32_t)cm_idx(d, t0, 64) * 2;
#pragma unroll
    for (int part = 0; part < 3; ++part)
        *reinterpret_cast<uint4*>(buf + part * 16384 + off) = make_uint4(p[part][0], p[part][1], p[part][2], p[part][3]);
}

// 512 threads: thread (blk, d) = (tid / 128, tid % 128) owns channel d (= TMEM lane d) of the 16-row
// block blk, so that a warp covers exactly one guard tile, everything along the token axis of a
// block is register-local, and four warps per scheduler hide each other's latencies.
// CONVB: the backward of the short convolutions of q and k runs here too (KdaParams.grad_conv_*): dq, dk of the
// convolved rows stay in shared memory and grad_q, grad_k receive the gradients of the projections.
template <bool CONVB>
__global__ void __launch_bounds__(bi::NTHR, 1) kda_bwd_intra(const KdaParams p, const __grid_constant__ RowMaps maps) {
    const WsLayout L = ws_layout(p.NT, p.H, p.dk, p.dv, p.dtype);
    using namespace bi;
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ uint64_t barA, barB, barH, mma1, mma2, mma3;
    __shared__ uint32_t tmem_s;
    const __nv_bfloat16* sQ = reinterpret_cast<const __nv_bfloat16*>(dyn + SQ);
    const __nv_bfloat16* sK = reinterpret_cast<const __nv_bfloat16*>(dyn + SK);
    float* sG = reinterpret_cast<float*>(dyn + SG);
    const __nv_bfloat16* sB = reinterpret_cast<const __nv_bfloat16*>(dyn + SB);
    float* stg = reinterpret_cast<float*>(dyn + STG);
    const __nv_bfloat16* spf = reinterpret_cast<const __nv_bfloat16*>(dyn + PF);
    float* sdb = reinterpret_cast<float*>(dyn + SDB);
    float* sdiag = reinterpret_cast<float*>(dyn + SDIAG);
    float* smid = reinterpret_cast<float*>(dyn + SMID);
    float* stot = reinterpret_cast<float*>(dyn + STOT);
    float* sscr = reinterpret_cast<float*>(dyn + SSCR);
    float* sred = reinterpret_cast<float*>(dyn + SRED);
    int* srej = reinterpret_cast<int*>(dyn + SREJ);
    float* fD = reinterpret_cast<float*>(dyn + FD);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, d = tid & 127, blk = tid >> 7, cg = warp & 3;
    const int wu = __shfl_sync(0xffffffffu, warp, 0);  // the warp index as a warp-uniform value (MMA issue)
    const int b0 = B * blk;
    char* sc = (char*)p.bwd_scratch;
    const bool l2 = p.flags & KDA_FLAG_QK_L2NORM, gate = p.flags & KDA_FLAG_GATE, sig = p.flags & KDA_FLAG_BETA_SIGMOID;
    const float scale = p.scale;
    KDA_PHASE_BEGIN();
    if (warp == 0) {
        tmem_alloc(&tmem_s, TMEM_COLS);
        tmem_relinquish();
    }
    if (tid == 0) {
        mbar_init(&barA, 1);
        mbar_init(&barB, 1);
        mbar_init(&barH, 1);
        mbar_init(&mma1, 4);  // four issuing threads commit each MMA group (one accumulator block each)
        mbar_init(&mma2, 4);
        mbar_init(&mma3, 4);
        mbar_fence_init();
    }
    pdl_wait();
    tc_fence_before();
    __syncthreads();  // barrier initialisation and the TMEM base address are visible
    tc_fence_after();
    const uint32_t tmem0 = tmem_s;
    const uint32_t tlane = tmem0 + ((uint32_t)(32 * cg) << 16);  // this warp's lane quadrant
    const uint32_t sb = smem_u32(dyn);

    // The CTA walks the units blockIdx.x, blockIdx.x + gridDim.x, ...: tensor memory, barriers and the CTA itself
    // are set up once.  Unit u = (chunk u / H, head (u + chunk) % H), so that the units of one CTA cycle through
    // all heads whatever the stride (heads differ in cost: rejected tiles take the exact path).
    // What the operands are built from: G, the normalised q and k, the row norms and beta kept by the forward.  With the
    // convolution fused, the NEXT unit's are requested as soon as this one is done with them, before the convolution's
    // backward (12288 units: 1530 us; requested before the row stage, with its rows in registers, 1567).
    constexpr bool AHEAD = CONVB;
    auto request_A = [&](size_t r, bool second) {
        const char* ws = (const char*)p.workspace;
        if (tid != 0) return;
        mbar_expect_tx(&barA, C * D * 4 + 2 * C * D * 2 + 3 * C * 4);
        tma_load_1d(dyn + SG, (const float*)(ws + L.Gc) + r * C * D, C * D * 4, &barA);
        tma_load_1d(dyn + SQ, (const __nv_bfloat16*)(ws + L.Qn) + r * C * D, C * D * 2, &barA);
        tma_load_1d(dyn + SK, (const __nv_bfloat16*)(ws + L.Kn) + r * C * D, C * D * 2, &barA);
        tma_load_1d(dyn + (second ? SAUX2 : SAUX), (const float*)(ws + L.aux) + r * 3 * C, 3 * C * 4, &barA);
    };
    const int n_units = p.NT * p.H;
    bool ok = true, ahead = false;
    uint32_t it = 0;
    UnitWalk uw;
    uw.init(blockIdx.x, gridDim.x, p.H);
    for (; uw.unit < n_units; uw.next(), ++it) {
    const uint32_t par = it & 1;
    const float* srq = reinterpret_cast<const float*>(dyn + (AHEAD && par ? SAUX2 : SAUX));  // aux record order: 1/|q|, 1/|k|, beta
    const float* srk = srq + 64;
    const float* sbeta = srq + 128;
    ahead = false;
    const int c = uw.c, hd = uw.head();
    const ChunkInfo ci = chunk_info(p, c);
    const size_t rec = (size_t)c * p.H + hd;
    const float expA = gate ? expf(p.A_log[hd]) : 1.f;  // requested at the start of the unit: used only in the gate chain at the end
    auto tok = [&](int i) { return ((size_t)(ci.tok0 + i) * p.H + hd); };
    // ---- everything the kernel reads arrives by bulk TMA: on barA what the operands are built from
    //      (G, the normalised q and k, the row norms and beta kept by the forward), on barB the split
    //      dAqk / dM tiles and the diagonal of dAqk from bwd_wy; the three [64][128] hand-over arrays
    //      that only the assembly needs follow on barH once an operand buffer is free
    if (!AHEAD || it == 0) request_A(rec, false);
    if (tid == 0) {
        mbar_expect_tx(&barB, 6 * C * C * 2 + C * 4);
        tma_load_1d(dyn + SB, (const __nv_bfloat16*)(sc + L.dAM) + rec * 6 * C * C, 6 * C * C * 2, &barB);
        tma_load_1d(sdiag, (const float*)(sc + L.dAd) + rec * C, C * 4, &barB);
        // (the hand-over arrays follow half a unit later: the hint hides their way from DRAM, 308 -> 303 us at 3072 units; from the
        //  middle of the unit, or for the next unit's dA and dM, hints cost as much as they give)
        l2_prefetch_bulk((const __nv_bfloat16*)(sc + L.dQt) + rec * C * D, C * D * 2);
        l2_prefetch_bulk((const __nv_bfloat16*)(sc + L.dKh) + rec * C * D, C * D * 2);
        l2_prefetch_bulk((const __nv_bfloat16*)(sc + L.dKb) + rec * C * D, C * D * 2);
    }
    if (tid < C) sdb[tid] = ((const float*)(sc + L.dbp))[rec * C + tid];
    const float carry_in = ((const float*)(sc + L.gC))[rec * D + d];
    ok = mbar_wait(&barA, par, p, 64);
    KDA_PHASE(0);

    // ---- my block: G of my channel, guard and references; operand step 1: KN_j = k_j 2^(ref - G_j) -> X
    float mid;
    float2 G2[B / 2];  // rows 2 i, 2 i + 1
    bool pass;
    {
        float G[B];
#pragma unroll
        for (int r = 0; r < B; ++r) G[r] = sG[swz_f32(b0 + r, d)];
        pass = guard_tile(G, fminf(p.guard_span, TC_SPAN), mid);
#pragma unroll
        for (int r = 0; r < B; r += 2) G2[r / 2] = make_float2(G[r], G[r + 1]);
    }
    auto k2 = [&](int i) { return make_float2(__bfloat162float(sK[swz_bf16(b0 + 2 * i, d)]), __bfloat162float(sK[swz_bf16(b0 + 2 * i + 1, d)])); };
    auto q2 = [&](int i) { return make_float2(__bfloat162float(sQ[swz_bf16(b0 + 2 * i, d)]), __bfloat162float(sQ[swz_bf16(b0 + 2 * i + 1, d)])); };
    auto beta2 = [&](int i) { return *reinterpret_cast<const float2*>(sbeta + b0 + 2 * i); };
    const float gl = sG[swz_f32(C - 1, d)];                          // G of the chunk's last row
    const float gprev = blk > 0 ? sG[swz_f32(b0 - 1, d)] : 0.f;      // G of the row before my block
    {
        // references of my rows as keys / as queries: the midpoint, or first rows when there is none
        // (block 3 has no later rows: zero keys)
        const float kref = pass ? mid : (blk < 3 ? sG[swz_f32(b0 + B, d)] : -INFINITY), qref = pass ? mid : G2[0].x;
        smid[blk * D + d] = kref;
        smid[(4 + blk) * D + d] = qref;
        if (lane == 0) srej[blk * 4 + cg] = pass ? 0 : 1;
#pragma unroll
        for (int g8 = 0; g8 < 2; ++g8) {
            float2 v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = __fmul2_rn(k2(4 * g8 + j), ex2_2(sub2(both(kref + SHIFT), G2[4 * g8 + j])));
            store_parts(dyn + XB, d, b0 + 8 * g8, v);
        }
    }
    if constexpr (!CONVB) tma_store_wait_read();
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    ok = ok && mbar_wait(&barB, par, p, 64);
    KDA_PHASE(1);
    constexpr int PA[6] = {0, 0, 1, 1, 0, 2}, PB[6] = {0, 1, 0, 1, 2, 0};
    // (descriptors: one base per buffer, the tile / part / block offset is added to its 14-bit address field)
    const uint64_t dX = make_desc(sb + XB, 128, 1024), dY = make_desc(sb + YB, 128, 1024);
    const uint64_t dBk = make_desc(sb + SB, 128, 1024), dBm = make_desc(sb + SB, 1024, 128);
    // An elected lane of warp J issues the MMAs of accumulator block J: the blocks are independent, and no warp
    // falls a whole issue sequence behind the others.
    if (wu < 4 && elect_one() && ok) {  // row side: accR_J = KN_J^T dA[i >= 16 J, J]^T (and dM), six passes each
        tc_fence_after();
#pragma unroll
        for (int J = 0; J < 4; ++J)
            if (J == wu) {
                const int N = 64 - B * J;
                const uint32_t id = make_idesc(128, N, false, false);
#pragma unroll
                for (int mat = 0; mat < 2; ++mat)
#pragma unroll
                    for (int ps = 0; ps < 6; ++ps)
                        mma_ss(tmem0 + rcol(J) + mat * N, dX + ((PA[ps] * 16384 + 256 * J) >> 4),
                               dBk + (((mat * 3 + PB[ps]) * 8192 + 2304 * J) >> 4), id, ps > 0);
            }
        mma_commit(&mma1);
    }
    // references of all four blocks for my channel, guard decisions for my channel group
    float kr4[4], qr4[4];
    bool any_rej = false;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        kr4[b] = smid[b * D + d];
        qr4[b] = smid[(4 + b) * D + d];
    }
#pragma unroll
    for (int b = 0; b < 16; ++b) any_rej = any_rej || srej[b] != 0;
    // ---- operand step 2: QP_i = scale q_i 2^(G_i - ref) -> Y (which the last unit's gate gradient has left: the threads that issued
    //      its copies wait for that before the barrier above)
    {
        const float qref = (pass ? mid : G2[0].x) - SHIFT;
#pragma unroll
        for (int g8 = 0; g8 < 2; ++g8) {
            float2 v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                v[j] = __fmul2_rn(__fmul2_rn(both(scale), q2(4 * g8 + j)), ex2_2(__fadd2_rn(G2[4 * g8 + j], both(-qref))));
            store_parts(dyn + YB, d, b0 + 8 * g8, v);
        }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    KDA_PHASE(2);
    if (wu < 4 && elect_one() && ok) {  // column side, first half: accC_I = QP_I^T dA[I, j < 16 (I+1)]
        tc_fence_after();
#pragma unroll
        for (int I = 0; I < 4; ++I)
            if (I == wu) {
                const uint32_t id = make_idesc(128, B * (I + 1), false, true);
#pragma unroll
                for (int ps = 0; ps < 6; ++ps)
                    mma_ss(tmem0 + ccol(I), dY + ((PA[ps] * 16384 + 256 * I) >> 4), dBm + ((PB[ps] * 8192 + 2048 * I) >> 4), id, ps > 0);
            }
        mma_commit(&mma2);
    }
    // ---- operand step 3: KP_i = beta_i k_i 2^(G_i - ref) -> X, once the row-side MMAs have read X
    ok = ok && mbar_wait(&mma1, par, p, 64);
    tc_fence_after();
    {
        const float qref = (pass ? mid : G2[0].x) - SHIFT;
#pragma unroll
        for (int g8 = 0; g8 < 2; ++g8) {
            float2 v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                v[j] = __fmul2_rn(__fmul2_rn(beta2(4 * g8 + j), k2(4 * g8 + j)), ex2_2(__fadd2_rn(G2[4 * g8 + j], both(-qref))));
            store_parts(dyn + XB, d, b0 + 8 * g8, v);
        }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    KDA_PHASE(3);
    if (wu < 4 && elect_one() && ok) {  // column side, second half: accC_I += KP_I^T dM[I, j < 16 (I+1)]
        tc_fence_after();
#pragma unroll
        for (int I = 0; I < 4; ++I)
            if (I == wu) {
                const uint32_t id = make_idesc(128, B * (I + 1), false, true);
#pragma unroll
                for (int ps = 0; ps < 6; ++ps)
                    mma_ss(tmem0 + ccol(I), dX + ((PA[ps] * 16384 + 256 * I) >> 4), dBm + (((3 + PB[ps]) * 8192 + 2048 * I) >> 4), id, true);
            }
        mma_commit(&mma3);
    }
    // ---- row sums of my block from the accumulators while the column-side MMAs run (the pairs inside my
    //      own block only if its tile passed the guard)
    float2 a1[B / 2], a2[B / 2], c1[B / 2];
#pragma unroll
    for (int i = 0; i < B / 2; ++i) a1[i] = a2[i] = c1[i] = both(0.f);
    auto pair = [](const uint32_t (&r)[16], int i) { return make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])); };
    if (ok) {
#pragma unroll
        for (int J = 0; J < 4; ++J)
            if (J < blk || (J == blk && pass)) {
                uint32_t ra[16], rm[16];
                const uint32_t col = tlane + rcol(J) + B * (blk - J);
                tmem_ld16(col, ra);
                tmem_ld16(col + 64 - B * J, rm);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < B / 2; ++i) {
                    const float2 f = ex2_2(__fadd2_rn(G2[i], both(-kr4[J] - SHIFT)));
                    a1[i] = __ffma2_rn(f, pair(ra, i), a1[i]);
                    a2[i] = __ffma2_rn(f, pair(rm, i), a2[i]);
                }
            }
    }
    KDA_PHASE(4);
    // ---- the hand-over arrays may land in Y as soon as the MMAs that read Y are done
    ok = ok && mbar_wait(&mma2, par, p, 64);
    if (tid == 0 && ok) {
        mbar_expect_tx(&barH, 3 * C * D * 2);
        tma_load_1d(dyn + PF, (const __nv_bfloat16*)(sc + L.dQt) + rec * C * D, C * D * 2, &barH);
        tma_load_1d(dyn + PF + C * D * 2, (const __nv_bfloat16*)(sc + L.dKh) + rec * C * D, C * D * 2, &barH);
        tma_load_1d(dyn + PF + 2 * C * D * 2, (const __nv_bfloat16*)(sc + L.dKb) + rec * C * D, C * D * 2, &barH);
    }
    // The next unit of this CTA finds what it needs first in L2: the hints go out here, in the middle of the unit,
    // when the copy unit has nothing else to do (there is no shared memory left to receive the records themselves).
    if (tid == 5 * 32) {
        UnitWalk un = uw;  // the next unit of this CTA
        un.next();
        if (un.unit < n_units) {
            const char* ws = (const char*)p.workspace;
            const size_t rn = un.rec();
            l2_prefetch_bulk((const float*)(ws + L.Gc) + rn * C * D, C * D * 4);
            l2_prefetch_bulk((const __nv_bfloat16*)(ws + L.Kn) + rn * C * D, C * D * 2);
            l2_prefetch_bulk((const __nv_bfloat16*)(ws + L.Qn) + rn * C * D, C * D * 2);
        }
    }
    ok = ok && mbar_wait(&mma3, par, p, 64);
    tc_fence_after();
    KDA_PHASE(5);
    // ---- column sums of my block
    if (ok) {
#pragma unroll
        for (int Ip = 0; Ip < 4; ++Ip)
            if (Ip > blk || (Ip == blk && pass)) {
                uint32_t rc[16];
                tmem_ld16(tlane + ccol(Ip) + b0, rc);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < B / 2; ++i) c1[i] = __ffma2_rn(ex2_2(sub2(both(qr4[Ip] - SHIFT), G2[i])), pair(rc, i), c1[i]);
            }
    }
    KDA_PHASE(6);
    if (any_rej) {  // uniform over the CTA: the diagonal blocks back to FP32 (x = p0 + p1 + p2) for the CUDA-core sums
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = tid + NTHR * u, mat = e >> 10, bb = (e >> 8) & 3, j = (e >> 4) & 15, r = e & 15;
            const __nv_bfloat16* t = sB + mat * 3 * C * C + cm_idx(B * bb + r, B * bb + j, C);
            fD[e] = (__bfloat162float(t[0]) + __bfloat162float(t[C * C])) + __bfloat162float(t[2 * C * C]);
        }
    }
    ok = ok && mbar_wait(&barH, par, p, 64);
    ok = __syncthreads_and(ok);  // (also: the rebuilt blocks are visible; the split tiles and X are dead -> staging area)
    KDA_PHASE(7);

    if (ok) {
        // ---- my tile was rejected: the pairs inside the block in FP32 on the CUDA cores, one exp2 per pair.
        //      Pair (r, j), j < r, feeds the row sums of r and the column sum of j with the same decay
        //      2^(G_r - G_j).  The key row j is the rolled loop (two segments, so that half of the unrolled rows
        //      above the diagonal are not masked off but left out); its column sum goes through my
        //      own column of the G tile, which nobody else reads any more.
        if (!pass) {
            const float* dA = fD + blk * B * B;
            const float* dM = fD + (4 + blk) * B * B;
            float2 qs[B / 2], kb[B / 2];
#pragma unroll
            for (int i = 0; i < B / 2; ++i) {
                qs[i] = __fmul2_rn(both(scale), q2(i));
                kb[i] = __fmul2_rn(beta2(i), k2(i));
            }
            // keys R0 .. R0 + 7 against the rows from R0 on (dA, dM are zero on and above the diagonal; two segments, because four
            // spill: 1580 against 1530 us with the convolution, 12288 units)
            auto segment = [&](auto r0c) {
                constexpr int R0 = decltype(r0c)::value;
#pragma unroll 1
                for (int j = R0; j < R0 + 8; ++j) {
                    const float kj = __bfloat162float(sK[swz_bf16(b0 + j, d)]), gj = sG[swz_f32(b0 + j, d)];
                    float2 cj = both(0.f);
#pragma unroll
                    for (int r = R0; r < B; r += 4) {
                        const float4 a4 = *reinterpret_cast<const float4*>(dA + j * B + r), m4 = *reinterpret_cast<const float4*>(dM + j * B + r);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int i = r / 2 + h;
                            const float2 a = h ? make_float2(a4.z, a4.w) : make_float2(a4.x, a4.y), m = h ? make_float2(m4.z, m4.w) : make_float2(m4.x, m4.y);
                            float2 e = ex2_2(__fadd2_rn(G2[i], both(-gj)));
                            if (r < R0 + 8) e = make_float2(2 * i > j ? e.x : 0.f, 2 * i + 1 > j ? e.y : 0.f);  // (rows before the key may overflow)
                            const float2 kp = __fmul2_rn(both(kj), e);
                            a1[i] = __ffma2_rn(a, kp, a1[i]);
                            a2[i] = __ffma2_rn(m, kp, a2[i]);
                            cj = __ffma2_rn(__ffma2_rn(a, qs[i], __fmul2_rn(m, kb[i])), e, cj);
                        }
                    }
                    sG[swz_f32(b0 + j, d)] = cj.x + cj.y;
                }
            };
            segment(std::integral_constant<int, 0>{});
            segment(std::integral_constant<int, 8>{});
#pragma unroll
            for (int i = 0; i < B / 2; ++i) c1[i] = __fadd2_rn(c1[i], make_float2(sG[swz_f32(b0 + 2 * i, d)], i < 7 ? sG[swz_f32(b0 + 2 * i + 1, d)] : 0.f));
        }
        KDA_PHASE(8);
        // ---- assembly of my block, last row first; a1 is reused for the running sum of dG
        {
            float acc = 0.f, tail = 0.f;
            // my 16 rows of the three hand-over arrays (channel-major, handover_idx): eight rows = one 16-byte word
#pragma unroll
            for (int hf = 1; hf >= 0; --hf) {
                const int o = handover_idx(b0 + 8 * hf, d);
                const uint4 uq = *reinterpret_cast<const uint4*>(spf + o), ukh = *reinterpret_cast<const uint4*>(spf + C * D + o),
                            ukb = *reinterpret_cast<const uint4*>(spf + 2 * C * D + o);
                const uint32_t hq[4] = {uq.x, uq.y, uq.z, uq.w}, hkh[4] = {ukh.x, ukh.y, ukh.z, ukh.w}, hkb[4] = {ukb.x, ukb.y, ukb.z, ukb.w};
#pragma unroll
                for (int r2 = 3; r2 >= 0; --r2) {
                    const int i = 4 * hf + r2, ii = b0 + 2 * i;
                    const float2 qi = q2(i), ki = k2(i), be = beta2(i), dg = __fmul2_rn(both(scale), *reinterpret_cast<const float2*>(sdiag + ii));
                    const float2 gam = ex2_2(G2[i]), he = __fmul2_rn(bf2(hkh[r2]), ex2_2(sub2(both(gl), G2[i])));  // dKh 2^(G_last - G)
                    const float2 kg = __fmul2_rn(bf2(hkb[r2]), gam);                                               // d(beta K~) 2^G
                    const float2 rq = __fmul2_rn(both(scale), __ffma2_rn(bf2(hq[r2]), gam, a1[i]));                 // row side of dq
                    const float2 am = __fadd2_rn(a2[i], kg), rk = __fmul2_rn(be, am), cs = __fadd2_rn(c1[i], he);   // row side of dk, the rest
                    const float2 dq = __ffma2_rn(dg, ki, rq), dk = __fadd2_rn(__ffma2_rn(dg, qi, rk), cs), db = __fmul2_rn(ki, am);
                    const float2 khe = __fmul2_rn(ki, he);  // the last row also collects sum_i dKh_i Kh_i
                    const float2 term = __ffma2_rn(qi, rq, __fmul2_rn(ki, sub2(rk, cs)));
                    stg[(0 * C + ii) * D + d] = dq.x;
                    stg[(0 * C + ii + 1) * D + d] = dq.y;
                    stg[(1 * C + ii) * D + d] = dk.x;
                    stg[(1 * C + ii + 1) * D + d] = dk.y;
                    stg[(2 * C + ii) * D + d] = db.x;
                    stg[(2 * C + ii + 1) * D + d] = db.y;
                    tail += khe.x + khe.y;
                    a1[i].y = acc + term.y;
                    acc = a1[i].y + term.x;
                    a1[i].x = acc;
                }
            }
            stot[blk * D + d] = acc;
            sscr[blk * D + d] = tail;
        }
        KDA_PHASE(9);
        const int c4 = (tid & 15) * 4;
        __syncthreads();
        KDA_PHASE(10);
        if constexpr (CONVB) {  // the hand-over arrays in Y are dead: fetch the projection rows the convolution backward needs
            const __nv_bfloat16* xq = (const __nv_bfloat16*)p.q;
            const __nv_bfloat16* xk = (const __nv_bfloat16*)p.k;
            __nv_bfloat16* sxq = reinterpret_cast<__nv_bfloat16*>(dyn + CXQ);
            __nv_bfloat16* sxk = reinterpret_cast<__nv_bfloat16*>(dyn + CXK);
            for (int qq = tid; qq < 67 * (D / 8); qq += NTHR) {
                const int r = qq >> 4, e8 = (qq & 15) * 8;
                const bool valid = r >= 3 ? r - 3 < ci.len : ci.lc > 0;
                const size_t src = ((size_t)(ci.tok0 + (valid ? r - 3 : 0)) * p.H + hd) * D + e8;
                cp_async16_z(sxq + r * D + e8, xq + src, valid);
                cp_async16_z(sxk + r * D + e8, xk + src, valid);
            }
            // (the filter taps of this head travel with them: thread t < 256 fetches tensor t / 128, channel t % 128)
            if (tid < 2 * D) stage_taps(reinterpret_cast<float4*>(dyn + CTAPS) + tid, tid < D ? p.conv_q : p.conv_k, hd, tid & (D - 1), p.conv_ksize);
            cp_async_commit();
        }
        // ---- reverse cumulative sum across the blocks and the gate chain
        float dA_acc = 0.f, dbias_acc = 0.f;
        {
            float base = carry_in + ((sscr[d] + sscr[D + d]) + (sscr[2 * D + d] + sscr[3 * D + d]));
#pragma unroll
            for (int b = 1; b < 4; ++b)
                if (b > blk) base += stot[b * D + d];
            const float negA = -expA, arg = LOG2E / expA;
            float2 dA2 = both(0.f), dbias2 = both(0.f);
            // (rows past the end of a partial chunk have a constant G, hence a zero decay and zero terms:
            //  only their stores are masked, so that the rows do not end up in sixteen basic blocks)
            __nv_bfloat16* dgp = (__nv_bfloat16*)p.grad_g + tok(b0) * D + d;
            __nv_bfloat16* sdg = reinterpret_cast<__nv_bfloat16*>(dyn + DG) + b0 * D + d;
            const size_t rstride = (size_t)p.H * D;
#pragma unroll
            for (int i = B / 2 - 1; i >= 0; --i) {
                const float2 run = __fadd2_rn(both(base), a1[i]);
                float2 outv = run;
                if (gate) {
                    // per-token log decay g = (G_i - G_{i-1}) ln 2; sigmoid(x + b) = 1 - exp(-softplus) = -expm1(g / e^A)
                    const float2 gnat = __fmul2_rn(sub2(G2[i], make_float2(i > 0 ? G2[i > 0 ? i - 1 : 0].y : gprev, G2[i].x)), both(0.6931471805599453f));
                    dA2 = __ffma2_rn(run, gnat, dA2);
                    outv = __fmul2_rn(__fmul2_rn(run, both(negA)), sub2(both(1.f), ex2_2(__fmul2_rn(gnat, both(arg)))));
                    dbias2 = __fadd2_rn(dbias2, outv);
                }
                if constexpr (!CONVB) {
                    sdg[2 * i * D] = __float2bfloat16_rn(outv.x);
                    sdg[(2 * i + 1) * D] = __float2bfloat16_rn(outv.y);
                } else {
                    if (b0 + 2 * i < ci.len) dgp[2 * i * rstride] = __float2bfloat16_rn(outv.x);
                    if (b0 + 2 * i + 1 < ci.len) dgp[(2 * i + 1) * rstride] = __float2bfloat16_rn(outv.y);
                }
            }
            dA_acc = dA2.x + dA2.y;
            dbias_acc = dbias2.x + dbias2.y;
        }
        if constexpr (!CONVB) {  // (one copy of the tile; sixteen 2-byte stores per thread took 0.6 us longer)
            fence_async_smem();
            __syncthreads();
            if (maps.ok && ci.len == C) {
                if (tid == NTHR - 32) tma_store_tile(&maps.m[0], hd * D, (int)ci.tok0, dyn + DG);
            } else if (tid >= NTHR - C && tid - (NTHR - C) < ci.len) {
                tma_store_1d((__nv_bfloat16*)p.grad_g + tok(tid - (NTHR - C)) * D, dyn + DG + (tid - (NTHR - C)) * D * 2, D * 2);
            }
            tma_store_commit();
        }
        KDA_PHASE(11);
        // ---- row-wise (one half warp per row, 64 rows): L2-norm chain, beta gradient.  Lane l of the half
        //      warp owns channels 4l .. 4l+3 and 64+4l .. 64+4l+3, so that its 16-byte staging loads and
        //      8-byte q / k loads are contiguous over the half warp (no bank conflicts)
        {
            __nv_bfloat16* dq_out = (__nv_bfloat16*)p.grad_q;
            __nv_bfloat16* dk_out = (__nv_bfloat16*)p.grad_k;
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const int ii = (tid >> 4) + 32 * m;
                float dq8[8], dk8[8], q8[8], k8[8], db = 0.f, dotq = 0.f, dotk = 0.f;
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    const int ch = 64 * hf + c4;
                    const float4 a = *reinterpret_cast<const float4*>(stg + (0 * C + ii) * D + ch);
                    const float4 b = *reinterpret_cast<const float4*>(stg + (1 * C + ii) * D + ch);
                    const float4 e = *reinterpret_cast<const float4*>(stg + (2 * C + ii) * D + ch);
                    const uint2 qu = *reinterpret_cast<const uint2*>(sQ + swz_bf16(ii, ch));
                    const uint2 ku = *reinterpret_cast<const uint2*>(sK + swz_bf16(ii, ch));
                    const float2 q01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&qu.x));
                    const float2 q23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&qu.y));
                    const float2 k01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ku.x));
                    const float2 k23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ku.y));
                    dq8[4 * hf] = a.x; dq8[4 * hf + 1] = a.y; dq8[4 * hf + 2] = a.z; dq8[4 * hf + 3] = a.w;
                    dk8[4 * hf] = b.x; dk8[4 * hf + 1] = b.y; dk8[4 * hf + 2] = b.z; dk8[4 * hf + 3] = b.w;
                    q8[4 * hf] = q01.x; q8[4 * hf + 1] = q01.y; q8[4 * hf + 2] = q23.x; q8[4 * hf + 3] = q23.y;
                    k8[4 * hf] = k01.x; k8[4 * hf + 1] = k01.y; k8[4 * hf + 2] = k23.x; k8[4 * hf + 3] = k23.y;
                    db += (e.x + e.y) + (e.z + e.w);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    dotq = fmaf(q8[j], dq8[j], dotq);
                    dotk = fmaf(k8[j], dk8[j], dotk);
                }
                db = half_warp_sum(db);
                if (l2) {
                    dotq = half_warp_sum(dotq);
                    dotk = half_warp_sum(dotk);
                    const float rq = srq[ii], rk = srk[ii];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        dq8[j] = (dq8[j] - q8[j] * dotq) * rq;
                        dk8[j] = (dk8[j] - k8[j] * dotk) * rk;
                    }
                }
                if constexpr (CONVB) {  // rows of the convolved tensors' gradients stay on chip (zero past the end)
                    __nv_bfloat16* sdyq = reinterpret_cast<__nv_bfloat16*>(dyn + CDYQ);
                    __nv_bfloat16* sdyk = reinterpret_cast<__nv_bfloat16*>(dyn + CDYK);
                    const bool valid = ii < ci.len;
                    __syncwarp();  // every lane has read its part of the staged rows that are overwritten here
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        *reinterpret_cast<uint2*>(sdyq + ii * CDS + 64 * hf + c4) =
                            valid ? make_uint2(pack_bf16(dq8[4 * hf], dq8[4 * hf + 1]), pack_bf16(dq8[4 * hf + 2], dq8[4 * hf + 3]))
                                  : make_uint2(0u, 0u);
                        *reinterpret_cast<uint2*>(sdyk + ii * CDS + 64 * hf + c4) =
                            valid ? make_uint2(pack_bf16(dk8[4 * hf], dk8[4 * hf + 1]), pack_bf16(dk8[4 * hf + 2], dk8[4 * hf + 3]))
                                  : make_uint2(0u, 0u);
                    }
                }
                if (ii < ci.len) {
                    const size_t row = tok(ii);
                    if constexpr (!CONVB) {
#pragma unroll
                        for (int hf = 0; hf < 2; ++hf) {
                            *reinterpret_cast<uint2*>(dq_out + row * D + 64 * hf + c4) =
                                make_uint2(pack_bf16(dq8[4 * hf], dq8[4 * hf + 1]), pack_bf16(dq8[4 * hf + 2], dq8[4 * hf + 3]));
                            *reinterpret_cast<uint2*>(dk_out + row * D + 64 * hf + c4) =
                                make_uint2(pack_bf16(dk8[4 * hf], dk8[4 * hf + 1]), pack_bf16(dk8[4 * hf + 2], dk8[4 * hf + 3]));
                        }
                    }
                    if ((tid & 15) == 0) {
                        float b = sbeta[ii], v = sdb[ii] + db;
                        if (sig) v *= b * (1.f - b);
                        ((__nv_bfloat16*)p.grad_beta)[row] = __float2bfloat16_rn(v);
                    }
                }
            }
        }
        KDA_PHASE(12);
        if constexpr (CONVB) {
            // ---- backward of the short convolutions of q and k: thread (channel, 16-row block) walks its rows of both
            //      tensors; dx replaces dy in shared memory and leaves in whole rows
            cp_async_wait<0>();
            fence_async_smem();
            __syncthreads();  // the projection rows have landed, dq / dk of the convolved rows are complete; G, q^ and k^ are dead
            UnitWalk un = uw;
            un.next();
            ahead = un.unit < n_units;
            if (ahead) request_A(un.rec(), par == 0);
            const __nv_bfloat16* sxq = reinterpret_cast<const __nv_bfloat16*>(dyn + CXQ);
            const __nv_bfloat16* sxk = reinterpret_cast<const __nv_bfloat16*>(dyn + CXK);
            __nv_bfloat16* sdyq = reinterpret_cast<__nv_bfloat16*>(dyn + CDYQ);
            __nv_bfloat16* sdyk = reinterpret_cast<__nv_bfloat16*>(dyn + CDYK);
            float* sdw = reinterpret_cast<float*>(dyn + CDW);  // [2][4][128][4]
            int c0s, ncs;
            seq_chunks(p, ci.seq, c0s, ncs);
            const bool has_next = ci.lc + 1 < ncs;
            float wq[4], wk[4], dwq[4] = {0.f, 0.f, 0.f, 0.f}, dwk[4] = {0.f, 0.f, 0.f, 0.f};
            uint32_t oq[8], ok_[8];
            {
                const float4 tq = reinterpret_cast<const float4*>(dyn + CTAPS)[d], tk = reinterpret_cast<const float4*>(dyn + CTAPS)[D + d];
                wq[0] = tq.x; wq[1] = tq.y; wq[2] = tq.z; wq[3] = tq.w;
                wk[0] = tk.x; wk[1] = tk.y; wk[2] = tk.z; wk[3] = tk.w;
            }
            float* cvh = (float*)(sc + L.cv_head) + (rec * 3 * 3) * D;
            float* cvt = (float*)(sc + L.cv_tail) + (rec * 3 * 3) * D;
            auto walk = [&](const __nv_bfloat16* sx, const __nv_bfloat16* sdy, const float(&w)[4], int tensor, float(&dw)[4], uint32_t(&o)[8]) {
                float out[16];
                conv_bwd_block<CDS>(sx, sx + 3 * D, sdy, w, d, blk, cvh + tensor * 3 * D, cvt + tensor * 3 * D, dw, out);
#pragma unroll
                for (int r = 0; r < 8; ++r) o[r] = pack_bf16(out[2 * r], out[2 * r + 1]);
            };
            walk(sxq, sdyq, wq, 0, dwq, oq);
            walk(sxk, sdyk, wk, 1, dwk, ok_);
            *reinterpret_cast<float4*>(sdw + (blk * D + d) * 4) = make_float4(dwq[0], dwq[1], dwq[2], dwq[3]);
            *reinterpret_cast<float4*>(sdw + ((4 + blk) * D + d) * 4) = make_float4(dwk[0], dwk[1], dwk[2], dwk[3]);
            __syncthreads();  // every read of dy is done, the filter-gradient shares are visible
#pragma unroll
            for (int r = 0; r < B; ++r) {
                reinterpret_cast<unsigned short*>(sdyq)[(b0 + r) * CDS + d] = (unsigned short)(oq[r / 2] >> (16 * (r & 1)));
                reinterpret_cast<unsigned short*>(sdyk)[(b0 + r) * CDS + d] = (unsigned short)(ok_[r / 2] >> (16 * (r & 1)));
            }
            if (blk < 2) {  // block 0 threads reduce the q filter, block 1 threads the k filter (fixed order)
                const float* src = sdw + (4 * blk * D + d) * 4;
                float4 t = *reinterpret_cast<const float4*>(src);
#pragma unroll
                for (int b = 1; b < 4; ++b) {
                    const float4 u = *reinterpret_cast<const float4*>(src + b * D * 4);
                    t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
                }
                *reinterpret_cast<float4*>((float*)(sc + L.cv_part) + ((rec * 3 + blk) * D + d) * 4) = t;
            }
            __syncthreads();
            const int lim = has_next ? 61 : ci.len;  // rows 61..63 of a chunk with a successor wait for the fix-up
            __nv_bfloat16* dq_o = (__nv_bfloat16*)p.grad_q;
            __nv_bfloat16* dk_o = (__nv_bfloat16*)p.grad_k;
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const int ii = (tid >> 4) + 32 * m, e8 = (tid & 15) * 8;
                if (ii < lim) {
                    const size_t row = tok(ii);
                    *reinterpret_cast<uint4*>(dq_o + row * D + e8) = *reinterpret_cast<const uint4*>(sdyq + ii * CDS + e8);
                    *reinterpret_cast<uint4*>(dk_o + row * D + e8) = *reinterpret_cast<const uint4*>(sdyk + ii * CDS + e8);
                }
            }
        }
        if (gate) {
            fD[blk * D + d] = dbias_acc;  // (the rebuilt diagonal blocks are dead since the assembly: their space is free)
            dA_acc = warp_sum(dA_acc);
            if (lane == 0) sred[warp] = dA_acc;
            __syncthreads();
            if (blk == 0) ((float*)(sc + L.dbias_part))[rec * D + d] = (fD[d] + fD[D + d]) + (fD[2 * D + d] + fD[3 * D + d]);
            if (tid == 0) {
                float t = 0.f;
                for (int w = 0; w < 16; ++w) t += sred[w];
                ((float*)(sc + L.dA_part))[rec] = t;
            }
        }
    }
    KDA_PHASE(13);
    fence_async_smem();  // (the tiles this unit wrote are about to receive the next unit's bulk copies)
    tc_fence_before();
    ok = __syncthreads_and(ok);
    if (!ok) break;  // a wait gave up (recorded in the status word): no further unit is started
    }
    if constexpr (!CONVB) tma_store_wait_all();
    if (!ok && ahead) {  // the next unit's copies are in flight
        mbar_wait(&barA, (it + 1) & 1, p, 64);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem0, TMEM_COLS);
}

// The rows a chunk could not finish (61..63 when it has a successor): dx from dpre of its last three rows and
// of the successor's first three, in the FMA order of conv_bwd_block.  Warp = (chunk, head, tensor), lane = four
// channels.  (One channel per thread and a CTA per chunk was bound by starting CTAs: 2048 chunks x 6 heads, three tensors 47 -> 23 us.)
__global__ void __launch_bounds__(128) conv_bwd_fixup_kernel(const KdaParams p) {
    const int c = blockIdx.x * 4 + (threadIdx.x >> 5), h = blockIdx.y, t = blockIdx.z, ch = (threadIdx.x & 31) * 4;
    pdl_wait();
    if (c >= p.NT) return;
    const ChunkInfo ci = chunk_info(p, c);
    int c0s, ncs;
    seq_chunks(p, ci.seq, c0s, ncs);
    if (ci.lc + 1 >= ncs) return;  // the last chunk of a sequence finished all its rows itself
    const WsLayout L = ws_layout(p.NT, p.H, p.dk, p.dv, p.dtype);
    const char* sc = (const char*)p.bwd_scratch;
    const size_t rec = (size_t)c * p.H + h, nxt = (size_t)(c + 1) * p.H + h;
    const float* tl = (const float*)(sc + L.cv_tail) + ((rec * 3 + t) * 3) * 128 + ch;
    const float* hdp = (const float*)(sc + L.cv_head) + ((nxt * 3 + t) * 3) * 128 + ch;
    float dp[6][4], w[4][4];  // dpre of rows 61 .. 66; taps [channel][tap]
#pragma unroll
    for (int r = 0; r < 6; ++r) {
        const float4 v = *reinterpret_cast<const float4*>(r < 3 ? tl + r * 128 : hdp + (r - 3) * 128);
        dp[r][0] = v.x; dp[r][1] = v.y; dp[r][2] = v.z; dp[r][3] = v.w;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) conv_taps(t == 0 ? p.conv_q : t == 1 ? p.conv_k : p.conv_v, h, ch + j, p.conv_ksize, w[j]);
    __nv_bfloat16* dst = (__nv_bfloat16*)(t == 0 ? p.grad_q : t == 1 ? p.grad_k : p.grad_v) + ((size_t)(ci.tok0 + 61) * p.H + h) * 128 + ch;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        float o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = fmaf(w[j][0], dp[r + 3][j], fmaf(w[j][1], dp[r + 2][j], fmaf(w[j][2], dp[r + 1][j], w[j][3] * dp[r][j])));
        *reinterpret_cast<uint2*>(dst + (size_t)r * p.H * 128) = make_uint2(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]));
    }
}

// Filter gradients: fixed-order sum of the per-chunk shares.  Grid (head, tensor), 8 groups of 128 threads sum
// every 8th chunk, then the 8 group sums are added in order (the scheme of kda_param_reduce).
__global__ void __launch_bounds__(1024) conv_bwd_reduce_kernel(const KdaParams p) {
    constexpr int CH = 16, G = 64;  // channels of a CTA (256 contiguous bytes of a record), groups of chunks
    __shared__ float4 sb[G][CH];
    const WsLayout L = ws_layout(p.NT, p.H, p.dk, p.dv, p.dtype);
    const float4* part = (const float4*)((const char*)p.bwd_scratch + L.cv_part);
    const int h = blockIdx.x, t = blockIdx.y, cl = threadIdx.x % CH, ch = CH * blockIdx.z + cl, grp = threadIdx.x / CH;
    pdl_wait();
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    // (eight loads in flight per thread, added in chunk order: the loop is a chain of round trips otherwise)
    for (int c0 = grp; c0 < p.NT; c0 += G * 8) {
        float4 u[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int c = c0 + G * q;
            u[q] = c < p.NT ? part[(((size_t)c * p.H + h) * 3 + t) * 128 + ch] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) { s.x += u[q].x; s.y += u[q].y; s.z += u[q].z; s.w += u[q].w; }
    }
    sb[grp][cl] = s;
    __syncthreads();
    if (grp == 0) {
        float4 a = sb[0][cl];
        for (int gi = 1; gi < G; ++gi) {
            a.x += sb[gi][cl].x; a.y += sb[gi][cl].y; a.z += sb[gi][cl].z; a.w += sb[gi][cl].w;
        }
        const int K = p.conv_ksize;
        float* dst = (t == 0 ? p.grad_conv_q : t == 1 ? p.grad_conv_k : p.grad_conv_v) + (size_t)(h * 128 + ch) * K;
        const float v4[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j >= 4 - K) dst[j - (4 - K)] = v4[j];
    }
}

cudaError_t launch_bwd_intra(const KdaParams& p, cudaStream_t s) {
    const bool convb = p.grad_conv_q != nullptr;
    auto kern = convb ? kda_bwd_intra<true> : kda_bwd_intra<false>;
    cudaError_t e = allow_smem(kern, (int)bi::TOTAL);
    if (e != cudaSuccess) return e;
    const int units = p.NT * p.H, sms = sm_count();
    RowMaps maps = {};
    maps.ok = !(p.flags & KDA_FLAG_ROW_COPIES) && make_row_map(&maps.m[0], p.grad_g, (long long)p.B * p.T, p.H, C);
    if ((e = launch_dependent(kern, units < sms ? units : sms, bi::NTHR, bi::TOTAL, s, p, maps)) != cudaSuccess) return e;
    if (convb) {
        if ((e = launch_dependent(conv_bwd_fixup_kernel, dim3((p.NT + 3) / 4, p.H, 3), 128, 0, s, p)) != cudaSuccess) return e;
        if ((e = launch_dependent(conv_bwd_reduce_kernel, dim3(p.H, 3, 8), 1024, 0, s, p)) != cudaSuccess) return e;
    }
    return cudaGetLastError();
}


// ---------------------------------------------------------------------------------------
// Stand-alone form of the guarded diagonal tile with the reference's own interface
// (experiments/kda_sm90/guarded_diagonal_oracle.py:57-180): gate, q, k [N,16,32], beta [N,16],
// dAqk, dAkk [N,16,16] -> dq, dk, dkt [N,16,32], hits [N].  One warp per tile, one lane per
// channel; same guard (guard_tile) and the same two evaluation rules as kda_bwd_intra.
//   dq[i]  = sum_{j<=i} dAqk[i][j] k[j] 2^(g_i-g_j)       dk[i] = sum_{j<=i} dAkk[i][j] k[j] 2^(g_i-g_j)
//   dkt[i] = sum_{j>=i} (dAqk[i][j] q[j] + dAkk[i][j] beta[j] k[j]) 2^(g_j-g_i)
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(32) kda_diag_tile_kernel(const float* __restrict__ gate, const float* __restrict__ q,
                                                           const float* __restrict__ k, const float* __restrict__ beta,
                                                           const float* __restrict__ dAqk, const float* __restrict__ dAkk,
                                                           float* __restrict__ dq, float* __restrict__ dk,
                                                           float* __restrict__ dkt, int* __restrict__ hits, float limit) {
    const int n = blockIdx.x, ch = threadIdx.x;
    float G[16], Q[16], K[16], Bt[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        G[r] = gate[(n * 16 + r) * 32 + ch];
        Q[r] = q[(n * 16 + r) * 32 + ch];
        K[r] = k[(n * 16 + r) * 32 + ch];
        Bt[r] = beta[n * 16 + r];
    }
    float mid;
    const bool pass = guard_tile(G, limit, mid);
    if (ch == 0) hits[n] = pass ? 1 : 0;
    const float* A = dAqk + n * 256;
    const float* M = dAkk + n * 256;
    float P[16], N[16];
    if (pass) {
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            P[r] = ex2_approx(G[r] - mid);
            N[r] = ex2_approx(mid - G[r]);
        }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        float sq = 0.f, sk = 0.f, st = 0.f;
        if (pass) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (j <= i) {
                    sq = fmaf(A[i * 16 + j], K[j] * N[j], sq);
                    sk = fmaf(M[i * 16 + j], K[j] * N[j], sk);
                }
                if (j >= i) st = fmaf(A[i * 16 + j], Q[j] * P[j], fmaf(M[i * 16 + j], Bt[j] * K[j] * P[j], st));
            }
            sq *= P[i];
            sk *= P[i];
            st *= N[i];
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (j <= i) {
                    const float kp = K[j] * ex2_approx(G[i] - G[j]);
                    sq = fmaf(A[i * 16 + j], kp, sq);
                    sk = fmaf(M[i * 16 + j], kp, sk);
                }
                if (j >= i) st = fmaf(A[i * 16 + j] * Q[j] + M[i * 16 + j] * (Bt[j] * K[j]), ex2_approx(G[j] - G[i]), st);
            }
        }
        dq[(n * 16 + i) * 32 + ch] = sq;
        dk[(n * 16 + i) * 32 + ch] = sk;
        dkt[(n * 16 + i) * 32 + ch] = st;
    }
}

}  // namespace kda

extern "C" int kda_guarded_diagonal_tiles(const float* gate, const float* q, const float* k, const float* beta,
                                          const float* dAqk, const float* dAkk, float* dq, float* dk, float* dkt, int* hits,
                                          int n_tiles, float max_log2_span, void* stream) {
    if (!gate || !q || !k || !beta || !dAqk || !dAkk || !dq || !dk || !dkt || !hits) return KDA_ERR_NULL;
    if (n_tiles <= 0) return KDA_ERR_SHAPE;
    if (!(max_log2_span < 0.f) && !(isfinite(max_log2_span) && max_log2_span < 252.f)) return KDA_ERR_GUARD;
    kda::kda_diag_tile_kernel<<<n_tiles, 32, 0, (cudaStream_t)stream>>>(gate, q, k, beta, dAqk, dAkk, dq, dk, dkt, hits,
                                                                       max_log2_span);
    return cudaGetLastError() == cudaSuccess ? KDA_OK : KDA_ERR_LAUNCH;
}

KDA_PHASE_EXPORT(kda_debug_phases_bwd_intra)
