// Float32 attention on the tensor cores: every operand is the sum of three bf16 parts (split_f32.cuh), a product of
// two operands six tcgen05 products of their parts, small ones first, accumulated in float32 over at most 64 terms in
// tensor memory and then added into float32 registers. Probabilities and score gradients are split the same way in
// registers, so nothing is held or multiplied with less than 24 bits. Parts are of 2^16 times a value (a power of its own for score
// gradients), so that small ones keep all of theirs; where a result leaves the accumulators that is undone.
//
// The CUDA-core kernels (attn_simt.cu) do the same products at the FMA pipe's rate, 128 per clock and SM; six bf16 products for
// each leave 683 per clock. Whole calls (split included), 16 units x L1024, causal: d 64 forward 93 -> 32 us, backward 215 -> 64; d 128, 8
// units: 105 -> 36 and 234 -> 100. What bounds them now: the compute warps (exponentials, splitting of 128 x 64 probabilities) and the
// hand-overs between them and the products. A tile takes, of its MMAs' clocks: forward 1930 of 1536 (d 64), 4160 of 3072 (d 128); backward, a
// query block's 3940 of 2688 and 9300 of 5500 (one pair of tiles, loaded without overlap).
// Errors against float64 (relative 2-norm, CUDA cores -> here): 16 units x L1024 d 64 causal: o 2.1e-7 -> 0.9e-7, dq 3.3e-7 ->
// 2.6e-7, dk 7.8e-7 -> 2.9e-7, dv 7.7e-7 -> 2.2e-7, log-sum-exp 3.2e-8 both; 8 x 777 x 1301 d 80: o 6.5e-7 -> 1.3e-7, dq 7.1e-7 -> 3.2e-7, dk
// 5.7e-7 -> 3.1e-7, dv 5.5e-7 -> 2.7e-7, log-sum-exp 2.9e-8 both.
//
// Common to the kernels: 128 rows of one operand belong to a CTA (a row per tensor-memory lane) and lie in tensor memory as
// the A operand of the score product, tiles of 64 rows of the other operand's planes are streamed by TMA, eight compute
// warps (two warpgroups) own the rows' softmax, two warps issue, one loads.
#include <float.h>
#include <math.h>

#include <initializer_list>

#include "common.cuh"
#include "kernels.cuh"
#include "ptx.cuh"
#include "split_f32.cuh"

namespace ember {

namespace {

using namespace ptx;

constexpr int F32_THREADS = 384;       // warps 0-7 compute, 8 and 10 MMA issue, 9 TMA, 11 allocation
constexpr float LOG2E_T = 1.4426950408889634f;
constexpr int SUB = 64 * 128;          // 64 rows x 128 bytes: one TMA box
constexpr int TN = 64;                 // rows of a streamed tile
constexpr int subs(int hd) { return (hd + 63) / 64; }  // 64-column sub-tiles

enum { WF_Q = 301, WF_K, WF_V, WF_S, WF_P, WF_O, WF_OFREE, WF_KEMPTY, WF_VEMPTY, WB_A, WB_B0, WB_B1, WB_S, WB_P, WB_DP, WB_DS, WB_ACC, WB_FREE, WB_E0, WB_E1, WB_SMEM };

__device__ __forceinline__ float exp_nat(float x) { return ex2(x * LOG2E_T); }

// e^x of the backward, which has no division by the sum for errors common to a row to cancel in: what the product with log2(e) is
// rounded by is put back to first order, 2^(y + r) = 2^y (1 + r ln 2). x log2(e) is finite (kMostScore), and x at most a rounding
// error of a score above 0, since scores come out as the forward's did.
__device__ __forceinline__ f32x2 exp_pair(f32x2 x)
{
    const f32x2 y = mul2(x, pack2(LOG2E_T, LOG2E_T)), neg = mul2(x, pack2(-LOG2E_T, -LOG2E_T));
    // log2(e) = LOG2E_T + 1.925963e-8
    const f32x2 r = fma2(x, pack2(1.925963033500e-8f, 1.925963033500e-8f), fma2(x, pack2(LOG2E_T, LOG2E_T), neg));
    float a, b;
    unpack2(y, a, b);
    const f32x2 v = pack2(ex2(a), ex2(b));
    return fma2(v, mul2(r, pack2(0.69314718f, 0.69314718f)), v);
}

// Row `src` (d columns in memory; null: zeros), columns [col0, col0 + 32 * n32) -> the three parts in tensor memory, part q at
// column taddr + q * plane, or the low part (`low` given) in shared memory: row r of sub-tiles of 128 rows x 64 columns, as TMA would lay them.
__device__ __forceinline__ void row_to_tmem(const float *src, int d, bool vec, int col0, int n32, uint32_t taddr, int plane, uint8_t *low, int r)
{
    for (int h = 0; h < n32; h++) {
        const int c0 = col0 + h * 32;
        float v[32];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int c = c0 + i * 4;
            float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
            if (src) {
                if (vec) {
                    if (c < d) f = *reinterpret_cast<const float4 *>(src + c);
                } else {
                    if (c < d) f.x = src[c];
                    if (c + 1 < d) f.y = src[c + 1];
                    if (c + 2 < d) f.z = src[c + 2];
                    if (c + 3 < d) f.w = src[c + 3];
                }
            }
            v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
        }
        uint32_t a[16], b[16], c[16];
#pragma unroll
        for (int i = 0; i < 16; i++) split_pair(pack2(v[2 * i] * kSplitUp, v[2 * i + 1] * kSplitUp), a[i], b[i], c[i]);
        const uint32_t t = taddr + (uint32_t)(c0 / 2);
        tmem_st_32x32b_x16(t, a);
        tmem_st_32x32b_x16(t + plane, b);
        if (low) {
            uint8_t *row = low + c0 / 64 * (2 * SUB) + r * 128;
#pragma unroll
            for (int i = 0; i < 4; i++)
                *reinterpret_cast<uint4 *>(row + (((c0 % 64 / 8 + i) ^ (r & 7)) << 4)) = make_uint4(c[4 * i], c[4 * i + 1], c[4 * i + 2], c[4 * i + 3]);
        } else {
            tmem_st_32x32b_x16(t + 2 * plane, c);
        }
    }
    if (low) fence_proxy_async();
    tmem_wait_st();
}

// Scores, and the parts of what is made of them, share a region of tensor memory; of a tile's 64 columns each half may belong to
// other threads, so the parts of one may not overwrite scores of the other. 32 values of a part are 16 columns, the A operand of one MMA (16
// values) 8. One accumulator: 64 scores in columns [16, 80) of 96; the parts of half h in [48 h, 48 h + 48). TWO side by side (the first 64
// columns of the contraction, and the others) in 128; the parts of half h in 16 columns each from 32 h, 32 h + 16 and 64 + 32 h.
template <bool TWO>
struct Region {
    static constexpr int COLS = TWO ? 128 : 96, SCORES = TWO ? 0 : 16, HALF = TWO ? 32 : 48, LOW = TWO ? 64 : 32;
    static __device__ __forceinline__ constexpr uint32_t step(int k16) { return (uint32_t)((k16 / 2) * HALF + (k16 % 2) * 8); }
    static __device__ __forceinline__ uint32_t part(uint32_t q) { return q == 2 ? LOW : q * 16; }
};

// 32 values of a row -> their parts in tensor memory, in a half of a region. UP: of 2^16 times the values.
template <typename R, bool UP>
__device__ __forceinline__ void split_to_tmem(const f32x2 *v, uint32_t taddr)
{
    uint32_t a[16], b[16], c[16];
#pragma unroll
    for (int i = 0; i < 16; i++) split_pair(UP ? mul2(v[i], pack2(kSplitUp, kSplitUp)) : v[i], a[i], b[i], c[i]);
    tmem_st_32x32b_x16(taddr, a);
    tmem_st_32x32b_x16(taddr + 16, b);
    tmem_st_32x32b_x16(taddr + R::LOW, c);
}

// 32 neighbouring scores of a row, as pairs. ADD: added to those that are there.
template <bool ADD>
__device__ __forceinline__ void load_scores(uint32_t taddr, f32x2 *s)
{
    uint32_t u[32];
    tmem_ld_32x32b_x32(taddr, u);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const f32x2 x = pack2(__uint_as_float(u[2 * i]), __uint_as_float(u[2 * i + 1]));
        s[i] = ADD ? add2(s[i], x) : x;
    }
}

// A chain of four or (four == 0) two MMAs of 16 contraction steps, A in tensor memory (AO* columns further each) or in shared memory (AO* in
// units of 16 bytes), B BO* further each. Products of parts are short MMAs (64 columns: 32 clocks), so what one costs to issue
// decides: `elected` is taken once per tile and four MMAs make one asm block (an elect.sync and a branch on the
// number of steps for each took 85 clocks an MMA), and the last two are predicated off where two do (a second asm block for that: 4 us
// of the forward's 37 at 16 units x L1024 d 64).
#define EMBER_CHAIN_HEAD "{\n.reg .pred p, q;\n.reg .b64 da, db;\n.reg .b32 t, u;\nsetp.ne.b32 q, %4, 0;\nsetp.ne.b32 p, %5, 0;\n"
#define EMBER_CHAIN_REST "setp.ne.and.b32 q, %13, 0, q;\n"
template <int A1, int A2, int A3, int B1, int B2, int B3>
__device__ __forceinline__ void chain_ts(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t elected, uint32_t acc, uint32_t four)
{
    asm volatile(EMBER_CHAIN_HEAD
                 "mov.b64 db, {%2, %6};\n@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\nsetp.eq.u32 p, 0, 0;\n"
                 "add.u32 t, %2, %10;\nadd.u32 u, %1, %7;\nmov.b64 db, {t, %6};\n@q tcgen05.mma.cta_group::1.kind::f16 [%0], [u], db, %3, p;\n" EMBER_CHAIN_REST
                 "add.u32 t, %2, %11;\nadd.u32 u, %1, %8;\nmov.b64 db, {t, %6};\n@q tcgen05.mma.cta_group::1.kind::f16 [%0], [u], db, %3, p;\n"
                 "add.u32 t, %2, %12;\nadd.u32 u, %1, %9;\nmov.b64 db, {t, %6};\n@q tcgen05.mma.cta_group::1.kind::f16 [%0], [u], db, %3, p;\n}\n"
                 ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"(elected), "r"(acc), "r"(kDescHiSw128), "n"(A1), "n"(A2), "n"(A3), "n"(B1), "n"(B2), "n"(B3), "r"(four) : "memory");
}
template <int A1, int A2, int A3, int B1, int B2, int B3>
__device__ __forceinline__ void chain_ss(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t elected, uint32_t acc, uint32_t four)
{
    asm volatile(EMBER_CHAIN_HEAD
                 "mov.b64 db, {%2, %6};\nmov.b64 da, {%1, %6};\n@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\nsetp.eq.u32 p, 0, 0;\n"
                 "add.u32 t, %2, %10;\nadd.u32 u, %1, %7;\nmov.b64 db, {t, %6};\nmov.b64 da, {u, %6};\n@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n" EMBER_CHAIN_REST
                 "add.u32 t, %2, %11;\nadd.u32 u, %1, %8;\nmov.b64 db, {t, %6};\nmov.b64 da, {u, %6};\n@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n"
                 "add.u32 t, %2, %12;\nadd.u32 u, %1, %9;\nmov.b64 db, {t, %6};\nmov.b64 da, {u, %6};\n@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n}\n"
                 ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"(elected), "r"(acc), "r"(kDescHiSw128), "n"(A1), "n"(A2), "n"(A3), "n"(B1), "n"(B2), "n"(B3), "r"(four) : "memory");
}

// Scores: D (128 x 64) = A * B^T over the 64-column sub-tiles [sub0, sub1) of the contraction, each into 64 columns of its own: an
// accumulator collects no more (128 terms of one sign lost 1.9e-7 of their sum to the truncation, in two accumulators 1.1e-7). B: a
// tile of 64 rows, planes PLANE bytes apart. A: A_TMEM tensor memory, parts HD / 2 columns apart; A_LOW the same, but the low part in
// shared memory at low_smem; A_SMEM all of it in shared memory: 128 rows, planes 2 * PLANE bytes apart, sub-tiles 2 * SUB. The contraction
// stops at the end of the 32 columns that hold the last of d (zeros past d). `mirrored`: the tile is the queries' and A the keys'.
enum AKind { A_TMEM, A_LOW, A_SMEM };
template <int HD, AKind KIND>
__device__ __forceinline__ void mma_scores(uint32_t d, uint32_t a, uint32_t low_smem, uint32_t b_smem, int sub0, int sub1, int ksteps, uint32_t elected, bool mirrored)
{
    constexpr uint32_t IDESC = idesc_bf16_f32(128, TN, 0, 0);
    constexpr int PLANE = subs(HD) * SUB;
    const uint32_t b_lo = desc_lo(b_smem, 16), a_lo = KIND == A_SMEM ? desc_lo(a, 16) : a, low = desc_lo(low_smem, 16);
#pragma unroll 1
    for (int i = 0; i < kSplitProducts; i++) {
        const uint32_t pa = split_part_a(i, mirrored), b = b_lo + split_part_b(i, mirrored) * (PLANE >> 4);
#pragma unroll
        for (int sub = sub0; sub < sub1; sub++) {
            const uint32_t at = d + (sub - sub0) * 64, four = ksteps - sub * 4 > 2, bs = b + ((sub * SUB) >> 4);
            if (KIND == A_SMEM) chain_ss<2, 4, 6, 2, 4, 6>(at, a_lo + pa * ((2 * PLANE) >> 4) + ((sub * 2 * SUB) >> 4), bs, IDESC, elected, i > 0, four);
            else if (KIND == A_LOW && pa == 2) chain_ss<2, 4, 6, 2, 4, 6>(at, low + ((sub * 2 * SUB) >> 4), bs, IDESC, elected, i > 0, four);
            else chain_ts<8, 16, 24, 2, 4, 6>(at, a_lo + pa * (HD / 2) + sub * 32, bs, IDESC, elected, i > 0, four);
        }
    }
}
// Results: D (128 x n) = P (parts in a region of tensor memory, 64 columns of the product) * B (the tile's 64 rows x n columns).
template <int HD, typename R>
__device__ __forceinline__ void mma_results(uint32_t d, uint32_t region, uint32_t b_smem, uint32_t idesc, uint32_t elected)
{
    constexpr int PLANE = subs(HD) * SUB;
    const uint32_t b_lo = desc_lo(b_smem, SUB);
#pragma unroll 1
    for (int i = 0; i < kSplitProducts; i++)
        chain_ts<R::step(1), R::step(2), R::step(3), 128, 256, 384>(d, region + R::part(split_part_a(i)), b_lo + split_part_b(i) * (PLANE >> 4), idesc, elected, i > 0, true);
}

// Loads a 64-row tile's three planes.
template <int HD>
__device__ __forceinline__ void load_planes(uint32_t dst, const CUtensorMap *map, uint32_t bar, int row, int unit, int units)
{
    mbar_arrive_expect_tx(bar, 3 * subs(HD) * SUB);
    for (int pl = 0; pl < 3; pl++)
        for (int s = 0; s < subs(HD); s++) tma_load_3d(dst + (pl * subs(HD) + s) * SUB, map, bar, s * 64, row, pl * units + unit);
}

// Adds a partial result's first n columns (rounded up to 32) into registers: acc = acc * alpha + part.
template <int N32, bool SCALE>
__device__ __forceinline__ void flush(f32x2 (&acc)[N32 * 16], uint32_t taddr, int n, float alpha)
{
    const f32x2 al = pack2(alpha, alpha);
#pragma unroll
    for (int c = 0; c < N32; c++) {
        if (c * 32 < n) {
            uint32_t u[32];
            tmem_ld_32x32b_x32(taddr + c * 32, u);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const f32x2 part = pack2(__uint_as_float(u[2 * i]), __uint_as_float(u[2 * i + 1]));
                acc[c * 16 + i] = SCALE ? fma2(acc[c * 16 + i], al, part) : add2(acc[c * 16 + i], part);
            }
        }
    }
}

template <int N, int M>
__device__ __forceinline__ void store_cols(float *dst, const f32x2 (&v2)[M], float down, float scale, int col0, int d, bool vec, const void *base, size_t bytes,
                                           DeviceStatus *status)
{
    (void)base; (void)bytes; (void)status;
#pragma unroll
    for (int c = 0; c < N; c += 4) {
        float v[4];
        unpack2(v2[c / 2], v[0], v[1]);
        unpack2(v2[c / 2 + 1], v[2], v[3]);
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = v[i] * down * scale;
        if (vec) {
            if (col0 + c < d && EMBER_STORE_OK(dst + col0 + c, base, bytes, 16, status))
                *reinterpret_cast<float4 *>(dst + col0 + c) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (col0 + c + i < d && EMBER_STORE_OK(dst + col0 + c + i, base, bytes, 4, status)) dst[col0 + c + i] = v[i];
        }
    }
}

// ---------------------------------------------------------------- forward
// The two warpgroups take the key tiles in turn, each with its own running maximum, sum and output, which are put together at
// the end: while one forms its probabilities, the tensor core works for the other. Tensor memory: the query rows' parts,
// scores and probabilities for each warpgroup (at 128 columns over one another), and the partial output.
// Two warps issue, one the score products and one the others: beside the compute warps, which evict its few instructions from
// the scheduler's own cache, an issuing warp needs 50 clocks for an MMA that takes 32 (alone 16), and one for both held a tile at 3570 clocks.
template <int HD>
struct F32FwdCfg {
    static constexpr int TILE = 3 * subs(HD) * SUB;  // 24 or 48 KB
    static constexpr int KST = HD == 64 ? 3 : 2, VST = KST;
    static constexpr int OFF_K = 0, OFF_V = KST * TILE, OFF_BAR = OFF_V + VST * TILE;
    static constexpr int USED = OFF_BAR + 256, SMEM = USED + 1024;
    // LATE, HD 64: one score buffer, read out at once, apart from the probabilities, and a partial output for each warpgroup, added up
    // a turn later. Above: scores under the probabilities, one partial output, added up before the next one's product. HD 96: both accumulators
    // of scores side by side. HALVES, HD 128: the two halves of the contraction formed and read one after the other (side by side they
    // fit only with the queries' low part in shared memory, and a product with that, between others, held a tile up for 800 clocks:
    // 1 x 32 x 2048, 87 us against 81; one after the other 8 x 842 d 96 takes 41.6 us, side by side 39.0).
    static constexpr bool LATE = HD == 64, HALVES = HD == 128;
    using R = Region<false>;
    static constexpr int R_STEP = HD == 96 ? 128 : R::COLS, SCORES = HD == 96 ? 0 : R::SCORES;
    static constexpr int T_Q = 0, T_P = 3 * HD / 2 + (LATE ? TN : 0), T_S = LATE ? 3 * HD / 2 : T_P + SCORES, S_STEP = LATE ? 0 : R_STEP;
    static constexpr int T_O = T_P + 2 * R_STEP, O_STEP = LATE ? HD : 0;
    static_assert(T_O + HD + O_STEP <= 512, "");
    enum { B_Q, B_KFULL, B_KEMPTY = B_KFULL + KST, B_VFULL = B_KEMPTY + KST, B_VEMPTY = B_VFULL + VST, B_S = B_VEMPTY + VST, B_P = B_S + 2, B_O = B_P + 2, B_OFREE = B_O + 2, B_SREAD = B_OFREE + 2, NUM_BARS };
    static_assert(8 * NUM_BARS + 8 + 4 * kSplitMaxTensors <= 256, "");
};

struct F32FwdParams {
    const float *q;
    float *out, *lse;
    int lq, lk, d, causal;
    bool vec_q, vec_o;
    float scale;
    SplitGuard guard;
    DeviceStatus *status;
    WorkOrder order;
    int paired;  // items that two CTAs share
};

// PAIR: where query blocks would leave SMs without one, two CTAs share a block's keys and put their results together through one another's shared
// memory (no memory of the call's, no second launch; about 1.7 us).
template <int HD, bool PAIR>
__global__ void __launch_bounds__(F32_THREADS, 1)
    sm100_f32_fwd_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const F32FwdParams p)
{
    using C = F32FwdCfg<HD>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar0 = smem_base + C::OFF_BAR;
    auto BAR = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem_gen + C::OFF_BAR + 8 * C::NUM_BARS);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    int unit, rank;
    // PAIR: the first p.paired items have a cluster each, whose two CTAs share the queries: the first takes the earlier half of their tiles, the
    // second the rest (of one tile: none). Behind them a cluster holds two items that know nothing of each other.
    const bool pair = PAIR && blockIdx.x < 2u * p.paired;
    const unsigned item = !PAIR ? blockIdx.x : pair ? blockIdx.x / 2 : blockIdx.x - p.paired;
    if (PAIR && item >= (unsigned)p.order.units * p.order.blocks) {  // there is an odd number of items
        pdl_wait();
        return;
    }
    work_item(p.order, (int)item, unit, rank);
    const int q0 = (p.order.blocks - 1 - rank) * 128, off = p.lk - p.lq;  // heaviest (latest) causal rows first
    const int tiles = ((p.causal ? min(p.lk, q0 + 128 + off) : p.lk) + TN - 1) / TN;
    const int half = pair ? (int)cluster_ctarank() : 0, first = half * ((tiles + 1) / 2);
    const int n = !pair ? tiles : half ? tiles - first : (tiles + 1) / 2;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        mbar_init(BAR(C::B_Q), 8);
        for (int s = 0; s < C::KST; s++) { mbar_init(BAR(C::B_KFULL + s), 1); mbar_init(BAR(C::B_KEMPTY + s), 1); }
        for (int s = 0; s < C::VST; s++) { mbar_init(BAR(C::B_VFULL + s), 1); mbar_init(BAR(C::B_VEMPTY + s), 1); }
        for (int w = 0; w < 2; w++) {
            mbar_init(BAR(C::B_S + w), 1);
            mbar_init(BAR(C::B_P + w), 4);
            mbar_init(BAR(C::B_O + w), 1);
            mbar_init(BAR(C::B_OFREE + w), 4);
        }
        mbar_init(BAR(C::B_SREAD), 4);
        fence_mbar_init();
    }
    if (warp == 11) {
        tmem_alloc(smem_u32(tmem_slot), 512);
        tmem_relinquish();
    }
    if (warp == 9 && lane == 0) {
        prefetch_tensormap(&tm_k);
        prefetch_tensormap(&tm_v);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    const bool leave = split_out_of_range(p.guard, tmem_slot + 2);
    // The CUDA-core kernel behind this one is let go by the end of a block that leaves: placed while these blocks still hold their shared memory, its
    // own would stand on few SMs (3 units x 411 x 411, d 64, values of 1e6, backward 54 -> 99 us; 20 x 289 x 338, d 32, forward 29 -> 36).
    if (!leave) pdl_launch_dependents();

    if (leave) {
        // the kernel behind this one does the work
    } else if (warp >= 8) {
        reg_dealloc_40();
        if (warp == 9 && lane == 0) {
            // ------------------------------------------------------------ TMA producer
            int k_issued = 0, v_issued = 0;
            for (int j = 0; j < n; j++) {
                const int ks = j % C::KST, vs = j % C::VST;
                if (!mbar_wait(BAR(C::B_KEMPTY + ks), ((j / C::KST) & 1) ^ 1, abort_flag, p.status, WF_KEMPTY)) break;
                load_planes<HD>(smem_base + C::OFF_K + ks * C::TILE, &tm_k, BAR(C::B_KFULL + ks), (first + j) * TN, unit, p.order.units);
                k_issued = j + 1;
                if (!mbar_wait(BAR(C::B_VEMPTY + vs), ((j / C::VST) & 1) ^ 1, abort_flag, p.status, WF_VEMPTY)) break;
                load_planes<HD>(smem_base + C::OFF_V + vs * C::TILE, &tm_v, BAR(C::B_VFULL + vs), (first + j) * TN, unit, p.order.units);
                v_issued = j + 1;
            }
            // do not leave while a copy is still landing in shared memory
            const long long t0 = clock64();
            for (int j = max(0, k_issued - C::KST); j < k_issued; j++)
                while (!mbar_try_wait(BAR(C::B_KFULL + j % C::KST), (j / C::KST) & 1) && clock64() - t0 < kWaitLimitCycles) {}
            for (int j = max(0, v_issued - C::VST); j < v_issued; j++)
                while (!mbar_try_wait(BAR(C::B_VFULL + j % C::VST), (j / C::VST) & 1) && clock64() - t0 < kWaitLimitCycles) {}
        } else if (warp == 8) {
            // ------------------------------------------------------------ score products
            const int ksteps = (p.d + 15) / 16;
            const uint32_t elected = elect_one();
            bool ok = mbar_wait(BAR(C::B_Q), 0, abort_flag, p.status, WF_Q);
            for (int j = 0; j < n && ok; j++) {
                const int w = j & 1;
                ok = ok && mbar_wait(BAR(C::B_KFULL + j % C::KST), (j / C::KST) & 1, abort_flag, p.status, WF_K);
                // the last scores here have been read, or (in the same columns) their probabilities multiplied
                if (C::LATE && j > 0) ok = ok && mbar_wait(BAR(C::B_SREAD), (j - 1) & 1, abort_flag, p.status, WF_P);
                if (!C::LATE && j > 1) ok = ok && mbar_wait(BAR(C::B_O + w), ((j - 2) >> 1) & 1, abort_flag, p.status, WF_P);
                tc_fence_after();
                const uint32_t at = tmem + C::T_S + w * C::S_STEP, k_smem = smem_base + C::OFF_K + (j % C::KST) * C::TILE;
                mma_scores<HD, A_TMEM>(at, tmem + C::T_Q, 0, k_smem, 0, C::HALVES ? 1 : subs(HD), ksteps, elected, false);
                tc_commit_elect(BAR(C::B_S + w));
                if (C::HALVES) {
                    ok = ok && mbar_wait(BAR(C::B_SREAD), j & 1, abort_flag, p.status, WF_P);
                    tc_fence_after();
                    mma_scores<HD, A_TMEM>(at, tmem + C::T_Q, 0, k_smem, 1, 2, ksteps, elected, false);
                    tc_commit_elect(BAR(C::B_S + w));
                }
                tc_commit_elect(BAR(C::B_KEMPTY + j % C::KST));
            }
        } else if (warp == 10) {
            // ------------------------------------------------------------ probabilities x V
            const uint32_t idesc_o = idesc_bf16_f32(128, (p.d + 15) / 16 * 16, 0, 1);
            const uint32_t elected = elect_one();
            bool ok = true;
            for (int j = 0; j < n && ok; j++) {
                const int w = j & 1;
                ok = ok && mbar_wait(BAR(C::B_VFULL + j % C::VST), (j / C::VST) & 1, abort_flag, p.status, WF_V);
                ok = ok && mbar_wait(BAR(C::B_P + w), (j >> 1) & 1, abort_flag, p.status, WF_P);
                // the partial output has been added up (LATE: this warpgroup did so before it wrote its probabilities)
                if (!C::LATE && j > 0) ok = ok && mbar_wait(BAR(C::B_OFREE + (w ^ 1)), ((j - 1) >> 1) & 1, abort_flag, p.status, WF_OFREE);
                tc_fence_after();
                mma_results<HD, typename C::R>(tmem + C::T_O + w * C::O_STEP, tmem + C::T_P + w * C::R_STEP, smem_base + C::OFF_V + (j % C::VST) * C::TILE, idesc_o, elected);
                tc_commit_elect(BAR(C::B_O + w));
                tc_commit_elect(BAR(C::B_VEMPTY + j % C::VST));
            }
        }
    } else {
        // ---------------------------------------------------------------- softmax and output
        reg_alloc_232();
        const int w = warp / 4, r = threadIdx.x % 128, row = q0 + r;
        const uint32_t lane_sel = (uint32_t)((warp % 4) * 32) << 16;
        const float *src = row < p.lq ? p.q + ((size_t)unit * p.lq + row) * p.d : nullptr;
        row_to_tmem(src, p.d, p.vec_q, HD == 64 ? w * 32 : w * 64, HD == 64 || (HD == 96 && w == 1) ? 1 : 2, tmem + lane_sel + C::T_Q, HD / 2, nullptr, r);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR(C::B_Q));

        const uint32_t scores = tmem + lane_sel + C::T_S + w * C::S_STEP, region = tmem + lane_sel + C::T_P + w * C::R_STEP, to = tmem + lane_sel + C::T_O + w * C::O_STEP;
        const int limit_row = p.causal ? min(p.lk - 1, row + off) : p.lk - 1;
        const int limit_tile = p.causal ? min(p.lk - 1, q0 + off) : p.lk - 1;
        const int cols = (p.d + 15) / 16 * 16;
        float m = -INFINITY, l = 0.f, late_alpha = 1.f;
        int late = -1;  // LATE: the tile whose partial output is still to be added, with this factor for what it is added to
        f32x2 o[HD / 2];
#pragma unroll
        for (int i = 0; i < HD / 2; i++) o[i] = 0;
        const f32x2 scale2 = pack2(p.scale * kSplitDown2, p.scale * kSplitDown2), l2e = pack2(LOG2E_T, LOG2E_T);
        bool ok = true;
        for (int j = w; j < n && ok; j += 2) {
            const int k0 = (first + j) * TN;
            ok = ok && mbar_wait(BAR(C::B_S + w), C::HALVES ? 0 : (j >> 1) & 1, abort_flag, p.status, WF_S);
            tc_fence_after();
            f32x2 s[32];
            load_scores<false>(scores, s);
            load_scores<false>(scores + 32, s + 16);
            if (C::LATE || C::HALVES) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR(C::B_SREAD));
            }
            if (C::HALVES) {
                ok = ok && mbar_wait(BAR(C::B_S + w), 1, abort_flag, p.status, WF_S);
                tc_fence_after();
            }
            if (!C::LATE) {  // the other half of the contraction
                load_scores<true>(scores + (C::HALVES ? 0 : 64), s);
                load_scores<true>(scores + (C::HALVES ? 32 : 96), s + 16);
            }
#pragma unroll
            for (int i = 0; i < 32; i++) s[i] = mul2(s[i], scale2);
            if (k0 + TN - 1 > limit_tile) {
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    float x, y;
                    unpack2(s[i], x, y);
                    s[i] = pack2(k0 + 2 * i > limit_row ? -INFINITY : x, k0 + 2 * i + 1 > limit_row ? -INFINITY : y);
                }
            }
            float m4[4] = {m, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < 32; i++) {
                float x, y;
                unpack2(s[i], x, y);
                m4[i & 3] = max3(m4[i & 3], x, y);
            }
            const float m_new = fmaxf(max3(m4[0], m4[1], m4[2]), m4[3]);
            const float ref = m_new == -INFINITY ? 0.f : m_new;  // masked keys alone so far: weights of 0
            const float alpha = exp_nat(m - ref);
            m = m_new;
            const f32x2 ref2 = pack2(ref, ref);
            f32x2 sum[2] = {0, 0};
#pragma unroll
            for (int h = 0; h < 2; h++) {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    float x, y;
                    unpack2(mul2(sub2(s[h * 16 + i], ref2), l2e), x, y);
                    s[h * 16 + i] = pack2(ex2(x), ex2(y));
                    sum[i & 1] = add2(sum[i & 1], s[h * 16 + i]);
                }
                if (C::LATE && h == 0 && late >= 0) {  // before the first probabilities: what they overwrite has been multiplied
                    ok = ok && mbar_wait(BAR(C::B_O + w), (late >> 1) & 1, abort_flag, p.status, WF_O);
                    tc_fence_after();
                    flush<HD / 32, true>(o, to, cols, late_alpha);
                }
                split_to_tmem<typename C::R, true>(s + h * 16, region + h * C::R::HALF);
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR(C::B_P + w));
            {
                float x, y;
                unpack2(add2(sum[0], sum[1]), x, y);
                l = l * alpha + (x + y);
            }
            if (C::LATE) {
                late = j;
                late_alpha = alpha;
            } else {
                ok = ok && mbar_wait(BAR(C::B_O + w), (j >> 1) & 1, abort_flag, p.status, WF_O);
                tc_fence_after();
                flush<HD / 32, true>(o, to, cols, alpha);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR(C::B_OFREE + w));
            }
        }
        if (C::LATE && late >= 0) {
            ok = ok && mbar_wait(BAR(C::B_O + w), (late >> 1) & 1, abort_flag, p.status, WF_O);
            tc_fence_after();
            flush<HD / 32, true>(o, to, cols, late_alpha);
        }
        // ---- the two warpgroups' results: each finishes half of the columns, the other half goes to the other one through shared
        // memory (no copy is in flight any more, and after the barrier no product either)
        constexpr int HALF = HD / 2, ROWB = HALF * 4, SWZ = HD == 96 ? 3 : 7;
        float2 *state = reinterpret_cast<float2 *>(smem_gen);                    // [2][128] maximum and sum
        uint8_t *xo = smem_gen + 2048;                                           // [2][128][HALF]: the half that warpgroup w finishes
        named_bar_sync(1, 256);
        state[w * 128 + r] = make_float2(m, l);
        {
            uint8_t *dst = xo + ((w ^ 1) * 128 + r) * ROWB;
#pragma unroll
            for (int c = 0; c < HALF / 4; c++) {
                const int i = 2 * c;
                const ulonglong2 v = w == 0 ? make_ulonglong2(o[HALF / 2 + i], o[HALF / 2 + i + 1]) : make_ulonglong2(o[i], o[i + 1]);
                *reinterpret_cast<ulonglong2 *>(dst + (((c & ~SWZ) | ((c ^ r) & SWZ)) << 4)) = v;
            }
        }
        named_bar_sync(1, 256);
        const float2 other = state[(w ^ 1) * 128 + r];
        float mm = fmaxf(m, other.x);
        const float ref = pair && mm == -INFINITY ? 0.f : mm;  // the other CTA's keys may be the only ones that a row sees
        const float a_own = exp_nat(m - ref), a_other = exp_nat(other.x - ref);
        float ll = w == 0 ? l * a_own + other.y * a_other : other.y * a_other + l * a_own;
        f32x2 res[HALF / 2];
        {
            const uint8_t *from = xo + (w * 128 + r) * ROWB;
            const f32x2 own2 = pack2(a_own, a_own), other2 = pack2(a_other, a_other);
#pragma unroll
            for (int c = 0; c < HALF / 4; c++) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(from + (((c & ~SWZ) | ((c ^ r) & SWZ)) << 4));
                const int i = 2 * c;
                res[i] = fma2(w == 0 ? o[i] : o[HALF / 2 + i], own2, mul2(v.x, other2));
                res[i + 1] = fma2(w == 0 ? o[i + 1] : o[HALF / 2 + i + 1], own2, mul2(v.y, other2));
            }
        }
        const bool stores = ok && row < p.lq;
        const size_t at = (size_t)unit * p.lq + row, o_bytes = (size_t)p.order.units * p.lq * p.d * 4;
        if (PAIR && pair) {
            // ---- each CTA of the pair finishes half of every thread's columns; what the other one needs, it reads from here
            constexpr int PART = HALF / 2;
            uint8_t *state2 = xo + 2 * 128 * ROWB, *xo2 = state2 + 1024;         // [128] maximum and sum, [PART / 4][256] 16 bytes
            if (w == 0) reinterpret_cast<float2 *>(state2)[r] = make_float2(mm, ll);
#pragma unroll
            for (int c = 0; c < PART / 4; c++) {
                const int i = 2 * c;
                reinterpret_cast<ulonglong2 *>(xo2)[c * 256 + threadIdx.x] = half == 0 ? make_ulonglong2(res[PART / 2 + i], res[PART / 2 + i + 1]) : make_ulonglong2(res[i], res[i + 1]);
            }
            cluster_arrive();
            cluster_wait();
            const uint32_t there = map_to_cta(smem_u32(state2), half ^ 1);
            const float4 st2 = ld_cluster4(there + r / 2 * 16);
            float4 v[PART / 4];
#pragma unroll
            for (int c = 0; c < PART / 4; c++) v[c] = ld_cluster4(there + 1024 + (c * 256 + threadIdx.x) * 16);
            const float m2 = r % 2 ? st2.z : st2.x, l2 = r % 2 ? st2.w : st2.y, top = fmaxf(mm, m2);
            const float a_here = exp_nat(mm - top), a_there = exp_nat(m2 - top);
            ll = half == 0 ? ll * a_here + l2 * a_there : l2 * a_there + ll * a_here;
            mm = top;
            const f32x2 here2 = pack2(a_here, a_here), there2 = pack2(a_there, a_there);
#pragma unroll
            for (int c = 0; c < PART / 4; c++) {
                const int i = 2 * c;
                res[i] = fma2(half == 0 ? res[i] : res[PART / 2 + i], here2, mul2(pack2(v[c].x, v[c].y), there2));
                res[i + 1] = fma2(half == 0 ? res[i + 1] : res[PART / 2 + i + 1], here2, mul2(pack2(v[c].z, v[c].w), there2));
            }
            if (stores) store_cols<PART>(p.out + at * p.d, res, kSplitDown2, 1.f / ll, w * HALF + half * PART, p.d, p.vec_o, p.out, o_bytes, p.status);
        } else if (stores) {
            store_cols<HALF>(p.out + at * p.d, res, kSplitDown2, 1.f / ll, w * HALF, p.d, p.vec_o, p.out, o_bytes, p.status);
        }
        if (stores && p.lse && w == 0 && half == 0 && EMBER_STORE_OK(p.lse + at, p.lse, (size_t)p.order.units * p.lq * 4, 4, p.status)) p.lse[at] = mm + logf(ll);
    }
    if (PAIR && pair && !leave) {
        __syncwarp();
        if (warp >= 8) {  // the compute warps' first meeting
            cluster_arrive();
            cluster_wait();
        }
        cluster_arrive();
        cluster_wait();   // the other CTA has read what it needs
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 11) tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------- backward
// Work items (roles). A CTA owns 128 rows of one side and streams the other side's tiles:
//   DKDV (HD 64)   keys:    S^T = K Q^T, P; dP^T = V dO^T, dS;  dV += P dO, dK += dS Q
//   DK, DV (HD 128) the same, one result each (tensor memory holds one 128-column result beside the parts)
//   DQ             queries: S = Q K^T, dP = dO V^T, dS;         dQ += dS K
// so there is one form: A0 and A1 are the CTA's rows, B0 and B1 the streamed tiles, S = A0 B0^T, dP = A1 B1^T, results P B1 and
// dS B0. Both products of a tile recompute P from the log-sum-exp; no atomics, results repeat bit for bit.
// A warpgroup takes 32 of a tile's 64 columns.
enum Role { R_DKDV = 0, R_DQ = 1, R_DK = 2, R_DV = 3 };

template <int HD>
struct F32BwdCfg {
    static constexpr int TILE = 3 * (HD / 64) * SUB;
    static constexpr int A_BYTES = 2 * TILE;                       // 128 rows (A1 at HD 128)
    // A ring of 3 pairs of tiles beside A1 (HD 64), one pair (HD 128), or (DV, which needs no A1) 2.
    static constexpr int MAXST = HD == 64 ? 3 : 2, STAGES = HD == 64 ? 3 : 1;
    static constexpr int OFF_B = 0, OFF_A1 = STAGES * 2 * TILE;    // TILE pairs, A1
    static constexpr int OFF_LOW = OFF_A1 + A_BYTES;               // HD 128: the low parts of A0
    static constexpr int OFF_VEC = OFF_LOW + (HD == 64 ? 0 : 4 * SUB);  // per warp: 32 log-sum-exps, 32 deltas
    static constexpr int OFF_BAR = OFF_VEC + 8 * 256, USED = OFF_BAR + 256;
    static constexpr int SMEM = HD == 64 ? USED + 1024 : 232448;   // 128: the base is checked in the kernel
    static_assert(HD == 64 || OFF_LOW == MAXST * 2 * TILE, "");
    // Columns. HD 64: A0, S, P, dP / dS, two results; S is apart from P, so that the next S does not wait for the product of P
    // (with A1 in tensor memory and S under P a tile took 5700 clocks). HD 128: A0, S, dP / dS, result; DV: A0, two regions
    // of S / P, result; two accumulators of S and dP each leave no room for A0's low part, which lies in shared memory (the products of
    // both halves with a part of A come one after the other: 16 x 1024 x 2048 d 128 488 us, half after half 507).
    using R = Region<HD == 128>;
    static constexpr int T_A0 = 0, T_S = HD == 64 ? 96 : 128, T_P = HD == 64 ? 160 : 128, T_D = 256, T_R = T_D + R::COLS;
    enum { B_A, B_FULL0, B_FULL1 = B_FULL0 + MAXST, B_EMPTY0 = B_FULL1 + MAXST, B_EMPTY1 = B_EMPTY0 + MAXST, B_S = B_EMPTY1 + MAXST, B_P, B_DP, B_DS, B_R0, B_R1, B_F0, B_F1, NUM_BARS,
           B_S1 = B_DP };  // DV: scores of odd tiles (the next tile's may be there before this one's have been waited for)
    static_assert(8 * NUM_BARS + 8 + 4 * kSplitMaxTensors <= 256, "");
};

struct F32BwdParams {
    const float *q, *k, *v, *dout, *lse, *delta;
    float *dq, *dk, *dv;
    int units, lq, lk, d, causal;
    int kblocks, qblocks;
    bool vec_in, vec_out;
    float scale;
    SplitGuard guard;
    DeviceStatus *status;
    WorkOrder order;
    int paired;  // items that two CTAs share
};

// Which role and block the rank-th heaviest item of a unit is.
template <int HD>
EMBER_HD void bwd_item(int rank, int kb, int qb, int &role, int &blk)
{
    constexpr int NR = HD == 64 ? 2 : 3;
    const int m = kb < qb ? kb : qb;
    if (rank < NR * m) {
        const int i = rank % NR;
        blk = rank / NR;
        role = i == 1 ? R_DQ : HD == 64 ? R_DKDV : i == 0 ? R_DK : R_DV;
    } else if (qb > kb) {
        role = R_DQ;
        blk = m + rank - NR * m;
    } else if (HD == 64) {
        role = R_DKDV;
        blk = m + rank - NR * m;
    } else {
        const int i = rank - NR * m;
        role = i % 2 ? R_DV : R_DK;
        blk = m + i / 2;
    }
}

// PAIR: as in the forward, two CTAs share the tiles that an item's 128 rows meet, and add up their results.
template <int HD, bool PAIR>
__global__ void __launch_bounds__(F32_THREADS, 1)
    sm100_f32_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                         const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do, const F32BwdParams p)
{
    using C = F32BwdCfg<HD>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    if (HD == 128) {  // every thread takes the same decision, before any barrier exists
        uint32_t dyn;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        if (smem_base + C::USED > smem_u32(smem_raw) + dyn) {
            if (threadIdx.x == 0 && atomicCAS(&p.status->code, 0, EMBER_ERR_UNSUPPORTED) == 0) {
                p.status->where = WB_SMEM;
                p.status->block = blockIdx.x;
                p.status->extra = (int)(smem_base - smem_u32(smem_raw));
            }
            pdl_wait();  // also a kernel that does nothing ends after all before it
            return;
        }
    }
    const uint32_t bar0 = smem_base + C::OFF_BAR;
    auto BAR = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem_gen + C::OFF_BAR + 8 * C::NUM_BARS);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    int unit, rank, role, blk;
    const bool pair = PAIR && blockIdx.x < 2u * p.paired;  // the items as in the forward
    const unsigned item = !PAIR ? blockIdx.x : pair ? blockIdx.x / 2 : blockIdx.x - p.paired;
    if (PAIR && item >= (unsigned)p.order.units * p.order.blocks) {
        pdl_wait();
        return;
    }
    work_item(p.order, (int)item, unit, rank);
    bwd_item<HD>(rank, p.kblocks, p.qblocks, role, blk);
    const bool is_q = role == R_DQ;
    const bool has_p = role == R_DKDV || role == R_DV, has_ds = role != R_DV;  // which results
    const int off = p.lk - p.lq;
    const int row0 = (is_q ? p.qblocks - 1 - blk : blk) * 128;  // heaviest first: the last queries, the first keys
    // the streamed tiles: rows [first, ...) of the other side
    const int start = is_q || !p.causal ? 0 : max(0, (row0 - off) / TN) * TN;
    const int end = is_q ? (p.causal ? min(p.lk, row0 + 128 + off) : p.lk) : p.lq;
    const int tiles = (end - start + TN - 1) / TN, half = pair ? (int)cluster_ctarank() : 0, first = start + half * ((tiles + 1) / 2) * TN;
    const int n = !pair ? tiles : half ? tiles - (tiles + 1) / 2 : (tiles + 1) / 2;
    const int stages = role == R_DV ? 2 : C::STAGES;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        mbar_init(BAR(C::B_A), has_ds ? 9 : 8);  // the compute warps, and the copies of A1
        for (int s = 0; s < C::MAXST; s++) {
            mbar_init(BAR(C::B_FULL0 + s), 1);
            mbar_init(BAR(C::B_FULL1 + s), 1);
            mbar_init(BAR(C::B_EMPTY0 + s), 1);
            mbar_init(BAR(C::B_EMPTY1 + s), role == R_DKDV ? 2 : 1);  // read by both issuing warps' products
        }
        mbar_init(BAR(C::B_S), 1);
        mbar_init(BAR(C::B_P), 8);
        mbar_init(BAR(C::B_DP), 1);
        mbar_init(BAR(C::B_DS), 8);
        mbar_init(BAR(C::B_R0), 1);
        mbar_init(BAR(C::B_R1), 1);
        mbar_init(BAR(C::B_F0), role == R_DKDV ? 4 : 8);
        mbar_init(BAR(C::B_F1), 4);
        fence_mbar_init();
    }
    if (warp == 11) {
        tmem_alloc(smem_u32(tmem_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    const bool leave = split_out_of_range(p.guard, tmem_slot + 2);
    if (!leave) pdl_launch_dependents();  // as in the forward

    const uint32_t t_s = tmem + C::T_S, t_p = tmem + C::T_P, t_d = tmem + C::T_D, t_r = tmem + C::T_R;
    // At 64 columns the queries' role, which multiplies no P, has dP in P's columns: the next tile's may be formed as soon as this one's has been read
    // (B_DS), and not only when the product with the dS that would lie over it is done.
    const bool dp_apart = HD == 64 && is_q;
    const uint32_t t_dp = dp_apart ? t_p : t_d + C::R::SCORES;
    if (leave) {
        // the kernel behind this one does the work
    } else if (warp >= 8) {
        reg_dealloc_40();
        if (warp == 9 && lane == 0) {
            // ------------------------------------------------------------ TMA producer
            const CUtensorMap *b0 = is_q ? &tm_k : &tm_q, *b1 = is_q ? &tm_v : &tm_do;
            if (has_ds) {  // A1: 128 rows as boxes of 64
                const CUtensorMap *a1 = is_q ? &tm_do : &tm_v;
                mbar_arrive_expect_tx(BAR(C::B_A), C::A_BYTES);
                for (int pl = 0; pl < 3; pl++)
                    for (int s = 0; s < HD / 64; s++)
                        for (int h = 0; h < 2; h++)
                            tma_load_3d(smem_base + C::OFF_A1 + ((pl * (HD / 64) + s) * 2 + h) * SUB, a1, BAR(C::B_A), s * 64, row0 + h * 64, pl * p.units + unit);
            }
            int issued0 = 0, issued1 = 0;
            for (int j = 0; j < n; j++) {
                const int s = j % stages, ph = ((j / stages) & 1) ^ 1;
                const uint32_t dst = smem_base + C::OFF_B + s * 2 * C::TILE;
                // one pair of tiles alone: B1 is free before B0 is (its product comes before the one that reads B0 last)
                if (stages == 1 && j > 0) {
                    if (!mbar_wait(BAR(C::B_EMPTY1), ph, abort_flag, p.status, WB_E1)) break;
                    load_planes<HD>(dst + C::TILE, b1, BAR(C::B_FULL1), first + j * TN, unit, p.units);
                    issued1 = j + 1;
                }
                if (!mbar_wait(BAR(C::B_EMPTY0 + s), ph, abort_flag, p.status, WB_E0)) break;
                load_planes<HD>(dst, b0, BAR(C::B_FULL0 + s), first + j * TN, unit, p.units);
                issued0 = j + 1;
                if (stages > 1 || j == 0) {
                    if (!mbar_wait(BAR(C::B_EMPTY1 + s), ph, abort_flag, p.status, WB_E1)) break;
                    load_planes<HD>(dst + C::TILE, b1, BAR(C::B_FULL1 + s), first + j * TN, unit, p.units);
                    issued1 = j + 1;
                }
            }
            // do not leave while a copy is still landing in shared memory
            const long long t0 = clock64();
            for (int j = max(0, issued0 - stages); j < issued0; j++)
                while (!mbar_try_wait(BAR(C::B_FULL0 + j % stages), (j / stages) & 1) && clock64() - t0 < kWaitLimitCycles) {}
            for (int j = max(0, issued1 - stages); j < issued1; j++)
                while (!mbar_try_wait(BAR(C::B_FULL1 + j % stages), (j / stages) & 1) && clock64() - t0 < kWaitLimitCycles) {}
            while (has_ds && !mbar_try_wait(BAR(C::B_A), 0) && clock64() - t0 < kWaitLimitCycles) {}
        } else if (warp == 8) {
            // ------------------------------------------------------------ S and dP
            const int ksteps = (p.d + 15) / 16;
            const uint32_t elected = elect_one();
            bool ok = mbar_wait(BAR(C::B_A), 0, abort_flag, p.status, WB_A);
            auto wait = [&](int bar, int phase, int where) { ok = ok && mbar_wait(BAR(bar), phase & 1, abort_flag, p.status, where); };
            for (int j = 0; j < n && ok; j++) {
                const int s = j % stages;
                const uint32_t b0 = smem_base + C::OFF_B + s * 2 * C::TILE;
                // the scores that these overwrite have been read (DV: their probabilities multiplied)
                uint32_t at = t_s;
                int done = C::B_S;
                wait(C::B_FULL0 + s, j / stages, WB_B0);
                if (role == R_DV) {  // two regions in turn
                    at += (j & 1) * C::R::COLS;
                    done = j & 1 ? C::B_S1 : C::B_S;
                    if (j > 1) wait(j & 1 ? C::B_R1 : C::B_R0, (j - 2) >> 1, WB_ACC);
                } else if (j > 0) {
                    wait(C::B_P, j - 1, WB_ACC);
                }
                tc_fence_after();
                mma_scores<HD, HD == 64 ? A_TMEM : A_LOW>(at, tmem + C::T_A0, smem_base + C::OFF_LOW, b0, 0, HD / 64, ksteps, elected, !is_q);  // the forward's scores, bit for bit
                tc_commit_elect(BAR(done));
                if (!has_ds) {
                    tc_commit_elect(BAR(C::B_EMPTY0 + s));
                    continue;
                }
                wait(C::B_FULL1 + s, j / stages, WB_B1);
                if (j > 0) wait(dp_apart ? C::B_DS : role == R_DKDV ? C::B_R1 : C::B_R0, j - 1, WB_ACC);  // over dS, or over the last dP
                tc_fence_after();
                mma_scores<HD, A_SMEM>(t_dp, smem_base + C::OFF_A1, 0, b0 + C::TILE, 0, HD / 64, ksteps, elected, false);
                tc_commit_elect(BAR(C::B_DP));
                tc_commit_elect(BAR(C::B_EMPTY1 + s));
            }
        } else if (warp == 10) {
            // ------------------------------------------------------------ P B1 and dS B0
            const uint32_t idesc_r = idesc_bf16_f32(128, (p.d + 15) / 16 * 16, 0, 1);
            const uint32_t elected = elect_one();
            bool ok = true;
            auto wait = [&](int bar, int phase, int where) { ok = ok && mbar_wait(BAR(bar), phase & 1, abort_flag, p.status, where); };
            for (int j = 0; j < n && ok; j++) {
                const int s = j % stages;
                const uint32_t b0 = smem_base + C::OFF_B + s * 2 * C::TILE;
                if (has_p) {
                    wait(C::B_P, j, WB_P);
                    wait(C::B_FULL1 + s, j / stages, WB_B1);
                    if (j > 0) wait(C::B_F0, j - 1, WB_FREE);
                    tc_fence_after();
                    mma_results<HD, typename C::R>(t_r, t_p + (role == R_DV ? (j & 1) * C::R::COLS : 0), b0 + C::TILE, idesc_r, elected);
                    tc_commit_elect(BAR(role == R_DV && (j & 1) ? C::B_R1 : C::B_R0));
                    tc_commit_elect(BAR(C::B_EMPTY1 + s));
                }
                if (has_ds) {
                    wait(C::B_DS, j, WB_DS);
                    wait(C::B_FULL0 + s, j / stages, WB_B0);
                    if (j > 0) wait(role == R_DKDV ? C::B_F1 : C::B_F0, j - 1, WB_FREE);
                    tc_fence_after();
                    mma_results<HD, typename C::R>(t_r + (role == R_DKDV ? 64 : 0), t_d, b0, idesc_r, elected);
                    tc_commit_elect(BAR(role == R_DKDV ? C::B_R1 : C::B_R0));
                    tc_commit_elect(BAR(C::B_EMPTY0 + s));
                }
            }
        }
    } else {
        // ---------------------------------------------------------------- probabilities, score gradients, results
        reg_alloc_232();
        const int w = warp / 4, r = threadIdx.x % 128, row = row0 + r;
        const uint32_t lane_sel = (uint32_t)((warp % 4) * 32) << 16;
        const int rows = is_q ? p.lq : p.lk;
        const float *a0 = is_q ? p.q : p.k;
        const size_t row_at = ((size_t)unit * rows + row) * p.d;
        row_to_tmem(row < rows ? a0 + row_at : nullptr, p.d, p.vec_in, w * (HD / 2), HD / 64, tmem + lane_sel + C::T_A0, HD / 2, HD == 64 ? nullptr : smem_gen + C::OFF_LOW, r);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR(C::B_A));

        const float *lse = p.lse + (size_t)unit * p.lq, *delta = p.delta + (size_t)unit * p.lq;
        float *vec = reinterpret_cast<float *>(smem_gen + C::OFF_VEC + warp * 256);  // this warp's 32 columns
        // Negative log-sum-exp and delta of a query; past the end (and where a row has no weight at all) P is 0: finite, since
        // the exponential below would make NaN of an infinity, and beyond every score (kMostScore).
        auto neg_lse = [&](int qi) {
            const float x = qi < p.lq ? lse[qi] : 1e30f;
            return x > 1e30f ? -1e30f : -x;
        };
        // Score gradients, products of four tensors' values, are split as 2^ds_shift times themselves: the range in which their
        // products' sums stay well inside float32 (with weights up to 2^20) depends on those tensors (0 to 4: q, dO, k, v, delta).
        const uint32_t *most = tmem_slot + 2;
        const int e_dp = max(split_exponent(most[1]) + split_exponent(most[3]) + 7, split_exponent(most[4])) + 1;
        const int e_sum = max(0, max(split_exponent(most[0]), split_exponent(most[2])) + kSplitShift + 32 - __clz(max(p.lq, p.lk)));
        const int ds_shift = max(-60, min(100, 100 - e_dp - e_sum));
        const float ds_up = __int_as_float((127 + ds_shift) << 23), ds_down = __int_as_float((127 - ds_shift - kSplitShift) << 23);
        const f32x2 dp_scale2 = pack2(ds_up * kSplitDown2, ds_up * kSplitDown2);
        auto neg_delta = [&](int qi) { return has_ds && qi < p.lq ? -delta[qi] * ds_up : 0.f; };
        const float nl_row = is_q ? neg_lse(row) : 0.f, nd_row = is_q ? neg_delta(row) : 0.f;
        const int cols = (p.d + 15) / 16 * 16;
        // results in registers: DKDV: warpgroup 0 dV, 1 dK; otherwise half of the columns each
        f32x2 acc[32];
#pragma unroll
        for (int i = 0; i < 32; i++) acc[i] = 0;
        const f32x2 scale2 = pack2(p.scale * kSplitDown2, p.scale * kSplitDown2);
        const int acc_col0 = role == R_DKDV ? 0 : w * (HD / 2);
        const int acc_cols = min(role == R_DKDV ? cols : HD / 2, cols - acc_col0);
        const uint32_t acc_at = t_r + lane_sel + (role == R_DKDV ? w * 64 : acc_col0);
        const int bar_r = role == R_DKDV && w == 1 ? C::B_R1 : C::B_R0, bar_f = role == R_DKDV && w == 1 ? C::B_F1 : C::B_F0;
        bool ok = true;
        auto add_result = [&](int j) {
            if (role == R_DV) ok = ok && mbar_wait(BAR(j & 1 ? C::B_R1 : C::B_R0), (j >> 1) & 1, abort_flag, p.status, WB_ACC);
            else ok = ok && mbar_wait(BAR(bar_r), j & 1, abort_flag, p.status, WB_ACC);
            tc_fence_after();
            if (acc_cols > 0) flush<2, false>(acc, acc_at, acc_cols, 1.f);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR(bar_f));
        };
        const bool first_flush = role == R_DKDV && w == 0;  // dV(j - 1) is there before S(j), dK(j - 1) about when P(j) is
        for (int j = 0; j < n && ok; j++) {
            const int c0 = first + j * TN + w * 32;  // this warpgroup's first column of the tile
            if (!is_q) {                             // columns are queries
                __syncwarp();
                const int qi = c0 + lane;
                vec[lane] = neg_lse(qi);
                vec[32 + lane] = neg_delta(qi);
                __syncwarp();
            }
            // which columns are masked: keys past the row's limit, or queries before the row's key
            const int hi = is_q ? (p.causal ? min(p.lk - 1, row + off) : p.lk - 1) : p.lq - 1;
            const int lo = !is_q && p.causal ? row - off : 0;
            const bool edge = is_q ? first + j * TN + TN - 1 > (p.causal ? min(p.lk - 1, row0 + off) : p.lk - 1)
                                   : p.causal && row0 + 127 - off > first + j * TN;
            if (j > 0 && first_flush) add_result(j - 1);
            if (role == R_DV) ok = ok && mbar_wait(BAR(j & 1 ? C::B_S1 : C::B_S), (j >> 1) & 1, abort_flag, p.status, WB_S);
            else ok = ok && mbar_wait(BAR(C::B_S), j & 1, abort_flag, p.status, WB_S);
            tc_fence_after();
            const uint32_t turn = lane_sel + (role == R_DV ? (j & 1) * C::R::COLS : 0);
            f32x2 e[16];
            {
                load_scores<false>(t_s + turn + w * 32, e);
                if (HD == 128) load_scores<true>(t_s + turn + 64 + w * 32, e);
#pragma unroll
                for (int i = 0; i < 16; i += 2) {
                    const ulonglong2 nl = is_q ? make_ulonglong2(pack2(nl_row, nl_row), pack2(nl_row, nl_row)) : *reinterpret_cast<const ulonglong2 *>(vec + i * 2);
                    e[i] = exp_pair(fma2(e[i], scale2, nl.x));
                    e[i + 1] = exp_pair(fma2(e[i + 1], scale2, nl.y));
                }
                if (edge) {
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        const int c = c0 + 2 * i;
                        float x, y;
                        unpack2(e[i], x, y);
                        e[i] = pack2(c > hi || c < lo ? 0.f : x, c + 1 > hi || c + 1 < lo ? 0.f : y);
                    }
                }
            }
            if (has_p) {
                if (role == R_DKDV && w == 1 && j > 0) {  // the last P has been multiplied (warpgroup 0 has waited for dV, DV's S for its region)
                    ok = ok && mbar_wait(BAR(C::B_R0), (j - 1) & 1, abort_flag, p.status, WB_ACC);
                    tc_fence_after();
                }
                split_to_tmem<typename C::R, true>(e, t_p + turn + w * C::R::HALF);
                tmem_wait_st();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR(C::B_P));  // P is written, or at least S is read
            if (j > 0 && !first_flush) add_result(j - 1);
            if (has_ds) {
                ok = ok && mbar_wait(BAR(C::B_DP), j & 1, abort_flag, p.status, WB_DP);
                tc_fence_after();
                f32x2 dp[16];
                load_scores<false>(t_dp + lane_sel + w * 32, dp);
                if (HD == 128) load_scores<true>(t_d + lane_sel + 64 + w * 32, dp);
#pragma unroll
                for (int i = 0; i < 16; i += 2) {
                    const ulonglong2 nd = is_q ? make_ulonglong2(pack2(nd_row, nd_row), pack2(nd_row, nd_row)) : *reinterpret_cast<const ulonglong2 *>(vec + 32 + i * 2);
                    e[i] = mul2(e[i], fma2(dp[i], dp_scale2, nd.x));
                    e[i + 1] = mul2(e[i + 1], fma2(dp[i + 1], dp_scale2, nd.y));
                }
                split_to_tmem<typename C::R, false>(e, t_d + lane_sel + w * C::R::HALF);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR(C::B_DS));
            }
        }
        if (ok && n > 0) add_result(n - 1);
        float *dst = is_q ? p.dq : role == R_DKDV ? (w == 0 ? p.dv : p.dk) : role == R_DK ? p.dk : p.dv;
        const bool is_dv = role == R_DV || (role == R_DKDV && w == 0), stores = ok && row < rows && acc_cols > 0;
        const float down = is_dv ? kSplitDown2 : ds_down, scale = is_dv ? 1.f : p.scale;
        const int limit = role == R_DKDV ? p.d : min(p.d, acc_col0 + HD / 2);
        const size_t bytes = (size_t)p.units * rows * p.d * 4;
        if (PAIR && pair) {
            // ---- each CTA of the pair finishes half of every thread's columns. The tiles have been multiplied, by both warpgroups' last results
            ulonglong2 *mine = reinterpret_cast<ulonglong2 *>(smem_gen + C::OFF_B);  // [8][256] 16 bytes
            named_bar_sync(1, 256);
#pragma unroll
            for (int c = 0; c < 8; c++) mine[c * 256 + threadIdx.x] = half == 0 ? make_ulonglong2(acc[16 + 2 * c], acc[17 + 2 * c]) : make_ulonglong2(acc[2 * c], acc[2 * c + 1]);
            cluster_arrive();
            cluster_wait();
            const uint32_t there = map_to_cta(smem_u32(mine), half ^ 1);
            f32x2 res[16];
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const float4 v = ld_cluster4(there + (c * 256 + threadIdx.x) * 16);
                res[2 * c] = add2(half == 0 ? acc[2 * c] : acc[16 + 2 * c], pack2(v.x, v.y));
                res[2 * c + 1] = add2(half == 0 ? acc[2 * c + 1] : acc[17 + 2 * c], pack2(v.z, v.w));
            }
            if (stores) store_cols<32>(dst + row_at, res, down, scale, acc_col0 + half * 32, limit, p.vec_out, dst, bytes, p.status);
        } else if (stores) {
            store_cols<64>(dst + row_at, acc, down, scale, acc_col0, limit, p.vec_out, dst, bytes, p.status);
        }
    }
    if (PAIR && pair && !leave) {
        __syncwarp();
        if (warp >= 8) {  // the compute warps' first meeting
            cluster_arrive();
            cluster_wait();
        }
        cluster_arrive();
        cluster_wait();   // the other CTA has read what it needs
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 11) tmem_dealloc(tmem, 512);
}

int plane_map(CUtensorMap *m, const void *planes, int d, int rows, int units)
{
    return make_tensor_map_bf16_3d(m, planes, (uint64_t)((d + 7) / 8 * 8), (uint64_t)rows, 3ull * units, 64, 64);
}

bool vec_rows(const void *a, const void *b, const void *c, const void *d, int cols)
{
    return cols % 4 == 0 && (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d) & 15) == 0;
}

cudaError_t launch_cfg(cudaLaunchConfig_t &cfg, LaunchAttrs &attrs, long long grid, size_t smem, cudaStream_t s)
{
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(F32_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attrs.pdl().set(cfg);
    return cudaSuccess;
}

// How many query blocks, from the longest on, two CTAs share: all, where that still is one wave, or as many as there are SMs left, where the mask
// makes blocks of different lengths and the longest that stays whole is then enough shorter. us, calls back to back, whole / shared:
//   all    d 64   1 x 512 17.4 / 15.0   8 x 1024 causal 33 / 24.5   4 x 2048 causal 47.3 / 32.9   22 x 5 x 2171 50.1 / 35.4   1 x 23 x 5882 101 / 60
//          d 128  1 x 512 30 / 23   8 x 1024 causal 50.2 / 35.4   28 x 21 x 4542 209 / 139
//   some   d 64   16 x 1024 31.5 / 30.2   8 x 2048 48.2 / 45.8   6 x 1686 41.0 / 30.3   12 x 1095 31.3 / 27.3   d 128  16 x 1024 53.4 / 50.1   3 x 4594 170 / 117
// Up to four tiles (64 columns) or two, what the two spend on each other is what they save (36 x 221, d 48, 14.8 / 15.1). So it is where one tile
// fewer is left (22 x 544 21.6 / 22.5) or little of many (45 x 215 x 3049 86 / 91). In two waves a start and an end more cost as much as the better
// balance gives: 92 blocks x 4711 keys 94.5 / 106, 364 x 775 58 / 77, all of 16 x 1024 causal 31.3 / 33.4 (160 x 5010, d 128, 373 / 304, is the exception).
int fwd_paired(const AttnArgs &a, const WorkOrder &order, int sms)
{
    const long long items = (long long)order.units * order.blocks;
    if (a.lk <= (a.d <= 64 ? 4 : 2) * TN) return 0;
    if (2 * items <= sms) return (int)items;
    if (!a.causal || order.ngroups != 1 || items + order.units > sms) return 0;
    const int left = (int)(sms - items), whole = order.blocks - 1 - left / order.units;  // the last block that stays whole
    const auto tiles = [&](int block) { return (min((long long)a.lk, (block + 1) * 128LL + a.lk - a.lq) + TN - 1) / TN; };
    const long long most = tiles(order.blocks - 1), saved = most - tiles(whole);
    return saved >= 2 && 12 * saved >= most ? left : 0;
}

template <int HD, bool PAIR>
int launch_fwd_form(const CUtensorMap &tk, const CUtensorMap &tv, const F32FwdParams &p, cudaStream_t s)
{
    auto kern = sm100_f32_fwd_kernel<HD, PAIR>;
    static SmemOptIn opt_in;
    EMBER_CUDA_TRY(opt_in(kern, F32FwdCfg<HD>::SMEM));
    cudaLaunchConfig_t cfg = {};
    LaunchAttrs attrs;
    attrs.cluster(PAIR ? 2 : 1);
    const long long ctas = (long long)p.order.units * p.order.blocks + p.paired;
    launch_cfg(cfg, attrs, PAIR ? (ctas + 1) / 2 * 2 : ctas, F32FwdCfg<HD>::SMEM, s);
    EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tk, tv, p));
    return EMBER_OK;
}

template <int HD>
int launch_fwd(const AttnArgs &a, const void *kp, const void *vp, const SplitGuard &guard, DeviceState *st, cudaStream_t s)
{
    CUtensorMap tk, tv;
    int rc;
    if ((rc = plane_map(&tk, kp, a.d, a.lk, a.bh)) != EMBER_OK || (rc = plane_map(&tv, vp, a.d, a.lk, a.bh)) != EMBER_OK) return rc;
    F32FwdParams p = {};
    p.q = (const float *)a.q;
    p.out = (float *)a.out;
    p.lse = a.lse;
    p.lq = a.lq; p.lk = a.lk; p.d = a.d; p.causal = a.causal;
    p.vec_q = vec_rows(a.q, nullptr, nullptr, nullptr, a.d);
    p.vec_o = vec_rows(a.out, nullptr, nullptr, nullptr, a.d);
    p.scale = a.scale;
    p.guard = guard;
    p.status = st->status;
    p.order = make_work_order(a.bh, (a.lq + 127) / 128, st->sm_count, (size_t)a.lk * a.d * 12 + (size_t)a.lq * a.d * 8, a.causal != 0);
    p.paired = fwd_paired(a, p.order, st->sm_count);
    return p.paired > 0 ? launch_fwd_form<HD, true>(tk, tv, p, s) : launch_fwd_form<HD, false>(tk, tv, p, s);
}

// How many items, from the longest on, two CTAs share: the forward's rule over both kinds of rows. us, calls back to back, whole / shared:
//   all    d 64   1 x 512 causal 28.7 / 21.4   4 x 1024 causal 49.6 / 33.7   1 x 2048 causal 81.6 / 48.1   17 x 203, d 48, 20.7 / 18.0
//          d 128  1 x 442 46.9 / 33.3   2 x 1024 causal 93.0 / 54.8   1 x 1533 x 3558, d 72, 263 / 140
//   some   d 64   6 x 1024 51.3 / 34.6   3 x 2414 100.5 / 73.1   14 x 346 28.5 / 23.0   d 128  1 x 3278 269 / 144   4 x 438 x 1647, d 96, 127 / 115.5
// Over 87 sizes with more than two tiles, 0.53 to 0.91 of the time.
template <int HD>
int bwd_paired(const F32BwdParams &p, int sms)
{
    const long long items = (long long)p.order.units * p.order.blocks;
    if ((p.lk > p.lq ? p.lk : p.lq) <= 2 * TN) return 0;
    if (2 * items <= sms) return (int)items;
    if (!p.causal || p.order.ngroups != 1 || items + p.order.units > sms) return 0;
    const auto tiles = [&](int rank) {
        int role, blk;
        bwd_item<HD>(rank, p.kblocks, p.qblocks, role, blk);
        const long long off = p.lk - p.lq, row0 = 128LL * (role == R_DQ ? p.qblocks - 1 - blk : blk);
        const long long begin = role == R_DQ || row0 < off ? 0 : (row0 - off) / TN * TN, end = role != R_DQ ? p.lq : row0 + 128 + off < p.lk ? row0 + 128 + off : p.lk;
        return (end - begin + TN - 1) / TN;
    };
    const int left = (int)(sms - items), whole = left / p.order.units;  // rank of the first item that stays whole
    long long most = 0, rest = 0;
    for (int r = 0; r < p.order.blocks; r++) {
        const long long t = tiles(r);
        most = most > t ? most : t;
        if (r >= whole) rest = rest > t ? rest : t;
    }
    return most - rest >= 2 && 12 * (most - rest) >= most ? left : 0;
}

template <int HD, bool PAIR>
int launch_bwd_form(const CUtensorMap &tq, const CUtensorMap &tk, const CUtensorMap &tv, const CUtensorMap &tg, const F32BwdParams &p, cudaStream_t s)
{
    auto kern = sm100_f32_bwd_kernel<HD, PAIR>;
    static SmemOptIn opt_in;
    EMBER_CUDA_TRY(opt_in(kern, F32BwdCfg<HD>::SMEM));
    cudaLaunchConfig_t cfg = {};
    LaunchAttrs attrs;
    attrs.cluster(PAIR ? 2 : 1);
    const long long ctas = (long long)p.order.units * p.order.blocks + p.paired;
    launch_cfg(cfg, attrs, PAIR ? (ctas + 1) / 2 * 2 : ctas, F32BwdCfg<HD>::SMEM, s);
    EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tq, tk, tv, tg, p));
    return EMBER_OK;
}

template <int HD>
int launch_bwd(const AttnArgs &a, const float *delta, const void *qp, const void *kp, const void *vp, const void *gp, const SplitGuard &guard,
               DeviceState *st, cudaStream_t s)
{
    using C = F32BwdCfg<HD>;
    CUtensorMap tq, tk, tv, tg;
    int rc;
    if ((rc = plane_map(&tq, qp, a.d, a.lq, a.bh)) != EMBER_OK || (rc = plane_map(&tk, kp, a.d, a.lk, a.bh)) != EMBER_OK ||
        (rc = plane_map(&tv, vp, a.d, a.lk, a.bh)) != EMBER_OK || (rc = plane_map(&tg, gp, a.d, a.lq, a.bh)) != EMBER_OK)
        return rc;
    F32BwdParams p = {};
    p.q = (const float *)a.q; p.k = (const float *)a.k; p.v = (const float *)a.v; p.dout = (const float *)a.dout;
    p.lse = a.lse; p.delta = delta;
    p.dq = (float *)a.dq; p.dk = (float *)a.dk; p.dv = (float *)a.dv;
    p.units = a.bh; p.lq = a.lq; p.lk = a.lk; p.d = a.d; p.causal = a.causal;
    p.kblocks = (a.lk + 127) / 128;
    p.qblocks = (a.lq + 127) / 128;
    p.vec_in = vec_rows(a.q, a.k, a.v, a.dout, a.d);
    p.vec_out = vec_rows(a.dq, a.dk, a.dv, nullptr, a.d);
    p.scale = a.scale;
    p.guard = guard;
    p.status = st->status;
    p.order = make_work_order(a.bh, (HD == 64 ? 1 : 2) * p.kblocks + p.qblocks, st->sm_count, ((size_t)a.lk + a.lq) * a.d * 24, a.causal != 0);
    p.paired = bwd_paired<HD>(p, st->sm_count);
    return p.paired > 0 ? launch_bwd_form<HD, true>(tq, tk, tv, tg, p, s) : launch_bwd_form<HD, false>(tq, tk, tv, tg, p, s);
}

// What scores may reach (columns x the largest elements of q and k x scale) before the CUDA cores take over. 2^96 keeps them below the
// 1e30 that stands for an infinite log-sum-exp. The backward's weights e^(score - log-sum-exp) carry the score's rounding error, unless
// forward and backward form the same bits: both tensor-core kernels do, both CUDA-core kernels do, one of each does not (values'
// gradients off by 1e-4 of their norm at scores of 1e4, 7e-3 at 1e6, NaN at 1e12). Where sizes send the two directions to different
// kernels, 2^12 keeps that below 5e-4. Units may be split over calls in one direction and not in the other (ember_attention_fwd_host
// does), so sizes count as sending both here only if they do with one unit as well (from L 512 on, d 64 and 128).
constexpr double kMostScore = 7.9e28, kMostScoreMixed = 4096;

// Scales below 2^-60 times 2^-32 (the parts' factors) would end in float32's smallest exponents, those beyond 2^20 could take scores
// of operands below 2^32 to the limit above.
bool takes(const AttnArgs &a)
{
    return a.dtype == EMBER_F32 && a.d <= 128 && fabsf(a.scale) <= 1048576.f && (a.scale == 0 || fabsf(a.scale) >= 8.7e-19f) && (long long)a.bh * 3 <= 0x7fffffffLL;
}

}  // namespace

// Which kernels take a call: both sides' times are estimated, in us, from measured launches. The tensor-core side has a fixed part (the
// split, three launches, start and end of a CTA) and works in 128-row blocks, so short or few rows stay on the CUDA cores; its
// planes cost passes over memory that a few rows against long keys do not pay back. Measured, CUDA cores / tensor cores, causal, forward
// (F) and backward (B):
//   d 64    8 x 128 F 10 / 19 B 17 / 21    32 x 128 F 12 / 17 B 28 / 23   1 x 256 F 15 / 18 B 26 / 24    32 x 256 F 25 / 21 B 64 / 29
//           1 x 512 F 25 / 23 B 43 / 33    8 x 1024 F 74 / 34 B 206 / 56  4 x 2048 F 141 / 52 B 393 / 92  512 x 128 F 56 / 66 B 172 / 145
//   d 128   8 x 256 F 23 / 27 B 52 / 39    1 x 512 F 39 / 34 B 68 / 57    8 x 1024 F 105 / 56 B 234 / 103 4 x 2048 F 197 / 89 B 444 / 182
//   rows against keys, d 64   512 x 32 x 2048 F 293 / 411 B 1668 / 1165   128 x 32 x 2048 F 121 / 106 B 483 / 318   512 x 64 x 64 F 26 / 44 B 67 / 87
// The estimates are within a quarter of these. They know nothing of blocks that two CTAs share, which are up to 1.9 times as fast: what goes to the tensor
// cores is better there than they say (back to back, causal, d 64: 1 x 512 F 22 / 15 B 40 / 21, 8 x 256 B 28 / 18.5), and some forwards of few blocks stay on the
// CUDA cores that would be quicker on the others (1 x 384 without a mask 17.4; 2 x 384, which go, 17.4 / 14.1).
namespace {
struct Shape {
    double units, lq, lk, d, visible;  // visible: the share of (query, key) pairs under the mask
    double qb, kb, qt, kt;             // blocks of 128 rows, tiles of 64
    bool wide;                         // more than 64 columns
    double dpad;                       // columns the CUDA-core kernels work on
    explicit Shape(const AttnArgs &a)
        : units(a.bh), lq(a.lq), lk(a.lk), d(a.d), visible(a.causal ? 1.0 - (a.lq - 1.0) / (2.0 * a.lk) : 1.0), qb((a.lq + 127) / 128), kb((a.lk + 127) / 128),
          qt((a.lq + 63) / 64), kt((a.lk + 63) / 64), wide(a.d > 64), dpad(a.d <= 32 ? 32 : a.d <= 64 ? 64 : 128)
    {
    }
};
double longest(double a, double b) { return a > b ? a : b; }
}  // namespace

bool sm100_f32_fwd_preferred(const AttnArgs &a, int sms)
{
    if (!takes(a) || (long long)a.bh * ((a.lq + 127) / 128) > 0x7fffffffLL) return false;
    const Shape s(a);
    const double tile = s.wide ? 2.1 : 1.13, cta = s.wide ? 7.0 : 5.5, waves = s.units * s.qb / (sms > 0 ? sms : 148);
    const double tensor = 10.0 + longest(cta + tile * s.kt, waves * (cta + tile * (s.visible * s.kt + 0.5))) + s.units * s.lk * s.d * 32.0 / 7.5e6;
    const double rows = (a.lq + 15) / 16 * 16.0;
    const double cores = 5.0 + s.lk * (s.wide ? 0.0665 : s.dpad > 32 ? 0.041 : 0.028) + 35e-9 * 4.0 * s.units * rows * s.lk * s.dpad * s.visible;
    return tensor < cores;
}

bool sm100_f32_bwd_preferred(const AttnArgs &a, int sms)
{
    if (!takes(a) || (long long)a.bh * (2 * ((a.lk + 127LL) / 128) + (a.lq + 127) / 128) > 0x7fffffffLL) return false;
    const Shape s(a);
    const double tile = s.wide ? 4.9 : 2.29, cta = s.wide ? 9.5 : 6.5, kinds = s.wide ? 2.0 : 1.0, blocks = kinds * s.kb + s.qb;
    const double mean = s.visible * (kinds * s.kb * s.qt + s.qb * s.kt) / blocks;
    const double tensor = 8.0 + longest(cta + tile * longest(s.qt, s.kt), s.units * blocks / (sms > 0 ? sms : 148) * (cta + tile * mean)) +
                          s.units * (s.lq + s.lk) * s.d * 32.0 / 7.5e6;
    const double rows = 0.57 * s.qt * 64.0 + 0.43 * ((a.lq + 15) / 16 * 16.0);
    const double cores = 8.0 + longest(s.lq, s.lk) * (s.wide ? 0.117 : s.dpad > 32 ? 0.07 : 0.05) + 33e-9 * 14.0 * s.units * rows * s.lk * s.dpad * s.visible;
    return tensor < 0.95 * cores;
}

namespace {
// The guard's limit for the largest elements of q and k.
float score_limit(const AttnArgs &a, int sms)
{
    AttnArgs one = a;
    one.bh = 1;
    bool both = true;
    for (const AttnArgs *p : {(const AttnArgs *)&one, &a}) both = both && sm100_f32_fwd_preferred(*p, sms) && sm100_f32_bwd_preferred(*p, sms);
    const double most = both ? kMostScore : kMostScoreMixed;
    const double limit = a.scale != 0 ? most / (a.d * fabs((double)a.scale)) : FLT_MAX;
    return limit < FLT_MAX ? (float)limit : FLT_MAX;
}
}  // namespace

int sm100_f32_attention_fwd(const AttnArgs &a, DeviceState *st, cudaStream_t s)
{
    const long long q_rows = (long long)a.bh * a.lq, k_rows = (long long)a.bh * a.lk;
    const size_t k_bytes = split_bytes(k_rows, a.d);
    char *mem = nullptr;
    if (!scratch_alloc((void **)&mem, kSplitGuardBytes + 2 * k_bytes, s)) return EMBER_ERR_NOMEM;
    const SplitJob jobs[3] = {{(const float *)a.k, mem, k_rows, a.d}, {(const float *)a.v, mem + k_bytes, k_rows, a.d}, {(const float *)a.q, nullptr, q_rows, a.d}};
    SplitGuard guard;
    int rc = split_f32(jobs, 3, nullptr, mem + 2 * k_bytes, &guard, s);
    guard.pair[1] = 2;  // k or q, and the other one
    guard.pair_limit = score_limit(a, st->sm_count);
    if (rc == EMBER_OK)
        rc = a.d <= 64 ? launch_fwd<64>(a, mem, mem + k_bytes, guard, st, s)
             : a.d <= 96 ? launch_fwd<96>(a, mem, mem + k_bytes, guard, st, s)
                         : launch_fwd<128>(a, mem, mem + k_bytes, guard, st, s);
    if (rc == EMBER_OK) {
        AttnArgs t = a;
        t.only_if = guard.fallback;
        rc = simt_attention_fwd(t, st, s);
    }
    cudaFreeAsync(mem, s);
    return rc;
}

int sm100_f32_attention_bwd(const AttnArgs &a, float *delta, DeviceState *st, cudaStream_t s)
{
    const long long q_rows = (long long)a.bh * a.lq, k_rows = (long long)a.bh * a.lk;
    const size_t q_bytes = split_bytes(q_rows, a.d), k_bytes = split_bytes(k_rows, a.d);
    char *mem = nullptr;
    if (!scratch_alloc((void **)&mem, kSplitGuardBytes + 2 * q_bytes + 2 * k_bytes, s)) return EMBER_ERR_NOMEM;
    char *qp = mem, *gp = qp + q_bytes, *kp = gp + q_bytes, *vp = kp + k_bytes, *words = vp + k_bytes;
    const SplitJob jobs[4] = {{(const float *)a.q, qp, q_rows, a.d}, {(const float *)a.dout, gp, q_rows, a.d}, {(const float *)a.k, kp, k_rows, a.d}, {(const float *)a.v, vp, k_rows, a.d}};
    const SplitDelta dl = {(const float *)a.out, (const float *)a.dout, delta, q_rows, a.d};
    SplitGuard guard;
    int rc = split_f32(jobs, 4, &dl, words, &guard, s);
    guard.pair[1] = 2;  // k or q, and the other one
    guard.pair_limit = score_limit(a, st->sm_count);
    if (rc == EMBER_OK)
        rc = a.d <= 64 ? launch_bwd<64>(a, delta, qp, kp, vp, gp, guard, st, s) : launch_bwd<128>(a, delta, qp, kp, vp, gp, guard, st, s);
    if (rc == EMBER_OK) {
        AttnArgs t = a;
        t.only_if = guard.fallback;
        rc = simt_attention_bwd(t, delta, true, st, s);
    }
    cudaFreeAsync(mem, s);
    return rc;
}

}  // namespace ember
