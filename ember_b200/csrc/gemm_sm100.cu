// Projection GEMM for sm_100a: C (m x n) = op(A) * op(B) [+ bias], bf16 in and out, float32
// accumulation in tensor memory. It serves the Linear layers either side of attention:
//   forward          y  = x * w + b          (NN; y may be written head-major: the layout attention reads)
//   input gradient   dx = dy * w^T           (NT)
//   weight gradient  dw = x^T * dy           (TN)
// where x, dy and y may lie head-major (parts, batch, heads, seq, dim) instead of row-major, so that
// no transpose kernel runs between a projection and attention.
//
// Persistent kernel, one CTA per SM, CTAs in PAIRS (clusters of two, cta_group::2): a pair computes
// 256 x 256 output tiles, K in steps of 64. Each CTA of a pair
//   * loads its own 128 rows of A and its own 128 of the tile's 256 columns of B (its own TMA copies;
//     the completion bytes of both CTAs are counted by rank 0's barrier),
//   * receives its 128 rows x 256 columns of the result in its own tensor memory and writes them out.
// Rank 0 issues tcgen05.mma M=256 N=256 K=16 for both. A single CTA working alone on 128 x 256
// tiles reads 12 KB of operands per MMA and receives 48 KB per K step through the same 128 bytes
// per clock of shared-memory bandwidth, about 190 bytes per clock of demand: that form measured
// 0.70-0.76 of the library GEMM. In a pair each SM reads 8 KB per MMA and receives 32 KB per step.
//   warps 0-3  epilogue: accumulator (TMEM) + bias -> bf16 -> shared memory -> coalesced rows
//   warp  4    TMEM allocation (both CTAs), then MMA issue (rank 0; warp-collective, one elected lane)
//   warp  5    TMA producer (one lane): a ring of 6 stages of A (16 KB) and B (16 KB) tiles
// Two accumulators of 256 columns (all 512 TMEM columns): the MMAs of the next tile run while the
// epilogue drains the previous one.
// Operand tiles in shared memory use the 128-byte swizzle. An operand whose contraction index runs
// along its memory rows (K-major: A of NN/NT, B of NT) is one TMA box of 64 k x 128 rows;
// one whose contraction index runs across rows (MN-major: A of TN, B of NN/TN) is stored as
// sub-tiles of 64 k-rows x 64 columns, 8 KB apart.
#include "common.cuh"
#include "gemm_tiles.cuh"
#include "kernels.cuh"
#include "ptx.cuh"

namespace ember {

namespace {

using namespace ptx;

constexpr int STAGES = 6;
constexpr int A_BYTES = BM * BK * 2;
constexpr int SUB_BYTES = 64 * 128;           // 64 rows x 128 bytes
constexpr int GEMM_THREADS = 192;

// BN: columns of a pair's tile, 256, or 128 for results of few tiles: see launch. The epilogue stages OUT columns at a time: 128, or 64 where
// column sums run beside the product, so that what is left of an SM's 228 KB of shared memory holds a block of column_sum_kernel. (64 where
// nothing does: forward of 8192 rows x 512 x 16384 137 -> 145 us, 2048 x 128 x 32768 64 -> 68.)
template <int BN, int OUT>
struct GemmCfg {
    static constexpr int BNH = BN / 2;                     // B columns held by one CTA of a pair
    static constexpr int STAGE_BYTES = A_BYTES + BNH * BK * 2;
    static constexpr int OFF_OUT = STAGES * STAGE_BYTES;   // 128 rows x OUT columns of bf16 for the epilogue
    static constexpr int OFF_BIAS = OFF_OUT + BM * OUT * 2;  // BN floats
    static constexpr int OFF_BAR = OFF_BIAS + BN * 4;
    static constexpr int USED_BYTES = OFF_BAR + 128;
    static constexpr int SMEM_BYTES = USED_BYTES + 1024 < 232448 ? USED_BYTES + 1024 : 232448;  // at most the opt-in limit; the base is checked in the kernel
};

enum { B_FULL = 0, B_EMPTY = B_FULL + STAGES, B_ACCFULL = B_EMPTY + STAGES, B_ACCEMPTY = B_ACCFULL + 2, NUM_BARS = B_ACCEMPTY + 2 };
enum { WG_EMPTY = 201, WG_FULL, WG_ACCEMPTY, WG_ACCFULL, WG_SMEM };

struct GemmParams {
    int n, kblocks;
    int tiles_m, tiles_n;
    // The result's rows: `batch` entries of `seq` rows, walked in blocks of 128 rows that never cross an
    // entry, i.e. in a row space where an entry takes seq_pad rows. One entry of all m rows unless an operand
    // or the result lies head-major with a seq that is no multiple of the boxes.
    int batch, seq, seq_pad;
    ViewGeom a, b;
    MatView c;
    int c_vec;  // rows of c are 16-byte aligned: 16-byte stores
    // Beside the kernel before (GemmArgs::beside): the first `head_pairs` pairs, which find SMs at once, take `head_tiles` tiles each
    // before the common order begins.
    int late_wait, head_pairs, head_tiles;
    const __nv_bfloat16 *bias;
    DeviceStatus *status;
};

// SIDE: one of a backward call's products that run side by side, or with column sums beside it.
template <int MODE, int BN, int OUT, bool SIDE>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    sm100_gemm_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                      const GemmParams p)
{
    using C = GemmCfg<BN, OUT>;
    constexpr int CPR = OUT / 8;  // CPR: 16-byte chunks of a staged row
    constexpr int BNH = C::BNH, STAGE_BYTES = C::STAGE_BYTES, OFF_OUT = C::OFF_OUT, OFF_BIAS = C::OFF_BIAS, OFF_BAR = C::OFF_BAR,
                  USED_BYTES = C::USED_BYTES;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    {   // every thread takes the same decision, before any barrier exists
        uint32_t dyn;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        if (smem_base + USED_BYTES > smem_u32(smem_raw) + dyn) {
            if (threadIdx.x == 0 && atomicCAS(&p.status->code, 0, EMBER_ERR_UNSUPPORTED) == 0) {
                p.status->where = WG_SMEM;
                p.status->block = blockIdx.x;
                p.status->extra = (int)(smem_base - smem_u32(smem_raw));
            }
            pdl_wait();  // also a kernel that does nothing ends after all before it
            return;
        }
    }
    const uint32_t bar0 = smem_base + OFF_BAR;
    auto BAR = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem_gen + OFF_BAR + 8 * NUM_BARS);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    float *bias_s = reinterpret_cast<float *>(smem_gen + OFF_BIAS);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int num_tiles = p.tiles_m * p.tiles_n;  // tiles of 2*BM x BN, one per CTA pair at a time
    const int kblocks = p.kblocks;
    const uint32_t rank = cluster_ctarank();      // 0 issues the MMAs
    const int pair = blockIdx.x / 2, npairs = gridDim.x / 2;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < STAGES; s++) {
            mbar_init(BAR(B_FULL + s), 1);   // rank 0: its producer's arrive + the bytes of both CTAs
            mbar_init(BAR(B_EMPTY + s), 1);  // one commit (delivered to both CTAs)
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(BAR(B_ACCFULL + b), 1);
            mbar_init(BAR(B_ACCEMPTY + b), 8);  // rank 0: one arrival per epilogue warp of both CTAs
        }
        fence_mbar_init();
    }
    if (warp == 4) {
        tmem_alloc_pair(smem_u32(tmem_slot), 512);
        tmem_relinquish_pair();
    }
    if (warp == 5 && lane == 0) {
        prefetch_tensormap(&tm_a);
        prefetch_tensormap(&tm_b);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers exist before either signals the other's
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // What is launched behind a SIDE kernel may read what this one reads before it has waited itself (late_wait, column_sum_kernel), so it
    // is let go only once the kernels before this one are done; a kernel with late_wait was let go that way and passes it on.
    if (!SIDE) pdl_launch_dependents();
    if (!SIDE || !p.late_wait) pdl_wait();
    if (SIDE) pdl_launch_dependents();
    // the pair's i-th tile, num_tiles or more when there is none
    auto tile_of = [&](int i) {
        if (!SIDE || p.head_pairs == 0) return i * npairs + pair;
        if (pair < p.head_pairs) {
            if (i < p.head_tiles) return i * p.head_pairs + pair;
            i -= p.head_tiles;
        }
        return p.head_pairs * p.head_tiles + i * npairs + (npairs - 1 - pair);  // those with a head come last in a round
    };

    if (warp == 5) {
        if (lane == 0) {
            // ------------------------------------------------------------ TMA producer (both CTAs)
            int it = 0;
            bool ok = true;
            for (int i = 0, tile; (tile = tile_of(i)) < num_tiles && ok; i++) {
                int tm, tn;
                tile_coords(p.tiles_m, p.tiles_n, tile, tm, tn);
                const int m0 = tm * 2 * BM + (int)rank * BM, n0 = tn * BN + (int)rank * BNH;  // this CTA's A rows and B columns
                constexpr int NA = MODE == GEMM_TN ? BM / 64 : 1, NB = MODE == GEMM_NT ? 1 : BNH / 64;
                BoxWalker wa[NA], wb[NB];
#pragma unroll
                for (int sub = 0; sub < NA; sub++)  // TN: A view is (k x m), boxes of 64 k-rows x 64 m-columns
                    wa[sub].init(p.a, MODE == GEMM_TN ? 0 : m0, MODE == GEMM_TN ? m0 + sub * 64 : 0);
#pragma unroll
                for (int sub = 0; sub < NB; sub++)  // NN, TN: B view is (k x n), boxes of 64 k-rows x 64 n-columns
                    wb[sub].init(p.b, MODE == GEMM_NT ? n0 : 0, MODE == GEMM_NT ? 0 : n0 + sub * 64);
                for (int kb = 0; kb < kblocks; kb++, it++) {
                    const int s = it % STAGES;
                    if (!(ok = mbar_wait(BAR(B_EMPTY + s), ((it / STAGES) & 1) ^ 1, abort_flag, p.status, WG_EMPTY))) break;
                    const uint32_t a_dst = smem_base + s * STAGE_BYTES, b_dst = a_dst + A_BYTES;
                    if (rank == 0) mbar_arrive_expect_tx(BAR(B_FULL + s), 2 * STAGE_BYTES);
#pragma unroll
                    for (int sub = 0; sub < NA; sub++) {
                        wa[sub].load(a_dst + sub * SUB_BYTES, &tm_a, BAR(B_FULL + s));
                        if (MODE == GEMM_TN) wa[sub].step_rows(); else wa[sub].step_cols();
                    }
#pragma unroll
                    for (int sub = 0; sub < NB; sub++) {
                        wb[sub].load(b_dst + sub * SUB_BYTES, &tm_b, BAR(B_FULL + s));
                        if (MODE == GEMM_NT) wb[sub].step_cols(); else wb[sub].step_rows();
                    }
                }
            }
            // Do not leave while a copy of this pair is still landing in shared memory: rank 0's
            // barriers count the bytes of both CTAs, and the cluster barrier below keeps rank 1 here
            // until rank 0 has seen them.
            if (rank == 0) {
                const long long t0 = clock64();
                for (int j = max(0, it - STAGES); j < it; j++)
                    while (!mbar_try_wait(BAR(B_FULL + j % STAGES), (j / STAGES) & 1) && clock64() - t0 < kWaitLimitCycles) {}
            }
        }
    } else if (warp == 4) {
        // ---------------------------------------------------------------- MMA issue (rank 0 for the pair)
        if (rank == 0) {
            constexpr uint32_t IDESC = idesc_bf16_f32(2 * BM, BN, MODE == GEMM_TN ? 1 : 0, MODE == GEMM_NT ? 0 : 1);
            constexpr uint32_t A_LBO = MODE == GEMM_TN ? SUB_BYTES : 16, A_STEP = (MODE == GEMM_TN ? 2048 : 32) >> 4;
            constexpr uint32_t B_LBO = MODE == GEMM_NT ? 16 : SUB_BYTES, B_STEP = (MODE == GEMM_NT ? 32 : 2048) >> 4;
            int it = 0, tcount = 0;
            bool ok = true;
            for (; tile_of(tcount) < num_tiles; tcount++) {
                const int buf = tcount & 1;
                ok = ok && mbar_wait(BAR(B_ACCEMPTY + buf), ((tcount >> 1) & 1) ^ 1, abort_flag, p.status, WG_ACCEMPTY);
                tc_fence_after();
                for (int kb = 0; kb < kblocks; kb++, it++) {
                    const int s = it % STAGES;
                    ok = ok && mbar_wait(BAR(B_FULL + s), (it / STAGES) & 1, abort_flag, p.status, WG_FULL);
                    tc_fence_after();
                    const uint32_t a_lo = desc_lo(smem_base + s * STAGE_BYTES, A_LBO);
                    const uint32_t b_lo = desc_lo(smem_base + s * STAGE_BYTES + A_BYTES, B_LBO);
#pragma unroll
                    for (int k16 = 0; k16 < BK / 16; k16++)
                        mma_ss_lo_pair(tmem + buf * BN, a_lo + k16 * A_STEP, b_lo + k16 * B_STEP, IDESC, (kb > 0 || k16 > 0) ? 1u : 0u);
                    tc_commit_pair(BAR(B_EMPTY + s), 3);  // the stage is free in both CTAs
                }
                tc_commit_pair(BAR(B_ACCFULL + buf), 3);
            }
        }
    } else {
        // -------------------------------------------------------------------- epilogue (warps 0-3, both CTAs)
        const int r = threadIdx.x;  // row inside this CTA's half of the tile == TMEM lane
        const uint32_t lane_sel = (uint32_t)(warp * 32) << 16;
        uint8_t *stage = smem_gen + OFF_OUT;
        __nv_bfloat16 *cptr = (__nv_bfloat16 *)p.c.ptr;
        const uint32_t accempty0 = map_to_cta(BAR(B_ACCEMPTY), 0);  // rank 0's barriers, as cluster addresses
        int tcount = 0;
        bool ok = true;
        for (int tile; (tile = tile_of(tcount)) < num_tiles; tcount++) {
            int tm, tn;
            tile_coords(p.tiles_m, p.tiles_n, tile, tm, tn);
            const int buf = tcount & 1;
            const int m0 = (tm * 2 + (int)rank) * BM, entry = m0 / p.seq_pad, l0 = m0 - entry * p.seq_pad;
            const int rows_valid = entry < p.batch ? min(BM, p.seq - l0) : 0;  // may be <= 0: padding alone
            const int n0 = tn * BN;
            named_bar_sync(1, 128);  // the previous tile's bias has been read by every thread
            for (int j = r; j < BN; j += 128)
                bias_s[j] = (p.bias && n0 + j < p.n) ? __bfloat162float(p.bias[n0 + j]) : 0.f;
            named_bar_sync(1, 128);
            ok = ok && mbar_wait(BAR(B_ACCFULL + buf), (tcount >> 1) & 1, abort_flag, p.status, WG_ACCFULL);
            tc_fence_after();
            const uint32_t tacc = tmem + lane_sel + buf * BN;
#pragma unroll 1
            for (int part = 0; part < BN / OUT; part++) {
#pragma unroll
                for (int ch = 0; ch < OUT / 32; ch++) {
                    uint32_t u[32];
                    tmem_ld_32x32b_x32(tacc + part * OUT + ch * 32, u);
                    tmem_wait_ld();
                    if (part == BN / OUT - 1 && ch == OUT / 32 - 1) {  // the accumulator is in registers: the next tile may use it
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster(accempty0 + 8u * (uint32_t)buf);
                    }
                    const float *bs = bias_s + part * OUT + ch * 32;
#pragma unroll
                    for (int q4 = 0; q4 < 4; q4++) {  // 8 columns = one 16-byte chunk
                        uint4 wv;
                        wv.x = pack_bf16(__uint_as_float(u[q4 * 8 + 0]) + bs[q4 * 8 + 0], __uint_as_float(u[q4 * 8 + 1]) + bs[q4 * 8 + 1]);
                        wv.y = pack_bf16(__uint_as_float(u[q4 * 8 + 2]) + bs[q4 * 8 + 2], __uint_as_float(u[q4 * 8 + 3]) + bs[q4 * 8 + 3]);
                        wv.z = pack_bf16(__uint_as_float(u[q4 * 8 + 4]) + bs[q4 * 8 + 4], __uint_as_float(u[q4 * 8 + 5]) + bs[q4 * 8 + 5]);
                        wv.w = pack_bf16(__uint_as_float(u[q4 * 8 + 6]) + bs[q4 * 8 + 6], __uint_as_float(u[q4 * 8 + 7]) + bs[q4 * 8 + 7]);
                        const int chunk = ch * 4 + q4;
                        const int sw = (chunk & ~7) | ((chunk ^ r) & 7);
                        *reinterpret_cast<uint4 *>(stage + r * (OUT * 2) + sw * 16) = wv;
                    }
                }
                __syncwarp();
                // Each warp copies its own 32 rows: two (four) rows of 16 (8) chunks per instruction. The destination
                // of a chunk is found without divisions in the loop: this thread's column is fixed, and
                // the 128 rows of a CTA's tile lie inside one batch entry and therefore at one distance
                // from each other (row-major: `cols` apart; head-major: `dim`).
                if (!p.c_vec) {
                    // Rows at any alignment (row-major, columns no multiple of 8): one element per lane,
                    // 64 contiguous bytes per store instruction.
                    if (rows_valid > 0) {
                        __nv_bfloat16 *crow = cptr + ((size_t)l0 + warp * 32) * p.c.cols + n0 + part * OUT;
                        const int rows_here = min(32, rows_valid - warp * 32), cols_here = min(OUT, p.n - n0 - part * OUT);
#pragma unroll 4
                        for (int rr = 0; rr < rows_here; rr++) {
                            const int tr = warp * 32 + rr;
#pragma unroll
                            for (int i = 0; i < OUT / 32; i++) {
                                const int e = i * 32 + lane, chunk = e / 8, sw = (chunk & ~7) | ((chunk ^ tr) & 7);
                                const __nv_bfloat16 v = *reinterpret_cast<const __nv_bfloat16 *>(stage + tr * (OUT * 2) + sw * 16 + (e % 8) * 2);
                                if (ok && e < cols_here) crow[(size_t)rr * p.c.cols + e] = v;
                            }
                        }
                    }
                    __syncwarp();
                    continue;
                }
                const int chunk = lane % CPR;
                const int col = n0 + part * OUT + chunk * 8;
                const size_t row_stride = p.c.heads == 0 ? (size_t)p.c.cols : (size_t)p.c.dim;
                const size_t base = (rows_valid > 0 && col < p.n) ? view_offset(p.c, (long long)entry * p.seq + l0, col) : 0;
#pragma unroll 4
                for (int it2 = 0; it2 < CPR; it2++) {
                    const int rr = warp * 32 + it2 * (32 / CPR) + lane / CPR;
                    const int sw = (chunk & ~7) | ((chunk ^ rr) & 7);
                    const uint4 wv = *reinterpret_cast<const uint4 *>(stage + rr * (OUT * 2) + sw * 16);
                    if (ok && rr < rows_valid && col < p.n) *reinterpret_cast<uint4 *>(cptr + base + (size_t)rr * row_stride) = wv;
                }
                __syncwarp();
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // neither CTA leaves while the other may still signal its barriers or use the shared allocation
    if (warp == 4) tmem_dealloc_pair(tmem, 512);
    if (SIDE && p.late_wait) pdl_wait();  // this kernel's end stands for the end of all before it
}

// Tiles of 256 rows and 256 (or 128) columns, and the steps of the contraction.
struct Tiling {
    long long tiles_m, tiles_n;
    int kblocks, bn;
};

Tiling tiling(const GemmArgs &g, int sms)
{
    const RowPlan rows = row_plan(g);
    Tiling t;
    t.tiles_m = ((g.mode == GEMM_TN ? g.m : (long long)rows.batch * rows.seq_pad) + 2 * BM - 1) / (2 * BM);
    t.kblocks = g.mode == GEMM_TN && rows.by_entry ? rows.batch * (rows.seq_pad / BK) : (g.k + BK - 1) / BK;
    t.bn = t.tiles_m * ((g.n + 255) / 256) * 2 <= sms / 2 ? 128 : 256;
    t.tiles_n = (g.n + t.bn - 1) / t.bn;
    return t;
}

// A product beside the one before it finds the SMs at once that the other's last round leaves idle. The first `pairs` CTA pairs get
// there first; they take `tiles` tiles each ahead of the rest, as many as make the end come soonest. false: no end comes sooner for it.
// sums: the bias gradient runs behind both, beside this product, and so begins the sooner.
bool head_of(const Tiling &before, const Tiling &t, int npairs, bool sums, int &pairs, int &tiles)  // npairs: what the SMs hold
{
    pairs = tiles = 0;
    const long long all = t.tiles_m * t.tiles_n, idle = npairs - before.tiles_m * before.tiles_n % npairs;
    if (idle >= npairs) return false;
    // At most a tile each. With SMs free at once for all of them; for the bias gradient's sake also else (both gradients and bias of 1542 x 2048 x 6144
    // 79 -> 71 us; without bias 2208 x 1024 x 1024 in 32 sequences 37 -> 39, 264 x 1024 x 1024 in 11 18.8 -> 19.8).
    if (all <= (sums ? npairs : idle)) return true;
    const double late = (double)before.kblocks * before.bn / ((double)t.kblocks * t.bn);  // the others' start, in tiles
    const double alone = late + (all + npairs - 1) / npairs;
    double best = alone;
    for (int x = 0; x <= late + 1 && x * idle <= all; x++) {
        const long long rest = all - x * idle, full = rest / npairs, rem = rest % npairs;
        const double end = fmax(late + full + (rem > 0), x + full + (rem > npairs - idle));
        if (end < best - 1e-9) {
            best = end;
            pairs = (int)idle;
            tiles = x;
        }
    }
    if (tiles == 0) pairs = 0;
    return best < alone - 1e-9;
}

bool c_rows_aligned(const GemmArgs &g) { return g.n % 8 == 0 && ((uintptr_t)g.c.ptr & 15) == 0; }

template <int MODE, int BN, int OUT, bool SIDE>
int launch_tile(const GemmArgs &g, DeviceState *st, cudaStream_t s)
{
    using C = GemmCfg<BN, OUT>;
    constexpr int BNH = C::BNH, SMEM_BYTES = C::SMEM_BYTES;
    const RowPlan rows = row_plan(g);
    MatView va = g.a, vb = g.b;
    ViewGeom ga = {va.heads, va.seq, va.dim}, gb = {vb.heads, vb.seq, vb.dim};
    auto by_entry = [&](MatView &v, ViewGeom &geom) {
        if (v.heads == 0) { v.heads = 1; v.seq = rows.seq; v.dim = v.cols; }
        geom = {v.heads, rows.seq_pad, v.dim};
    };
    if (rows.by_entry) {
        by_entry(va, ga);
        if (MODE == GEMM_TN) by_entry(vb, gb);
    }
    CUtensorMap ta, tb;
    int rc;
    if ((rc = make_tensor_map_bf16_view(&ta, va, 64, MODE == GEMM_TN ? 64 : BM)) != EMBER_OK) return rc;
    if ((rc = make_tensor_map_bf16_view(&tb, vb, 64, MODE == GEMM_NT ? BNH : 64)) != EMBER_OK) return rc;
    GemmParams p;
    p.n = g.n;
    if (MODE == GEMM_TN) {  // the result's rows are columns of A: one entry
        p.tiles_m = (int)((g.m + 2 * BM - 1) / (2 * BM));
        p.kblocks = rows.by_entry ? rows.batch * (rows.seq_pad / BK) : (g.k + BK - 1) / BK;
        p.batch = 1;
        p.seq = (int)g.m;
        p.seq_pad = p.tiles_m * 2 * BM;
    } else {
        p.batch = rows.batch;
        p.seq = rows.seq;
        p.seq_pad = rows.seq_pad;
        p.tiles_m = (int)(((long long)p.batch * p.seq_pad + 2 * BM - 1) / (2 * BM));
        p.kblocks = (g.k + BK - 1) / BK;
    }
    p.tiles_n = (g.n + BN - 1) / BN;
    p.a = ga;
    p.b = gb;
    p.c = g.c;
    p.c_vec = c_rows_aligned(g);
    p.bias = (const __nv_bfloat16 *)g.bias;
    p.status = st->status;
    auto kern = sm100_gemm_kernel<MODE, BN, OUT, SIDE>;
    static SmemOptIn opt_in;
    EMBER_CUDA_TRY(opt_in(kern, SMEM_BYTES));
    const long long tiles = (long long)p.tiles_m * p.tiles_n;
    const int sms = st->sm_count > 0 ? st->sm_count : 148;
    const int pairs = (int)(tiles < sms / 2 ? tiles : sms / 2);
    p.late_wait = g.beside != nullptr;
    p.head_pairs = p.head_tiles = 0;
    if (g.beside) head_of(tiling(*g.beside, sms), tiling(g, sms), sms / 2, g.leaves_room, p.head_pairs, p.head_tiles);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = s;
    LaunchAttrs attrs;  // consecutive CTAs 2i, 2i+1 form a pair
    attrs.cluster(2).pdl().set(cfg);
    EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, ta, tb, p));
    return EMBER_OK;
}

// Tiles of 128 columns where those of 256 would leave half of the CTA pairs without one: twice the pairs, half
// the products and half the epilogue each. Beyond that the wider tile is the better one: an MMA of 128 columns
// and its copies want more shared-memory bandwidth (192 bytes per clock) than there is. Measured: forward and
// backward of a block of 2 x 500 x 512 (4 to 24 tiles) 127 -> 116 us; with the line at twice as many tiles a block of
// 2 x 1024 x 1536 (48 to 144 tiles) 224 -> 248 us.
template <int MODE>
int launch(const GemmArgs &g, DeviceState *st, cudaStream_t s)
{
    const int sms = st->sm_count > 0 ? st->sm_count : 148;
    const bool narrow = tiling(g, sms).bn == 128;
    if constexpr (MODE != GEMM_NN) {  // nothing runs beside a forward product
        if (g.leaves_room) return narrow ? launch_tile<MODE, 128, 64, true>(g, st, s) : launch_tile<MODE, 256, 64, true>(g, st, s);
        if (g.held || g.beside) return narrow ? launch_tile<MODE, 128, 128, true>(g, st, s) : launch_tile<MODE, 256, 128, true>(g, st, s);
    }
    return narrow ? launch_tile<MODE, 128, 128, false>(g, st, s) : launch_tile<MODE, 256, 128, false>(g, st, s);
}

}  // namespace

bool sm100_gemm_supported(const GemmArgs &g)
{
    if (g.dtype != EMBER_BF16 || g.m <= 0 || g.n <= 0 || g.k <= 0) return false;
    if (g.m > 0x7fffff00LL || g.a.rows > 0x7fffff00LL || g.b.rows > 0x7fffff00LL) return false;  // 32-bit box coordinates
    if ((g.m + 2 * BM - 1) / (2 * BM) * (long long)((g.n + 255) / 256) > 0x7fffffffLL) return false;
    if (g.c.heads > 0 && (g.c.dim % 8 != 0 || !c_rows_aligned(g))) return false;  // 16-byte output chunks
    if (!view_ok(g.a) || !view_ok(g.b)) return false;
    if (g.mode != GEMM_TN && g.b.heads != 0) return false;  // no caller has a head-major weight
    const RowPlan rows = row_plan(g);
    if (!rows.by_entry) return true;
    if (g.mode != GEMM_TN && !c_rows_aligned(g)) return false;  // element stores know one batch entry only
    // Every head-major view on the row axis has the same entries. Padding an entry to whole boxes pays
    // while the tensor core still beats the CUDA cores on the valid rows: they run at 20 to 25 TFLOP/s, this
    // kernel at 600 and more, so from one row in sixteen.
    for (const MatView *v : {&g.a, g.mode == GEMM_TN ? &g.b : &g.c})
        if (v->heads > 0 && v->seq != rows.seq) return false;
    const long long padded = (long long)rows.batch * rows.seq_pad;
    const long long total = g.mode == GEMM_TN ? g.k : g.m;
    if ((long long)rows.batch * rows.seq != total || rows.seq * 16LL < rows.seq_pad) return false;
    return padded <= 0x7fffff00LL && (g.mode == GEMM_TN || (padded + 2 * BM - 1) / (2 * BM) * (long long)((g.n + 255) / 256) <= 0x7fffffffLL);
}

// dst (rows x 8*chunks) = src (rows x cols) with zeros past the last column. The source has rows at any
// alignment: a lane makes 16 bytes of a row from 4 words, or from 3 words and the halves at the two ends.
// A block takes 8 rows x 256 chunks, a warp one row, so that short and long rows both spread over the SMs (rows longer than
// 65535 such pieces, 134 million columns: every 65535th of them).
__global__ void __launch_bounds__(256) pack_rows_kernel(const unsigned short *__restrict__ src, uint4 *__restrict__ dst, long long rows,
                                                        int cols, int chunks)
{
    ptx::pdl_launch_dependents();
    ptx::pdl_wait();
    const long long row = (long long)blockIdx.x * 8 + threadIdx.x / 32;
    if (row >= rows) return;
    const unsigned short *r = src + (size_t)row * cols;
    const bool odd = ((uintptr_t)r & 2) != 0;  // rows are 2-byte aligned
    for (int c0 = blockIdx.y * 256; c0 < chunks; c0 += gridDim.y * 256) {
        const int end = min(chunks, c0 + 256);
#pragma unroll 4
        for (int c = c0 + threadIdx.x % 32; c < end; c += 32) {
            uint32_t w[4];
            const unsigned short *e = r + (size_t)c * 8;
            if (c * 8 + 8 > cols) {
                unsigned short h[8];
#pragma unroll
                for (int i = 0; i < 8; i++) h[i] = c * 8 + i < cols ? e[i] : (unsigned short)0;
#pragma unroll
                for (int i = 0; i < 4; i++) w[i] = (uint32_t)h[2 * i] | (uint32_t)h[2 * i + 1] << 16;
            } else if (odd) {
                const uint32_t *m = reinterpret_cast<const uint32_t *>(e + 1);
                const uint32_t first = e[0], a = m[0], b = m[1], d = m[2], last = e[7];
                w[0] = first | a << 16;
                w[1] = a >> 16 | b << 16;
                w[2] = b >> 16 | d << 16;
                w[3] = d >> 16 | last << 16;
            } else {
                const uint32_t *m = reinterpret_cast<const uint32_t *>(e);
#pragma unroll
                for (int i = 0; i < 4; i++) w[i] = m[i];
            }
            dst[(size_t)row * chunks + c] = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

int pack_rows(const MatView &v, void *dst, cudaStream_t s)
{
    const int chunks = (v.cols + 7) / 8, pieces = (chunks + 255) / 256;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((v.rows + 7) / 8), (unsigned)(pieces < 65535 ? pieces : 65535));
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    LaunchAttrs attrs;
    attrs.pdl().set(cfg);
    EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, pack_rows_kernel, (const unsigned short *)v.ptr, (uint4 *)dst, v.rows, v.cols, chunks));
    return EMBER_OK;
}

bool sm100_gemm_gains_beside(const GemmArgs &before, const GemmArgs &g, DeviceState *st)
{
    const int sms = st->sm_count > 0 ? st->sm_count : 148;
    int pairs, head;
    return head_of(tiling(before, sms), tiling(g, sms), sms / 2, g.leaves_room, pairs, head);
}

int sm100_gemm(const GemmArgs &g, DeviceState *st, cudaStream_t s)
{
    switch (g.mode) {
    case GEMM_NN: return launch<GEMM_NN>(g, st, s);
    case GEMM_NT: return launch<GEMM_NT>(g, st, s);
    default: return launch<GEMM_TN>(g, st, s);
    }
}

}  // namespace ember
