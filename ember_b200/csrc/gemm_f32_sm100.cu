// Float32 matrix products of the Linear layers on the tensor cores: C (m x n) = op(A) * op(B) [+ bias], operands as three bf16
// planes (split_f32.cuh), six tcgen05 products for one float32 product, float32 results. Modes and views as in gemm_sm100.cu, whose
// CTA pairs, boxes and walks along batch entries it shares (gemm_tiles.cuh).
//
// What differs: one accumulator holds one contraction step of 64 only, since the tensor core adds with truncation. The six products
// of the planes, four MMAs each, go into one of two accumulators, small products first; eight epilogue warps add it into float32
// registers (64 or 128 per thread) while the next step fills the other one. A step is 24 MMAs of 128 clocks (256 columns),
// adding it up 200 to 300, so the tensor core is never waited for.
//   warps 0-7  epilogue: row (warp % 4) * 32 + lane of this CTA's 128, columns by half (warp / 4)
//   warp  8    tensor-memory allocation, MMA issue (even rank of a pair)
//   warp  9    TMA producer: a ring of 2 or 3 stages of three planes of A and B
// Results of few tiles are split along the contraction: a cluster of 2 or 4 pairs of CTAs, a pair per part, whose partial tiles
// are added in order through distributed shared memory, so results repeat bit for bit.
#include "common.cuh"
#include "gemm_tiles.cuh"
#include "kernels.cuh"
#include "ptx.cuh"
#include "split_f32.cuh"

namespace ember {

namespace {

using namespace ptx;

constexpr int THREADS = 320, MAX_STAGES = 3;
constexpr int A_PLANE = BM * BK * 2, SUB_BYTES = 64 * 128;

template <int BN>
struct Cfg {
    static constexpr int BNH = BN / 2;
    static constexpr int B_PLANE = BNH * BK * 2, STAGE = 3 * (A_PLANE + B_PLANE);
    // 256 columns: results pass through 4 KB per epilogue warp. 128: a third stage instead (a step is half as long, and
    // with two its loads were waited for: 4096 x 72 x 4096, both gradients, 63 us each), and results, which are few, go out from registers.
    static constexpr int STAGES = BN == 256 ? 2 : 3;
    static constexpr int OFF_OUT = STAGES * STAGE;
    static constexpr int OFF_BAR = OFF_OUT + (BN == 256 ? 8 * 4096 : 0), USED = OFF_BAR + 128;
    static constexpr int SMEM = BN == 256 ? 232448 : USED + 1024;  // 256: the base is checked in the kernel
    static constexpr int HALF = BN / 2;                       // columns of an epilogue warp
};

enum { B_FULL = 0, B_EMPTY = B_FULL + MAX_STAGES, B_ACCFULL = B_EMPTY + MAX_STAGES, B_ACCEMPTY = B_ACCFULL + 2, NUM_BARS = B_ACCEMPTY + 2 };
static_assert(8 * NUM_BARS + 8 + 4 * kSplitMaxTensors <= 128, "");
enum { WS_EMPTY = 401, WS_FULL, WS_ACCEMPTY, WS_ACCFULL, WS_SMEM };

struct Params {
    int n, kblocks, tiles_m, tiles_n;
    int batch, seq, seq_pad;  // the result's rows, as in gemm_sm100.cu
    ViewGeom a, b;
    int parts_a, parts_b;     // parts of a plane
    MatView c;
    int c_vec;
    const float *bias;
    int splits;
    SplitGuard guard;
    DeviceStatus *status;
};

// Four MMAs of 16 contraction steps of a pair.
template <int A_STEP, int B_STEP>
__device__ __forceinline__ void chain_pair(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t elected, uint32_t acc)
{
    asm volatile("{\n.reg .pred p, q;\n.reg .b64 da, db;\n.reg .b32 t, u;\nsetp.ne.b32 q, %4, 0;\nsetp.ne.b32 p, %5, 0;\n"
                 "mov.b64 da, {%1, %6};\nmov.b64 db, {%2, %6};\n@q tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\nsetp.eq.u32 p, 0, 0;\n"
                 "add.u32 u, %1, %7;\nadd.u32 t, %2, %10;\nmov.b64 da, {u, %6};\nmov.b64 db, {t, %6};\n@q tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n"
                 "add.u32 u, %1, %8;\nadd.u32 t, %2, %11;\nmov.b64 da, {u, %6};\nmov.b64 db, {t, %6};\n@q tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n"
                 "add.u32 u, %1, %9;\nadd.u32 t, %2, %12;\nmov.b64 da, {u, %6};\nmov.b64 db, {t, %6};\n@q tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n}\n"
                 ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"(elected), "r"(acc), "r"(kDescHiSw128), "n"(A_STEP), "n"(2 * A_STEP), "n"(3 * A_STEP), "n"(B_STEP),
                 "n"(2 * B_STEP), "n"(3 * B_STEP)
                 : "memory");
}

template <int MODE, int BN>
__global__ void __launch_bounds__(THREADS, 1)
    sm100_f32_gemm_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const Params p)
{
    using C = Cfg<BN>;
    constexpr int BNH = C::BNH, STAGES = C::STAGES;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    {   // every thread takes the same decision, before any barrier exists
        uint32_t dyn;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        if (smem_base + C::USED > smem_u32(smem_raw) + dyn) {
            if (threadIdx.x == 0 && atomicCAS(&p.status->code, 0, EMBER_ERR_UNSUPPORTED) == 0) {
                p.status->where = WS_SMEM;
                p.status->block = blockIdx.x;
                p.status->extra = (int)(smem_base - smem_u32(smem_raw));
            }
            pdl_wait();  // also a kernel that does nothing ends after all before it
            return;
        }
    }
    const uint32_t bar0 = smem_base + C::OFF_BAR;
    auto BAR = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem_gen + C::OFF_BAR + 8 * NUM_BARS);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int num_tiles = p.tiles_m * p.tiles_n;
    const uint32_t crank = cluster_ctarank(), rank = crank & 1, even = crank & ~1u;  // rank 0 of a pair issues
    const int split = (int)(crank / 2), cluster = blockIdx.x / (2 * p.splits), clusters = gridDim.x / (2 * p.splits);
    const int kb0 = (int)((long long)p.kblocks * split / p.splits), kb1 = (int)((long long)p.kblocks * (split + 1) / p.splits);

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < STAGES; s++) {
            mbar_init(BAR(B_FULL + s), 1);
            mbar_init(BAR(B_EMPTY + s), 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(BAR(B_ACCFULL + b), 1);
            mbar_init(BAR(B_ACCEMPTY + b), 16);  // the epilogue warps of both CTAs
        }
        fence_mbar_init();
    }
    if (warp == 8) {
        tmem_alloc_pair(smem_u32(tmem_slot), 2 * BN);
        tmem_relinquish_pair();
    }
    if (warp == 9 && lane == 0) {
        prefetch_tensormap(&tm_a);
        prefetch_tensormap(&tm_b);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_launch_dependents();
    pdl_wait();
    const bool leave = split_out_of_range(p.guard, tmem_slot + 2);

    if (leave) {
        // the kernel behind this one does the work
    } else if (warp == 9) {
        if (lane == 0) {
            // ------------------------------------------------------------ TMA producer
            int it = 0;
            bool ok = true;
            for (int tile = cluster; tile < num_tiles && ok; tile += clusters) {
                int tm, tn;
                tile_coords(p.tiles_m, p.tiles_n, tile, tm, tn);
                const int m0 = tm * 2 * BM + (int)rank * BM, n0 = tn * BN + (int)rank * BNH;
                constexpr int NA = MODE == GEMM_TN ? BM / 64 : 1, NB = MODE == GEMM_NT ? 1 : BNH / 64;
                BoxWalker wa[NA], wb[NB];
#pragma unroll
                for (int sub = 0; sub < NA; sub++) wa[sub].init(p.a, MODE == GEMM_TN ? kb0 * BK : m0, MODE == GEMM_TN ? m0 + sub * 64 : kb0 * BK);
#pragma unroll
                for (int sub = 0; sub < NB; sub++) wb[sub].init(p.b, MODE == GEMM_NT ? n0 : kb0 * BK, MODE == GEMM_NT ? kb0 * BK : n0 + sub * 64);
                for (int kb = kb0; kb < kb1; kb++, it++) {
                    const int s = it % STAGES;
                    if (!(ok = mbar_wait(BAR(B_EMPTY + s), ((it / STAGES) & 1) ^ 1, abort_flag, p.status, WS_EMPTY))) break;
                    const uint32_t a_dst = smem_base + s * C::STAGE, b_dst = a_dst + 3 * A_PLANE;
                    if (rank == 0) mbar_arrive_expect_tx(BAR(B_FULL + s), 2 * C::STAGE);
#pragma unroll
                    for (int sub = 0; sub < NA; sub++) {
#pragma unroll
                        for (int pl = 0; pl < 3; pl++) wa[sub].load(a_dst + pl * A_PLANE + sub * SUB_BYTES, &tm_a, BAR(B_FULL + s), pl * p.parts_a);
                        if (MODE == GEMM_TN) wa[sub].step_rows(); else wa[sub].step_cols();
                    }
#pragma unroll
                    for (int sub = 0; sub < NB; sub++) {
#pragma unroll
                        for (int pl = 0; pl < 3; pl++) wb[sub].load(b_dst + pl * C::B_PLANE + sub * SUB_BYTES, &tm_b, BAR(B_FULL + s), pl * p.parts_b);
                        if (MODE == GEMM_NT) wb[sub].step_cols(); else wb[sub].step_rows();
                    }
                }
            }
            // do not leave while a copy of this pair is still landing in shared memory (rank 0 counts both CTAs')
            if (rank == 0) {
                const long long t0 = clock64();
                for (int j = max(0, it - STAGES); j < it; j++)
                    while (!mbar_try_wait(BAR(B_FULL + j % STAGES), (j / STAGES) & 1) && clock64() - t0 < kWaitLimitCycles) {}
            }
        }
    } else if (warp == 8) {
        // ---------------------------------------------------------------- MMA issue (rank 0 for the pair)
        if (rank == 0) {
            constexpr uint32_t IDESC = idesc_bf16_f32(2 * BM, BN, MODE == GEMM_TN ? 1 : 0, MODE == GEMM_NT ? 0 : 1);
            constexpr uint32_t A_LBO = MODE == GEMM_TN ? SUB_BYTES : 16, A_STEP = (MODE == GEMM_TN ? 2048 : 32) >> 4;
            constexpr uint32_t B_LBO = MODE == GEMM_NT ? 16 : SUB_BYTES, B_STEP = (MODE == GEMM_NT ? 32 : 2048) >> 4;
            const uint32_t elected = elect_one();
            const uint16_t both = (uint16_t)(3u << even);
            int it = 0;
            bool ok = true;
            for (int tile = cluster; tile < num_tiles; tile += clusters)
                for (int kb = kb0; kb < kb1; kb++, it++) {
                    const int s = it % STAGES, buf = it & 1;
                    ok = ok && mbar_wait(BAR(B_ACCEMPTY + buf), ((it >> 1) & 1) ^ 1, abort_flag, p.status, WS_ACCEMPTY);
                    ok = ok && mbar_wait(BAR(B_FULL + s), (it / STAGES) & 1, abort_flag, p.status, WS_FULL);
                    tc_fence_after();
                    const uint32_t a_lo = desc_lo(smem_base + s * C::STAGE, A_LBO), b_lo = desc_lo(smem_base + s * C::STAGE + 3 * A_PLANE, B_LBO);
#pragma unroll 1
                    for (int i = 0; i < kSplitProducts; i++)
                        chain_pair<A_STEP, B_STEP>(tmem + buf * BN, a_lo + split_part_a(i) * (A_PLANE >> 4), b_lo + split_part_b(i) * (C::B_PLANE >> 4), IDESC, elected, i > 0);
                    tc_commit_pair(BAR(B_EMPTY + s), both);
                    tc_commit_pair(BAR(B_ACCFULL + buf), both);
                }
        }
    } else {
        // -------------------------------------------------------------------- epilogue (warps 0-7, both CTAs)
        const int r = (warp % 4) * 32 + lane, half = warp / 4;
        const uint32_t lane_sel = (uint32_t)((warp % 4) * 32) << 16;
        float *cptr = (float *)p.c.ptr;
        const uint32_t accempty = map_to_cta(BAR(B_ACCEMPTY), even);
        int it = 0;
        bool ok = true;
        for (int tile = cluster; tile < num_tiles; tile += clusters) {
            int tm, tn;
            tile_coords(p.tiles_m, p.tiles_n, tile, tm, tn);
            const int m0 = (tm * 2 + (int)rank) * BM, entry = m0 / p.seq_pad, l0 = m0 - entry * p.seq_pad;
            const int rows_valid = entry < p.batch ? min(BM, p.seq - l0) : 0;  // may be <= 0: padding alone
            const int n0 = tn * BN;
            f32x2 acc[C::HALF / 2];
#pragma unroll
            for (int i = 0; i < C::HALF / 2; i++) acc[i] = 0;
            for (int kb = kb0; kb < kb1; kb++, it++) {
                const int buf = it & 1;
                ok = ok && mbar_wait(BAR(B_ACCFULL + buf), (it >> 1) & 1, abort_flag, p.status, WS_ACCFULL);
                tc_fence_after();
                const uint32_t t = tmem + lane_sel + buf * BN + half * C::HALF;
#pragma unroll
                for (int c = 0; c < C::HALF / 32; c++) {
                    uint32_t u[32];
                    tmem_ld_32x32b_x32(t + c * 32, u);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 16; i++) acc[c * 16 + i] = add2(acc[c * 16 + i], pack2(__uint_as_float(u[2 * i]), __uint_as_float(u[2 * i + 1])));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(accempty + 8u * (uint32_t)buf);
            }
            // Rows lie at one distance from each other in a CTA's tile (one batch entry), columns of 4 in one head. The loops stay loops:
            // with every store and its address unrolled the epilogue missed the instruction cache throughout, 14 us a tile.
            const size_t row_stride = p.c.heads == 0 ? (size_t)p.c.cols : (size_t)p.c.dim;
            const long long row0 = (long long)entry * p.seq + l0;
            auto column = [&](int col) {  // row 0 of this CTA's tile
                return cptr + (p.c.heads == 0 ? (size_t)row0 * p.c.cols + col : view_offset(p.c, row0, col));
            };
            auto bias4 = [&](int col) {
                return p.bias ? make_float4(p.bias[col], p.bias[col + 1], p.bias[col + 2], p.bias[col + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
            };
            auto with_bias = [](const float4 &v, const float4 &b) {
                return make_float4(fmaf(v.x, kSplitDown2, b.x), fmaf(v.y, kSplitDown2, b.y), fmaf(v.z, kSplitDown2, b.z), fmaf(v.w, kSplitDown2, b.w));
            };
            auto store1 = [&](float *dst, int col, const float4 &v) {  // columns one by one (row-major)
                const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (col + i < p.n) dst[i] = fmaf(x[i], kSplitDown2, p.bias ? p.bias[col + i] : 0.f);
            };
            const int rows_here = ok ? rows_valid : 0;
            if (BN == 128 && p.splits == 1) {
                const int col = n0 + half * C::HALF;  // 64 columns, inside one head
                if (r < rows_here && col < p.n) {
                    float *dst = column(col) + (size_t)r * row_stride;
#pragma unroll
                    for (int q = 0; q < C::HALF / 4; q++) {
                        float4 v;
                        unpack2(acc[2 * q], v.x, v.y);
                        unpack2(acc[2 * q + 1], v.z, v.w);
                        if (col + q * 4 >= p.n) continue;
                        if (p.c_vec) {
                            *reinterpret_cast<float4 *>(dst + q * 4) = with_bias(v, bias4(col + q * 4));
                        } else {
                            store1(dst + q * 4, col + q * 4, v);
                        }
                    }
                }
            } else if (p.splits == 1) {
                uint8_t *stage = smem_gen + C::OFF_OUT + warp * 4096;  // 32 rows x 32 columns
#pragma unroll
                for (int c = 0; c < C::HALF / 32; c++) {
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < 8; q++)
                        *reinterpret_cast<ulonglong2 *>(stage + lane * 128 + ((q ^ (lane & 7)) << 4)) = make_ulonglong2(acc[c * 16 + 2 * q], acc[c * 16 + 2 * q + 1]);
                    __syncwarp();
                    const int col = n0 + half * C::HALF + c * 32 + (lane % 8) * 4, first = (warp % 4) * 32 + lane / 8;
                    if (rows_here <= 0 || col >= p.n) continue;
                    const uint8_t *from = stage + (lane / 8) * 128;
                    float *dst = column(col) + (size_t)first * row_stride;
                    if (p.c_vec) {
                        const float4 b = bias4(col);
#pragma unroll 4
                        for (int i = 0; i < 8; i++) {
                            const float4 v = *reinterpret_cast<const float4 *>(from + i * 512 + (((lane % 8) ^ ((i * 4 + lane / 8) & 7)) << 4));
                            if (first + i * 4 < rows_here) *reinterpret_cast<float4 *>(dst + (size_t)(i * 4) * row_stride) = with_bias(v, b);
                        }
                    } else {
#pragma unroll 1
                        for (int i = 0; i < 8; i++)
                            if (first + i * 4 < rows_here)
                                store1(dst + (size_t)(i * 4) * row_stride, col, *reinterpret_cast<const float4 *>(from + i * 512 + (((lane % 8) ^ ((i * 4 + lane / 8) & 7)) << 4)));
                    }
                }
            } else {
                // Every CTA leaves its partial tile (128 rows x BN columns) where the ring was (all products have been formed), then adds
                // the rows that are its share, part 0 first.
                uint8_t *mine = smem_gen + r * (BN * 4);
#pragma unroll
                for (int q = 0; q < C::HALF / 4; q++) {
                    const int chunk = half * (C::HALF / 4) + q;
                    *reinterpret_cast<ulonglong2 *>(mine + ((chunk ^ (r & 7)) << 4)) = make_ulonglong2(acc[2 * q], acc[2 * q + 1]);
                }
                cluster_arrive();
                cluster_wait();
                const int rows = BM / p.splits;
                for (int e = threadIdx.x; e < rows * (BN / 4); e += 256) {
                    const int row = split * rows + e / (BN / 4), chunk = e % (BN / 4);
                    const uint32_t at = smem_base + row * (BN * 4) + ((chunk ^ (row & 7)) << 4);
                    float4 v = ld_cluster4(map_to_cta(at, rank));
                    for (int s = 1; s < p.splits; s++) {
                        const float4 x = ld_cluster4(map_to_cta(at, 2 * s + rank));
                        v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
                    }
                    const int col = n0 + chunk * 4;
                    if (row >= rows_here || col >= p.n) continue;
                    float *dst = column(col) + (size_t)row * row_stride;
                    if (p.c_vec) {
                        *reinterpret_cast<float4 *>(dst) = with_bias(v, bias4(col));
                    } else {
                        store1(dst, col, v);
                    }
                }
            }
        }
    }
    if (!leave && p.splits > 1 && warp >= 8) {  // the barrier between the partial tiles' writing and reading is the whole cluster's
        __syncwarp();
        cluster_arrive();
        cluster_wait();
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // nobody leaves while others may still signal its barriers or read its shared memory
    if (warp == 8) tmem_dealloc_pair(tmem, 2 * BN);
}

bool c_vec(const GemmArgs &g) { return g.n % 4 == 0 && ((uintptr_t)g.c.ptr & 15) == 0; }

// The planes of a view: row-major rows are padded to 8 columns, a head-major tensor stays as it is.
MatView planes_of(const MatView &v, const void *planes)
{
    MatView t = v;
    t.ptr = planes;
    if (t.heads == 0) t.cols = (t.cols + 7) / 8 * 8;
    return t;
}

template <int MODE, int BN>
int launch_tile(const GemmArgs &g, const void *a_planes, const void *b_planes, int splits, const SplitGuard &guard, DeviceStatus *status, int sms, cudaStream_t s)
{
    using C = Cfg<BN>;
    const RowPlan rows = row_plan(g);
    MatView va = planes_of(g.a, a_planes), vb = planes_of(g.b, b_planes);
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
    if ((rc = make_tensor_map_bf16_view(&ta, va, 64, MODE == GEMM_TN ? 64 : BM, 3)) != EMBER_OK) return rc;
    if ((rc = make_tensor_map_bf16_view(&tb, vb, 64, MODE == GEMM_NT ? C::BNH : 64, 3)) != EMBER_OK) return rc;
    Params p = {};
    p.n = g.n;
    if (MODE == GEMM_TN) {
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
    p.parts_a = va.heads ? va.cols / (va.heads * va.dim) : 1;
    p.parts_b = vb.heads ? vb.cols / (vb.heads * vb.dim) : 1;
    p.c = g.c;
    p.c_vec = c_vec(g);
    p.bias = (const float *)g.bias;
    p.splits = splits < p.kblocks ? splits : 1;
    p.guard = guard;
    p.status = status;
    auto kern = sm100_f32_gemm_kernel<MODE, BN>;
    static SmemOptIn opt_in;
    EMBER_CUDA_TRY(opt_in(kern, C::SMEM));
    const long long tiles = (long long)p.tiles_m * p.tiles_n;
    const int clusters = p.splits > 1 ? (int)tiles : (int)(tiles < sms / 2 ? tiles : sms / 2);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * p.splits * clusters));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = s;
    LaunchAttrs attrs;
    attrs.cluster(2 * p.splits).pdl().set(cfg);
    EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, ta, tb, p));
    return EMBER_OK;
}

struct Plan {
    int bn, splits;
    double us;  // estimate, without the splitting of the operands
};

// Tiles of 128 columns where those of 256 would leave half of the pairs without one, and the contraction over 2 or 4 pairs while
// all find room at once and each has four steps. Clusters of 8 CTAs find room up to 12 or so (512 x 1024 x 1024, 16 tiles: 23 us with
// two parts, 30 with four; 256 x 1000 x 1024, 8 tiles: 23 and 18).
Plan plan(const GemmArgs &g, int sms)
{
    const RowPlan rows = row_plan(g);
    const long long m = g.mode == GEMM_TN ? g.m : (long long)rows.batch * rows.seq_pad;
    const long long k = g.mode == GEMM_TN && rows.by_entry ? (long long)rows.batch * rows.seq_pad : g.k;
    const double pairs = sms > 1 ? sms / 2 : 74;
    const double tm = (double)((m + 2 * BM - 1) / (2 * BM)), steps = (double)((k + BK - 1) / BK);
    Plan p;
    p.bn = tm * ((g.n + 255) / 256) * 2 <= pairs ? 128 : 256;
    const double tiles = tm * ((g.n + p.bn - 1) / p.bn);
    p.splits = 1;
    if (p.bn == 128) {
        if (tiles <= 12 && steps >= 16) p.splits = 4;
        else if (tiles * 2 <= 0.9 * pairs && steps >= 8) p.splits = 2;
    }
    const double waves = p.splits > 1 ? 1.0 : (double)(long long)((tiles + pairs - 1) / pairs);
    p.us = waves * (steps / p.splits * (p.bn == 256 ? 1.75 : 0.95) + (p.bn == 256 ? 4.0 : 2.0));  // steps, start and end of a tile
    return p;
}

template <int MODE>
int launch(const GemmArgs &g, const void *a, const void *b, const SplitGuard &guard, DeviceState *st, cudaStream_t s)
{
    const int sms = st->sm_count > 0 ? st->sm_count : 148;
    const Plan p = plan(g, sms);
    return p.bn == 128 ? launch_tile<MODE, 128>(g, a, b, p.splits, guard, st->status, sms, s) : launch_tile<MODE, 256>(g, a, b, 1, guard, st->status, sms, s);
}

// Whether the planes of a view can be walked: asked of a stand-in at an aligned address.
bool planes_ok(const MatView &v) { return view_ok(planes_of(v, (const void *)(uintptr_t)256)); }

}  // namespace

bool sm100_f32_gemm_supported(const GemmArgs &g)
{
    if (g.dtype != EMBER_F32 || g.m <= 0 || g.n <= 0 || g.k <= 0) return false;
    if (g.m > 0x7fffff00LL || g.a.rows > 0x7fffff00LL || g.b.rows > 0x7fffff00LL || g.a.cols > 0x7ffffff0 || g.b.cols > 0x7ffffff0) return false;
    if ((g.m + 2 * BM - 1) / (2 * BM) * (long long)((g.n + 127) / 128) > 0x3fffffffLL) return false;
    if (g.c.heads > 0 && (g.c.dim % 64 != 0 || !c_vec(g))) return false;
    if (!planes_ok(g.a) || !planes_ok(g.b)) return false;
    if (g.mode != GEMM_TN && g.b.heads != 0) return false;
    const RowPlan rows = row_plan(g);
    if (!rows.by_entry) return true;
    if (g.mode != GEMM_TN && !c_vec(g)) return false;  // element stores know one batch entry only
    for (const MatView *v : {&g.a, g.mode == GEMM_TN ? &g.b : &g.c})
        if (v->heads > 0 && v->seq != rows.seq) return false;
    const long long padded = (long long)rows.batch * rows.seq_pad, total = g.mode == GEMM_TN ? g.k : g.m;
    if ((long long)rows.batch * rows.seq != total || rows.seq * 4LL < rows.seq_pad) return false;
    return padded <= 0x7fffff00LL && (g.mode == GEMM_TN || (padded + 2 * BM - 1) / (2 * BM) * (long long)((g.n + 127) / 128) <= 0x3fffffffLL);
}

double sm100_f32_gemm_us(const GemmArgs &g, int sms) { return plan(g, sms).us; }

int sm100_f32_gemm(const GemmArgs &g, const void *a_planes, const void *b_planes, const SplitGuard &guard, DeviceState *st, cudaStream_t s)
{
    switch (g.mode) {
    case GEMM_NN: return launch<GEMM_NN>(g, a_planes, b_planes, guard, st, s);
    case GEMM_NT: return launch<GEMM_NT>(g, a_planes, b_planes, guard, st, s);
    default: return launch<GEMM_TN>(g, a_planes, b_planes, guard, st, s);
    }
}

}  // namespace ember
