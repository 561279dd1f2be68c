// Products with few rows for sm_100a: y (m x n) = x (m x k) * op(w) [+ bias] with m <= 128, bf16 in and
// out, float32 accumulation. This is a decode step's projection (m = sequences): 2 m flops per weight
// byte, so the bound is reading w once, and the kernel is shaped for that, not for the tensor pipe:
//   - the product is computed TRANSPOSED, y^T = op(w)^T x^T: 128 outputs (columns of y) are the M rows
//     of a tcgen05.mma and the m rows of x are its N columns (padded to 16, 32, 64 or 128). A tile of
//     256 x 256 of the kernel for large products would be 97 % padding at m = 8, and CUDA cores need
//     m FMAs per weight, more than the FMA pipe has above m = 8.
//   - w streams through a ring of 64 x 128 tiles (16 KB TMA boxes, 96 KB in flight per CTA, two CTAs per
//     SM), each tile read from HBM exactly once.
//   - the contraction is split over a cluster of up to 8 CTAs, so that a 2048 x 2048 weight matrix still
//     gives 128 CTAs their own 64 KB of it; the float32 partials are added in rank order through
//     distributed shared memory (the stage buffers, dead by then): no workspace, no second kernel, and
//     the same bits on every run.
// Warps 0-3: accumulator -> shared memory -> sum over the cluster -> y. Warp 4: tensor memory, MMA
// issue. Warp 5: TMA.
// Measured (m 8, bf16): outputs x contraction 6144 x 2048 14.4 us, 8192 x 8192 36.9 us (3.7 TB/s), 32768 x 2048 34.9 us; with 128 rows
// 22.5, 45.1 and 47.1. Where the kernel for large products is quicker: see sm100_skinny_gemm_preferred.
#include "common.cuh"
#include "kernels.cuh"
#include "ptx.cuh"

namespace ember {

namespace {

using namespace ptx;

constexpr int TILE_N = 128;                 // outputs per CTA
constexpr int KB = 64;                      // contraction step
constexpr int W_BYTES = TILE_N * KB * 2, SUB_BYTES = 64 * 128;
constexpr int THREADS = 192;
constexpr int MAX_SPLIT = 8;

template <int MP>
struct Cfg {
    static constexpr int X_BYTES = MP * KB * 2, STAGE_BYTES = W_BYTES + X_BYTES;
    static constexpr int STAGES = MP <= 16 ? 6 : MP <= 32 ? 5 : MP <= 64 ? 4 : 3;  // about 100 KB: two CTAs per SM
    static constexpr int OFF_BAR = STAGES * STAGE_BYTES;  // >= MP * 128 * 4, the float32 partials that reuse the stages
    static constexpr int USED_BYTES = OFF_BAR + 8 * (2 * STAGES + 1) + 16;
    static constexpr int SMEM_BYTES = USED_BYTES + 1024;
    static_assert(OFF_BAR >= MP * TILE_N * 4, "the partial sums reuse the stage buffers");
};

enum { WS_EMPTY = 251, WS_FULL, WS_ACC };

struct SkinnyParams {
    int m, n, k, splits;
    MatView y;
    const __nv_bfloat16 *bias;
    CacheRows cache;  // k null: none
    DeviceStatus *status;
};

__device__ __forceinline__ float ld_cluster_f32(uint32_t addr)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

// TRANS_W = false: w is (k x n), outputs contiguous (forward). true: w is (n x k), the contraction contiguous
// (input gradient, where "n" counts the input features).
// STEP: a projection of a decode step, behind an attention kernel or another layer: the first tiles of w come into L2 while that one ends, and
// results may go into a cache. Layers of a step with weights of their own (batch 2, 2048 wide, 435 positions) 17.4 -> 16.6 us each. Projections that
// follow one another have nothing to wait for, and the prefetches stand before their copies: 26 x 2872 x 9256 19.7 -> 21.9 us, 1 x 6072 x
// 2160 8.4 -> 9.3; the rows' choice of a destination costs them 0.1 to 0.2 us more (140 sizes, 4.5 % in all). They have a form without either.
template <int MP, bool TRANS_W, bool STEP>
__global__ void __launch_bounds__(THREADS) skinny_gemm_kernel(const __grid_constant__ CUtensorMap tm_w,
                                                              const __grid_constant__ CUtensorMap tm_x, const SkinnyParams p)
{
    using C = Cfg<MP>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar0 = smem_base + C::OFF_BAR;
    auto FULL = [&](int s) { return bar0 + 8u * (uint32_t)s; };
    auto EMPTY = [&](int s) { return bar0 + 8u * (uint32_t)(C::STAGES + s); };
    const uint32_t ACC = bar0 + 8u * (2 * C::STAGES);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem_gen + C::OFF_BAR + 8 * (2 * C::STAGES + 1));
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    constexpr int TMEM_COLS = MP < 32 ? 32 : MP;

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int rank = p.splits > 1 ? (int)cluster_ctarank() : 0;
    const int n0 = (blockIdx.x / p.splits) * TILE_N;
    const int kblocks = (p.k + KB - 1) / KB;
    const int kb0 = (int)((long long)kblocks * rank / p.splits), nkb = (int)((long long)kblocks * (rank + 1) / p.splits) - kb0;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < C::STAGES; s++) {
            mbar_init(FULL(s), 1);
            mbar_init(EMPTY(s), 1);
        }
        mbar_init(ACC, 1);
        fence_mbar_init();
    }
    if (warp == 4) {
        tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
        tmem_relinquish();
    }
    if (warp == 5 && lane == 0) {
        prefetch_tensormap(&tm_w);
        prefetch_tensormap(&tm_x);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_launch_dependents();
    if (STEP && warp == 5 && lane == 0)
        for (int i = 0; i < min(nkb, C::STAGES); i++) {
            const int kk = (kb0 + i) * KB;
            tma_prefetch_5d(&tm_w, TRANS_W ? kk : n0, TRANS_W ? n0 : kk, 0, 0, 0);
            if (!TRANS_W) tma_prefetch_5d(&tm_w, n0 + 64, kk, 0, 0, 0);
        }
    pdl_wait();

    if (warp == 5) {
        if (lane == 0) {
            int issued = 0;
            for (int i = 0; i < nkb; i++, issued++) {
                const int s = i % C::STAGES, kk = (kb0 + i) * KB;
                if (!mbar_wait(EMPTY(s), ((i / C::STAGES) & 1) ^ 1, abort_flag, p.status, WS_EMPTY)) break;
                const uint32_t w_dst = smem_base + s * C::STAGE_BYTES, x_dst = w_dst + W_BYTES;
                mbar_arrive_expect_tx(FULL(s), C::STAGE_BYTES);
                if (TRANS_W) {
                    tma_load_5d(w_dst, &tm_w, FULL(s), kk, n0, 0, 0, 0);
                } else {
                    tma_load_5d(w_dst, &tm_w, FULL(s), n0, kk, 0, 0, 0);
                    tma_load_5d(w_dst + SUB_BYTES, &tm_w, FULL(s), n0 + 64, kk, 0, 0, 0);
                }
                tma_load_5d(x_dst, &tm_x, FULL(s), kk, 0, 0, 0, 0);
            }
            // stay until every copy of this CTA has landed (bounded; a copy that was issued completes)
            const long long t0 = clock64();
            for (int i = max(0, issued - C::STAGES); i < issued; i++)
                while (!mbar_try_wait(FULL(i % C::STAGES), (i / C::STAGES) & 1) && clock64() - t0 < kWaitLimitCycles) {}
        }
    } else if (warp == 4) {
        constexpr uint32_t IDESC = idesc_bf16_f32(TILE_N, MP, TRANS_W ? 0 : 1, 0);
        constexpr uint32_t W_LBO = TRANS_W ? 16 : SUB_BYTES, W_STEP = (TRANS_W ? 32 : 2048) >> 4;
        bool ok = true;
        for (int i = 0; i < nkb && ok; i++) {
            const int s = i % C::STAGES;
            ok = mbar_wait(FULL(s), (i / C::STAGES) & 1, abort_flag, p.status, WS_FULL);
            tc_fence_after();
            const uint32_t w_lo = desc_lo(smem_base + s * C::STAGE_BYTES, W_LBO);
            const uint32_t x_lo = desc_lo(smem_base + s * C::STAGE_BYTES + W_BYTES, 16);
#pragma unroll
            for (int k16 = 0; k16 < KB / 16; k16++)
                mma_ss_lo(tmem, w_lo + k16 * W_STEP, x_lo + k16 * 2, IDESC, (i > 0 || k16 > 0) ? 1u : 0u);
            tc_commit_elect(EMPTY(s));
        }
        tc_commit_elect(ACC);
    }
    bool ok = true;
    float *part = reinterpret_cast<float *>(smem_gen);  // [MP rows of x][128 outputs]
    if (warp < 4) {
        ok = mbar_wait(ACC, 0, abort_flag, p.status, WS_ACC);
        tc_fence_after();
        const uint32_t tacc = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll
        for (int c0 = 0; c0 < MP; c0 += 16) {
            uint32_t u[16];
            tmem_ld_32x32b_x16(tacc + c0, u);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (c0 + i < p.m) part[(c0 + i) * TILE_N + threadIdx.x] = __uint_as_float(u[i]);
        }
        tc_fence_before();
    }
    __syncwarp();
    // every CTA's partial sums are in its shared memory (and, within a CTA, all its warps are past their copies)
    if (p.splits > 1) cluster_sync_all(); else __syncthreads();
    if (warp < 4) {
        const int col = n0 + (int)threadIdx.x;
        if (col < p.n && ok) {
            const float b = p.bias ? __bfloat162float(p.bias[col]) : 0.f;
            __nv_bfloat16 *y = (__nv_bfloat16 *)p.y.ptr + view_offset(p.y, 0, col);  // rows and columns of a view address independently
            const bool cached = STEP && p.cache.k && col >= p.cache.from;
            if (cached) {
                const int c = col % p.cache.from;
                y = (__nv_bfloat16 *)(col < 2 * p.cache.from ? p.cache.k : p.cache.v) + ((size_t)(c / p.cache.d) * p.cache.capacity + p.cache.pos) * p.cache.d + c % p.cache.d;
            }
            const size_t cache_step = STEP ? (size_t)p.cache.heads * p.cache.capacity * p.cache.d : 0;
            const uint32_t mine = smem_base + 4u * threadIdx.x;
            uint32_t peer[MAX_SPLIT];
#pragma unroll
            for (int r = 0; r < MAX_SPLIT; r++) peer[r] = r < p.splits && p.splits > 1 ? map_to_cta(mine, r) : 0;
            for (int row = rank; row < p.m; row += p.splits) {  // the cluster's CTAs share the rows
                float s;
                if (p.splits > 1) {
                    float v[MAX_SPLIT];
#pragma unroll
                    for (int r = 0; r < MAX_SPLIT; r++) v[r] = r < p.splits ? ld_cluster_f32(peer[r] + row * TILE_N * 4) : 0.f;
                    s = v[0];
#pragma unroll
                    for (int r = 1; r < MAX_SPLIT; r++) s += v[r];
                } else {
                    s = part[row * TILE_N + threadIdx.x];
                }
                y[cached ? row * cache_step : view_offset(p.y, row, 0)] = __float2bfloat16_rn(s + b);
            }
        }
    }
    tc_fence_before();
    if (p.splits > 1) cluster_sync_all(); else __syncthreads();  // nobody reads this CTA's shared memory any more
    if (warp == 4) tmem_dealloc(tmem, TMEM_COLS);
}

template <int MP, bool TRANS_W, bool STEP = false>
int launch_mp(const GemmArgs &g, DeviceState *st, cudaStream_t s)
{
    using C = Cfg<MP>;
    if constexpr (!TRANS_W && !STEP)
        if (g.cache || g.a.heads) return launch_mp<MP, TRANS_W, true>(g, st, s);  // head-major x: what a step's attention wrote
    MatView x = g.a;
    x.heads = 0;  // head-major rows of sequences of length 1 lie row-major
    CUtensorMap tw, tx;
    int rc;
    if ((rc = make_tensor_map_bf16_view(&tw, g.b, 64, TRANS_W ? TILE_N : KB)) != EMBER_OK) return rc;
    if ((rc = make_tensor_map_bf16_view(&tx, x, KB, MP)) != EMBER_OK) return rc;
    const int sms = st->sm_count > 0 ? st->sm_count : 148;
    const int tiles = (g.n + TILE_N - 1) / TILE_N, kblocks = (g.k + KB - 1) / KB;
    int splits = 1;  // as many CTAs as two per SM hold, each with at least two contraction steps
    // (a GPC's SMs do not divide into clusters of 8 without rest: 36 tiles in 8 parts 9.2 us, in 4 5.9, 8 x 1536 x 4608)
    auto fit = [&](int parts) { return tiles * parts <= (parts == 8 ? 2 * sms * 7 / 8 : 2 * sms); };
    while (splits < MAX_SPLIT && fit(splits * 2) && kblocks >= splits * 4) splits *= 2;
    const CacheRows none = {};
    SkinnyParams p = {(int)g.m, g.n, g.k, splits, g.c, (const __nv_bfloat16 *)g.bias, g.cache ? *g.cache : none, st->status};
    auto kern = skinny_gemm_kernel<MP, TRANS_W, STEP>;
    static SmemOptIn opt_in;
    EMBER_CUDA_TRY(opt_in(kern, C::SMEM_BYTES));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * splits));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = s;
    LaunchAttrs attrs;
    attrs.cluster((unsigned)splits).pdl().set(cfg);
    EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tw, tx, p));
    return EMBER_OK;
}

template <bool TRANS_W>
int launch(const GemmArgs &g, DeviceState *st, cudaStream_t s)
{
    if (g.m <= 16) return launch_mp<16, TRANS_W>(g, st, s);
    if (g.m <= 32) return launch_mp<32, TRANS_W>(g, st, s);
    if (g.m <= 64) return launch_mp<64, TRANS_W>(g, st, s);
    return launch_mp<128, TRANS_W>(g, st, s);
}

}  // namespace

// bf16, at most 128 rows, 16-byte rows of w and x. x may lie head-major only where that is the same as
// row-major (sequences of length 1, a decode step); y may lie any way and at any alignment.
bool sm100_skinny_gemm_supported(const GemmArgs &g)
{
    if (g.dtype != EMBER_BF16 || g.mode == GEMM_TN || g.m <= 0 || g.m > 128 || g.n <= 0 || g.k <= 0) return false;
    if (g.b.heads != 0 || (g.a.heads != 0 && g.a.seq != 1)) return false;
    if (g.a.heads != 0 && g.a.cols != g.a.heads * g.a.dim) return false;  // several parts do not lie side by side
    if (g.a.cols % 8 != 0 || g.b.cols % 8 != 0) return false;
    return (((uintptr_t)g.a.ptr | (uintptr_t)g.b.ptr) & 15) == 0;
}

// Whether a product that both tensor-core kernels take is the quicker here. Up to 32 rows it always is (or level: 64 x 64 10.3 us
// both, 128256 x 2048 108 both). Beyond that the results leave by one thread per output, row after row, while the other
// kernel's tiles fill up, but that one walks the whole contraction in one CTA pair. us, this kernel / the other, outputs x
// contraction: at 48 rows 64 x 64 12 / 10, 16384 x 1024 23 / 20, 32768 x 2048 39 / 41, 128256 x 2048 121 / 109; at 64 rows 2048 x 512 14 / 12,
// 4096 x 1024 14 both, 8192 x 2048 20 both, 6144 x 2048 18 / 20, 1024 x 1024 12 / 14; at 128 rows 1024 x 1024 14 both,
// 2048 x 2048 16 / 18, 4096 x 1024 16 / 14, 6144 x 2048 23 / 20, 2048 x 8192 23 / 43, 8192 x 8192 45 / 51, 50304 x 1024 57 / 37; rows of
// results at odd addresses, at 64 rows 50257 x 1024 84 / 88, 1000001 x 64 303 / 510, at 96 rows 92 / 88, 379 / 513.
bool sm100_skinny_gemm_preferred(const GemmArgs &g)
{
    if (g.m <= 32) return true;
    const bool odd_results = g.n % 8 != 0 || ((uintptr_t)g.c.ptr & 15) != 0;
    if (odd_results && (g.m <= 64 || g.k <= 256)) return true;  // the other stores such rows element by element, too
    return g.k >= 1024 && g.n <= (g.m <= 48 && g.k >= 2048 ? 16LL : g.m <= 64 ? 8LL : 2LL) * g.k;
}

int sm100_skinny_gemm(const GemmArgs &g, DeviceState *st, cudaStream_t s)
{
    return g.mode == GEMM_NT ? launch<true>(g, st, s) : launch<false>(g, st, s);
}

}  // namespace ember
