// CUDA-core matrix products for the Linear layers: float32 arithmetic, f32 or bf16 storage, any
// shape and any view (row-major or head-major operands): small float32 products, float32 values that the tensor-core
// kernel's planes (gemm_f32_sm100.cu) cannot hold, and shapes that the tcgen05 kernels do not take.
#include "common.cuh"
#include "kernels.cuh"
#include "ptx.cuh"

namespace ember {

namespace {

__device__ __forceinline__ float ld(const float *p, size_t i) { return p[i]; }
__device__ __forceinline__ float ld(const __nv_bfloat16 *p, size_t i) { return __bfloat162float(p[i]); }
__device__ __forceinline__ void st(float *p, size_t i, float v) { p[i] = v; }
__device__ __forceinline__ void st(__nv_bfloat16 *p, size_t i, float v) { p[i] = __float2bfloat16_rn(v); }

// Matrix products on the FMA pipe. A block owns a TM x TN tile of the result and walks the contraction in
// slabs of KG * KD; its 256 threads are KG groups, each of which multiplies its own KD rows of every slab
// over the whole tile, 8 x 8 results per thread: 2 + 2 shared-memory loads of 16 bytes for 32 packed FMAs.
//   128 x 128, KG = 1   enough tiles to fill the SMs
//    64 x  64, KG = 1   64 threads: many tiles of a short contraction, or along a narrow result
//    64 x  64, KG = 4
//    32 x  32, KG = 16  small results: one slab is 128 deep (32 for the shortest contractions), so a contraction of 784 is 7 rounds of loads
//                       instead of the 49 of a 64 x 64 tile with 16-deep steps
// and when even the 32 x 32 tiles leave SMs idle, a cluster of up to 8 blocks splits the contraction and adds
// the partial tiles in rank order through distributed shared memory. The partial sums of the groups are added
// in a fixed order too, so results repeat bit for bit.
// A product of a short contraction is bound by its stores. Results are stored four columns at a time where their addresses
// allow, otherwise the tile goes through shared memory and neighbouring threads store neighbouring columns (f32, k 8: 2048 x 2048
// 10.6 -> 5.3 us, k 4: 4096 x 4097 35 -> 23, against the four columns of a thread one after the other).
// Slabs lie k-major in shared memory; the next one is loaded into registers while this one is multiplied.
using ptx::f32x2;

template <int TM_, int TN_, int KD_, int NT_ = 256>
struct Tile {
    static constexpr int TM = TM_, TN = TN_, KD = KD_, NT = NT_;
    static constexpr int GT = (TM / 8) * (TN / 8), KG = NT / GT, SLAB = KG * KD;   // threads per group, groups, slab depth
    static constexpr int PA = TM + 4, PB = TN + 4;                                   // padded rows of the slabs
    static constexpr int UA = TM * SLAB / 4 / NT, UB = TN * SLAB / 4 / NT;            // 4-element loads per thread and slab
    static constexpr int SLAB_FLOATS = SLAB * (PA + PB);
    static constexpr int PITCH = TN + 4, PART = TM * PITCH;                           // a group's partial tile
    static constexpr int STORE_FLOATS = KG > 1 ? KG * PART : 32 * PITCH;              // what the results pass through
    static constexpr int FLOATS = STORE_FLOATS > SLAB_FLOATS ? STORE_FLOATS : SLAB_FLOATS;
    static_assert(UA >= 1 && UB >= 1 && GT * KG == NT, "");
};

// One 4-element load of an operand. KC: the contraction runs along memory (rows of the view are tile rows);
// otherwise the tile's rows do. FAST: float32, 16-byte pieces that lie inside a row or head and are aligned.
template <typename T, bool KC, bool FAST, int EXT>
struct Operand {
    static __device__ __forceinline__ void coords(int u, int &mn, int &kk)
    {
        if constexpr (KC) {
            mn = u % EXT;
            kk = u / EXT * 4;
        } else {
            mn = u % (EXT / 4) * 4;
            kk = u / (EXT / 4);
        }
    }
    static __device__ __forceinline__ float4 load(const MatView &v, long long mn, int kk, long long mn_end, int k_end)
    {
        const T *p = (const T *)v.ptr;
        const long long row = KC ? mn : kk, row_end = KC ? mn_end : k_end;
        const long long col = KC ? kk : mn, col_end = KC ? k_end : mn_end;
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row >= row_end) return r;
        if constexpr (FAST) {
            if (col < col_end) r = *reinterpret_cast<const float4 *>(p + view_offset(v, row, (int)col));
        } else {
            if (col < col_end) r.x = ld(p, view_offset(v, row, (int)col));
            if (col + 1 < col_end) r.y = ld(p, view_offset(v, row, (int)col + 1));
            if (col + 2 < col_end) r.z = ld(p, view_offset(v, row, (int)col + 2));
            if (col + 3 < col_end) r.w = ld(p, view_offset(v, row, (int)col + 3));
        }
        return r;
    }
    static __device__ __forceinline__ void store(float *slab, int pitch, int mn, int kk, const float4 &r)
    {
        if constexpr (KC) {
            slab[kk * pitch + mn] = r.x;
            slab[(kk + 1) * pitch + mn] = r.y;
            slab[(kk + 2) * pitch + mn] = r.z;
            slab[(kk + 3) * pitch + mn] = r.w;
        } else {
            *reinterpret_cast<float4 *>(slab + kk * pitch + mn) = r;
        }
    }
};

__device__ __forceinline__ void st4(float *p, const float (&v)[4]) { *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void st4(__nv_bfloat16 *p, const float (&v)[4])
{
    *reinterpret_cast<uint2 *>(p) = make_uint2(ptx::pack_bf16(v[0], v[1]), ptx::pack_bf16(v[2], v[3]));
}

// CV: results are stored four columns at a time, else neighbouring columns by neighbouring threads.
template <typename T, int MODE, bool FA, bool FB, bool CV, typename C>
__global__ void __launch_bounds__(C::NT, 512 / C::NT) simt_gemm_kernel(const MatView a, const MatView b, const MatView c, const T *bias,
                                                        const long long m, const int n, const int k, const int tiles_n,
                                                        const int splits, const int *only_if)
{
    using OA = Operand<T, MODE != GEMM_TN, FA, C::TM>;
    using OB = Operand<T, MODE == GEMM_NT, FB, C::TN>;
    ptx::pdl_launch_dependents();
    ptx::pdl_wait();
    if (only_if && *only_if == 0) return;  // the tensor-core kernel before this one did the work
    extern __shared__ __align__(16) float sm[];
    float *as = sm, *bs = sm + C::SLAB * C::PA;
    const int rank = splits > 1 ? (int)ptx::cluster_ctarank() : 0;
    const int tile = blockIdx.x / splits;
    const long long m0 = (long long)(tile / tiles_n) * C::TM;
    const int n0 = (tile % tiles_n) * C::TN;
    const int slabs = (k + C::SLAB - 1) / C::SLAB;
    const int s0 = (int)((long long)slabs * rank / splits), s1 = (int)((long long)slabs * (rank + 1) / splits);
    const int group = threadIdx.x / C::GT, t = threadIdx.x % C::GT;
    const int tx = t % (C::TN / 8), ty = t / (C::TN / 8);

    f32x2 acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0;
    float4 ra[C::UA], rb[C::UB];
    auto fetch = [&](int slab) {
        const int k0 = slab * C::SLAB;
#pragma unroll
        for (int i = 0; i < C::UA; i++) {
            int mn, kk;
            OA::coords(threadIdx.x + i * C::NT, mn, kk);
            ra[i] = OA::load(a, m0 + mn, k0 + kk, m, k);
        }
#pragma unroll
        for (int i = 0; i < C::UB; i++) {
            int mn, kk;
            OB::coords(threadIdx.x + i * C::NT, mn, kk);
            rb[i] = OB::load(b, n0 + mn, k0 + kk, n, k);
        }
    };
    if (s0 < s1) fetch(s0);
    for (int slab = s0; slab < s1; slab++) {
        if (slab != s0) __syncthreads();
#pragma unroll
        for (int i = 0; i < C::UA; i++) {
            int mn, kk;
            OA::coords(threadIdx.x + i * C::NT, mn, kk);
            OA::store(as, C::PA, mn, kk, ra[i]);
        }
#pragma unroll
        for (int i = 0; i < C::UB; i++) {
            int mn, kk;
            OB::coords(threadIdx.x + i * C::NT, mn, kk);
            OB::store(bs, C::PB, mn, kk, rb[i]);
        }
        __syncthreads();
        if (slab + 1 < s1) fetch(slab + 1);
        const float *ga = as + group * C::KD * C::PA + ty * 4, *gb = bs + group * C::KD * C::PB + tx * 4;
#pragma unroll
        for (int kk = 0; kk < C::KD; kk++) {
            // rows ty*4 + {0..3} and TM/2 + the same, columns likewise: 16-byte loads, no bank conflicts
            const float4 a0 = *reinterpret_cast<const float4 *>(ga + kk * C::PA), a1 = *reinterpret_cast<const float4 *>(ga + kk * C::PA + C::TM / 2);
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2 *>(gb + kk * C::PB), b1 = *reinterpret_cast<const ulonglong2 *>(gb + kk * C::PB + C::TN / 2);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const f32x2 bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const f32x2 aa = ptx::pack2(av[i], av[i]);
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = ptx::fma2(aa, bv[j], acc[i][j]);
            }
        }
    }
    auto row_of = [&](int i) { return (i / 4) * (C::TM / 2) + ty * 4 + i % 4; };
    auto col_of = [&](int j) { return (j / 2) * (C::TN / 2) + tx * 4 + (j % 2) * 2; };

    T *cp = (T *)c.ptr;
    // Columns gj .. gj + 3 of result row gi, which lie side by side, aligned to their size (CV).
    auto store4 = [&](long long gi, int gj, float4 s) {
        if (gi >= m || gj >= n) return;
        float v[4] = {s.x, s.y, s.z, s.w};
        if (bias) {
#pragma unroll
            for (int h = 0; h < 4; h++) v[h] += ld(bias, (size_t)(gj + h));
        }
        st4(cp + view_offset(c, gi, gj), v);
    };
    auto store1 = [&](long long gi, int gj, float s) {
        if (gi < m && gj < n) st(cp, view_offset(c, gi, gj), s + (bias ? ld(bias, (size_t)gj) : 0.f));
    };
    if constexpr (C::KG == 1) {
        if constexpr (CV) {
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                    float4 v;
                    ptx::unpack2(acc[i][j], v.x, v.y);
                    ptx::unpack2(acc[i][j + 1], v.z, v.w);
                    store4(m0 + row_of(i), n0 + col_of(j), v);
                }
        } else {
            // 32 rows at a time, in the slabs' memory: those of half the threads' first or last four rows
            constexpr int Q = C::TM / 64;  // rounds of 32 rows per half of the tile
#pragma unroll
            for (int q = 0; q < 2 * Q; q++) {
                __syncthreads();
                if (ty / 8 == q % Q) {
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            *reinterpret_cast<f32x2 *>(sm + ((ty % 8) * 4 + i) * C::PITCH + col_of(j)) = acc[(q / Q) * 4 + i][j];
                }
                __syncthreads();
                for (int e = threadIdx.x; e < 32 * C::TN; e += C::NT)
                    store1(m0 + q * 32 + e / C::TN, n0 + e % C::TN, sm[e / C::TN * C::PITCH + e % C::TN]);
            }
        }
    } else {
        // Every group leaves its partial tile in shared memory; then all 256 threads add them, group 0 first.
        __syncthreads();
        float *mine = sm + group * C::PART;
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) *reinterpret_cast<f32x2 *>(mine + row_of(i) * C::PITCH + col_of(j)) = acc[i][j];
        __syncthreads();
        auto add4 = [](float4 &s, const float4 &v) {
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        };
        auto store = [&](int e, const float4 &s) {
            const int row = e / (C::TN / 4), col = e % (C::TN / 4) * 4;
            if constexpr (CV) {
                store4(m0 + row, n0 + col, s);
                return;
            }
            if (m0 + row >= m) return;
            const size_t row_off = view_offset(c, m0 + row, 0);  // rows and columns of a view address independently
            const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const int gj = n0 + col + h;
                if (gj < n) st(cp, row_off + view_offset(c, 0, gj), v[h] + (bias ? ld(bias, (size_t)gj) : 0.f));
            }
        };
        for (int e = threadIdx.x; e < C::TM * C::TN / 4; e += 256) {
            float *p = sm + e / (C::TN / 4) * C::PITCH + e % (C::TN / 4) * 4;
            float4 s = *reinterpret_cast<const float4 *>(p);
#pragma unroll
            for (int g = 1; g < C::KG; g++) add4(s, *reinterpret_cast<const float4 *>(p + g * C::PART));
            if (splits == 1) store(e, s);
            else *reinterpret_cast<float4 *>(p) = s;  // only this thread reads this place of group 0's tile
        }
        if (splits > 1) {
            // ---- the cluster's tiles, rank 0 first; every block adds its share of the elements
            ptx::cluster_sync_all();
            for (int e = rank * 256 + threadIdx.x; e < C::TM * C::TN / 4; e += splits * 256) {
                const uint32_t at = ptx::smem_u32(sm + e / (C::TN / 4) * C::PITCH + e % (C::TN / 4) * 4);
                float4 s = ptx::ld_cluster4(ptx::map_to_cta(at, 0));
                for (int r = 1; r < splits; r++) add4(s, ptx::ld_cluster4(ptx::map_to_cta(at, (uint32_t)r)));
                store(e, s);
            }
            ptx::cluster_sync_all();  // nobody reads this block's shared memory any more
        }
    }
}

bool view_fast(const MatView &v, size_t align)  // pieces of 4 elements stay inside a row or head, and their addresses are aligned
{
    return ((uintptr_t)v.ptr & (align - 1)) == 0 && (v.heads ? v.dim % 4 == 0 : v.cols % 4 == 0);
}

template <typename T, int MODE, bool FA, bool FB, bool CV, typename C>
int launch_store(const GemmArgs &g, int splits, cudaStream_t s)
{
    const long long tiles_m = (g.m + C::TM - 1) / C::TM, tiles_n = (g.n + C::TN - 1) / C::TN;
    if (tiles_m * tiles_n * splits > 0x7fffffffLL) {
        set_error("linear: %lld x %d results are too many for the CUDA-core kernel", g.m, g.n);
        return EMBER_ERR_UNSUPPORTED;
    }
    auto kern = simt_gemm_kernel<T, MODE, FA, FB, CV, C>;
    static SmemOptIn opt_in;
    EMBER_CUDA_TRY(opt_in(kern, C::FLOATS * sizeof(float)));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles_m * tiles_n * splits));
    cfg.blockDim = dim3(C::NT);
    cfg.dynamicSmemBytes = C::FLOATS * sizeof(float);
    cfg.stream = s;
    LaunchAttrs attrs;
    attrs.cluster((unsigned)splits);
    if (cfg.gridDim.x <= (unsigned)kPdlMaxGrid) attrs.pdl();
    attrs.set(cfg);
    EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, g.a, g.b, g.c, (const T *)g.bias, g.m, g.n, g.k, (int)tiles_n, splits, g.only_if));
    return EMBER_OK;
}

// A kernel of its own for each kind of store (with both in one its main loop spills, 4 % at 2048^3); float32 operands that are not
// fast to load have one kernel, whose stores are coalesced all the same.
template <typename T, int MODE, bool FA, bool FB, typename C>
int launch_tile(const GemmArgs &g, int splits, cudaStream_t s)
{
    if constexpr (sizeof(T) == 2 || (FA && FB))
        if (view_fast(g.c, 4 * sizeof(T))) return launch_store<T, MODE, FA, FB, true, C>(g, splits, s);
    return launch_store<T, MODE, FA, FB, false, C>(g, splits, s);
}

template <typename T, int MODE, bool FA, bool FB>
int launch_mode(const GemmArgs &g, int sms, cudaStream_t s)
{
    auto tiles = [&](int t) { return (g.m + t - 1) / t * (long long)((g.n + t - 1) / t); };
    // Short contractions are bound by the start and the end of a block, and a narrow side would leave half of a larger tile
    // empty: small blocks, eight to an SM. us, tiles of 128 -> these: f32 65536 x 64, contraction 64: 29 -> 21; 100000 x 10, 64: 59 ->
    // 37; bf16 10^6 x 64, 10: 187 -> 123; 4096 x 4097, 4: 49 -> 31; but 65536 x 96, 31: 33 -> 44.
    if (tiles(64) >= 4LL * sms && (g.k <= 16 || g.m <= 64 || g.n <= 64)) return launch_tile<T, MODE, FA, FB, Tile<64, 64, 8, 64>>(g, 1, s);
    // The largest tile that still gives (nearly) every SM one block.
    if (tiles(128) >= sms) return launch_tile<T, MODE, FA, FB, Tile<128, 128, 16>>(g, 1, s);
    if (4 * tiles(64) >= 3LL * sms) return launch_tile<T, MODE, FA, FB, Tile<64, 64, 8>>(g, 1, s);
    if (g.k <= 64) return launch_tile<T, MODE, FA, FB, Tile<32, 32, 2>>(g, 1, s);  // a slab of 128 would be mostly padding
    // 32 x 32, and the contraction over a cluster while that still leaves every block a slab
    int splits = 1;
    while (splits < 8 && tiles(32) * splits * 2 <= 2LL * sms && g.k > 128LL * splits) splits *= 2;
    return launch_tile<T, MODE, FA, FB, Tile<32, 32, 8>>(g, splits, s);
}

template <typename T, int MODE>
int launch_views(const GemmArgs &g, int sms, cudaStream_t s)
{
    if constexpr (sizeof(T) == 4) {
        const bool fa = view_fast(g.a, 16), fb = view_fast(g.b, 16);
        if (fa && fb) return launch_mode<T, MODE, true, true>(g, sms, s);
        if (fa) return launch_mode<T, MODE, true, false>(g, sms, s);
        if (fb) return launch_mode<T, MODE, false, true>(g, sms, s);
    }
    return launch_mode<T, MODE, false, false>(g, sms, s);
}

template <typename T>
int launch_gemm(const GemmArgs &g, int sms, cudaStream_t s)
{
    if (g.mode == GEMM_NN) return launch_views<T, GEMM_NN>(g, sms, s);
    if (g.mode == GEMM_NT) return launch_views<T, GEMM_NT>(g, sms, s);
    return launch_views<T, GEMM_TN>(g, sms, s);
}

}  // namespace

int simt_gemm(const GemmArgs &g, DeviceState *st, cudaStream_t s)
{
    const int sms = st->sm_count > 0 ? st->sm_count : 148;
    return g.dtype == EMBER_BF16 ? launch_gemm<__nv_bfloat16>(g, sms, s) : launch_gemm<float>(g, sms, s);
}

}  // namespace ember
