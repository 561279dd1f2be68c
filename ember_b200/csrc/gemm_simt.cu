// CUDA-core matrix products for the Linear layers: float32 arithmetic, f32 or bf16 storage, any
// shape and any view (row-major or head-major operands). This is the float32 mode of the layers
// (bf16 tensor-core products would use up its 1e-3 tolerance) and the path for shapes the tcgen05
// kernel does not take. Also the column sums that give the bias gradient.
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
//    64 x  64, KG = 4
//    32 x  32, KG = 16  small results: one slab is 128 deep (32 for the shortest contractions), so a contraction of 784 is 7 rounds of loads
//                       instead of the 49 of a 64 x 64 tile with 16-deep steps
// and when even the 32 x 32 tiles leave SMs idle, a cluster of up to 8 blocks splits the contraction and adds
// the partial tiles in rank order through distributed shared memory. The partial sums of the groups are added
// in a fixed order too, so results repeat bit for bit.
// Slabs lie k-major in shared memory; the next one is loaded into registers while this one is multiplied.
using ptx::f32x2;

template <int TM_, int TN_, int KD_>
struct Tile {
    static constexpr int TM = TM_, TN = TN_, KD = KD_;
    static constexpr int GT = (TM / 8) * (TN / 8), KG = 256 / GT, SLAB = KG * KD;  // threads per group, groups, slab depth
    static constexpr int PA = TM + 4, PB = TN + 4;                                   // padded rows of the slabs
    static constexpr int UA = TM * SLAB / 4 / 256, UB = TN * SLAB / 4 / 256;          // 4-element loads per thread and slab
    static constexpr int SLAB_FLOATS = SLAB * (PA + PB);
    static constexpr int PITCH = TN + 4, PART = TM * PITCH;                           // a group's partial tile
    static constexpr int FLOATS = KG > 1 && KG * PART > SLAB_FLOATS ? KG * PART : SLAB_FLOATS;
    static_assert(UA >= 1 && UB >= 1 && GT * KG == 256, "");
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

__device__ __forceinline__ float4 ld_cluster4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

template <typename T, int MODE, bool FA, bool FB, typename C>
__global__ void __launch_bounds__(256, 2) simt_gemm_kernel(const MatView a, const MatView b, const MatView c, const T *bias,
                                                        const long long m, const int n, const int k, const int tiles_n,
                                                        const int splits)
{
    using OA = Operand<T, MODE != GEMM_TN, FA, C::TM>;
    using OB = Operand<T, MODE == GEMM_NT, FB, C::TN>;
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
            OA::coords(threadIdx.x + i * 256, mn, kk);
            ra[i] = OA::load(a, m0 + mn, k0 + kk, m, k);
        }
#pragma unroll
        for (int i = 0; i < C::UB; i++) {
            int mn, kk;
            OB::coords(threadIdx.x + i * 256, mn, kk);
            rb[i] = OB::load(b, n0 + mn, k0 + kk, n, k);
        }
    };
    if (s0 < s1) fetch(s0);
    for (int slab = s0; slab < s1; slab++) {
        if (slab != s0) __syncthreads();
#pragma unroll
        for (int i = 0; i < C::UA; i++) {
            int mn, kk;
            OA::coords(threadIdx.x + i * 256, mn, kk);
            OA::store(as, C::PA, mn, kk, ra[i]);
        }
#pragma unroll
        for (int i = 0; i < C::UB; i++) {
            int mn, kk;
            OB::coords(threadIdx.x + i * 256, mn, kk);
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
    if constexpr (C::KG == 1) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const long long gi = m0 + row_of(i);
            if (gi >= m) continue;
            const size_t row_off = view_offset(c, gi, 0);  // rows and columns of a view address independently
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float v[2];
                ptx::unpack2(acc[i][j], v[0], v[1]);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int gj = n0 + col_of(j) + h;
                    if (gj < n) st(cp, row_off + view_offset(c, 0, gj), v[h] + (bias ? ld(bias, (size_t)gj) : 0.f));
                }
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
        auto store4 = [&](int e, const float4 &s) {
            const long long gi = m0 + e / (C::TN / 4);
            const int gj = n0 + e % (C::TN / 4) * 4;
            if (gi >= m) return;
            const size_t row_off = view_offset(c, gi, 0);
            const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
            for (int h = 0; h < 4; h++)
                if (gj + h < n) st(cp, row_off + view_offset(c, 0, gj + h), v[h] + (bias ? ld(bias, (size_t)(gj + h)) : 0.f));
        };
        auto add4 = [](float4 &s, const float4 &v) {
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        };
        for (int e = threadIdx.x; e < C::TM * C::TN / 4; e += 256) {
            float *p = sm + e / (C::TN / 4) * C::PITCH + e % (C::TN / 4) * 4;
            float4 s = *reinterpret_cast<const float4 *>(p);
#pragma unroll
            for (int g = 1; g < C::KG; g++) add4(s, *reinterpret_cast<const float4 *>(p + g * C::PART));
            if (splits == 1) store4(e, s);
            else *reinterpret_cast<float4 *>(p) = s;  // only this thread reads this place of group 0's tile
        }
        if (splits > 1) {
            // ---- the cluster's tiles, rank 0 first; every block adds its share of the elements
            ptx::cluster_sync_all();
            for (int e = rank * 256 + threadIdx.x; e < C::TM * C::TN / 4; e += splits * 256) {
                const uint32_t at = ptx::smem_u32(sm + e / (C::TN / 4) * C::PITCH + e % (C::TN / 4) * 4);
                float4 s = ld_cluster4(ptx::map_to_cta(at, 0));
                for (int r = 1; r < splits; r++) add4(s, ld_cluster4(ptx::map_to_cta(at, (uint32_t)r)));
                store4(e, s);
            }
            ptx::cluster_sync_all();  // nobody reads this block's shared memory any more
        }
    }
}

// out[j] = sum over the rows of a(:, j). One block owns 32 consecutive columns and all the rows:
// 4 threads read the 32 columns of a row as 8-element vectors (whole 64- or 128-byte segments), 64
// rows at a time; every thread keeps 8 float32 partial sums over the rows it visits (rows t, t + 64,
// ...), and shared memory adds the 64 partials of a column in a fixed order. Needs 8-element groups
// that do not straddle a head (cols, or the head dimension, a multiple of 8) and a 16-byte aligned
// base; other shapes take the element-wise kernel below.
template <typename T>
__global__ void __launch_bounds__(256) column_sum_vec_kernel(MatView a, T *out)
{
    __shared__ float part[64][33];
    const int part_col = (threadIdx.x % 4) * 8, rt = threadIdx.x / 4;
    const int col = blockIdx.x * 32 + part_col;
    const T *ap = (const T *)a.ptr;
    float s[8] = {};
    if (col < a.cols) {
        for (long long r = rt; r < a.rows; r += 64) {
            const T *src = ap + view_offset(a, r, col);
            if constexpr (sizeof(T) == 2) {
                const uint4 v = *reinterpret_cast<const uint4 *>(src);
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    s[2 * i] += __uint_as_float(w[i] << 16);
                    s[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
                }
            } else {
                const float4 v0 = *reinterpret_cast<const float4 *>(src), v1 = *reinterpret_cast<const float4 *>(src + 4);
                s[0] += v0.x; s[1] += v0.y; s[2] += v0.z; s[3] += v0.w;
                s[4] += v1.x; s[5] += v1.y; s[6] += v1.z; s[7] += v1.w;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) part[rt][part_col + i] = s[i];
    __syncthreads();
    if (threadIdx.x < 32) {
        float t = 0.f;
        for (int r = 0; r < 64; r++) t += part[r][threadIdx.x];
        const int c = blockIdx.x * 32 + threadIdx.x;
        if (c < a.cols) st(out, (size_t)c, t);
    }
}

// Element-wise variant for any shape: one warp per column, lane t takes rows t, t + 32, ...
template <typename T>
__global__ void __launch_bounds__(256) column_sum_kernel(MatView a, T *out)
{
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int col = blockIdx.x * 8 + warp;
    if (col >= a.cols) return;
    const T *ap = (const T *)a.ptr;
    float s = 0.f;
    for (long long r = lane; r < a.rows; r += 32) s += ld(ap, view_offset(a, r, col));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) st(out, (size_t)col, s);
}

template <typename T, int MODE, bool FA, bool FB, typename C>
int launch_tile(const GemmArgs &g, int splits, cudaStream_t s)
{
    const long long tiles_m = (g.m + C::TM - 1) / C::TM, tiles_n = (g.n + C::TN - 1) / C::TN;
    if (tiles_m * tiles_n * splits > 0x7fffffffLL) {
        set_error("linear: %lld x %d results are too many for the CUDA-core kernel", g.m, g.n);
        return EMBER_ERR_UNSUPPORTED;
    }
    auto kern = simt_gemm_kernel<T, MODE, FA, FB, C>;
    static SmemOptIn opt_in;
    EMBER_CUDA_TRY(opt_in(kern, C::FLOATS * sizeof(float)));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles_m * tiles_n * splits));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = C::FLOATS * sizeof(float);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = splits > 1 ? 1 : 0;
    EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, g.a, g.b, g.c, (const T *)g.bias, g.m, g.n, g.k, (int)tiles_n, splits));
    return EMBER_OK;
}

template <typename T, int MODE, bool FA, bool FB>
int launch_mode(const GemmArgs &g, int sms, cudaStream_t s)
{
    auto tiles = [&](int t) { return (g.m + t - 1) / t * (long long)((g.n + t - 1) / t); };
    // The largest tile that still gives (nearly) every SM one block.
    if (tiles(128) >= sms) return launch_tile<T, MODE, FA, FB, Tile<128, 128, 16>>(g, 1, s);
    if (4 * tiles(64) >= 3LL * sms) return launch_tile<T, MODE, FA, FB, Tile<64, 64, 8>>(g, 1, s);
    if (g.k <= 64) return launch_tile<T, MODE, FA, FB, Tile<32, 32, 2>>(g, 1, s);  // a slab of 128 would be mostly padding
    // 32 x 32, and the contraction over a cluster while that still leaves every block a slab
    int splits = 1;
    while (splits < 8 && tiles(32) * splits * 2 <= 2LL * sms && g.k > 128LL * splits) splits *= 2;
    return launch_tile<T, MODE, FA, FB, Tile<32, 32, 8>>(g, splits, s);
}

bool view_fast(const MatView &v)  // 4-element float pieces stay inside a row or head, 16-byte aligned
{
    return ((uintptr_t)v.ptr & 15) == 0 && (v.heads ? v.dim % 4 == 0 : v.cols % 4 == 0);
}

template <typename T, int MODE>
int launch_views(const GemmArgs &g, int sms, cudaStream_t s)
{
    if constexpr (sizeof(T) == 4) {
        const bool fa = view_fast(g.a), fb = view_fast(g.b);
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

// Column sums of a large bf16 matrix in two passes, both coalesced: the rows are cut into chunks; a block
// of 8 warps takes 256 columns of one chunk (a warp reads 512 contiguous bytes of a row, lane t its
// columns 8t..8t+7; the offset of a view element splits into a column part, computed once per lane,
// and a row part that is walked without divisions), adds its rows in float32 and writes one partial
// per column; a second kernel adds the partials of a column in a fixed order. The one-pass kernel
// above gives a block only 32 columns, i.e. 64-byte pieces of every row.
__global__ void __launch_bounds__(256) column_partial_kernel(MatView a, float *__restrict__ partial, int rows_per_chunk)
{
    __shared__ float red[8][256];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int col = blockIdx.x * 256 + lane * 8;
    const long long r0 = (long long)blockIdx.y * rows_per_chunk, r1 = min(a.rows, r0 + rows_per_chunk);
    float s[8] = {};
    if (col < a.cols) {
        const __nv_bfloat16 *ap = (const __nv_bfloat16 *)a.ptr;
        const size_t col_off = view_offset(a, 0, col);  // rows and columns of a view address independently
        // row part of the offset: row-major r * cols; head-major (b * heads * seq + l) * dim with r = b * seq + l
        long long r = r0 + warp;
        long long b = a.heads ? r / a.seq : 0;
        int l = a.heads ? (int)(r - b * a.seq) : 0;
#pragma unroll 4
        for (; r < r1; r += 8) {
            const size_t row_off = a.heads ? ((size_t)b * a.heads * a.seq + l) * a.dim : (size_t)r * a.cols;
            const uint4 v = *reinterpret_cast<const uint4 *>(ap + col_off + row_off);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                s[2 * i] += __uint_as_float(w[i] << 16);
                s[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
            }
            if (a.heads) {
                l += 8;
                if (l >= a.seq) { l -= a.seq; b++; }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) red[warp][lane * 8 + i] = s[i];
    __syncthreads();
    const int c = blockIdx.x * 256 + threadIdx.x;
    if (c < a.cols) {
        float t = 0.f;
#pragma unroll
        for (int w8 = 0; w8 < 8; w8++) t += red[w8][threadIdx.x];
        partial[(size_t)blockIdx.y * a.cols + c] = t;
    }
}

__global__ void __launch_bounds__(256) column_final_kernel(const float *__restrict__ partial, __nv_bfloat16 *__restrict__ out, int cols,
                                                           int chunks)
{
    const int c = blockIdx.x * 256 + threadIdx.x;
    if (c >= cols) return;
    float t = 0.f;
    for (int k = 0; k < chunks; k++) t += partial[(size_t)k * cols + c];
    out[c] = __float2bfloat16_rn(t);
}

int column_sums(const MatView &a, void *out, int dtype, cudaStream_t s)
{
    const bool vec = ((uintptr_t)a.ptr & 15) == 0 && (a.heads ? a.dim % 8 == 0 : a.cols % 8 == 0);
    if (vec && dtype == EMBER_BF16 && a.rows >= 4096 && (a.heads == 0 || a.seq % 8 == 0)) {
        const int chunks = 64;
        const int rows_per_chunk = (int)((a.rows + chunks - 1) / chunks + 7) / 8 * 8;
        float *partial = nullptr;
        EMBER_CUDA_TRY(cudaMallocAsync((void **)&partial, (size_t)chunks * a.cols * sizeof(float), s));
        column_partial_kernel<<<dim3((a.cols + 255) / 256, chunks), 256, 0, s>>>(a, partial, rows_per_chunk);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) {
            column_final_kernel<<<(a.cols + 255) / 256, 256, 0, s>>>(partial, (__nv_bfloat16 *)out, a.cols, chunks);
            e = cudaGetLastError();
        }
        cudaFreeAsync(partial, s);
        EMBER_CUDA_TRY(e);
        return EMBER_OK;
    }
    if (vec) {
        const int grid = (a.cols + 31) / 32;
        if (dtype == EMBER_BF16)
            column_sum_vec_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(a, (__nv_bfloat16 *)out);
        else
            column_sum_vec_kernel<float><<<grid, 256, 0, s>>>(a, (float *)out);
    } else {
        const int grid = (a.cols + 7) / 8;
        if (dtype == EMBER_BF16)
            column_sum_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(a, (__nv_bfloat16 *)out);
        else
            column_sum_kernel<float><<<grid, 256, 0, s>>>(a, (float *)out);
    }
    EMBER_CUDA_TRY(cudaGetLastError());
    return EMBER_OK;
}

}  // namespace ember
