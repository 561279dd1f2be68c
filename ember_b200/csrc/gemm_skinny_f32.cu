// Float32 y = x w + b for at most 16 rows of x (a decode step's projections): CUDA cores, w streamed once.
//
// Bound: the bytes of w (2048 x 16384, 134 MB: 4.8 TB/s with 1 row, 3.9 with 8), from there on the shared-memory reads of x. The tiles of gemm_simt.cu load
// a slab of w and a slab of x, meet at a barrier and multiply, which left the memory idle for most of a round. Here a thread owns
// 4 columns of all rows and reads its rows of w straight into registers, the next ones while it multiplies; x lies transposed in shared
// memory, from where a step's rows are broadcast. 256 threads are 16 column groups x 16 contraction groups; a cluster of up to
// 8 blocks splits the contraction, and partial sums are added in a fixed order (through shared memory, then the cluster's).
// us, gemm_simt.cu -> here, 1 / 8 / 16 rows, call to call: 512 x 1536 7 / 7 / 8 -> 6 / 6 / 7; 1024 x 3072 15 / 15 / 16 -> 9 / 11 / 15; 2048 x 6144
// 42 / 43 / 46 -> 17 / 20 / 28; 2048 x 16384 110 / 111 / 112 -> 28 / 34 / 55. A form for 32 rows (2 columns a thread) took 13 to 14 where the
// tiles take 8 (512 x 1536) and 52 against 55 (2048 x 6144), four wavefronts of x for each of its reads, and was left out.
#include "common.cuh"
#include "kernels.cuh"
#include "ptx.cuh"

namespace ember {

namespace {

using namespace ptx;

constexpr int KG = 16;

struct SkinnyF32 {
    const float *x, *w, *bias;
    MatView y;
    int m, n, k, splits;
    int x_vec;  // rows of x in 16-byte pieces
};

template <int MR>
struct SkinnyCfg {
    static constexpr int PITCH = MR + 4;                       // floats of a row of x^T
    static constexpr int CPT = 4, COLS = 16 * CPT;             // columns of a thread, of a block
    static constexpr int U = MR <= 8 ? 8 : 4;                  // rows of w in flight per thread and round
    static constexpr int PART = 8 * MR * COLS;                // floats: a partial result per warp
    static __host__ __device__ int padded(int k_block) { return (k_block + U * KG - 1) / (U * KG) * (U * KG); }
    static size_t smem(int k_block) { return (size_t)(padded(k_block) * PITCH > PART ? padded(k_block) * PITCH : PART) * 4; }
};

template <int MR>
__global__ void __launch_bounds__(256, 2) skinny_f32_kernel(const SkinnyF32 p)
{
    using C = SkinnyCfg<MR>;
    constexpr int CPT = C::CPT, COLS = C::COLS;
    extern __shared__ __align__(16) float sm[];
    pdl_launch_dependents();
    pdl_wait();
    const int rank = p.splits > 1 ? (int)cluster_ctarank() : 0, strip = blockIdx.x / p.splits;
    const int k0 = (int)((long long)p.k * rank / p.splits) & ~3, k1 = rank + 1 == p.splits ? p.k : (int)((long long)p.k * (rank + 1) / p.splits) & ~3, kn = k1 - k0;
    const int pad = C::padded(kn);
    const int tx = threadIdx.x % 16, kg = threadIdx.x / 16, col = strip * COLS + tx * CPT;
    const bool have = col < p.n;  // n is a multiple of 4
    const float *w = p.w + (size_t)k0 * p.n + (have ? col : 0);

    // the first rows of w are on their way while x is laid out
    float4 cur[C::U], nxt[C::U];
    auto fetch = [&](float4 (&v)[C::U], int base) {
#pragma unroll
        for (int u = 0; u < C::U; u++) {
            const int kk = base + u * KG + kg;
            v[u] = kk < kn && have ? __ldcs(reinterpret_cast<const float4 *>(w + (size_t)kk * p.n)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    fetch(cur, 0);
    if (p.x_vec) {  // parts start at multiples of 4
#pragma unroll 4
        for (int i = threadIdx.x; i < MR * (kn / 4); i += 256) {
            const int r = i % MR, kk = i / MR * 4;
            const float4 v = r < p.m ? *reinterpret_cast<const float4 *>(p.x + (size_t)r * p.k + k0 + kk) : make_float4(0.f, 0.f, 0.f, 0.f);
            float *to = sm + kk * C::PITCH + r;
            to[0] = v.x; to[C::PITCH] = v.y; to[2 * C::PITCH] = v.z; to[3 * C::PITCH] = v.w;
        }
    } else {
        for (int i = threadIdx.x; i < MR * kn; i += 256) {
            const int r = i % MR, kk = i / MR;
            sm[kk * C::PITCH + r] = r < p.m ? p.x[(size_t)r * p.k + k0 + kk] : 0.f;
        }
    }
    // a round multiplies whole steps: zeros past the end
    for (int i = threadIdx.x; i < (pad - kn) * C::PITCH; i += 256) sm[kn * C::PITCH + i] = 0.f;
    __syncthreads();
    // packed along the rows: a pair of rows of x^T is read as it lies
    f32x2 acc[MR / 2][CPT];
#pragma unroll
    for (int r = 0; r < MR / 2; r++)
#pragma unroll
        for (int c = 0; c < CPT; c++) acc[r][c] = 0;
    for (int base = 0; base < kn; base += C::U * KG) {
        if (base + C::U * KG < kn) fetch(nxt, base + C::U * KG);
#pragma unroll
        for (int u = 0; u < C::U; u++) {
            f32x2 wv[CPT];
            wv[0] = pack2(cur[u].x, cur[u].x);
            wv[1] = pack2(cur[u].y, cur[u].y);
            wv[2] = pack2(cur[u].z, cur[u].z);
            wv[3] = pack2(cur[u].w, cur[u].w);
            const ulonglong2 *xr = reinterpret_cast<const ulonglong2 *>(sm + (base + u * KG + kg) * C::PITCH);
#pragma unroll
            for (int r4 = 0; r4 < MR / 4; r4++) {
                const ulonglong2 v = xr[r4];
#pragma unroll
                for (int c = 0; c < CPT; c++) acc[r4 * 2][c] = fma2(v.x, wv[c], acc[r4 * 2][c]);
#pragma unroll
                for (int c = 0; c < CPT; c++) acc[r4 * 2 + 1][c] = fma2(v.y, wv[c], acc[r4 * 2 + 1][c]);
            }
        }
#pragma unroll
        for (int u = 0; u < C::U; u++) cur[u] = nxt[u];
    }
    __syncthreads();  // x has been read
    // ---- the two contraction groups of a warp, then the warps
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
#pragma unroll
    for (int r = 0; r < MR; r += 2) {
        float lo[CPT], hi[CPT];
#pragma unroll
        for (int c = 0; c < CPT; c++) {
            unpack2(acc[r / 2][c], lo[c], hi[c]);
            lo[c] += __shfl_xor_sync(0xffffffffu, lo[c], 16);
            hi[c] += __shfl_xor_sync(0xffffffffu, hi[c], 16);
        }
        if (lane < 16) {
            float *at = sm + (warp * MR + r) * COLS + lane * CPT;
            *reinterpret_cast<float4 *>(at) = make_float4(lo[0], lo[1], lo[2], lo[3]);
            *reinterpret_cast<float4 *>(at + COLS) = make_float4(hi[0], hi[1], hi[2], hi[3]);
        }
    }
    __syncthreads();
    auto add = [](float4 &s, const float4 &v) { s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w; };
    auto store = [&](int e, float4 v) {
        const int r = e / (COLS / 4), c = strip * COLS + e % (COLS / 4) * 4;
        if (r >= p.m || c >= p.n) return;
        if (p.bias) add(v, make_float4(p.bias[c], p.bias[c + 1], p.bias[c + 2], p.bias[c + 3]));
        *reinterpret_cast<float4 *>((float *)p.y.ptr + view_offset(p.y, r, c)) = v;
    };
    for (int e = threadIdx.x; e < MR * COLS / 4; e += 256) {
        float *at = sm + e * 4;
        float4 v = *reinterpret_cast<const float4 *>(at);
#pragma unroll
        for (int g = 1; g < 8; g++) add(v, *reinterpret_cast<const float4 *>(at + g * MR * COLS));
        if (p.splits == 1) store(e, v);
        else *reinterpret_cast<float4 *>(at) = v;  // only this thread reads this place of warp 0's part
    }
    if (p.splits > 1) {
        cluster_sync_all();
        for (int e = rank * 256 + threadIdx.x; e < MR * COLS / 4; e += p.splits * 256) {
            const uint32_t at = smem_u32(sm + e * 4);
            float4 v = ld_cluster4(map_to_cta(at, 0));
            for (int r = 1; r < p.splits; r++) add(v, ld_cluster4(map_to_cta(at, (uint32_t)r)));
            store(e, v);
        }
        cluster_sync_all();  // nobody reads this block's shared memory any more
    }
}

bool plain_rows(const MatView &v) { return v.heads == 0 || (v.seq == 1 && v.cols == v.heads * v.dim); }

template <int MR>
int launch(const GemmArgs &g, int sms, cudaStream_t s)
{
    SkinnyF32 p = {(const float *)g.a.ptr, (const float *)g.b.ptr, (const float *)g.bias, g.c, (int)g.m, g.n, g.k, 1, g.k % 4 == 0 && ((uintptr_t)g.a.ptr & 15) == 0};
    constexpr int COLS = SkinnyCfg<MR>::COLS;
    const int strips = (g.n + COLS - 1) / COLS;
    // parts of the contraction: until two blocks per SM are there, while a part keeps 128, or 64 as long as SMs are without a
    // block (512 x 4096, 1 / 8 / 16 rows: 8 parts of 64 8 / 9.5 / 11.4 us, 4 of 128 4.3 / 5.1 / 6.9), and what a block keeps of x fits
    while (p.splits < 8 && (long long)strips * p.splits < ((g.k >= 256 * p.splits) ? 2LL * sms : (long long)sms) && g.k >= 128 * p.splits) p.splits *= 2;
    while (p.splits < 8 && SkinnyCfg<MR>::smem((g.k + p.splits - 1) / p.splits + 4) > 96 * 1024) p.splits *= 2;
    const size_t smem = SkinnyCfg<MR>::smem((g.k + p.splits - 1) / p.splits + 4);
    auto kern = skinny_f32_kernel<MR>;
    static SmemOptIn opt_in;
    EMBER_CUDA_TRY(opt_in(kern, 200 * 1024));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(strips * p.splits));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    LaunchAttrs attrs;
    attrs.cluster((unsigned)p.splits);
    if (cfg.gridDim.x <= (unsigned)kPdlMaxGrid) attrs.pdl();
    attrs.set(cfg);
    EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, p));
    return EMBER_OK;
}

}  // namespace

bool skinny_f32_supported(const GemmArgs &g)
{
    if (g.dtype != EMBER_F32 || g.mode != GEMM_NN || g.m <= 0 || g.m > 16 || g.n < 64 || g.n % 4 != 0 || g.k < 64) return false;
    if (g.k > 8 * 1024 || g.n > 0x7ffffe00 / 8) return false;  // 8 parts of x in shared memory; blocks of a launch
    if (!plain_rows(g.a) || g.b.heads != 0 || (((uintptr_t)g.b.ptr | (uintptr_t)g.c.ptr) & 15) != 0) return false;
    // Above 8 rows a round is 64 of the contraction: one that ends early in its second round does the work of 128 (16 x 100 x 512: 3.8 us
    // against 3.5 of gemm_simt.cu; 2048 columns 3.8 against 4.0).
    if (g.m > 8 && g.k > 64 && g.k < 128 && g.n < 2048) return false;
    return g.c.heads == 0 || g.c.dim % 4 == 0;  // stores of 4 columns stay inside a head
}

int skinny_f32_gemm(const GemmArgs &g, DeviceState *st, cudaStream_t s)
{
    const int sms = st->sm_count > 0 ? st->sm_count : 148;
    if (g.m <= 4) return launch<4>(g, sms, s);
    if (g.m <= 8) return launch<8>(g, sms, s);
    return launch<16>(g, sms, s);
}

}  // namespace ember
