// Float32 y = x w + b for at most 12 columns (a small classifier's logits): CUDA cores.
//
// Bound: latency. The products of 256 x 784 x 10 are 4 MFLOP on 0.8 MB; as tiles of 32 x 32 with the contraction over clusters
// (gemm_simt.cu) they were 64 blocks, two thirds of whose columns were padding, and rounds through shared memory, cluster barriers and
// strips: 10 us. Here a block owns four rows and its 256 threads share the contraction, four consecutive k each at a time: 16 bytes of
// each row of x and the 4 n floats of w that go with them, which lie side by side. All of a thread's loads are in flight at once, and
// the 4 n sums of a warp are formed by exchanging halves (as many shuffles as there are sums, not five times as many), then added over
// the eight warps in a fixed order.
// us, gemm_simt.cu -> here, call to call (6 is the host): 256 x 784 x 10 9.8 -> 6.0 (the kernel 10.3 -> 3.3), 8192 x 784 x 10 73 -> 19, 8192 x 2048 x 4 126 -> 20,
// 32768 x 2048 x 10 469 -> 103, 8192 x 512 x 2 46 -> 8.
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "ptx.cuh"

namespace ember {

namespace {

using namespace ptx;

constexpr int ROWS = 4;

template <int N>
__global__ void __launch_bounds__(256) narrow_f32_kernel(const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ bias,
                                                         float *__restrict__ y, int m, int k)
{
    __shared__ float part[8][ROWS * N];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, row0 = blockIdx.x * ROWS;
    float v[ROWS * N];
#pragma unroll
    for (int i = 0; i < ROWS * N; i++) v[i] = 0.f;
    for (int kk = threadIdx.x * 4; kk < k; kk += 1024) {
        float4 xv[ROWS], wv[N];
#pragma unroll
        for (int r = 0; r < ROWS; r++) xv[r] = *reinterpret_cast<const float4 *>(x + (size_t)min(row0 + r, m - 1) * k + kk);  // past the end: not stored
#pragma unroll
        for (int i = 0; i < N; i++) wv[i] = reinterpret_cast<const float4 *>(w + (size_t)kk * N)[i];
        const float *wf = reinterpret_cast<const float *>(wv);
#pragma unroll
        for (int r = 0; r < ROWS; r++)
#pragma unroll
            for (int c = 0; c < N; c++) {
                float s = xv[r].x * wf[c];
                s = fmaf(xv[r].y, wf[N + c], s);
                s = fmaf(xv[r].z, wf[2 * N + c], s);
                v[r * N + c] += fmaf(xv[r].w, wf[3 * N + c], s);
            }
    }
    // A lane keeps one half of its sums, [first, end), and gives the other away, five times. Lengths are rounded up: places past `end` hold nothing.
    constexpr int V0 = ROWS * N, V1 = (V0 + 1) / 2, V2 = (V1 + 1) / 2, V3 = (V2 + 1) / 2, V4 = (V3 + 1) / 2, V5 = (V4 + 1) / 2;
    int first = 0, end = V0;
    auto step = [&](auto count, int o) {
        constexpr int V = decltype(count)::value, H = (V + 1) / 2;
        const bool upper = lane & o;
#pragma unroll
        for (int i = 0; i < H; i++) {
            const float a = v[i], b = i + H < V ? v[i + H] : 0.f;
            v[i] = (upper ? b : a) + __shfl_xor_sync(0xffffffffu, upper ? a : b, o);
        }
        if (upper) first += H; else end = min(end, first + H);
    };
    step(std::integral_constant<int, V0>(), 16);
    step(std::integral_constant<int, V1>(), 8);
    step(std::integral_constant<int, V2>(), 4);
    step(std::integral_constant<int, V3>(), 2);
    step(std::integral_constant<int, V4>(), 1);
#pragma unroll
    for (int i = 0; i < V5; i++)
        if (first + i < end) part[warp][first + i] = v[i];
    __syncthreads();
    const int e = threadIdx.x, row = row0 + e / N;
    if (e < V0 && row < m) {
        const float s = ((part[0][e] + part[1][e]) + (part[2][e] + part[3][e])) + ((part[4][e] + part[5][e]) + (part[6][e] + part[7][e]));
        y[(size_t)row * N + e % N] = s + (bias ? bias[e % N] : 0.f);
    }
}

template <int N>
int launch(const GemmArgs &g, cudaStream_t s)
{
    if constexpr (N > 12) {
        return EMBER_ERR_UNSUPPORTED;
    } else {
        if (g.n != N) return launch<N + 1>(g, s);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)((g.m + ROWS - 1) / ROWS));
        cfg.blockDim = dim3(256);
        cfg.stream = s;
        LaunchAttrs attrs;
        if (cfg.gridDim.x <= (unsigned)kPdlMaxGrid) attrs.pdl();
        attrs.set(cfg);
        EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, narrow_f32_kernel<N>, (const float *)g.a.ptr, (const float *)g.b.ptr, (const float *)g.bias,
                                          (float *)g.c.ptr, (int)g.m, g.k));
        return EMBER_OK;
    }
}

// The backward of such a layer in one launch: grad_w = x^T grad_y and, with it, grad_b in the first `sum_blocks` blocks, grad_x = grad_y w^T in the others.
//
// Bound: latency again at a few hundred rows (three launches, of which the weight gradient's contraction over the rows was a chain of tiles on
// 25 blocks: 13 us for 784 x 256 x 10), the bytes of x and grad_x at thousands. A lane has four columns of x or grad_x, a warp 128 of them, so
// that every access of a row is 512 bytes in one piece; the N values of grad_y that go with a row are the same for the whole warp. The rows
// of a weight gradient are shared by a cluster of up to eight blocks of eight warps, whose sums are added in a fixed order: no atomics.
template <int N>
__device__ __forceinline__ void load_row(const float *p, float (&v)[N])
{
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N / 4; i++) {
            const float4 f = reinterpret_cast<const float4 *>(p)[i];
            v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
        }
    } else if constexpr (N % 2 == 0) {
#pragma unroll
        for (int i = 0; i < N / 2; i++) {
            const float2 f = reinterpret_cast<const float2 *>(p)[i];
            v[2 * i] = f.x; v[2 * i + 1] = f.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; i++) v[i] = p[i];
    }
}

struct NarrowBwd {
    const float *x, *w, *dy;
    float *dx, *dw, *db;  // dx, db: may be NULL
    int m, k, tiles;      // tiles of 128 columns
    int cluster;          // blocks that share the rows of a tile
    int sum_blocks, chunk_rows;
};

// what lies at `mine` in the shared memory of another block of the cluster
__device__ __forceinline__ float ld_cluster(const float *mine, int rank)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(map_to_cta(smem_u32(mine), rank)) : "memory");
    return v;
}
__device__ __forceinline__ double ld_cluster(const double *mine, int rank)
{
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(map_to_cta(smem_u32(mine), rank)) : "memory");
    return v;
}

// Two blocks an SM: 12 columns would take 167 registers and leave one (8055 x 2056 x 12 82 -> 50 us, 200 x 116552 x 12 193 -> 123).
template <int N>
__global__ void __launch_bounds__(256, 2) narrow_f32_bwd_kernel(const NarrowBwd p)
{
    extern __shared__ float red[];     // [8][N][128]: the warps' sums
    __shared__ float total[N * 128];   // the block's: [N][128]
    __shared__ double total_b[N], red_b[8][N];  // grad_b: a few sums of m values, in 64 bits for what that costs
    constexpr int U = 4;               // rows of a warp in flight
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    if ((int)blockIdx.x >= p.sum_blocks) {
        // ---------------------------------------------------------------- grad_x
        const int b = blockIdx.x - p.sum_blocks, tile = b % p.tiles, col = tile * 128 + lane * 4;
        const int r0 = b / p.tiles * p.chunk_rows, r1 = min(p.m, r0 + p.chunk_rows);
        if (r0 < p.m && col < p.k) {
            float wv[4 * N];
#pragma unroll
            for (int i = 0; i < N; i++) {
                const float4 f = reinterpret_cast<const float4 *>(p.w + (size_t)col * N)[i];
                wv[4 * i] = f.x; wv[4 * i + 1] = f.y; wv[4 * i + 2] = f.z; wv[4 * i + 3] = f.w;
            }
            for (int r = r0 + warp * U; r < r1; r += 8 * U) {
                float g[U][N];
#pragma unroll
                for (int u = 0; u < U; u++) load_row<N>(p.dy + (size_t)min(r + u, p.m - 1) * N, g[u]);
#pragma unroll
                for (int u = 0; u < U; u++) {
                    float o[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        // Above four columns in two sums, of every other column: one chain is off by more than the tiles' sums were
                        // (256 x 784 x 10 5.5e-8 of the norm as tiles, 6.0e-8 in one chain, 5.2e-8 in two; 64 x 784 x 12 5.8, 6.4, 5.5).
                        constexpr int CHAINS = N > 4 ? 2 : 1;
                        float s[CHAINS];
#pragma unroll
                        for (int c = 0; c < N; c++) s[c % CHAINS] = c < CHAINS ? g[u][c] * wv[j * N + c] : fmaf(g[u][c], wv[j * N + c], s[c % CHAINS]);
                        o[j] = CHAINS == 2 ? s[0] + s[CHAINS - 1] : s[0];
                    }
                    if (r + u < r1) *reinterpret_cast<float4 *>(p.dx + (size_t)(r + u) * p.k + col) = make_float4(o[0], o[1], o[2], o[3]);
                }
            }
        }
        return;  // (its cluster, if any, is of such blocks alone)
    }
    // -------------------------------------------------------------------- grad_w, grad_b
    const int rank = p.cluster > 1 ? (int)cluster_ctarank() : 0, tile = blockIdx.x / p.cluster, col = tile * 128 + lane * 4;
    const int r0 = (int)((long long)p.m * rank / p.cluster), r1 = (int)((long long)p.m * (rank + 1) / p.cluster);
    const bool sum_b = p.db && tile == 0;
    float acc[N][4] = {};
    double acc_b = 0.;
    for (int r = r0 + warp * U; r < r1; r += 8 * U) {
        float4 xv[U];
        float g[U][N];
#pragma unroll
        for (int u = 0; u < U; u++) {
            xv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r + u < r1 && col < p.k) xv[u] = *reinterpret_cast<const float4 *>(p.x + (size_t)(r + u) * p.k + col);
        }
#pragma unroll
        for (int u = 0; u < U; u++) load_row<N>(p.dy + (size_t)min(r + u, r1 - 1) * N, g[u]);
        float gb[U] = {};
        if (sum_b && lane < N) {
#pragma unroll
            for (int u = 0; u < U; u++)
                if (r + u < r1) gb[u] = p.dy[(size_t)(r + u) * N + lane];
        }
        if (sum_b) acc_b += ((double)gb[0] + gb[1]) + ((double)gb[2] + gb[3]);
#pragma unroll
        for (int u = 1; u < U; u++)
            if (r + u >= r1) {  // another row's values, which could be infinite
#pragma unroll
                for (int c = 0; c < N; c++) g[u][c] = 0.f;
            }
        // Four products are added up before they meet the sums: a chain of m / (32 cluster) additions instead of m / (8 cluster)
        // (8192 x 784 x 10, eight blocks: grad_w 1.3e-7 of its norm off; row by row 2.2e-7, gemm_simt.cu 1.7e-7). Wide layers, whose blocks have all
        // rows, have the longest: 16384 x 40000 x 8, 512 additions, 4.1e-7, gemm_simt.cu 2.3e-6; 1024 x 200000 x 10 1.2e-7 and 5.8e-7.
#pragma unroll
        for (int c = 0; c < N; c++) {
            acc[c][0] += fmaf(xv[3].x, g[3][c], fmaf(xv[2].x, g[2][c], fmaf(xv[1].x, g[1][c], xv[0].x * g[0][c])));
            acc[c][1] += fmaf(xv[3].y, g[3][c], fmaf(xv[2].y, g[2][c], fmaf(xv[1].y, g[1][c], xv[0].y * g[0][c])));
            acc[c][2] += fmaf(xv[3].z, g[3][c], fmaf(xv[2].z, g[2][c], fmaf(xv[1].z, g[1][c], xv[0].z * g[0][c])));
            acc[c][3] += fmaf(xv[3].w, g[3][c], fmaf(xv[2].w, g[2][c], fmaf(xv[1].w, g[1][c], xv[0].w * g[0][c])));
        }
    }
#pragma unroll
    for (int c = 0; c < N; c++) *reinterpret_cast<float4 *>(red + (warp * N + c) * 128 + lane * 4) = make_float4(acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
    if (sum_b && lane < N) red_b[warp][lane] = acc_b;
    __syncthreads();
    for (int e = threadIdx.x; e < N * 128; e += 256) {
        const float *a = red + e;
        constexpr int W = N * 128;
        total[e] = ((a[0] + a[W]) + (a[2 * W] + a[3 * W])) + ((a[4 * W] + a[5 * W]) + (a[6 * W] + a[7 * W]));
    }
    if (sum_b && threadIdx.x < N) {
        const int e = threadIdx.x;
        total_b[e] = ((red_b[0][e] + red_b[1][e]) + (red_b[2][e] + red_b[3][e])) + ((red_b[4][e] + red_b[5][e]) + (red_b[6][e] + red_b[7][e]));
    }
    if (p.cluster > 1) cluster_sync_all(); else __syncthreads();
    // element e of the tile's 128 x N results, as they lie in memory; a block of the cluster has every cluster-th run of 256
    for (int e = rank * 256 + threadIdx.x; e < 128 * N; e += p.cluster * 256) {
        const int j = e / N, c = e - j * N;
        if (tile * 128 + j >= p.k) break;
        float v = 0.f;
        for (int q = 0; q < p.cluster; q++) v += p.cluster > 1 ? ld_cluster(total + c * 128 + j, q) : total[c * 128 + j];
        p.dw[(size_t)tile * 128 * N + e] = v;
    }
    if (sum_b && rank == 0 && threadIdx.x < N) {
        double v = 0.;
        for (int q = 0; q < p.cluster; q++) v += p.cluster > 1 ? ld_cluster(total_b + threadIdx.x, q) : total_b[threadIdx.x];
        p.db[threadIdx.x] = (float)v;
    }
    if (p.cluster > 1) cluster_sync_all();  // no block leaves while another may read its sums
}

template <int N>
int launch_bwd(NarrowBwd p, int n, DeviceState *st, cudaStream_t s)
{
    if constexpr (N > 12) {
        return EMBER_ERR_UNSUPPORTED;
    } else {
        if (n != N) return launch_bwd<N + 1>(p, n, st, s);
        p.tiles = (p.k + 127) / 128;
        p.cluster = 1;
        // At least 32 rows each, four for a warp, and only until there are two blocks an SM: with few rows a block's end (its warps' sums added up, two
        // waits for the cluster) is most of its time (always up to eight / this: 362 x 12152 x 8 26.9 / 19.5 us, 282 x 29424 x 10 40.7 / 17.0, 800 x 149512 x 4 256 / 185).
        while (p.cluster < 8 && p.m >= p.cluster * 64 && p.tiles * p.cluster < 2 * st->sm_count) p.cluster *= 2;
        p.sum_blocks = p.tiles * p.cluster;
        long long blocks = p.sum_blocks;
        if (p.dx) {
            const int chunks = max(1, min((p.m + 31) / 32, 4 * st->sm_count / p.tiles));
            p.chunk_rows = ((p.m + chunks - 1) / chunks + 31) / 32 * 32;
            blocks += (long long)p.tiles * ((p.m + p.chunk_rows - 1) / p.chunk_rows);
        }
        blocks = (blocks + p.cluster - 1) / p.cluster * p.cluster;
        const int smem = 8 * N * 128 * (int)sizeof(float);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)blocks);
        cfg.blockDim = dim3(256);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        auto kern = narrow_f32_bwd_kernel<N>;
        static SmemOptIn opt_in;
        EMBER_CUDA_TRY(opt_in(kern, smem));
        LaunchAttrs attrs;
        attrs.cluster(p.cluster);
        if (cfg.gridDim.x <= (unsigned)kPdlMaxGrid) attrs.pdl();
        attrs.set(cfg);
        EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, p));
        return EMBER_OK;
    }
}

}  // namespace

bool narrow_f32_bwd_supported(const void *x, const void *w, const void *dy, const void *dx, const void *db, long long m, int n, int k)
{
    if (n > 12 || k % 4 != 0 || k > 0x7fffffff - 1024 || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)dy | (uintptr_t)dx) & 15) != 0) return false;
    // us, the kernels that took these calls before (gemm_simt.cu, from some sizes on gemm_f32_sm100.cu, column_sums.cu) / here, calls back to back in
    // a graph, grad_x, grad_w and grad_b: 256 x 784 x 10 14.8 / 5.7, 32 x 64 x 10 8.3 / 3.7, 1000 x 512 x 12 15.4 / 10, 8192 x 784 x 10 68 / 33,
    // 8192 x 2048 x 10 136 / 46; over 500 sizes (1 to 16384 rows, contractions of 4 to 2048) 0.44 of the time,
    // over 200 with contractions to 262144 (up to 2^27 elements of x) 0.43.
    // At most eight blocks share the rows of 128 columns, which is too few for tall matrices: 32768 x 784 x 10 231 / 213, 68047 x 536 x 11 420 / 444,
    // 122465 x 308 x 8 395 / 949; with 8 and 12 columns, which tiles move in pieces of 16 bytes, from 4097 rows on if they are also narrow (9277 x 8 x 12
    // 28 / 34, 14721 x 200 x 8 36 / 37.5). A weight gradient of 12 columns alone is quicker as tiles (95 x 220 4.1 / 5.2, 1576 x 156 7.7 / 9.3).
    // Few rows and a wide weight gradient without grad_x, with the same columns: a block then has little but its end to do (6 x 145280 x 8 8.2 / 10.1,
    // 12 x 167224 x 12 14.3 / 15.8).
    if (m > 16384 || ((n == 8 || n == 12) && (m > 4096 && k < 512 || m <= 16 && k > 32768 && !dx))) return false;
    return n != 12 || dx || db;
}

int narrow_f32_backward(const void *x, const void *w, const void *dy, void *dx, void *dw, void *db, long long m, int n, int k, DeviceState *st, cudaStream_t s)
{
    NarrowBwd p = {};
    p.x = (const float *)x;
    p.w = (const float *)w;
    p.dy = (const float *)dy;
    p.dx = (float *)dx;
    p.dw = (float *)dw;
    p.db = (float *)db;
    p.m = (int)m;
    p.k = k;
    return launch_bwd<1>(p, n, st, s);
}

bool narrow_f32_supported(const GemmArgs &g)
{
    if (g.dtype != EMBER_F32 || g.mode != GEMM_NN || g.m <= 0 || g.n <= 0 || g.n > 12 || g.k <= 0 || g.k % 4 != 0) return false;
    if (g.a.heads != 0 || g.b.heads != 0 || g.c.heads != 0 || (((uintptr_t)g.a.ptr | (uintptr_t)g.b.ptr) & 15) != 0) return false;
    if (g.m > 0x7ffffff0LL || g.k > 0x7fffffff - 1024) return false;  // the kernel counts in ints, 1024 at a time
    // us, the kernels that took these calls before (gemm_simt.cu, from some sizes on gemm_f32_sm100.cu) / here, calls back to back in a graph.
    // Few rows and long contractions stay here, although a block's contraction is a chain and there are only m / 4 blocks: 17 x 4096 x 10
    // 19.4 / 6.4, 17 x 65536 x 10 232 / 56, 1 x 65536 x 12 91 / 87, 1 x 262144 x 12 350 / 340, 256 x 65536 x 4 155 / 84.
    // Short contractions leave most of a block's threads without work: with more rows than two blocks an SM take at once the tiles are quicker
    // (2048 x 16 x 7 3.6 / 3.9, x 9 3.7 / 4.4, x 64 x 12 3.7 / 4.3; 1536 x 16 x 7 3.5 / 2.8, 2048 x 64 x 10 4.8 / 3.6; 8192 x 64 x 10 10.2 / 9.9, 65536 x 64 x 9 27 / 88).
    const bool slow = g.n == 8 || g.n == 9 || g.n == 12;  // tiles move 8 and 12 columns in pieces of 16 bytes; the sums of 9 divide unevenly among lanes
    if (g.m <= 1184) return true;
    if (g.m <= 2048) return g.k >= (g.n == 12 ? 96 : slow || g.n == 11 || (g.n >= 6 && g.n != 10 && g.m > 1536) ? 64 : 0);
    if (g.k < 256) return false;
    // 8 and 12 columns while the tiles that gemm_simt.cu takes by then fill the SMs: 6000 rows x 256 9.9 / 10.3 and 9.9 / 11, x 372 x 12 12.1 / 12.9, 16384 x 256 19 / 24 both, x 384
    // 26.6 / 27.5; on either side 3072 x 256 7.8 / 6.5, 8192 x 256 18 / 13, 12000 x 320 23 / 19.5, 18900 x 256 31 / 27, 32768 x 256 55 / 45.
    if (g.n == 8 || g.n == 12) {
        if (g.m >= 4096 && g.m <= 7040) return g.k >= 384;
        if (g.m > 13500 && g.m <= 147 * 128) return g.k >= (g.m > 15500 ? 512 : 320);
    }
    // Very tall: 61000 x 256 x 8 and 12 1.22, x 448 1.1 times as long here, 262144 x 660 x 8 1.17 (65536 x 768 x 8 197 / 172); other
    // widths 383000 x 256 x 4 1.22, x 6 1.37, x 10 1.2, x 11 1.46, x 320 1.02 to 1.24, from 384 on level or quicker here (65536 x 256 x 4 69 / 43, x 10 86 / 72).
    if (slow && g.m > 55000) return g.k >= 768;
    if (g.n >= 4 && g.m > 84000) return g.k >= 384;
    return true;  // from 13 columns on the registers hold fewer blocks (4096 x 784 x 16: 15.8 / 21.3)
}

int narrow_f32_gemm(const GemmArgs &g, cudaStream_t s) { return launch<1>(g, s); }

}  // namespace ember
