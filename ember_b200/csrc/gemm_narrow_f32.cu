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

}  // namespace

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
