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
    // Short contractions leave most of a block's threads without work: with many rows the tiles are quicker (8192 rows, 64 x 9: 10.3 us there, 15.5
    // here; 128 x 9: 15.9 and 16.4; 256 x 10: 27 and 14). From 13 columns on the registers hold fewer blocks (4096 x 784 x 16: 15.8 and 21.3).
    return g.m <= 0x7ffffff0LL && (g.k >= 256 || g.m <= 2048);
}

int narrow_f32_gemm(const GemmArgs &g, cudaStream_t s) { return launch<1>(g, s); }

}  // namespace ember
