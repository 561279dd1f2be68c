// Column sums: the bias gradient, out[j] = sum over the rows of a(:, j). HBM-bound: every element is read
// once and nothing else moves.
//
// One launch for every shape. A block takes a strip of columns 128 bytes wide (element by element: 32
// columns) and a cluster of up to 8 blocks shares the strip's rows, so that a bias of 2048 still gives 256
// blocks their own rows; the partial sums of a cluster are added in rank order through distributed shared
// memory. No workspace, and the same bits on every run. float32 arithmetic.
// Measured with cold caches, against one block per 32 columns (below 4096 rows) and two kernels with a workspace
// (from there): 2048 x 4608 bf16 26 -> 11 us, 2048 x 1536 8 -> 6, 8192 x 6144 30 -> 26, 8192 x 2048 15 -> 11.5.
// Tall matrices of few strips have at most 8 blocks per strip, so their blocks are of 1024 threads: see launch_size.
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "ptx.cuh"

namespace ember {

namespace {

using namespace ptx;

__device__ __forceinline__ float ld_peer_f32(uint32_t addr)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

// VEC: 16-byte pieces that are aligned and stay inside a row or head.
// BESIDE: beside the kernel before it (rules beside pdl_enabled), it reads before it waits. The kernels that wrote `a` are done by then and their
// writes in L2; the fence drops what this SM's L1 may still hold from before them, and nothing writes `a` while this kernel runs. (Loads past
// L1, or relaxed ones, in its place: 1946 x 512 x 1536 backward 18.5 -> 24.5 us, 2468 x 1024 x 3072 45 -> 50; with the fence as without it.)
template <typename T, bool VEC, int NTHR, bool BESIDE>
__global__ void __launch_bounds__(NTHR) column_sum_kernel(const MatView a, T *__restrict__ out, int splits)
{
    constexpr int NV = VEC ? 16 / (int)sizeof(T) : 1;  // columns per load
    constexpr int TX = VEC ? 8 : 32, TY = NTHR / TX;   // threads along a strip's columns, rows per pass
    constexpr int COLS = TX * NV;
    __shared__ float red[TY][COLS + 1];
    __shared__ float total[COLS];
    pdl_launch_dependents();
    if constexpr (BESIDE) __threadfence(); else pdl_wait();
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const int rank = splits > 1 ? (int)cluster_ctarank() : 0;
    const int col = ((int)blockIdx.x / splits) * COLS + tx * NV;
    const long long r0 = a.rows * rank / splits, r1 = a.rows * (rank + 1) / splits;
    float s[NV] = {};
    if (col < a.cols) {
        // rows and columns of a view address independently: offset = column part + row part, and the row
        // part of a head-major view is (b * heads * seq + l) * dim for row b * seq + l
        const T *ap = (const T *)a.ptr + view_offset(a, 0, col);
        long long r = r0 + ty, b = a.heads ? r / a.seq : 0;
        int l = a.heads ? (int)(r - b * a.seq) : 0;
        // Eight loads in flight, also over the last rows (WHOLE: all eight rows exist).
        constexpr int U = 8;
        auto pass = [&](auto whole) {
            constexpr bool WHOLE = decltype(whole)::value;
            uint4 v[U];
            float e[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                v[u] = make_uint4(0u, 0u, 0u, 0u);
                e[u] = 0.f;
                if (WHOLE || r + u * TY < r1) {
                    const T *src = ap + (a.heads ? ((size_t)b * a.heads * a.seq + l) * a.dim : (size_t)(r + u * TY) * a.cols);
                    if constexpr (VEC) v[u] = *reinterpret_cast<const uint4 *>(src);
                    else if constexpr (sizeof(T) == 2) e[u] = __bfloat162float(*src);
                    else e[u] = *src;
                }
                if (a.heads) {
                    l += TY;
                    if (l >= a.seq) {
                        const int over = l / a.seq;
                        b += over;
                        l -= over * a.seq;
                    }
                }
            }
            // a column's eight values are added pairwise: the chain that rounding errors grow along is an eighth as long
#pragma unroll
            for (int i = 0; i < NV; i++) {
                float x[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
                    if constexpr (!VEC) x[u] = e[u];
                    else if constexpr (sizeof(T) == 2) x[u] = __uint_as_float(i % 2 ? w[i / 2] & 0xffff0000u : w[i / 2] << 16);
                    else x[u] = __uint_as_float(w[i]);
                }
                s[i] += ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
            }
        };
        for (; r + (U - 1) * TY < r1; r += U * TY) pass(std::true_type());
        if (r < r1) pass(std::false_type());
    }
#pragma unroll
    for (int i = 0; i < NV; i++) red[ty][tx * NV + i] = s[i];
    __syncthreads();
    const int c = threadIdx.x;
    if (c < COLS) {
        float t = 0.f;
#pragma unroll 4
        for (int y = 0; y < TY; y += 8)
            t += ((red[y][c] + red[y + 1][c]) + (red[y + 2][c] + red[y + 3][c])) + ((red[y + 4][c] + red[y + 5][c]) + (red[y + 6][c] + red[y + 7][c]));
        total[c] = t;
    }
    if (splits > 1) {
        cluster_sync_all();
        if (rank == 0 && c < COLS) {
            float t = total[c];
            for (int p = 1; p < splits; p++) t += ld_peer_f32(map_to_cta(smem_u32(&total[c]), (uint32_t)p));
            total[c] = t;
        }
        cluster_sync_all();  // no block leaves while its partials are being read
    }
    const int oc = ((int)blockIdx.x / splits) * COLS + c;
    if (rank == 0 && c < COLS && oc < a.cols) {
        if constexpr (sizeof(T) == 2) out[oc] = __float2bfloat16_rn(total[c]); else out[oc] = total[c];
    }
    if constexpr (BESIDE) pdl_wait();  // this kernel's end stands for the end of all before it
}

template <typename T, bool VEC>
constexpr int strip_cols() { return VEC ? 128 / (int)sizeof(T) : 32; }

template <typename T, bool VEC, int NTHR>
int launch(const MatView &a, T *out, int sms, cudaStream_t s, bool beside)
{
    constexpr int TY = NTHR / (VEC ? 8 : 32);
    const long long strips = (a.cols + strip_cols<T, VEC>() - 1) / strip_cols<T, VEC>();
    // Up to 8 resident blocks (of 256 threads) per SM; a block keeps at least eight passes over its rows (a cluster costs a
    // microsecond to launch: 256 rows in two blocks 8.2 us, in one 7.2).
    int splits = 1;
    while (splits < 8 && strips * splits * 2 <= 8LL * sms && a.rows >= 16LL * TY * splits) splits *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(strips * splits));
    cfg.blockDim = dim3(NTHR);
    cfg.stream = s;
    LaunchAttrs attrs;
    attrs.cluster((unsigned)splits).pdl().set(cfg);
    EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, beside ? column_sum_kernel<T, VEC, NTHR, true> : column_sum_kernel<T, VEC, NTHR, false>, a, out, splits));
    return EMBER_OK;
}

// With up to 8 blocks for a strip, a tall matrix of few strips leaves most SMs idle and waits on what a block has in
// flight: blocks of 1024 threads while those of 256 would not give every second SM one.
template <typename T, bool VEC>
int launch_size(const MatView &a, T *out, int sms, cudaStream_t s, bool beside)
{
    const long long strips = (a.cols + strip_cols<T, VEC>() - 1) / strip_cols<T, VEC>();
    if (a.rows >= 32768 && strips * 8 * 2 <= sms) return launch<T, VEC, 1024>(a, out, sms, s, beside);
    return launch<T, VEC, 256>(a, out, sms, s, beside);
}

template <typename T>
int launch_any(const MatView &a, T *out, int sms, cudaStream_t s, bool beside)
{
    constexpr int NV = 16 / (int)sizeof(T);
    const bool vec = ((uintptr_t)a.ptr & 15) == 0 && (a.heads ? a.dim % NV == 0 : a.cols % NV == 0);
    return vec ? launch_size<T, true>(a, out, sms, s, beside) : launch_size<T, false>(a, out, sms, s, beside);
}

}  // namespace

int column_sums(const MatView &a, void *out, int dtype, DeviceState *st, cudaStream_t s, bool beside)
{
    const int sms = st->sm_count > 0 ? st->sm_count : 148;
    return dtype == EMBER_BF16 ? launch_any(a, (__nv_bfloat16 *)out, sms, s, beside) : launch_any(a, (float *)out, sms, s, beside);
}

}  // namespace ember
