// Attention on the CUDA cores: float32 arithmetic throughout, float32 or bf16 storage, any head
// dimension up to 128, any sequence lengths. These kernels serve small float32 calls, float32 values that the tensor-core
// kernels (attn_f32_sm100.cu) cannot hold, and the bf16 shapes that the tcgen05 kernels do not take.
//
// Bound: the float32 FMA pipe (128 per clock and SM). A product of two 64-row tiles over 64 columns is
// 2048 SM clocks of it, so everything is arranged to keep operands coming at that rate:
//   - every multiply-add is packed (fma.rn.f32x2, one issue slot per two), which leaves the other issue
//     slots to the shared-memory loads. A score product A B^T pairs the CONTRACTION index: both tiles
//     stay in their natural row-major layout, a thread reads 4 columns of a row as one 16-byte load and
//     accumulates even and odd columns apart (added at the end). A product P V pairs the output columns.
//   - a thread owns R rows x 4 columns of the score tile and R rows x DPAD/16 columns of an output tile
//     (128 threads: 8 row groups x 16 column groups). R = 8 costs 12 shared-memory loads per 64 packed
//     FMAs (16 wavefronts in 32 clocks of a scheduler's FMA time), R = 4 costs 8 per 32 (12 in 16), R = 2
//     is bound by those loads and only serves launches that cannot fill the SMs otherwise.
//   - tiles are swizzled: the 16-byte chunk c of row r lies at chunk c ^ ((r / 4) % 8), which keeps
//     the three ways a tile is read (rows of a thread, rows tx*4+c across the lanes, one row across the
//     lanes) free of bank conflicts without padding, and is one XOR per 4 columns.
//   - tiles arrive by cp.async, K while the previous tile's softmax and PV run, V while its scores are
//     formed; several blocks per SM hide what is left of the latency.
// The score tile is passed from the score product to the PV product through shared memory, but only
// between the 16 threads that share its rows: a __syncwarp, no block barrier.
#include <math.h>

#include "common.cuh"
#include "kernels.cuh"
#include "ptx.cuh"

namespace ember {

namespace {

using ptx::f32x2;
using ptx::fma2;
using ptx::pack2;
using ptx::unpack2;

constexpr int NT = 128;  // 8 row groups (ty) x 16 column groups (tx)
constexpr int TN = 64;   // columns of a score tile (4 per thread)
constexpr float LOG2E_S = 1.4426950408889634f;

// e^x of the forward. Scores, maxima and log-sum-exps stay in natural units and only their differences are scaled by
// log2(e): scaled beforehand, a score or a log-sum-exp of the size of 7 is rounded at 5e-7, which every weight of its
// row then carries, and a finite score above 2.3e38 overflows. What the approximation has in common for a row cancels in
// the forward's division by the sum; the backward has no such division and uses expf (1 to 2 % of its time).
// Errors against float64, relative 2-norm, 8 units x 64 x 2000, d 40: log-sum-exp 4.3e-8 -> 2.6e-8, dv 3.5e-7 -> 2.8e-7 (3.4e-7
// with this function), dk 3.8e-7 -> 3.1e-7. 16 units x L1024 D64 causal: forward 97 us both, backward 218 -> 222 us.
__device__ __forceinline__ float exp_nat(float x) { return ptx::ex2(x * LOG2E_S); }

template <typename T>
__device__ __forceinline__ float ld(const T *p)
{
    if constexpr (sizeof(T) == 4)
        return *p;
    else
        return __bfloat162float(*p);
}
template <typename T>
__device__ __forceinline__ void st(T *p, float v)
{
    if constexpr (sizeof(T) == 4)
        *p = v;
    else
        *p = __float2bfloat16_rn(v);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Byte offset of row r, chunk 0 of a swizzled tile of `row_bytes` rows; XOR with (chunk << 4).
__device__ __forceinline__ int row_off(int r, int row_bytes) { return r * row_bytes + (((r >> 2) & 7) << 4); }

// Rows [row0, row0 + ROWS) x columns [0, d) of a (nrows x d) matrix into a swizzled [ROWS][DPAD] float
// tile; rows past nrows and columns past d are zero. FAST: float32 rows of whole 16-byte chunks.
template <typename T, bool FAST, int DPAD, int ROWS>
__device__ __forceinline__ void load_tile(char *tile, const T *src, int row0, int nrows, int d)
{
    constexpr int CH = DPAD / 4;
    for (int idx = threadIdx.x; idx < ROWS * CH; idx += NT) {
        const int r = idx / CH, c = idx % CH;
        const bool row_ok = row0 + r < nrows;
        char *dst = tile + (row_off(r, DPAD * 4) ^ (c << 4));
        if constexpr (FAST) {
            const bool ok = row_ok && c * 4 < d;
            cp_async16(ptx::smem_u32(dst), ok ? (const void *)(src + (size_t)(row0 + r) * d + c * 4) : (const void *)src, ok);
        } else {
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; i++)
                v[i] = row_ok && c * 4 + i < d ? ld(src + (size_t)(row0 + r) * d + c * 4 + i) : 0.f;
            *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
}

// acc[r][c] = sum over columns of A[ty*R+r][:] * B[tx*4+c][:], nch chunks of 4 columns.
template <int R, int DPAD>
__device__ __forceinline__ void mm_abt(float (&acc)[R][4], const char *A, const char *B, int nch, int ty, int tx)
{
    constexpr int RB = DPAD * 4;
    f32x2 s[R][4];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) s[r][c] = 0;
    constexpr int G = (R + 3) / 4;  // groups of rows that share a swizzle
    int a_off[G];
#pragma unroll
    for (int g = 0; g < G; g++) a_off[g] = row_off(ty * R + g * 4, RB);
    const int b_off = row_off(tx * 4, RB);
#pragma unroll 2
    for (int j = 0; j < nch; j++) {
        const int jo = j << 4;
        ulonglong2 b[4];
#pragma unroll
        for (int c = 0; c < 4; c++) b[c] = *reinterpret_cast<const ulonglong2 *>(B + (b_off ^ jo) + c * RB);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(A + (a_off[r / 4] ^ jo) + (r % 4) * RB);
#pragma unroll
            for (int c = 0; c < 4; c++) s[r][c] = fma2(a.x, b[c].x, s[r][c]);
#pragma unroll
            for (int c = 0; c < 4; c++) s[r][c] = fma2(a.y, b[c].y, s[r][c]);
        }
    }
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            float lo, hi;
            unpack2(s[r][c], lo, hi);
            acc[r][c] = lo + hi;
        }
}

// The columns of an output row a thread owns, as NP packed pairs: chunks tx + 16 h (DPAD = 64, 128) or
// half a chunk (DPAD = 32).
template <int DPAD>
struct Cols {
    static constexpr int NP = DPAD / 32;
    static __device__ __forceinline__ int first(int tx, int pair)  // first column of a pair
    {
        return DPAD == 32 ? tx * 2 : tx * 4 + (pair / 2) * 64 + (pair % 2) * 2;
    }
    static __device__ __forceinline__ void load(f32x2 (&v)[NP], const char *row, int swz, int tx)
    {
        if constexpr (DPAD == 32) {
            v[0] = *reinterpret_cast<const f32x2 *>(row + (((tx >> 1) << 4) ^ swz) + (tx & 1) * 8);
        } else {
#pragma unroll
            for (int h = 0; h < DPAD / 64; h++) {
                const ulonglong2 u = *reinterpret_cast<const ulonglong2 *>(row + ((tx << 4) ^ swz) + h * 256);
                v[2 * h] = u.x;
                v[2 * h + 1] = u.y;
            }
        }
    }
};

// acc[r][:] += sum over k < TN of P[ty*R+r][k] * V[k][:]; P is [rows][64] swizzled, V [64][DPAD] swizzled.
template <int R, int DPAD>
__device__ __forceinline__ void mm_pv(f32x2 (&acc)[R][Cols<DPAD>::NP], const char *P, const char *V, int ty, int tx)
{
    constexpr int NP = Cols<DPAD>::NP, RB = DPAD * 4, G = (R + 3) / 4;
    int p_off[G];
#pragma unroll
    for (int g = 0; g < G; g++) p_off[g] = row_off(ty * R + g * 4, TN * 4);
#pragma unroll 2
    for (int jk = 0; jk < TN / 4; jk++) {
        float4 p[R];
#pragma unroll
        for (int r = 0; r < R; r++) p[r] = *reinterpret_cast<const float4 *>(P + (p_off[r / 4] ^ (jk << 4)) + (r % 4) * (TN * 4));
#pragma unroll
        for (int i = 0; i < 4; i++) {
            f32x2 v[NP];
            Cols<DPAD>::load(v, V + (jk * 4 + i) * RB, (jk & 7) << 4, tx);
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float pv = i == 0 ? p[r].x : i == 1 ? p[r].y : i == 2 ? p[r].z : p[r].w;
                const f32x2 pp = pack2(pv, pv);
#pragma unroll
                for (int n = 0; n < NP; n++) acc[r][n] = fma2(pp, v[n], acc[r][n]);
            }
        }
    }
}

template <int R>
__device__ __forceinline__ void store_p(char *P, const float (&s)[R][4], int ty, int tx)
{
#pragma unroll
    for (int r = 0; r < R; r++)
        *reinterpret_cast<float4 *>(P + (row_off(ty * R + r, TN * 4) ^ (tx << 4))) = make_float4(s[r][0], s[r][1], s[r][2], s[r][3]);
}

// Row `row` of an (nrows x d) result, this thread's columns, scaled.
template <typename T, bool FAST, int DPAD>
__device__ __forceinline__ void store_row(T *dst, const f32x2 (&v)[Cols<DPAD>::NP], float scale, int d, int tx)
{
    if constexpr (FAST && DPAD >= 64) {
#pragma unroll
        for (int h = 0; h < DPAD / 64; h++) {
            const int c = Cols<DPAD>::first(tx, 2 * h);
            float a, b, e, f;
            unpack2(v[2 * h], a, b);
            unpack2(v[2 * h + 1], e, f);
            if (c < d) *reinterpret_cast<float4 *>(dst + c) = make_float4(a * scale, b * scale, e * scale, f * scale);
        }
    } else {
#pragma unroll
        for (int n = 0; n < Cols<DPAD>::NP; n++) {
            const int c = Cols<DPAD>::first(tx, n);
            float a, b;
            unpack2(v[n], a, b);
            if (c < d) st(dst + c, a * scale);
            if (c + 1 < d) st(dst + c + 1, b * scale);
        }
    }
}

// Behind a tensor-core kernel these kernels are launched programmatically, to leave at once if it did the work (*only_if is 0).
__device__ __forceinline__ bool not_needed(const int *only_if)
{
    if (!only_if) return false;
    ptx::pdl_launch_dependents();
    ptx::pdl_wait();
    return *only_if == 0;
}

// Plain order otherwise: with blocks that wait on every SM 16 units x L1024 took 385 us instead of 305, forward and backward.
template <typename P>
int launch_simt(void (*kern)(P), long long grid, size_t smem, cudaStream_t s, const P &p)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    LaunchAttrs attrs;
    if (p.only_if) attrs.pdl();
    attrs.set(cfg);
    EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, p));
    return EMBER_OK;
}

struct SimtFwd {
    const void *q, *k, *v;
    void *out;
    float *lse;
    int bh, lq, lk, d, causal, blocks;
    float scale;
    const int *only_if;
};

template <typename T, bool FAST, int DPAD, int R>
__global__ void __launch_bounds__(NT) simt_fwd_kernel(const SimtFwd p)
{
    if (not_needed(p.only_if)) return;
    constexpr int BM = 8 * R, NP = Cols<DPAD>::NP;
    extern __shared__ __align__(1024) char smem[];
    char *Qs = smem, *Ks = Qs + BM * DPAD * 4, *Vs = Ks + TN * DPAD * 4, *Ps = Vs + TN * DPAD * 4;
    // blocks of all units, the heaviest (last, under a causal mask) query blocks first
    const int unit = blockIdx.x % p.bh, blk = p.blocks - 1 - blockIdx.x / p.bh;
    const int q0 = blk * BM, off = p.lk - p.lq, d = p.d;
    const int ty = threadIdx.x / 16, tx = threadIdx.x % 16, nch = (d + 3) / 4;
    const T *q = (const T *)p.q + (size_t)unit * p.lq * d, *k = (const T *)p.k + (size_t)unit * p.lk * d,
            *v = (const T *)p.v + (size_t)unit * p.lk * d;
    const int kend = p.causal ? min(p.lk, q0 + BM + off) : p.lk;  // keys visible to the last row of this block

    load_tile<T, FAST, DPAD, BM>(Qs, q, q0, p.lq, d);
    load_tile<T, FAST, DPAD, TN>(Ks, k, 0, p.lk, d);
    cp_commit();

    float m[R], l[R];
    f32x2 o[R][NP];
#pragma unroll
    for (int r = 0; r < R; r++) {
        m[r] = -INFINITY;
        l[r] = 0.f;
#pragma unroll
        for (int n = 0; n < NP; n++) o[r][n] = 0;
    }
    for (int k0 = 0; k0 < kend; k0 += TN) {
        cp_wait<0>();
        __syncthreads();  // K(k0) is here; the previous tile's V has been read by every thread
        load_tile<T, FAST, DPAD, TN>(Vs, v, k0, p.lk, d);
        cp_commit();
        float s[R][4];
        mm_abt<R, DPAD>(s, Qs, Ks, nch, ty, tx);
        __syncthreads();  // K(k0) has been read
        if (k0 + TN < kend) load_tile<T, FAST, DPAD, TN>(Ks, k, k0 + TN, p.lk, d);
        cp_commit();
        const bool edge = k0 + TN - 1 > (p.causal ? min(p.lk - 1, q0 + off) : p.lk - 1);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int row = q0 + ty * R + r, limit = p.causal ? min(p.lk - 1, row + off) : p.lk - 1;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                s[r][c] *= p.scale;
                if (edge && k0 + tx * 4 + c > limit) s[r][c] = -INFINITY;
            }
            float mx = fmaxf(fmaxf(s[r][0], s[r][1]), fmaxf(s[r][2], s[r][3]));
#pragma unroll
            for (int t = 8; t > 0; t >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, t));
            const float m_new = fmaxf(m[r], mx);
            // Every score so far may be -inf (padded keys at the front): 0 as the reference keeps inf - inf out, and
            // the weights are 0.
            const float ref = m_new == -INFINITY ? 0.f : m_new;
            const float alpha = exp_nat(m[r] - ref);
            m[r] = m_new;
#pragma unroll
            for (int c = 0; c < 4; c++) s[r][c] = exp_nat(s[r][c] - ref);
            l[r] = l[r] * alpha + ((s[r][0] + s[r][1]) + (s[r][2] + s[r][3]));  // this thread's columns only
            const f32x2 al2 = pack2(alpha, alpha);
#pragma unroll
            for (int n = 0; n < NP; n++) o[r][n] = ptx::mul2(o[r][n], al2);
        }
        store_p<R>(Ps, s, ty, tx);
        cp_wait<1>();
        __syncthreads();  // V(k0) is here (and the scores, which only this half-warp reads)
        mm_pv<R, DPAD>(o, Ps, Vs, ty, tx);
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
        float lr = l[r];
#pragma unroll
        for (int t = 8; t > 0; t >>= 1) lr += __shfl_xor_sync(0xffffffffu, lr, t);
        const int row = q0 + ty * R + r;
        if (row < p.lq) {
            store_row<T, FAST, DPAD>((T *)p.out + ((size_t)unit * p.lq + row) * d, o[r], 1.f / lr, d, tx);
            if (p.lse && tx == 0) p.lse[(size_t)unit * p.lq + row] = m[r] + logf(lr);
        }
    }
}

// delta[row] = sum_c dO[row][c] * O[row][c]; one warp per row.
template <typename T>
__global__ void delta_kernel(const T *__restrict__ out, const T *__restrict__ dout,
                             float *__restrict__ delta, size_t rows, int d)
{
    const size_t row = (size_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    if (row >= rows) return;
    const int lane = threadIdx.x % 32;
    float s = 0.f;
    for (int c = lane; c < d; c += 32) s += ld(out + row * d + c) * ld(dout + row * d + c);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) delta[row] = s;
}

struct SimtBwd {
    const void *q, *k, *v, *dout;
    const float *lse, *delta;
    void *dq, *dk, *dv;
    int bh, lq, lk, d, causal;
    int kblocks, qblocks;  // blocks of 8*R keys (dK, dV) and of 8*R queries (dQ) per unit
    float scale;
    const int *only_if;
};

// One launch, two kinds of blocks: the first bh * kblocks own 8*R keys each and form dK and dV over all
// queries that see them (4 products per tile), the others own 8*R queries and form dQ (3 products). They
// are independent, and together they fill the SMs of a small problem and share one tail. Both recompute
// P from the saved log-sum-exp; no atomics, so results repeat bit for bit.
template <typename T, bool FAST, int DPAD, int R>
__global__ void __launch_bounds__(NT) simt_bwd_kernel(const SimtBwd p)
{
    if (not_needed(p.only_if)) return;
    constexpr int BM = 8 * R, NP = Cols<DPAD>::NP;
    extern __shared__ __align__(1024) char smem[];
    // A0, A1: this block's rows (K and V, or Q and dO); B0, B1: the streamed 64-row tiles (Q and dO, or K and V)
    char *A0 = smem, *A1 = A0 + BM * DPAD * 4, *B0 = A1 + BM * DPAD * 4, *B1 = B0 + TN * DPAD * 4,
         *Ps = B1 + TN * DPAD * 4;
    float *lse_s = reinterpret_cast<float *>(Ps + BM * TN * 4), *delta_s = lse_s + 64;
    const int ty = threadIdx.x / 16, tx = threadIdx.x % 16, d = p.d, nch = (d + 3) / 4, off = p.lk - p.lq;
    const float sc = p.scale;
    const bool is_kv = blockIdx.x < (unsigned)(p.bh * p.kblocks);
    const int idx = is_kv ? blockIdx.x : blockIdx.x - p.bh * p.kblocks;
    const int unit = idx % p.bh;
    const T *q = (const T *)p.q + (size_t)unit * p.lq * d, *dout = (const T *)p.dout + (size_t)unit * p.lq * d,
            *k = (const T *)p.k + (size_t)unit * p.lk * d, *v = (const T *)p.v + (size_t)unit * p.lk * d;
    const float *lse = p.lse + (size_t)unit * p.lq, *delta = p.delta + (size_t)unit * p.lq;

    if (is_kv) {
        const int k0 = (idx / p.bh) * BM;  // under a causal mask the first keys are seen by the most queries
        load_tile<T, FAST, DPAD, BM>(A0, k, k0, p.lk, d);
        load_tile<T, FAST, DPAD, BM>(A1, v, k0, p.lk, d);
        f32x2 adk[R][NP], adv[R][NP];
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int n = 0; n < NP; n++) adk[r][n] = adv[r][n] = 0;
        const int qstart = p.causal ? max(0, (k0 - off) / TN) * TN : 0;  // first query tile that sees key k0
        for (int q0 = qstart; q0 < p.lq; q0 += TN) {
            if (q0 != qstart) __syncthreads();  // the previous tile has been read
            load_tile<T, FAST, DPAD, TN>(B0, q, q0, p.lq, d);
            load_tile<T, FAST, DPAD, TN>(B1, dout, q0, p.lq, d);
            cp_commit();
            if (threadIdx.x < 64) {
                const int row = q0 + threadIdx.x;
                lse_s[threadIdx.x] = row < p.lq ? lse[row] : INFINITY;  // rows past the end: P = 0
                delta_s[threadIdx.x] = row < p.lq ? delta[row] : 0.f;
            }
            cp_wait<0>();
            __syncthreads();
            float s[R][4], dp[R][4];  // transposed: keys x queries
            mm_abt<R, DPAD>(s, A0, B0, nch, ty, tx);
            mm_abt<R, DPAD>(dp, A1, B1, nch, ty, tx);
            const bool edge = k0 + BM > p.lk || (p.causal && k0 + BM - 1 > q0 + off);
            const float4 L4 = *reinterpret_cast<const float4 *>(lse_s + tx * 4), D4 = *reinterpret_cast<const float4 *>(delta_s + tx * 4);
            const float L[4] = {L4.x, L4.y, L4.z, L4.w}, dl[4] = {D4.x, D4.y, D4.z, D4.w};
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int key = k0 + ty * R + r;
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    float pr = expf(fmaf(s[r][c], sc, -L[c]));
                    if (edge && (key >= p.lk || (p.causal && key > q0 + tx * 4 + c + off))) pr = 0.f;
                    s[r][c] = pr;
                    dp[r][c] = pr * (dp[r][c] - dl[c]);
                }
            }
            store_p<R>(Ps, s, ty, tx);
            __syncwarp();
            mm_pv<R, DPAD>(adv, Ps, B1, ty, tx);
            __syncwarp();
            store_p<R>(Ps, dp, ty, tx);
            __syncwarp();
            mm_pv<R, DPAD>(adk, Ps, B0, ty, tx);
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int key = k0 + ty * R + r;
            if (key >= p.lk) continue;
            const size_t row = ((size_t)unit * p.lk + key) * d;
            store_row<T, FAST, DPAD>((T *)p.dk + row, adk[r], p.scale, d, tx);
            store_row<T, FAST, DPAD>((T *)p.dv + row, adv[r], 1.f, d, tx);
        }
    } else {
        const int q0 = (p.qblocks - 1 - idx / p.bh) * BM;  // the last queries see the most keys
        load_tile<T, FAST, DPAD, BM>(A0, q, q0, p.lq, d);
        load_tile<T, FAST, DPAD, BM>(A1, dout, q0, p.lq, d);
        float L[R], dl[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int row = q0 + ty * R + r;
            L[r] = row < p.lq ? lse[row] : INFINITY;
            dl[r] = row < p.lq ? delta[row] : 0.f;
        }
        f32x2 adq[R][NP];
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int n = 0; n < NP; n++) adq[r][n] = 0;
        const int kend = p.causal ? min(p.lk, q0 + BM + off) : p.lk;
        for (int k0 = 0; k0 < kend; k0 += TN) {
            if (k0 != 0) __syncthreads();
            load_tile<T, FAST, DPAD, TN>(B0, k, k0, p.lk, d);
            load_tile<T, FAST, DPAD, TN>(B1, v, k0, p.lk, d);
            cp_commit();
            cp_wait<0>();
            __syncthreads();
            float s[R][4], dp[R][4];
            mm_abt<R, DPAD>(s, A0, B0, nch, ty, tx);
            mm_abt<R, DPAD>(dp, A1, B1, nch, ty, tx);
            const bool edge = k0 + TN - 1 > (p.causal ? min(p.lk - 1, q0 + off) : p.lk - 1);
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int row = q0 + ty * R + r, limit = p.causal ? min(p.lk - 1, row + off) : p.lk - 1;
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    float pr = expf(fmaf(s[r][c], sc, -L[r]));
                    if (edge && k0 + tx * 4 + c > limit) pr = 0.f;
                    dp[r][c] = pr * (dp[r][c] - dl[r]);
                }
            }
            store_p<R>(Ps, dp, ty, tx);
            __syncwarp();
            mm_pv<R, DPAD>(adq, Ps, B0, ty, tx);
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int row = q0 + ty * R + r;
            if (row < p.lq) store_row<T, FAST, DPAD>((T *)p.dq + ((size_t)unit * p.lq + row) * d, adq[r], p.scale, d, tx);
        }
    }
}

int too_many_blocks()
{
    set_error("attention: too many (batch*head) units and blocks for one launch");
    return EMBER_ERR_UNSUPPORTED;
}

template <typename T, bool FAST, int DPAD, int R>
int launch_fwd(const AttnArgs &a, cudaStream_t s)
{
    constexpr int BM = 8 * R;
    const size_t smem = (size_t)(BM + 2 * TN) * DPAD * 4 + BM * TN * 4;
    auto kern = simt_fwd_kernel<T, FAST, DPAD, R>;
    static SmemOptIn opt_in;
    EMBER_CUDA_TRY(opt_in(kern, smem));
    SimtFwd p = {a.q, a.k, a.v, a.out, a.lse, a.bh, a.lq, a.lk, a.d, a.causal, (a.lq + BM - 1) / BM, a.scale, a.only_if};
    const long long grid = (long long)p.bh * p.blocks;
    if (grid > 0x7fffffffLL) return too_many_blocks();
    return launch_simt(kern, grid, smem, s, p);
}

template <typename T, bool FAST, int DPAD, int R>
int launch_bwd(const AttnArgs &a, const float *delta, cudaStream_t s)
{
    constexpr int BM = 8 * R;
    const size_t smem = (size_t)(2 * BM + 2 * TN) * DPAD * 4 + BM * TN * 4 + 512;
    auto kern = simt_bwd_kernel<T, FAST, DPAD, R>;
    static SmemOptIn opt_in;
    EMBER_CUDA_TRY(opt_in(kern, smem));
    SimtBwd p = {a.q, a.k, a.v, a.dout, a.lse, delta, a.dq, a.dk, a.dv, a.bh, a.lq, a.lk, a.d, a.causal,
                 (a.lk + BM - 1) / BM, (a.lq + BM - 1) / BM, a.scale, a.only_if};
    const long long grid = (long long)p.bh * ((long long)p.kblocks + p.qblocks);
    if (grid > 0x7fffffffLL) return too_many_blocks();
    return launch_simt(kern, grid, smem, s, p);
}

bool fast_rows(const AttnArgs &a)
{
    const uintptr_t bits = (uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.out | (uintptr_t)a.dout |
                           (uintptr_t)a.dq | (uintptr_t)a.dk | (uintptr_t)a.dv;
    return a.dtype == EMBER_F32 && a.d % 4 == 0 && (bits & 15) == 0;
}

// Rows per thread. More rows per thread cost fewer shared-memory loads per FMA, fewer give more and
// shorter blocks. Measured (us, R = 8 / 4 / 2), float32:
//   forward   16 units x L1024 D64 causal   105 /  93 / 101    8 x L2048 D64            271 / 288 / 354
//             16 x L1024 D128 causal        175 / 153 / 200    2 x L2048 D128 causal    291 / 190 / 169
//             8 x L128 D64                   17 /  11 /   9    4 x L333 D80 causal       52 /  34 /  27
//   backward  16 x L1024 D64 causal         211 / 230 / 311    16 x L1024 D128 causal   507 / 438 / 627
//             2 x L2048 D128 causal         633 / 438 / 352    8 x L128 D64              27 /  21 /  17
// so: 16-row blocks while 32-row blocks would not give every SM two, and 64-row blocks at up to 64
// columns (at 128 they leave one block per SM) once there are three per two SMs; the forward under a
// causal mask keeps 32-row blocks, whose last wave is better balanced.
int rows_per_thread(long long blocks32, long long blocks64, bool big_ok, int d, int sms)
{
    if (blocks32 < 2LL * sms) return 2;
    return big_ok && d <= 64 && 2 * blocks64 >= 3LL * sms ? 8 : 4;
}

template <int DPAD>
int dispatch_fwd(const AttnArgs &a, int sms, cudaStream_t s)
{
    if (a.dtype == EMBER_BF16) return launch_fwd<__nv_bfloat16, false, DPAD, 4>(a, s);
    if (!fast_rows(a)) return launch_fwd<float, false, DPAD, 4>(a, s);
    const long long bh = a.bh;
    const int r = rows_per_thread(bh * ((a.lq + 31) / 32), bh * ((a.lq + 63) / 64), !a.causal, a.d, sms);
    if (r == 2) return launch_fwd<float, true, DPAD, 2>(a, s);
    if constexpr (DPAD <= 64)
        if (r == 8) return launch_fwd<float, true, DPAD, 8>(a, s);
    return launch_fwd<float, true, DPAD, 4>(a, s);
}

template <int DPAD>
int dispatch_bwd(const AttnArgs &a, int sms, const float *delta, cudaStream_t s)
{
    if (a.dtype == EMBER_BF16) return launch_bwd<__nv_bfloat16, false, DPAD, 4>(a, delta, s);
    if (!fast_rows(a)) return launch_bwd<float, false, DPAD, 4>(a, delta, s);
    const long long bh = a.bh;
    const int r = rows_per_thread(bh * ((a.lq + 31) / 32 + (a.lk + 31) / 32), bh * ((a.lq + 63) / 64 + (a.lk + 63) / 64),
                                  true, a.d, sms);
    if (r == 2) return launch_bwd<float, true, DPAD, 2>(a, delta, s);
    if constexpr (DPAD <= 64)
        if (r == 8) return launch_bwd<float, true, DPAD, 8>(a, delta, s);
    return launch_bwd<float, true, DPAD, 4>(a, delta, s);
}

}  // namespace

int simt_attention_fwd(const AttnArgs &a, DeviceState *st, cudaStream_t s)
{
    if (a.d > 128) {
        set_error("head dimension %d > 128 is not supported", a.d);
        return EMBER_ERR_UNSUPPORTED;
    }
    const int sms = st->sm_count > 0 ? st->sm_count : 148;
    if (a.d <= 32) return dispatch_fwd<32>(a, sms, s);
    return a.d <= 64 ? dispatch_fwd<64>(a, sms, s) : dispatch_fwd<128>(a, sms, s);
}

int simt_attention_bwd(const AttnArgs &a, float *delta, bool delta_made, DeviceState *st, cudaStream_t s)
{
    if (a.d > 128) {
        set_error("head dimension %d > 128 is not supported", a.d);
        return EMBER_ERR_UNSUPPORTED;
    }
    const int rc = delta_made ? EMBER_OK : launch_delta(a, delta, s);
    if (rc != EMBER_OK) return rc;
    const int sms = st->sm_count > 0 ? st->sm_count : 148;
    if (a.d <= 32) return dispatch_bwd<32>(a, sms, delta, s);
    return a.d <= 64 ? dispatch_bwd<64>(a, sms, delta, s) : dispatch_bwd<128>(a, sms, delta, s);
}

int launch_delta(const AttnArgs &a, float *delta, cudaStream_t s)
{
    const size_t rows = (size_t)a.bh * a.lq;
    if (a.dtype == EMBER_F32)
        delta_kernel<float><<<(unsigned)((rows + 7) / 8), 256, 0, s>>>((const float *)a.out, (const float *)a.dout, delta, rows, a.d);
    else
        delta_kernel<__nv_bfloat16><<<(unsigned)((rows + 7) / 8), 256, 0, s>>>((const __nv_bfloat16 *)a.out, (const __nv_bfloat16 *)a.dout, delta, rows, a.d);
    EMBER_CUDA_TRY(cudaGetLastError());
    return EMBER_OK;
}

}  // namespace ember
