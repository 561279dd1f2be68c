// Internal interface between the C-ABI dispatcher and the kernel families.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace ember {

// Programmatic dependent launch: a kernel sets itself up (barriers, tensor memory, descriptors) on SMs that fall
// idle while the one before it drains, which saves 2 to 3 us a launch in chains of short kernels. Measured with
// and without it on the projections, the cache and the forward: a token through a 2048-wide block at batch 8, back to
// back on the same buffers, 41 -> 31 us, forward and backward of a block of 2 x 1024 x 1536 224 -> 200 us, of 16 units x L2048 92.5 -> 87.2 us.
// EMBER_PDL=0 (read once) launches every kernel in plain stream order.
// Rules of the kernels that are launched with it, which make any chain of them safe:
//   - every thread passes pdl_wait() before it reads or writes global memory (prefetching a tensor map and
//     setting up barriers and tensor memory may come before), so that a kernel's end implies the end of
//     all before it (the single-pass backward reads q, k, v and dO earlier: the delta kernel before it passes
//     pdl_wait() first and lets it start afterwards); that goes for blocks that leave early, too;
//   - a kernel that allocates tensor memory passes pdl_launch_dependents() after the allocation: a later kernel's
//     block can then never hold the columns that an earlier one's, which it waits for, still needs;
//   - sm100_gemm_kernel, where a call asks for it (GemmArgs::held, beside), passes pdl_wait() before pdl_launch_dependents(). What is launched behind it finds every
//     kernel before it done, and may begin without pdl_wait() if it neither reads nor overwrites anything of the product itself: the products and the bias gradient of one
//     backward call ("beside"). Such a kernel passes pdl_wait() last, so that its end, too, implies the end of all before it, and
//     pdl_launch_dependents() first, for another of its kind;
//   - what is read before pdl_wait() comes from L2: by TMA, or behind a fence that empties the SM's L1. Being let go early makes the writes of the
//     kernels before visible nowhere else, and L1 may hold older lines of recycled memory.
bool pdl_enabled();

struct LaunchAttrs {
    cudaLaunchAttribute attr[2];
    int count = 0;

    LaunchAttrs &cluster(unsigned x)
    {
        if (x > 1) {
            attr[count].id = cudaLaunchAttributeClusterDimension;
            attr[count].val.clusterDim.x = x;
            attr[count].val.clusterDim.y = 1;
            attr[count++].val.clusterDim.z = 1;
        }
        return *this;
    }
    LaunchAttrs &pdl()
    {
        if (pdl_enabled()) {
            attr[count].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[count++].val.programmaticStreamSerializationAllowed = 1;
        }
        return *this;
    }
    void set(cudaLaunchConfig_t &cfg)
    {
        cfg.attrs = attr;
        cfg.numAttrs = (unsigned)count;
    }
};

// For kernels without clusters. A grid of more than 8 blocks per SM (of 148) lasts longer than its start: plain order (with
// blocks that wait on every SM an 8192 x 32768 classifier step took 0.6 % longer).
constexpr int kPdlMaxGrid = 8 * 148;
template <typename... Params, typename... Args>
cudaError_t launch_pdl(void (*kern)(Params...), int grid, int block, size_t smem, cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    LaunchAttrs attrs;
    if (grid <= kPdlMaxGrid) attrs.pdl();
    attrs.set(cfg);
    return cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
}

struct AttnArgs {
    const void *q = nullptr, *k = nullptr, *v = nullptr;
    void *out = nullptr;
    float *lse = nullptr;
    const void *dout = nullptr;
    void *dq = nullptr, *dk = nullptr, *dv = nullptr;
    int bh = 0, lq = 0, lk = 0, d = 0;
    float scale = 1.f;
    int causal = 0;
    int dtype = EMBER_F32;
    const int *only_if = nullptr;  // CUDA-core kernels: return at once when this word of device memory is 0
};

// CUDA-core kernels (attn_simt.cu): float32 math, f32 or bf16 storage, d <= 128.
int simt_attention_fwd(const AttnArgs &a, DeviceState *st, cudaStream_t s);
// delta_made: delta holds the rows' sums already
int simt_attention_bwd(const AttnArgs &a, float *delta, bool delta_made, DeviceState *st, cudaStream_t s);
// Float32 storage on the tensor cores, each operand as three bf16 parts (attn_f32_sm100.cu). The scratch they allocate may be
// missing: EMBER_ERR_NOMEM, nothing launched.
bool sm100_f32_fwd_preferred(const AttnArgs &a, int sms);
int sm100_f32_attention_fwd(const AttnArgs &a, DeviceState *st, cudaStream_t s);
bool sm100_f32_bwd_preferred(const AttnArgs &a, int sms);
int sm100_f32_attention_bwd(const AttnArgs &a, float *delta, DeviceState *st, cudaStream_t s);
int launch_delta(const AttnArgs &a, float *delta, cudaStream_t s);

// tcgen05 kernels (attn_fwd_sm100.cu / attn_bwd_sm100.cu): bf16 storage, d in {64, 128}.
bool sm100_fwd_supported(const AttnArgs &a);
int sm100_fwd_set_block_rows(int rows);  // 0 = choose per call, 128, 256; returns the previous setting
int sm100_attention_fwd(const AttnArgs &a, DeviceState *st, cudaStream_t s);
bool sm100_bwd_supported(const AttnArgs &a);
// deterministic: two kernels (dK/dV, then dQ), bit-reproducible; otherwise one pass that adds its dQ
// contributions into dq_acc (sm100_bwd_accumulator_bytes of float32 scratch after the delta vector).
size_t sm100_bwd_accumulator_bytes(int bh, int lq, int d);
int sm100_attention_bwd(const AttnArgs &a, float *delta, float *dq_acc, bool deterministic, DeviceState *st, cudaStream_t s);

// Decode over a contiguous key/value cache with grouped-query heads on the tensor cores
// (attn_fwd_sm100.cu: the forward kernel with the group's query heads as the rows of one tile and the
// key axis cut into splits). chunk: keys per split, a multiple of 128; workspace: partial outputs.
struct CacheDecodeArgs {
    const void *q = nullptr, *k_cache = nullptr, *v_cache = nullptr;
    void *out = nullptr;
    float *lse = nullptr;
    int batch = 0, q_heads = 0, kv_heads = 0, lk = 0, capacity = 0, d = 0, dtype = EMBER_BF16;
    float scale = 1.f;
    const int *seq_lens = nullptr;
    int splits = 1, chunk = 0;
    void *workspace = nullptr;
};
bool sm100_cache_decode_supported(const CacheDecodeArgs &a);
size_t sm100_cache_decode_workspace_bytes(int units, int rows, int d, int splits);
int sm100_cache_decode(const CacheDecodeArgs &a, DeviceState *st, cudaStream_t s);

// Decode over a contiguous bf16 cache with up to 16 query heads per K/V head (decode_sm100.cu); splits,
// chunk are not used.
bool sm100_decode_supported(const CacheDecodeArgs &a);
size_t sm100_decode_workspace_bytes(int rows, int d, int sms);
int sm100_decode(const CacheDecodeArgs &a, DeviceState *st, cudaStream_t s);

// Split-KV decode (attn_decode.cu): lq == 1, bf16 or f32 storage, d <= 256 and d % 8 == 0.
int decode_pick_splits(int bh, int lk, int d, int dtype, int sm_count);
size_t decode_workspace_bytes(int bh, int d, int splits);
int decode_attention(const AttnArgs &a, int splits, void *workspace, DeviceState *st, cudaStream_t s);

// ---------------------------------------------------------------- projections either side of attention
// A logical (rows x cols) matrix and how it lies in memory.
//   heads == 0: row-major, leading dimension = cols.
//   heads  > 0: head-major (parts, batch, heads, seq, dim), the layout attention consumes:
//               row = b * seq + l, col = (part * heads + h) * dim + d, batch = rows / seq,
//               parts = cols / (heads * dim).
struct MatView {
    const void *ptr = nullptr;
    long long rows = 0;
    int cols = 0;
    int heads = 0, seq = 0, dim = 0;
};

__host__ __device__ inline size_t view_offset(const MatView &v, long long row, int col)
{
    if (v.heads == 0) return (size_t)row * v.cols + col;
    const long long b = row / v.seq, batch = v.rows / v.seq;
    const int l = (int)(row - b * v.seq), ph = col / v.dim, d = col - ph * v.dim;
    const int part = ph / v.heads, h = ph - part * v.heads;
    return ((((size_t)part * batch + b) * v.heads + h) * v.seq + l) * v.dim + d;
}

// C (m x n) = op(A) * op(B) [+ bias], bf16 or f32 storage, float32 accumulation.
enum GemmMode {
    GEMM_NN = 0,  // A view (m x k), B view (k x n)
    GEMM_NT = 1,  // A view (m x k), B view (n x k)
    GEMM_TN = 2   // A view (k x m), B view (k x n)
};
// Results of a few-row q/k/v projection that go straight into a key/value cache (batch, heads, capacity, d): columns
// from `from` on are k, then v, `from` each; row b of the product is row `pos` of sequence b.
struct CacheRows {
    void *k, *v;
    int from, heads, capacity, d, pos;
};

struct GemmArgs {
    int mode = GEMM_NN;
    MatView a, b, c;
    const void *bias = nullptr;  // n values of the storage dtype, or null
    long long m = 0;
    int n = 0, k = 0;
    int dtype = EMBER_F32;
    const CacheRows *cache = nullptr;  // gemm_skinny_sm100.cu
    // gemm_sm100.cu: the product launched just before this one, which neither reads this one's results nor writes what this one reads:
    // the two run side by side where SMs are free (rules beside pdl_enabled).
    const GemmArgs *beside = nullptr;
    bool held = false;         // gemm_sm100.cu: what is launched next runs beside this product
    bool leaves_room = false;  // the same, with room for blocks of column_sum_kernel on this product's SMs
    const int *only_if = nullptr;  // CUDA-core kernel: return at once when this word of device memory is 0
};

// CUDA-core kernels (gemm_simt.cu): float32 math, any shape and view.
int simt_gemm(const GemmArgs &g, DeviceState *st, cudaStream_t s);
// column_sums.cu: out[j] = sum over rows of a(:, j), any shape and view
// beside: the kernel launched just before neither writes a nor touches out and runs beside this one (rules beside pdl_enabled)
int column_sums(const MatView &a, void *out, int dtype, DeviceState *st, cudaStream_t s, bool beside = false);
// tcgen05 kernel (gemm_sm100.cu): bf16 storage; see sm100_gemm_supported for the shapes it takes.
bool sm100_gemm_supported(const GemmArgs &g);
int sm100_gemm(const GemmArgs &g, DeviceState *st, cudaStream_t s);
bool sm100_gemm_gains_beside(const GemmArgs &before, const GemmArgs &g, DeviceState *st);  // whether GemmArgs::beside makes g end sooner
// dst (bf16, 16-byte aligned, rows of v.cols rounded up to 8) = v (row-major, any alignment), zeros past v.cols
int pack_rows(const MatView &v, void *dst, cudaStream_t s);
// tcgen05 kernel for at most 128 rows (gemm_skinny_sm100.cu): a decode step's projections.
bool sm100_skinny_gemm_supported(const GemmArgs &g);
bool sm100_skinny_gemm_preferred(const GemmArgs &g);  // quicker than sm100_gemm, where that takes the product too
int sm100_skinny_gemm(const GemmArgs &g, DeviceState *st, cudaStream_t s);
// planes: so many copies of the view one after the other, counted along the parts
int make_tensor_map_bf16_view(CUtensorMap *map, const MatView &v, uint32_t box_cols, uint32_t box_rows, int planes = 1);
// Float32, at most 16 rows, y = x w + b (gemm_skinny_f32.cu): a decode step's projections on the CUDA cores.
bool skinny_f32_supported(const GemmArgs &g);
int skinny_f32_gemm(const GemmArgs &g, DeviceState *st, cudaStream_t s);

// Float32, at most 12 columns, y = x w + b (gemm_narrow_f32.cu): a small classifier's logits on the CUDA cores.
bool narrow_f32_supported(const GemmArgs &g);
int narrow_f32_gemm(const GemmArgs &g, cudaStream_t s);
// All gradients of such a layer (dx, db may be NULL) in one launch, where they lie apart from the operands and from one another.
bool narrow_f32_bwd_supported(const void *x, const void *w, const void *dy, const void *dx, const void *db, long long m, int n, int k);
int narrow_f32_backward(const void *x, const void *w, const void *dy, void *dx, void *dw, void *db, long long m, int n, int k, DeviceState *st, cudaStream_t s);
// Float32 storage on the tensor cores, operands as three bf16 planes each (gemm_f32_sm100.cu, split_f32.cuh): a row-major view's rows
// padded to 8 columns. _us: an estimate of the time, without the splitting.
struct SplitGuard;
bool sm100_f32_gemm_supported(const GemmArgs &g);
double sm100_f32_gemm_us(const GemmArgs &g, int sms);
int sm100_f32_gemm(const GemmArgs &g, const void *a_planes, const void *b_planes, const SplitGuard &guard, DeviceState *st, cudaStream_t s);

}  // namespace ember
