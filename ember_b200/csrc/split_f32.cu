// Splits float32 tensors into three bf16 planes for the tensor cores (see split_f32.cuh).
#include "split_f32.cuh"

namespace ember {

namespace {

struct SplitParams {
    SplitJob job[kSplitMaxJobs];
    int first[kSplitMaxJobs + 1];
    int count;
    uint32_t *slots;
    SplitDelta delta;
    int delta_blocks;
};

// The largest magnitude that this block saw, into its slot.
__device__ __forceinline__ void report(uint32_t *slots, uint32_t amax)
{
    __shared__ uint32_t most;
    if (threadIdx.x == 0) most = 0;
    __syncthreads();
    amax = __reduce_max_sync(0xffffffffu, amax);
    if (threadIdx.x % 32 == 0) atomicMax(&most, amax);
    __syncthreads();
    if (threadIdx.x == 0) slots[blockIdx.x] = most;
}

// Bound: one pass over memory, 4 bytes read and 6 written per element, mostly within L2 (the next kernel reads the planes at
// once). A thread makes 8 columns of the three planes (16-byte stores); a block takes every n-th piece of its tensor.
__global__ void __launch_bounds__(256) split_f32_kernel(const SplitParams p)
{
    ptx::pdl_launch_dependents();
    ptx::pdl_wait();
    const int total = p.first[p.count];
    if ((int)blockIdx.x >= total) {
        // ---- delta: 16 lanes per row
        const SplitDelta &d = p.delta;
        const int lane = threadIdx.x % 16;
        const bool vec = d.cols % 4 == 0 && (((uintptr_t)d.out | (uintptr_t)d.dout) & 15) == 0;
        const long long step = (long long)p.delta_blocks * 16;
        uint32_t amax = 0;
        for (long long row0 = (long long)((int)blockIdx.x - total) * 16; row0 < d.rows; row0 += step) {
            const long long row = row0 + threadIdx.x / 16;
            float s = 0.f;
            if (row < d.rows) {
                const float *a = d.out + row * d.cols, *b = d.dout + row * d.cols;
                if (vec) {
                    for (int c = lane * 4; c < d.cols; c += 64) {
                        const float4 x = *reinterpret_cast<const float4 *>(a + c), y = *reinterpret_cast<const float4 *>(b + c);
                        s += (x.x * y.x + x.y * y.y) + (x.z * y.z + x.w * y.w);
                    }
                } else {
                    for (int c = lane; c < d.cols; c += 16) s += a[c] * b[c];
                }
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (row < d.rows && lane == 0) {
                d.delta[row] = s;
                amax = max(amax, __float_as_uint(s) & 0x7fffffffu);
            }
        }
        report(p.slots, amax);
        return;
    }
    int j = 0;
    while ((int)blockIdx.x >= p.first[j + 1]) j++;
    const SplitJob &job = p.job[j];
    const int nblk = p.first[j + 1] - p.first[j], cpr = (job.cols + 7) / 8;
    const long long chunks = job.rows * cpr;
    const bool flat = job.cols % 8 == 0 && ((uintptr_t)job.src & 15) == 0;
    uint4 *dst = (uint4 *)job.dst;
    uint32_t amax = 0;
#pragma unroll 2
    for (long long c = (long long)((int)blockIdx.x - p.first[j]) * 256 + threadIdx.x; c < chunks; c += (long long)nblk * 256) {
        float v[8];
        if (flat) {
            const float4 a = reinterpret_cast<const float4 *>(job.src)[2 * c], b = reinterpret_cast<const float4 *>(job.src)[2 * c + 1];
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
            v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
            const long long row = c / cpr;
            const int col = (int)(c - row * cpr) * 8;
            const float *r = job.src + row * job.cols + col;
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = col + i < job.cols ? r[i] : 0.f;
        }
        uint32_t h[4], m[4], l[4];
#pragma unroll
        for (int i = 0; i < 8; i++) amax = max(amax, __float_as_uint(v[i]) & 0x7fffffffu);
        if (!dst) continue;
#pragma unroll
        for (int i = 0; i < 4; i++) split_pair(v[2 * i] * kSplitUp, v[2 * i + 1] * kSplitUp, h[i], m[i], l[i]);
        dst[c] = make_uint4(h[0], h[1], h[2], h[3]);
        dst[chunks + c] = make_uint4(m[0], m[1], m[2], m[3]);
        dst[2 * chunks + c] = make_uint4(l[0], l[1], l[2], l[3]);
    }
    report(p.slots, amax);
}

}  // namespace

int split_f32(const SplitJob *jobs, int count, const SplitDelta *delta, void *guard_mem, SplitGuard *guard, cudaStream_t s)
{
    SplitParams p = {};
    long long pieces[kSplitMaxJobs], all = 0;
    for (int i = 0; i < count; i++) {
        p.job[i] = jobs[i];
        pieces[i] = (jobs[i].rows * ((jobs[i].cols + 7) / 8) + 255) / 256;  // blocks' worth of 8-column pieces
        all += pieces[i];
    }
    const long long budget = kSplitMaxBlocks - kSplitMaxJobs;
    for (int i = 0; i < count; i++) {
        long long n = all <= budget ? pieces[i] : budget * pieces[i] / all + 1;
        if (n > pieces[i]) n = pieces[i];
        p.first[i + 1] = p.first[i] + (int)n;
    }
    p.count = count;
    p.slots = (uint32_t *)guard_mem;
    if (delta) {
        p.delta = *delta;
        const long long n = (delta->rows + 15) / 16;
        p.delta_blocks = (int)(n < kSplitMaxBlocks ? n : kSplitMaxBlocks);
    }
    guard->slots = p.slots;
    guard->count = count;
    for (int i = 0; i <= count; i++) guard->first[i] = p.first[i];
    if (delta) {
        guard->delta_at = guard->count++;
        guard->first[guard->count] = p.first[count] + p.delta_blocks;
    }
    guard->fallback = (int *)guard_mem + 2 * kSplitMaxBlocks;
    EMBER_CUDA_TRY(launch_pdl(split_f32_kernel, p.first[count] + p.delta_blocks, 256, 0, s, p));
    return EMBER_OK;
}

}  // namespace ember
