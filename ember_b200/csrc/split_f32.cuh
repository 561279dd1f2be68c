// Float32 operands for the tensor cores. A float32 value is the exact sum of three bf16 values (24 significand
// bits = 3 x 8): high, middle and low part, each the rounding of what the ones before left over. Of the nine products of
// two such sums the six largest are formed, all in float32; what is left out is below 2^-24 of the product, 2^-27 as a rule.
// The tensor core adds with truncation (a sum keeps 24 bits and loses the rest towards zero; within one MMA, terms are cut
// at 2^-25 of the largest), so an accumulator that collects a whole contraction drifts: relative error of random sums of 64 /
// 512 / 2048 terms 6.6e-8 / 4.7e-7 / 2.1e-6. The kernels therefore let it collect 64 terms at most, the
// small products first, and add it into float32 registers with rounding.
// Parts are made of the value times 2^16: bf16 ends at 2^-133 (tcgen05 multiplies those small ones as they are), where the low part of a
// value below 2^-110 would lose its last bits (a row of 1e-36 beside ordinary ones: 3e-5 of its results); 2^16 times the smallest float32 is
// just held. What is made of parts is divided by the powers of two again where it leaves the accumulators.
// Values that the parts cannot hold (infinities, NaN, 2^32 and above, whose sums of 2^31 products times 2^32 may pass float32) are
// found while the parts are made: the tensor-core kernel then leaves the work to the CUDA-core kernel that is launched behind it and
// otherwise returns at once.
#pragma once

#include "common.cuh"
#include "kernels.cuh"
#include "ptx.cuh"

namespace ember {

constexpr int kSplitMaxJobs = 4;
constexpr int kSplitMaxBlocks = 592;               // 4 blocks of 256 threads per SM
constexpr int kSplitMaxTensors = kSplitMaxJobs + 1;  // delta's largest magnitude is reported as well
constexpr uint32_t kSplitHuge = 0x4F800000u;       // 2^32
constexpr uint32_t kSplitHugeDelta = 0x67800000u;  // 2^80
constexpr int kSplitShift = 16;
constexpr float kSplitUp = 65536.f, kSplitDown2 = 1.f / 65536.f / 65536.f;  // a part's factor, and what undoes it in a product of two

// What a split launch leaves for the kernels behind it: the largest magnitude (as bits; a NaN is larger than all) that each of
// its blocks saw, by tensor, and the word through which the tensor-core kernel tells the CUDA-core kernel to run.
struct SplitGuard {
    const uint32_t *slots = nullptr;
    int first[kSplitMaxTensors + 1] = {};  // blocks [first[i], first[i + 1]) saw tensor i; the last may be delta
    int count = 0, delta_at = -1;
    int *fallback = nullptr;
    // Largest product of tensors pair[0]'s and pair[1]'s largest magnitudes that the kernel takes (attention: what it could score).
    int pair[2] = {};
    float pair_limit = 0;  // 0: any
};

#ifdef __CUDACC__
// Whether any tensor holds values that the parts cannot represent, or the pair's product is beyond its limit. All threads of the block
// call it; `words` is shared memory, kSplitMaxTensors words, in which the tensors' largest magnitudes stay (as bits).
__device__ __forceinline__ bool split_out_of_range(const SplitGuard &g, uint32_t *words)
{
    if (threadIdx.x < kSplitMaxTensors) words[threadIdx.x] = 0;
    __syncthreads();
    uint32_t m[kSplitMaxTensors] = {};
#pragma unroll 2
    for (int b = (int)threadIdx.x; b < g.first[g.count]; b += blockDim.x) {
        const uint32_t v = g.slots[b];
#pragma unroll
        for (int i = 0; i < kSplitMaxTensors; i++)
            if (i < g.count && b >= g.first[i] && b < g.first[i + 1]) m[i] = max(m[i], v);
    }
#pragma unroll
    for (int i = 0; i < kSplitMaxTensors; i++) {
        m[i] = __reduce_max_sync(0xffffffffu, m[i]);
        if (threadIdx.x % 32 == 0 && m[i] != 0) atomicMax(&words[i], m[i]);
    }
    __syncthreads();
    bool out = g.pair_limit > 0 && !(__uint_as_float(words[g.pair[0]]) * __uint_as_float(words[g.pair[1]]) <= g.pair_limit);
    for (int i = 0; i < g.count; i++) out = out || words[i] >= (i == g.delta_at ? kSplitHugeDelta : kSplitHuge);
    if (blockIdx.x == 0 && threadIdx.x == 0) *g.fallback = out ? 1 : 0;
    return out;
}

// A power of two above a magnitude given as bits: its exponent.
__device__ __forceinline__ int split_exponent(uint32_t bits) { return (int)(bits >> 23) - 126; }

// The six products of parts, small ones first: (part of A, part of B) = (2, 0) (1, 1) (0, 2) (1, 0) (0, 1) (0, 0), 0 = high. A
// loop and not straight code: with the four products of a backward step unrolled, issuing and computing warps together outgrew
// the instruction cache. With the two operands exchanged and `mirrored` the same six come in the same order, so that a product and its
// transpose are the same bits.
constexpr int kSplitProducts = 6;
__device__ __forceinline__ uint32_t split_part_a(int i, bool mirrored = false) { return ((mirrored ? 0x124u : 0x046u) >> (2 * i)) & 3u; }
__device__ __forceinline__ uint32_t split_part_b(int i, bool mirrored = false) { return ((mirrored ? 0x046u : 0x124u) >> (2 * i)) & 3u; }

// Two neighbouring columns -> one 32-bit word of each part.
__device__ __forceinline__ void split_pair(float a, float b, uint32_t &hi, uint32_t &mid, uint32_t &lo)
{
    hi = ptx::pack_bf16(a, b);
    a -= __uint_as_float(hi << 16);
    b -= __uint_as_float(hi & 0xffff0000u);
    mid = ptx::pack_bf16(a, b);
    a -= __uint_as_float(mid << 16);
    b -= __uint_as_float(mid & 0xffff0000u);
    lo = ptx::pack_bf16(a, b);
}
__device__ __forceinline__ void split_pair(ptx::f32x2 v, uint32_t &hi, uint32_t &mid, uint32_t &lo)
{
    float a, b;
    ptx::unpack2(v, a, b);
    hi = ptx::pack_bf16(a, b);
    v = ptx::sub2(v, ptx::pack2(__uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u)));
    ptx::unpack2(v, a, b);
    mid = ptx::pack_bf16(a, b);
    v = ptx::sub2(v, ptx::pack2(__uint_as_float(mid << 16), __uint_as_float(mid & 0xffff0000u)));
    ptx::unpack2(v, a, b);
    lo = ptx::pack_bf16(a, b);
}
#endif

// One tensor to split: rows x cols float32, row-major -> three bf16 planes (of 2^16 times its values) of rows x cols
// rounded up to 8 (zeros there), one after the other. dst null: only looked through for values out of range.
struct SplitJob {
    const float *src = nullptr;
    void *dst = nullptr;
    long long rows = 0;
    int cols = 0;
};
// delta[row] = sum of out * dout over the row, made by further blocks of the same launch (the backward needs both before it starts)
struct SplitDelta {
    const float *out = nullptr, *dout = nullptr;
    float *delta = nullptr;
    long long rows = 0;
    int cols = 0;
};

inline size_t split_plane_elems(long long rows, int cols) { return (size_t)rows * ((cols + 7) / 8 * 8); }
inline size_t split_bytes(long long rows, int cols) { return align_up(3 * split_plane_elems(rows, cols) * 2, 256); }
// scratch for the guard's words
constexpr size_t kSplitGuardBytes = (2 * kSplitMaxBlocks + 64) * 4;

// Splits up to four tensors in one launch. guard_mem: kSplitGuardBytes. Any alignment of src; dst 16-byte aligned.
int split_f32(const SplitJob *jobs, int count, const SplitDelta *delta, void *guard_mem, SplitGuard *guard, cudaStream_t s);

}  // namespace ember
