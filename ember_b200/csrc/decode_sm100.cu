// Decode over a contiguous bf16 key/value cache on the tensor cores (HBM-bound): one query row per
// (batch, query head), G = q_heads / kv_heads query heads read the same K/V head.
//
// The bound is reading the cache once, so the kernel is a stream: one CTA per SM, each with an equal
// share of ALL key tiles of the step (the (unit, 128-key tile) pairs of every batch entry and K/V head laid
// end to end and cut into equal slices; with sequences of their own lengths only the tiles that hold keys, which every
// CTA counts for itself), TMA producers running 3 K and 3 V tiles (192 KB) ahead, across the
// boundaries between units. A slice begins and ends inside a unit as a rule; those two segments leave
// float32 partials (output, maximum, sum) that a small second kernel merges, the units between them are
// finished by the CTA itself. Equal slices have no last wave: cutting every unit into splits of 512 keys
// left 1.7 waves of CTAs at 128 units x 4001 keys.
//
// The products are formed with the KEYS as the rows of the MMA, so that almost nothing is padding:
//   S^T (128 keys x 16)  = K (128 x D) Q^T      query heads are the 16 columns (N), zero-filled past G
//   O^T (D x 16)        += V^T (D x 128) P^T    V is the MN-major A operand straight from its TMA tile
// One thread owns one key: G scores to scale, exponentiate and write as bf16 into a 4 KB B operand. With
// the query heads as the 128 rows instead, every tile cost a full 128 x 128 softmax for G useful rows,
// 2850 clocks, about what the tile takes to arrive from HBM (5.5 TB/s); here it takes about 600.
// One query head per K/V head: its probabilities stay float32 in effect. A second column of P holds what the bf16
// rounding of the first left over (P = hi + lo to 2^-17, a column of the 16 that would be zero otherwise, so no
// more products and no more memory traffic), and the two columns of O are added when it is read. Rounded to bf16
// alone, the error of the results was 1.4 times that of the bf16 output itself (2.35e-3 against 1.65e-3 at 128 units x
// 4001 keys); with the second column it is 1.65e-3 again.
// A tile's maximum is taken over its 128 threads (shuffles, shared memory, one named barrier); the running
// reference moves, and O is rescaled in tensor memory, only when it grew by more than 2^8.
//
// Warps 0-3: softmax and results. Warp 4: tensor memory, MMA issue. Warp 5: TMA.
#include <math.h>

#include "common.cuh"
#include "kernels.cuh"
#include "ptx.cuh"

namespace ember {

namespace {

using namespace ptx;

constexpr int THREADS = 192, NG = 16;  // NG: columns of the transposed products
constexpr float LOG2E_D = 1.4426950408889634f, LN2_D = 0.6931471805599453f, RESCALE_D = 8.f;

template <int HD>
struct Cfg {
    static constexpr int NSUB = HD / 64, SUB = 128 * 128, TILE = NSUB * SUB;
    static constexpr int ST = HD == 128 ? 3 : 6;  // stages of K and of V
    static constexpr int Q_BYTES = NSUB * NG * 128, P_BYTES = 2 * NG * 128;
    static constexpr int OFF_K = 0, OFF_V = OFF_K + ST * TILE, OFF_Q = OFF_V + ST * TILE, OFF_P = OFF_Q + 2 * Q_BYTES;
    static constexpr int OFF_RED = OFF_P + 2 * P_BYTES;  // [2][4 warps][16] maxima (and sums)
    static constexpr int OFF_BAR = OFF_RED + 2 * 4 * NG * 4;
    static constexpr int B_KFULL = 0, B_KEMPTY = B_KFULL + ST, B_VFULL = B_KEMPTY + ST, B_VEMPTY = B_VFULL + ST,
                         B_QFULL = B_VEMPTY + ST, B_QEMPTY = B_QFULL + 2, B_S = B_QEMPTY + 2, B_R = B_S + 2, B_P = B_R + 2,
                         B_O = B_P + 2, NUM_BARS = B_O + 2;
    static constexpr int USED = OFF_BAR + 8 * NUM_BARS + 16, SMEM = USED + 1024;
    static constexpr int TMEM_S = 0, TMEM_O = 32, TMEM_COLS = 64;
};

enum { WD_KEMPTY = 401, WD_VEMPTY, WD_QEMPTY, WD_K, WD_V, WD_Q, WD_R, WD_P, WD_S, WD_O };

// What a CTA leaves for the merge: the unit that its slice is the first to hold a tile of and does not finish.
struct SharedUnit {
    long long end, total;  // where the unit's tiles end, and all tiles, on the axis that is cut into slices
    int unit, slot;        // unit < 0: nothing to merge here; slot: which of this CTA's two partials is the unit's
};

struct DecParams {
    __nv_bfloat16 *out;
    float *lse, *part_o, *part_ml;
    SharedUnit *shared_unit;  // one per CTA
    const int *seq_lens;
    int batch, kv_heads, rows;  // rows: query heads per unit
    int lk;                     // keys of a sequence, or the most where seq_lens gives each its own
    bool whole_units;
    int segment_cost;           // tiles that the end of a unit's part counts for when the lengths differ, else 0
    float scale_log2;
    DeviceStatus *status;
};

__host__ __device__ inline long long slice_begin(long long total, int i, int n) { return total * i / n; }

__device__ __forceinline__ int sequence_length(const DecParams &p, int b) { return p.seq_lens ? max(0, min(p.lk, p.seq_lens[b])) : p.lk; }

// Slice of CTA i of n: tiles [begin, end) of the `total` tiles of all units laid end to end; the first of them is tile kt
// of batch entry b, K/V head h.
struct Slice {
    long long begin, end, total;
    int b, h, kt;

    // Sequences of one length; `whole`: slices of whole units.
    __device__ __forceinline__ void cut(const DecParams &p, int i, int n, bool whole)
    {
        const int tiles = (p.lk + 127) / 128, step = whole ? tiles : 1;
        total = (long long)p.batch * p.kv_heads * (tiles / step);
        begin = slice_begin(total, i, n) * step;
        end = slice_begin(total, i + 1, n) * step;
        const int unit = (int)(begin / tiles);
        kt = (int)(begin - (long long)unit * tiles);
        b = unit / p.kv_heads;
        h = unit - b * p.kv_heads;
    }
    // Sequences of their own lengths; the 32 lanes of a warp together, the result is the same in all of them. Cut over
    // the padded length instead, the CTAs that hold the long sequences' tiles do all the work: lengths {32768, 63 x 100} and
    // 8 K/V heads of 4 query heads 718 us (300 with a CTA per 512 keys). A unit counts segment_cost tiles more than it has, for
    // the end of a segment (sums, results), or a CTA of many short sequences is the last to finish: lengths {32768, 1, 1, 1}
    // and 32 K/V heads of 4 query heads 138 -> 112 us.
    __device__ __forceinline__ void cut_lengths(const DecParams &p, int i, int n, int lane)
    {
        auto slots_of = [&](int at) {
            const int tiles = at < p.batch ? (sequence_length(p, at) + 127) / 128 : 0;
            return tiles > 0 ? tiles + p.segment_cost : 0;
        };
        long long sum = 0;
#pragma unroll 4
        for (int at = lane; at < p.batch; at += 32) sum += slots_of(at);
#pragma unroll
        for (int t = 16; t > 0; t >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, t);
        total = sum * p.kv_heads;
        begin = slice_begin(total, i, n);
        end = slice_begin(total, i + 1, n);
        b = h = kt = 0;
        if (begin >= end) return;
        long long before = 0;  // tiles of the batch entries before these 32
        for (int at = 0; at < p.batch; at += 32) {
            const int slots = slots_of(at + lane);
            const long long mine = (long long)slots * p.kv_heads;
            long long upto = mine;
#pragma unroll
            for (int t = 1; t < 32; t <<= 1) {
                const long long v = __shfl_up_sync(0xffffffffu, upto, t);
                if (lane >= t) upto += v;
            }
            const unsigned past = __ballot_sync(0xffffffffu, before + upto > begin);
            if (past) {
                const int src = __ffs(past) - 1, unit_slots = __shfl_sync(0xffffffffu, slots, src);
                const long long r = begin - (before + __shfl_sync(0xffffffffu, upto - mine, src));
                b = at + src;
                h = (int)(r / unit_slots);
                kt = (int)(r - (long long)h * unit_slots);  // (past the unit's last tile: the slice begins with the next unit)
                return;
            }
            before += __shfl_sync(0xffffffffu, upto, 31);
        }
    }
};

// The tiles of a slice in order, unit by unit.
struct TileIter {
    long long left;                        // tiles of the slice past this unit
    int b, h, unit, kt, last, len, tiles;  // tile kt of the slice's part [.., last) of this unit; len, tiles: the unit's keys and tiles
    bool first;                            // first tile of this unit in the slice

    __device__ __forceinline__ void load(const DecParams &p)
    {
        len = sequence_length(p, b);
        tiles = (len + 127) / 128;
    }
    __device__ __forceinline__ void segment()
    {
        const int n = (int)min(left, (long long)(tiles - kt));
        last = kt + n;
        left -= n;
        first = true;
    }
    __device__ __forceinline__ bool start(const DecParams &p, const Slice &s)
    {
        left = s.end - s.begin;
        if (left <= 0) return false;
        b = s.b;
        h = s.h;
        kt = s.kt;
        unit = b * p.kv_heads + h;
        load(p);
        if (kt >= tiles) {
            left += kt - tiles;  // what is left of the unit's extra slots is next_unit's to take
            return next_unit(p);
        }
        segment();
        return true;
    }
    __device__ __forceinline__ bool next(const DecParams &p)
    {
        if (kt + 1 < last) {
            kt++;
            first = false;
            return true;
        }
        return next_unit(p);
    }
    __device__ __forceinline__ bool next_unit(const DecParams &p)
    {
        left -= p.segment_cost;
        if (left <= 0) return false;
        kt = 0;
        unit++;
        if (++h == p.kv_heads) {
            h = 0;
            do {
                if (++b >= p.batch) return false;
                load(p);
            } while (tiles == 0);
            unit = b * p.kv_heads;
        }
        segment();
        return true;
    }
};

template <int HD, int G>
__global__ void __launch_bounds__(THREADS, 1) decode_sm100_kernel(const __grid_constant__ CUtensorMap tm_q,
                                                                  const __grid_constant__ CUtensorMap tm_k,
                                                                  const __grid_constant__ CUtensorMap tm_v, const DecParams p)
{
    using C = Cfg<HD>;
    constexpr int GP = G == 1 ? 2 : G;  // columns of P and O in use (G = 1: high and low part)
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar0 = smem_base + C::OFF_BAR;
    auto BAR = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem_gen + C::OFF_BAR + 8 * C::NUM_BARS);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < C::NUM_BARS; i++) mbar_init(BAR(i), (i >= C::B_R && i < C::B_O) ? 4 : 1);  // R and P: one arrival per softmax warp
        fence_mbar_init();
    }
    if (warp == 4) {
        tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
        tmem_relinquish();
    }
    if (warp == 5 && lane == 0) {
        prefetch_tensormap(&tm_q);
        prefetch_tensormap(&tm_k);
        prefetch_tensormap(&tm_v);
    }
    // rows of P past the query heads stay zero
    for (int i = threadIdx.x; i < 2 * C::P_BYTES / 16; i += THREADS)
        *reinterpret_cast<uint4 *>(smem_gen + C::OFF_P + i * 16) = make_uint4(0, 0, 0, 0);
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_launch_dependents();
    // The first tiles come into L2 while the kernel before this one ends. A softmax warp, idle until the first scores, asks for them: from the
    // copying warp's hands they stood before its own copies where there was nothing to wait for (113 decode steps of a block 2 % longer).
    if (warp == 3 && lane == 0 && !p.seq_lens) {
        Slice ahead;
        TileIter ti;
        ahead.cut(p, blockIdx.x, gridDim.x, p.whole_units);
        int n = 0;
        for (bool more = ti.start(p, ahead); more && n < C::ST; more = ti.next(p), n++)
            for (int sub = 0; sub < C::NSUB; sub++) {
                tma_prefetch_3d(&tm_k, sub * 64, ti.kt * 128, ti.unit);
                tma_prefetch_3d(&tm_v, sub * 64, ti.kt * 128, ti.unit);
            }
    }
    pdl_wait();  // the cache's new rows may come from the kernel before this one

    Slice slice;
    if (p.seq_lens) {
        __shared__ Slice found;
        if (warp == 0) {
            slice.cut_lengths(p, blockIdx.x, gridDim.x, lane);
            if (lane == 0) found = slice;
        }
        __syncthreads();
        slice = found;
    } else {
        slice.cut(p, blockIdx.x, gridDim.x, p.whole_units);
    }

    if (warp == 5) {
        if (lane == 0) {
            // ------------------------------------------------------------ TMA producer
            TileIter ti;
            int it = 0, seg = 0;
            bool ok = true;
            for (bool more = ti.start(p, slice); more && ok; more = ti.next(p), it++) {
                const int s = it % C::ST, par = ((it / C::ST) & 1) ^ 1;
                if (ti.first) {
                    const int qs = seg & 1;
                    if (!(ok = mbar_wait(BAR(C::B_QEMPTY + qs), ((seg >> 1) & 1) ^ 1, abort_flag, p.status, WD_QEMPTY))) break;
                    mbar_arrive_expect_tx(BAR(C::B_QFULL + qs), C::Q_BYTES);
                    for (int sub = 0; sub < C::NSUB; sub++)
                        tma_load_3d(smem_base + C::OFF_Q + qs * C::Q_BYTES + sub * NG * 128, &tm_q, BAR(C::B_QFULL + qs), sub * 64, 0, ti.unit);
                    seg++;
                }
                if (!(ok = mbar_wait(BAR(C::B_KEMPTY + s), par, abort_flag, p.status, WD_KEMPTY))) break;
                mbar_arrive_expect_tx(BAR(C::B_KFULL + s), C::TILE);
                for (int sub = 0; sub < C::NSUB; sub++)
                    tma_load_3d(smem_base + C::OFF_K + s * C::TILE + sub * C::SUB, &tm_k, BAR(C::B_KFULL + s), sub * 64, ti.kt * 128, ti.unit);
                if (!(ok = mbar_wait(BAR(C::B_VEMPTY + s), par, abort_flag, p.status, WD_VEMPTY))) break;
                mbar_arrive_expect_tx(BAR(C::B_VFULL + s), C::TILE);
                for (int sub = 0; sub < C::NSUB; sub++)
                    tma_load_3d(smem_base + C::OFF_V + s * C::TILE + sub * C::SUB, &tm_v, BAR(C::B_VFULL + s), sub * 64, ti.kt * 128, ti.unit);
            }
            // A CTA that gave up stays until its copies have landed: every full barrier whose phase is open
            // is polled, bounded, for the last copies that were issued (it counts whole iterations, so
            // one more K tile may be in flight).
            const long long c0 = clock64();
            for (int j = max(0, it - C::ST); j < it + (ok ? 0 : 1); j++)
                for (int b = C::B_KFULL; b <= C::B_VFULL; b += C::B_VFULL - C::B_KFULL)
                    while (!mbar_try_wait(BAR(b + j % C::ST), (j / C::ST) & 1) && clock64() - c0 < kWaitLimitCycles && (ok || clock64() - c0 < 1000000)) {}
        }
    } else if (warp == 4) {
        // ---------------------------------------------------------------- MMA issue
        constexpr uint32_t IDESC_S = idesc_bf16_f32(128, NG, 0, 0), IDESC_O = idesc_bf16_f32(128, NG, 1, 0);
        TileIter ahead, cur;
        bool ok = true;
        int its = 0, seg = 0, it = 0;  // next score tile, its segment, current PV tile
        auto issue_s = [&]() {         // scores of tile `ahead`
            const int s = its % C::ST, b = its & 1;
            if (ahead.first) {
                ok = ok && mbar_wait(BAR(C::B_QFULL + (seg & 1)), (seg >> 1) & 1, abort_flag, p.status, WD_Q);
                seg++;
            }
            ok = ok && mbar_wait(BAR(C::B_KFULL + s), (its / C::ST) & 1, abort_flag, p.status, WD_K);
            if (its >= 2) ok = ok && mbar_wait(BAR(C::B_R + b), ((its >> 1) - 1) & 1, abort_flag, p.status, WD_R);
            tc_fence_after();
            const uint32_t k_lo = desc_lo(smem_base + C::OFF_K + s * C::TILE, 16);
            const uint32_t q_lo = desc_lo(smem_base + C::OFF_Q + ((seg - 1) & 1) * C::Q_BYTES, 16);
#pragma unroll
            for (int ks = 0; ks < HD / 16; ks++)
                mma_ss_lo(tmem + C::TMEM_S + b * NG, k_lo + (((ks / 4) * C::SUB + (ks % 4) * 32) >> 4),
                          q_lo + (((ks / 4) * NG * 128 + (ks % 4) * 32) >> 4), IDESC_S, ks > 0);
            tc_commit_elect(BAR(C::B_S + b));
            tc_commit_elect(BAR(C::B_KEMPTY + s));
            if (ahead.kt + 1 >= ahead.last) tc_commit_elect(BAR(C::B_QEMPTY + ((seg - 1) & 1)));
            its++;
        };
        bool more_s = ahead.start(p, slice);
        if (more_s) {
            issue_s();
            more_s = ahead.next(p);
        }
        for (bool more = cur.start(p, slice); more && ok; more = cur.next(p), it++) {
            if (more_s) {
                issue_s();
                more_s = ahead.next(p);
            }
            const int s = it % C::ST, b = it & 1;
            ok = ok && mbar_wait(BAR(C::B_VFULL + s), (it / C::ST) & 1, abort_flag, p.status, WD_V);
            if (p.seq_lens && cur.kt * 128 + 128 > cur.len) {
                // TMA zero-fills rows past the MAP's end only; between a sequence's own length and there
                // the cache may hold anything, and 0 * Inf would poison the product: zero those rows here
                uint8_t *vt = smem_gen + C::OFF_V + s * C::TILE;
                const int r0 = cur.len - cur.kt * 128;
                for (int i = lane; i < (128 - r0) * C::NSUB * 8; i += 32) {
                    const int rr = r0 + i / (C::NSUB * 8), sub = (i / 8) % C::NSUB, ch = i % 8;
                    *reinterpret_cast<uint4 *>(vt + sub * C::SUB + rr * 128 + ch * 16) = make_uint4(0, 0, 0, 0);
                }
                fence_proxy_async();
                __syncwarp();
            }
            ok = ok && mbar_wait(BAR(C::B_P + b), (it >> 1) & 1, abort_flag, p.status, WD_P);
            tc_fence_after();
            // HD = 64: the 64 columns of V stand in for rows 64-127 of the MMA a second time; nobody reads those
            const uint32_t v_lo = desc_lo(smem_base + C::OFF_V + s * C::TILE, HD == 128 ? C::SUB : 0);
            const uint32_t p_lo = desc_lo(smem_base + C::OFF_P + b * C::P_BYTES, 16);
#pragma unroll
            for (int ks = 0; ks < 8; ks++)
                mma_ss_lo(tmem + C::TMEM_O, v_lo + ks * (2048 >> 4), p_lo + (((ks / 4) * NG * 128 + (ks % 4) * 32) >> 4), IDESC_O,
                          (!cur.first || ks > 0) ? 1u : 0u);
            tc_commit_elect(BAR(C::B_VEMPTY + s));
            tc_commit_elect(BAR(C::B_O + b));
        }
    } else {
        // ---------------------------------------------------------------- softmax: one thread per key
        const uint32_t lane_sel = (uint32_t)(warp * 32) << 16;
        float *red = reinterpret_cast<float *>(smem_gen + C::OFF_RED);
        const int tid = threadIdx.x;
        TileIter ti;
        int it = 0;
        bool ok = true;
        float m[G], l[G];
        if (tid == 0) p.shared_unit[blockIdx.x].unit = -1;
        int segment = 0;
        // Tiles [kt0, kt1) of a unit are done: the result, or a partial of the units that other CTAs have a part of. A
        // CTA has at most two of those, the one its slice begins in (slot 0) and the one it ends in.
        auto finish = [&](int unit, int kt0, int kt1, int tiles) {
            uint32_t o[NG];
            ok = ok && mbar_wait(BAR(C::B_O + (it & 1)), (it >> 1) & 1, abort_flag, p.status, WD_O);
            tc_fence_after();
            tmem_ld_32x32b_x16(tmem + lane_sel + C::TMEM_O, o);
            tmem_wait_ld();
            tc_fence_before();
            // sums over the 128 keys' threads
            named_bar_sync(1, 128);
            float lt[G];
#pragma unroll
            for (int g = 0; g < G; g++) {
                float v = l[g];
#pragma unroll
                for (int t = 16; t > 0; t >>= 1) v += __shfl_xor_sync(0xffffffffu, v, t);
                if (lane == 0) red[warp * NG + g] = v;
            }
            named_bar_sync(1, 128);
#pragma unroll
            for (int g = 0; g < G; g++) lt[g] = (red[g] + red[NG + g]) + (red[2 * NG + g] + red[3 * NG + g]);
            named_bar_sync(1, 128);  // red is written again by the next tile
            const bool whole = kt0 == 0 && kt1 == tiles;
            const int slot = 2 * blockIdx.x + (segment == 0 ? 0 : 1);
            segment++;
            if (tid == 0 && kt0 == 0 && !whole) {  // the slice ends here, and the next one goes on with this unit
                const SharedUnit su = {slice.end + (tiles - kt1), slice.total, unit, slot & 1};
                p.shared_unit[blockIdx.x] = su;
            }
            // thread g has head g's maximum and sum to itself: one logarithm for all heads
            float m_own = m[0], l_own = lt[0];
#pragma unroll
            for (int g = 1; g < G; g++) {
                m_own = tid == g ? m[g] : m_own;
                l_own = tid == g ? lt[g] : l_own;
            }
            const size_t row0 = (whole ? (size_t)unit : (size_t)slot) * p.rows;
            if (ok && tid < p.rows) {
                if (!whole) *reinterpret_cast<float2 *>(p.part_ml + (row0 + tid) * 2) = make_float2(m_own, l_own);
                else if (p.lse) p.lse[row0 + tid] = l_own == 0.f ? -INFINITY : (m_own + log2f(l_own)) * LN2_D;
            }
#pragma unroll
            for (int g = 0; g < G; g++) {
                if (g >= p.rows || !ok || tid >= HD) continue;
                const float ov = G == 1 ? __uint_as_float(o[0]) + __uint_as_float(o[1]) : __uint_as_float(o[g]);
                if (whole) p.out[(row0 + g) * HD + tid] = __float2bfloat16_rn(lt[g] == 0.f ? 0.f : ov * (1.f / lt[g]));  // no weight anywhere: zeros
                else p.part_o[(row0 + g) * HD + tid] = ov;
            }
        };
        // A thread that gave up on a wait carries on, so that all 128 still meet at the named barriers.
        int kt0 = 0;
        for (bool more = ti.start(p, slice); more; more = ti.next(p), it++) {
            if (ti.first) kt0 = ti.kt;
            const int b = it & 1;
            ok = ok && mbar_wait(BAR(C::B_S + b), (it >> 1) & 1, abort_flag, p.status, WD_S);
            tc_fence_after();
            uint32_t u[NG];
            tmem_ld_32x32b_x16(tmem + lane_sel + C::TMEM_S + b * NG, u);
            tmem_wait_ld();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR(C::B_R + b));
            const bool valid = ti.kt * 128 + tid < ti.len;
            float x[G], mt[G];
#pragma unroll
            for (int g = 0; g < G; g++) {
                x[g] = valid ? __uint_as_float(u[g]) * p.scale_log2 : -INFINITY;
                float v = x[g];
#pragma unroll
                for (int t2 = 16; t2 > 0; t2 >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, t2));
                if (lane == 0) red[(b * 4 + warp) * NG + g] = v;
            }
            named_bar_sync(1, 128);
            bool grow = false;
#pragma unroll
            for (int g = 0; g < G; g++) {
                const float *r = red + b * 4 * NG + g;
                mt[g] = fmaxf(fmaxf(r[0], r[NG]), fmaxf(r[2 * NG], r[3 * NG]));  // -inf where no key of the tile has a score above it
                if (ti.first) {
                    m[g] = mt[g];
                    l[g] = 0.f;
                }
                grow = grow || mt[g] - m[g] > RESCALE_D;  // the same in all 128 threads
            }
            if (grow) {
                float alpha[G];
#pragma unroll
                for (int g = 0; g < G; g++) {
                    const float mn = fmaxf(m[g], mt[g]);
                    alpha[g] = m[g] == mn ? 1.f : ex2(m[g] - mn);  // (both -inf: another head's maximum grew)
                    m[g] = mn;
                    l[g] *= alpha[g];
                }
                ok = ok && mbar_wait(BAR(C::B_O + ((it - 1) & 1)), ((it - 1) >> 1) & 1, abort_flag, p.status, WD_O);
                tc_fence_after();
                uint32_t o[NG];
                tmem_ld_32x32b_x16(tmem + lane_sel + C::TMEM_O, o);
                tmem_wait_ld();
#pragma unroll
                for (int g = 0; g < GP; g++) o[g] = __float_as_uint(__uint_as_float(o[g]) * alpha[G == 1 ? 0 : g]);
                tmem_st_32x32b_x16(tmem + lane_sel + C::TMEM_O, o);
                tmem_wait_st();
                tc_fence_before();
            }
            if (it >= 2) ok = ok && mbar_wait(BAR(C::B_O + b), ((it >> 1) - 1) & 1, abort_flag, p.status, WD_O);  // P(it-2) has been read
            uint8_t *pb = smem_gen + C::OFF_P + b * C::P_BYTES + (tid / 64) * (NG * 128) + (tid % 8) * 2;
            auto store_p = [&](int col, __nv_bfloat16 v) {
                *reinterpret_cast<__nv_bfloat16 *>(pb + col * 128 + ((((tid % 64) / 8) ^ (col & 7)) << 4)) = v;
            };
#pragma unroll
            for (int g = 0; g < G; g++) {
                // every score so far is -inf: 0 as the reference keeps inf - inf out, the weights are 0
                const float pr = ex2(x[g] - (m[g] == -INFINITY ? 0.f : m[g]));
                l[g] += pr;
                const __nv_bfloat16 hi = __float2bfloat16_rn(pr);
                store_p(g, hi);
                if constexpr (G == 1) store_p(1, __float2bfloat16_rn(pr - __bfloat162float(hi)));
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR(C::B_P + b));
            if (ti.kt + 1 >= ti.last) finish(ti.unit, kt0, ti.last, ti.tiles);
        }
        // sequences without keys are on no slice: zeros and -inf
        for (int b = blockIdx.x; p.seq_lens && b < p.batch; b += gridDim.x) {
            if (sequence_length(p, b) > 0) continue;
            const size_t row0 = (size_t)b * p.kv_heads * p.rows;
            for (int i = tid; i < p.kv_heads * p.rows * HD; i += 128) p.out[row0 * HD + i] = __float2bfloat16_rn(0.f);
            for (int i = tid; p.lse && i < p.kv_heads * p.rows; i += 128) p.lse[row0 + i] = -INFINITY;
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 4) tmem_dealloc(tmem, C::TMEM_COLS);
}

// Merges the partial segments of the units that several CTAs share: one block per (CTA whose slice such a unit begins
// in, query head). Thread k reads slice k's maximum and sum, so that they take one memory latency, and the outputs are
// added with eight loads in flight; a unit of 32 tiles has 32 slices, and one after the other they took 20 us.
constexpr int MAX_SLICES = 256;

template <int HD>
__global__ void __launch_bounds__(128) decode_merge_kernel(const float *part_o, const float *part_ml,
                                                           const SharedUnit *shared_unit, __nv_bfloat16 *__restrict__ out,
                                                           float *__restrict__ lse, int rows, int ncta)
{
    __shared__ float sm_m[MAX_SLICES], sm_w[MAX_SLICES], red[4], half_sum[HD];
    __shared__ int sm_row[MAX_SLICES], count;
    const int i = blockIdx.x / rows, g = blockIdx.x - i * rows, tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    if (tid == 0) count = 0;
    pdl_launch_dependents();
    pdl_wait();
    const SharedUnit su = shared_unit[i];
    if (su.unit < 0) return;  // the same in all threads
    __syncthreads();
    float mx = -INFINITY;
    for (int k = tid; k < ncta - i; k += 128) {
        const long long begin = slice_begin(su.total, i + k, ncta);
        const bool used = begin < su.end && slice_begin(su.total, i + k + 1, ncta) > begin;
        const int row = (2 * (i + k) + (k == 0 ? su.slot : 0)) * rows + g;
        sm_row[k] = used ? row : -1;
        sm_m[k] = used ? part_ml[(size_t)row * 2] : -INFINITY;
        sm_w[k] = used ? part_ml[(size_t)row * 2 + 1] : 0.f;  // the sum, until the maximum is known
        mx = fmaxf(mx, sm_m[k]);
        if (used) atomicMax(&count, k + 1);
    }
#pragma unroll
    for (int t = 16; t > 0; t >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, t));
    if (lane == 0) red[warp] = mx;
    __syncthreads();
    mx = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    const int n = count;
    float l = 0.f;
    for (int k = tid; k < n; k += 128) {
        const float w = sm_m[k] == -INFINITY ? 0.f : exp2f(sm_m[k] - mx);
        l += sm_w[k] * w;  // (a NaN sum stays NaN)
        sm_w[k] = w;
    }
#pragma unroll
    for (int t = 16; t > 0; t >>= 1) l += __shfl_xor_sync(0xffffffffu, l, t);
    __syncthreads();
    if (lane == 0) red[warp] = l;
    __syncthreads();
    l = (red[0] + red[1]) + (red[2] + red[3]);
    constexpr int WAYS = 128 / HD;  // threads per column: they take every other slice
    const int c = tid % HD;
    float acc = 0.f;
#pragma unroll 8
    for (int k = tid / HD; k < n; k += WAYS)
        if (sm_row[k] >= 0) acc += part_o[(size_t)sm_row[k] * HD + c] * sm_w[k];
    if (WAYS == 2) {
        if (tid >= HD) half_sum[c] = acc;
        __syncthreads();
        acc += half_sum[c];
    }
    const size_t r = (size_t)su.unit * rows + g;
    if (tid < HD) out[r * HD + c] = __float2bfloat16_rn(l == 0.f ? 0.f : acc * (1.f / l));
    if (tid == 0 && lse) lse[r] = l == 0.f ? -INFINITY : (mx + log2f(l)) * LN2_D;
}

// Short sequences are not cut: the merge would take longer than a few tiles. us, cut -> whole, d 128: 128 units x 384 keys, group 1 / 16:
// 19 -> 15, 26 -> 17; 64 x 768 keys: 19 -> 15, 26 -> 18; 256 x 1001 keys: 40 -> 36, 46 -> 40; 16 units x 1001 keys 15 both, 17 -> 18.
bool whole_units(const CacheDecodeArgs &a)
{
    const int tiles = (a.lk + 127) / 128;
    return !a.seq_lens && (tiles <= 4 || (tiles <= 8 && a.batch * a.kv_heads >= 32));
}

int slices(const CacheDecodeArgs &a, int sms)
{
    const long long total = (long long)a.batch * a.kv_heads * (whole_units(a) ? 1 : (a.lk + 127) / 128);
    const int most = sms < MAX_SLICES ? sms : MAX_SLICES;
    return (int)(total < most ? total : most);
}

template <int HD, int G>
int launch(const CacheDecodeArgs &a, DeviceState *st, cudaStream_t s)
{
    using C = Cfg<HD>;
    const int units = a.batch * a.kv_heads, rows = a.q_heads / a.kv_heads;
    const int ncta = slices(a, st->sm_count > 0 ? st->sm_count : 148);
    CUtensorMap tq, tk, tv;
    int rc;
    if ((rc = make_tensor_map_bf16_3d(&tq, a.q, HD, rows, units, 64, NG)) != EMBER_OK) return rc;
    if ((rc = make_tensor_map_bf16_3d(&tk, a.k_cache, HD, a.lk, units, 64, 128, a.capacity)) != EMBER_OK) return rc;
    if ((rc = make_tensor_map_bf16_3d(&tv, a.v_cache, HD, a.lk, units, 64, 128, a.capacity)) != EMBER_OK) return rc;
    DecParams p;
    p.out = (__nv_bfloat16 *)a.out;
    p.lse = a.lse;
    p.part_o = (float *)a.workspace;
    p.part_ml = p.part_o + (size_t)2 * ncta * rows * HD;
    p.shared_unit = reinterpret_cast<SharedUnit *>(p.part_ml + (size_t)2 * ncta * rows * 2);
    p.seq_lens = a.seq_lens;
    p.batch = a.batch;
    p.kv_heads = a.kv_heads;
    p.rows = rows;
    p.lk = a.lk;
    p.whole_units = whole_units(a);
    p.segment_cost = !a.seq_lens ? 0 : rows <= 2 ? 1 : rows <= 8 ? 2 : 4;
    p.scale_log2 = a.scale * LOG2E_D;
    p.status = st->status;
    auto kern = decode_sm100_kernel<HD, G>;
    static SmemOptIn opt_in;
    EMBER_CUDA_TRY(opt_in(kern, C::SMEM));
    LaunchAttrs attrs;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ncta);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = s;
    attrs.pdl().set(cfg);
    EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tq, tk, tv, p));
    // a unit is shared whenever a slice begins inside it
    const int tiles = (a.lk + 127) / 128;
    const long long total = (long long)units * tiles;
    if (ncta > 1 && !p.whole_units && (a.seq_lens || total % ncta != 0 || (total / ncta) % tiles != 0)) {
        cfg.gridDim = dim3((unsigned)(ncta * rows));
        cfg.blockDim = dim3(128);
        cfg.dynamicSmemBytes = 0;
        EMBER_CUDA_TRY(cudaLaunchKernelEx(&cfg, decode_merge_kernel<HD>, (const float *)p.part_o, (const float *)p.part_ml,
                                          (const SharedUnit *)p.shared_unit, p.out, p.lse, rows, ncta));
    }
    return EMBER_OK;
}

template <int HD>
int dispatch(const CacheDecodeArgs &a, DeviceState *st, cudaStream_t s)
{
    const int rows = a.q_heads / a.kv_heads;
    if (rows == 1) return launch<HD, 1>(a, st, s);
    if (rows == 2) return launch<HD, 2>(a, st, s);
    if (rows <= 4) return launch<HD, 4>(a, st, s);
    if (rows <= 8) return launch<HD, 8>(a, st, s);
    return launch<HD, 16>(a, st, s);
}

}  // namespace

bool sm100_decode_supported(const CacheDecodeArgs &a)
{
    if (a.dtype != EMBER_BF16 || (a.d != 64 && a.d != 128)) return false;
    if (a.q_heads % a.kv_heads != 0 || a.q_heads / a.kv_heads > NG || !isfinite(a.scale)) return false;
    const uintptr_t bits = (uintptr_t)a.q | (uintptr_t)a.k_cache | (uintptr_t)a.v_cache;
    return (bits & 15) == 0;
}

size_t sm100_decode_workspace_bytes(int rows, int d, int sms)
{
    return (size_t)2 * sms * rows * (d + 2) * sizeof(float) + (size_t)sms * sizeof(SharedUnit);
}

int sm100_decode(const CacheDecodeArgs &a, DeviceState *st, cudaStream_t s)
{
    return a.d == 128 ? dispatch<128>(a, st, s) : dispatch<64>(a, st, s);
}

}  // namespace ember
