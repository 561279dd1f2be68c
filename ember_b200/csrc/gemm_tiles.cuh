// How the tensor-core projection kernels (gemm_sm100.cu, gemm_f32_sm100.cu) walk their operands: tiles of a CTA pair, boxes of
// operands that may lie head-major, batch entries that are no multiple of the boxes.
#pragma once

#include "common.cuh"
#include "kernels.cuh"
#include "ptx.cuh"

namespace ember {

constexpr int BM = 128, BK = 64;              // BM: rows per CTA; a pair covers 2 * BM
constexpr int GROUP_M = 16;                   // tiles that share B columns run together

// seq: rows from one batch entry to the next in the TILE's row space, see RowPlan::seq_pad
struct ViewGeom {
    int heads, seq, dim;
};

#ifdef __CUDACC__
// TMA coordinates of a 64-column box of a view, walked along the contraction index. The producer
// computes coordinates on the critical path of every stage, so the divisions that split a row into
// (batch, position) and a column into (part, head, element) are done once per tile and the walk
// itself only adds and carries (all steps are 64; the padded seq is a multiple of 64, dim too unless
// there is a single head: a row-major matrix walked by batch entries).
struct BoxWalker {
    int c0, c1, c2, c3, c4;  // column | element, row | position, head, batch, part
    int heads, seq, dim;

    __device__ __forceinline__ void init(const ViewGeom &g, int row0, int col0)
    {
        heads = g.heads;
        seq = g.seq;
        dim = g.dim;
        if (heads == 0) {
            c0 = col0; c1 = row0; c2 = c3 = c4 = 0;
        } else {
            c3 = row0 / seq; c1 = row0 - c3 * seq;
            const int ph = col0 / dim;
            c0 = col0 - ph * dim;
            c4 = ph / heads; c2 = ph - c4 * heads;
        }
    }
    __device__ __forceinline__ void step_rows()  // 64 rows further
    {
        c1 += 64;
        if (heads != 0 && c1 >= seq) { c1 -= seq; c3++; }
    }
    __device__ __forceinline__ void step_cols()  // 64 columns further
    {
        c0 += 64;
        if (heads != 0 && c0 >= dim) {
            c0 = 0;
            if (++c2 >= heads) { c2 = 0; c4++; }
        }
    }
    // part0: parts to skip (a plane of a split operand comes after all parts of the one before)
    __device__ __forceinline__ void load(uint32_t dst, const CUtensorMap *map, uint32_t bar, int part0 = 0) const
    {
        ptx::tma_load_5d_pair(dst, map, bar, c0, c1, c2, c3, c4 + part0);
    }
};

__device__ __forceinline__ void tile_coords(int tiles_m, int tiles_n, int tile, int &tm, int &tn)
{
    const int per_group = GROUP_M * tiles_n;
    const int g = tile / per_group, rem = tile - g * per_group;
    const int rows_here = min(GROUP_M, tiles_m - g * GROUP_M);
    tn = rem / rows_here;
    tm = g * GROUP_M + (rem - tn * rows_here);
}

#endif

// The batch entries the rows of a product are walked by. A head-major view whose seq is a multiple of the
// boxes' rows can be tiled as if its rows were consecutive; otherwise tiles (NN, NT: rows of A and C) or
// contraction steps (TN: rows of A and B) stop at the end of each entry, the copy engine fills the rest
// of the box with zeros, and what is computed for them is not stored. A row-major view on the same row
// axis is then described as one head of `cols` columns, so that its boxes end there too (with rows of the
// next entry in their place, an infinity among those would meet the other operand's zeros).
struct RowPlan {
    bool by_entry;
    int batch, seq, seq_pad;
};

inline RowPlan row_plan(const GemmArgs &g)
{
    const MatView *axis[2] = {&g.a, g.mode == GEMM_TN ? &g.b : &g.c};
    const long long rows = g.mode == GEMM_TN ? g.k : g.m;
    const int box = g.mode == GEMM_TN ? BK : BM;
    for (const MatView *v : axis)
        if (v->heads > 0 && v->seq % box != 0) return {true, (int)(rows / v->seq), v->seq, (v->seq + box - 1) / box * box};
    return {false, 1, (int)rows, (int)((rows + 2 * BM - 1) / (2 * BM) * (2 * BM))};
}

inline bool view_ok(const MatView &v)
{
    if (((uintptr_t)v.ptr & 15) != 0) return false;
    if (v.heads == 0) return v.cols % 8 == 0;
    // head-major: a box of 64 columns must stay inside one head
    return v.dim % 64 == 0 && v.rows % v.seq == 0 && v.cols % (v.heads * v.dim) == 0;
}

}  // namespace ember
