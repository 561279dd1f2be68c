// The extern "C" entry points of the Linear layers either side of attention: argument checks,
// then dispatch of each matrix product to the tcgen05 kernel (bf16, aligned views) or the CUDA-core
// kernel (float32 mode and everything else).
#include "common.cuh"
#include "kernels.cuh"
#include "split_f32.cuh"

using namespace ember;

namespace {

struct LinearShape {
    long long m;
    int n, k, dtype, x_heads, y_heads, seq, head_dim;
};

int check_linear(const char *fn, const LinearShape &s)
{
    EMBER_REQUIRE(s.dtype == EMBER_F32 || s.dtype == EMBER_BF16, "%s: unknown dtype %d", fn, s.dtype);
    EMBER_REQUIRE(s.m > 0 && s.n > 0 && s.k > 0, "%s: extents must be positive, got m=%lld n=%d k=%d", fn, s.m, s.n, s.k);
    EMBER_REQUIRE(s.x_heads >= 0 && s.y_heads >= 0, "%s: negative head count", fn);
    if (s.x_heads > 0 || s.y_heads > 0) {
        EMBER_REQUIRE(s.seq > 0 && s.head_dim > 0, "%s: head-major layout needs seq > 0 and head_dim > 0", fn);
        EMBER_REQUIRE(s.m % s.seq == 0, "%s: m=%lld is not a multiple of seq=%d", fn, s.m, s.seq);
    }
    if (s.x_heads > 0)
        EMBER_REQUIRE(s.k == s.x_heads * s.head_dim, "%s: k=%d must equal x_heads*head_dim=%d", fn, s.k,
                      s.x_heads * s.head_dim);
    if (s.y_heads > 0)
        EMBER_REQUIRE(s.n % (s.y_heads * s.head_dim) == 0, "%s: n=%d is not a multiple of y_heads*head_dim=%d", fn,
                      s.n, s.y_heads * s.head_dim);
    return EMBER_OK;
}

MatView view(const void *p, long long rows, int cols, int heads, const LinearShape &s)
{
    MatView v;
    v.ptr = p;
    v.rows = rows;
    v.cols = cols;
    v.heads = heads;
    v.seq = heads ? s.seq : 0;
    v.dim = heads ? s.head_dim : 0;
    return v;
}

// The three products of a layer: y (m x n) = x w, grad_w (k x n) = x^T dy, grad_x (m x k) = dy w^T.
enum { FORWARD = 0, GRAD_W = 1, GRAD_X = 2 };

GemmArgs product_of(int product, const LinearShape &s, const void *x, const void *w, const void *y_or_dy, const void *out)
{
    const MatView vx = view(x, s.m, s.k, s.x_heads, s), vw = view(w, s.k, s.n, 0, s), vdy = view(y_or_dy, s.m, s.n, s.y_heads, s);
    GemmArgs g;
    g.dtype = s.dtype;
    if (product == GRAD_W) {
        g.mode = GEMM_TN;
        g.a = vx; g.b = vdy; g.c = view(out, s.k, s.n, 0, s);
        g.m = s.k; g.n = s.n; g.k = (int)s.m;
    } else if (product == GRAD_X) {
        g.mode = GEMM_NT;
        g.a = vdy; g.b = vw; g.c = view(out, s.m, s.k, s.x_heads, s);
        g.m = s.m; g.n = s.k; g.k = s.n;
    } else {
        g.mode = GEMM_NN;
        g.a = vx; g.b = vw; g.c = vdy;
        g.m = s.m; g.n = s.n; g.k = s.k;
    }
    return g;
}

// Copies of operands whose rows are no multiple of 16 bytes (a vocabulary of 50257 columns, say), padded with
// zeros to rows that the copy engine can fetch. They live for one entry point's call, so that the two
// gradients of a backward call share the copy of dy, and are freed in stream order.
struct PackedOperands {
    cudaStream_t stream;
    int count = 0;
    MatView from[4], to[4];  // x, dy and w are all there are

    explicit PackedOperands(cudaStream_t s) : stream(s) {}
    PackedOperands(const PackedOperands &) = delete;
    PackedOperands &operator=(const PackedOperands &) = delete;
    ~PackedOperands()
    {
        for (int i = 0; i < count; i++) cudaFreeAsync(const_cast<void *>(to[i].ptr), stream);
    }
    // v becomes its copy. EMBER_ERR_NOMEM: there is no memory for one, v and the error state are as they were.
    int get(MatView &v)
    {
        for (int i = 0; i < count; i++)
            if (from[i].ptr == v.ptr && from[i].rows == v.rows && from[i].cols == v.cols) {
                v = to[i];
                return EMBER_OK;
            }
        MatView t = v;
        t.cols = (v.cols + 7) / 8 * 8;
        void *buf = nullptr;
        if (!scratch_alloc(&buf, (size_t)t.rows * t.cols * 2, stream)) return EMBER_ERR_NOMEM;
        t.ptr = buf;
        from[count] = v;
        to[count++] = t;
        const int rc = pack_rows(v, buf, stream);
        v = t;
        return rc;
    }
};

bool needs_packing(const MatView &v) { return v.heads == 0 && (v.cols % 8 != 0 || ((uintptr_t)v.ptr & 15) != 0); }

// Whether a product that the tensor-core kernels refuse for its operands' rows is to run on copies of them.
// A copy costs a launch or two, a tile of results with odd rows is stored element by element, and the CUDA-core kernel is
// quick on small products. Forward / both gradients, us, CUDA cores -> copies: 2.7e7 flop a product (256 x 101 x 512)
// 14 / 33 -> 21 / 39, 6.7e7 (256 x 513 x 256) 19 / 45 -> 19 / 43, 1.1e8 (512 x 101 x 1024) 29 / 50 -> 23 / 40, 2.1e9
// (1024 x 1001 x 1024) 160 / 268 -> 25 / 50, 1.2e10 (2000 x 3001 x 1024) 566 / 1372 -> 35 / 71.
// A contraction shorter than one step of the tensor-core kernel (64) leaves little but the tiles' stores: only results large on
// both sides gain, from 8 on; those with odd rows of their own, which are stored element by element, from 16 and more work on. us,
// CUDA cores -> copies (rows x columns of the result, contraction): odd rows 1024 x 3001, 16 and 32: 17 and 25 -> 25 and 23; 777 x
// 10001 (two copies), 8, 16 and 32: 19, 29 and 43 -> 35, 45 and 45; 1024 x 50257, 8 and 16: 86 and 125 -> 111 and 111; others
// 4096 x 16384, 1: 70 -> 76, 8192 x 2048, 10: 38 -> 29, 200000 x 128, 33: 98 -> 86; narrow ones 64 x 1000001, 32: 300 -> 484, 10^6 x 64, 10: 123 -> 340.
constexpr double kPackFlops = 8e7;
constexpr int kPackShort = 64;

bool worth_packing(const GemmArgs &g)
{
    const bool copy_a = needs_packing(g.a), copy_b = needs_packing(g.b);
    if (g.dtype != EMBER_BF16 || (!copy_a && !copy_b)) return false;
    double least = kPackFlops;
    if (g.k < kPackShort) {
        const bool odd_results = g.n % 8 != 0 || ((uintptr_t)g.c.ptr & 15) != 0;
        if (g.k < (odd_results ? 16 : 8)) return false;
        const int side = !odd_results && g.k >= 32 ? 128 : 512;
        if (g.m < side || g.n < side) return false;
        if (odd_results) least = copy_a && copy_b ? 4e8 : g.k == 16 ? 2e8 : least;
    }
    if (2.0 * (double)g.m * g.n * g.k < least) return false;
    if (g.a.rows > 0x7fffff00LL || g.b.rows > 0x7fffff00LL) return false;
    GemmArgs t = g;
    for (MatView *v : {&t.a, &t.b})
        if (needs_packing(*v)) {
            if (v->cols > 0x7ffffff0) return false;
            v->cols = (v->cols + 7) / 8 * 8;
            v->ptr = (const void *)(uintptr_t)256;
        }
    return sm100_skinny_gemm_supported(t) || sm100_gemm_supported(t);
}

// Float32 products on the tensor cores (gemm_f32_sm100.cu): the operands' planes are made in one launch for all products of an
// entry point, and the CUDA-core kernels behind them return at once unless an operand holds values that planes cannot.
//
// Which side takes a call: both times are estimated, in us. The tensor-core side starts at 17.5 for one product (split, product, the launch
// that returns) and 33 for two, splitting costs a pass (4 bytes read and 6 written an element, rows written as multiples of 8, at 5 TB/s), its tiles are 256 rows; the CUDA cores
// run at 40 TFLOP/s where tiles of 128 x 128 fill the SMs, at 17 to 34 below. Measured, CUDA cores / tensor cores, forward and both gradients
// (rows x contraction x columns):
//   300^3 10 / 18, 21 / 35      512^3 17 / 17, 35 / 33          1024^3 66 / 24, 153 / 46       2048^3 415 / 85, 831 / 168
//   256 x 1024 x 1000 30 / 18, 50 / 36      8192 x 64 x 1000 30 / 22, 128 / 80     4000 x 512 x 200 35 / 20, 87 / 50    2000 x 1024 x 3001 354 / 84, 1003 / 161
//   8192 x 512 x 64 34 / 22, 47 / 66        64 x 2048 x 8192 125 / 84, 183 / 155   32 x 1024 x 16384 61 / 75, 103 / 155
constexpr double kSplitUsPerByte = 1.0 / 5e6;

double simt_f32_us(const GemmArgs &g, int sms)
{
    const bool full = (double)((g.m + 127) / 128) * ((g.n + 127) / 128) >= sms;
    return 6.0 + 2.0 * (double)g.m * g.n * g.k / (full ? 4e7 : 2.4e7);
}

struct F32Products {
    GemmArgs g[2];
    int count = 0;
    MatView ops[3];
    int nops = 0;

    int operand(const MatView &v)
    {
        for (int i = 0; i < nops; i++)
            if (ops[i].ptr == v.ptr && ops[i].rows == v.rows && ops[i].cols == v.cols && ops[i].heads == v.heads) return i;
        ops[nops] = v;
        return nops++;
    }
    void add(const GemmArgs &p)
    {
        g[count++] = p;
        operand(p.a);
        operand(p.b);
    }
    bool preferred(int sms)
    {
        if (count == 0) return false;
        double tensor = count > 1 ? 20.0 : 12.0, cores = 0;
        for (int i = 0; i < count; i++) {
            if (!sm100_f32_gemm_supported(g[i])) return false;
            tensor += sm100_f32_gemm_us(g[i], sms);
            cores += simt_f32_us(g[i], sms);
        }
        for (int i = 0; i < nops; i++) tensor += (4.0 * ops[i].rows * ops[i].cols + 6.0 * split_plane_elems(ops[i].rows, ops[i].cols)) * kSplitUsPerByte;
        if (tensor < (count > 1 ? 33.0 : 17.5)) tensor = count > 1 ? 33.0 : 17.5;
        return tensor < cores;
    }
    // EMBER_ERR_NOMEM: no memory for the planes, nothing launched
    int run(DeviceState *st, cudaStream_t s)
    {
        size_t at[3], bytes = 0;
        for (int i = 0; i < nops; i++) {
            at[i] = bytes;
            bytes += split_bytes(ops[i].rows, ops[i].cols);
        }
        char *mem = nullptr;
        if (!scratch_alloc((void **)&mem, bytes + kSplitGuardBytes, s)) return EMBER_ERR_NOMEM;
        SplitJob jobs[3];
        for (int i = 0; i < nops; i++) {
            jobs[i].src = (const float *)ops[i].ptr;
            jobs[i].dst = mem + at[i];
            jobs[i].rows = ops[i].rows;  // a head-major tensor is as many elements in a row, of which planes keep the order
            jobs[i].cols = ops[i].cols;
        }
        SplitGuard guard;
        int rc = split_f32(jobs, nops, nullptr, mem + bytes, &guard, s);
        for (int i = 0; i < count && rc == EMBER_OK; i++) rc = sm100_f32_gemm(g[i], mem + at[operand(g[i].a)], mem + at[operand(g[i].b)], guard, st, s);
        for (int i = 0; i < count && rc == EMBER_OK; i++) {
            GemmArgs t = g[i];
            t.only_if = guard.fallback;
            rc = simt_gemm(t, st, s);
        }
        cudaFreeAsync(mem, s);
        return rc;
    }
};

// Whether run() hands a product to sm100_gemm as it is.
bool on_tile_kernel(const GemmArgs &g)
{
    return !worth_packing(g) && sm100_gemm_supported(g) && !(sm100_skinny_gemm_supported(g) && sm100_skinny_gemm_preferred(g));
}

bool apart(const void *a, size_t an, const void *b, size_t bn)
{
    return (uintptr_t)a + an <= (uintptr_t)b || (uintptr_t)b + bn <= (uintptr_t)a;
}

int run(GemmArgs g, DeviceState *st, cudaStream_t s, PackedOperands &packed)
{
    if (worth_packing(g)) {
        GemmArgs t = g;
        int rc = EMBER_OK;
        if (needs_packing(t.a)) rc = packed.get(t.a);
        if (rc == EMBER_OK && needs_packing(t.b)) rc = packed.get(t.b);
        if (rc == EMBER_OK) g = t;
        else if (rc != EMBER_ERR_NOMEM) return rc;  // without memory for copies: the CUDA cores, which need none
    }
    const bool large = sm100_gemm_supported(g);
    if (sm100_skinny_gemm_supported(g) && (!large || sm100_skinny_gemm_preferred(g))) return sm100_skinny_gemm(g, st, s);
    if (large) return sm100_gemm(g, st, s);
    if (skinny_f32_supported(g)) return skinny_f32_gemm(g, st, s);
    if (narrow_f32_supported(g)) return narrow_f32_gemm(g, s);
    return simt_gemm(g, st, s);
}

}  // namespace

extern "C" {

int ember_linear_fwd(const void *x, const void *w, const void *bias, void *y, long long m, int n, int k, int dtype,
                     int x_heads, int y_heads, int seq, int head_dim, void *stream)
{
    const LinearShape sh = {m, n, k, dtype, x_heads, y_heads, seq, head_dim};
    int rc = check_linear("ember_linear_fwd", sh);
    if (rc) return rc;
    EMBER_REQUIRE(x && w && y, "ember_linear_fwd: NULL tensor pointer");
    DeviceState *st = device_state();
    if (!st) return EMBER_ERR_CUDA;
    GemmArgs g = product_of(FORWARD, sh, x, w, y, nullptr);
    g.bias = bias;
    PackedOperands packed(pick_stream(stream, st));
    F32Products f32;
    if (dtype == EMBER_F32 && !skinny_f32_supported(g) && !narrow_f32_supported(g)) f32.add(g);
    if (f32.preferred(st->sm_count) && (rc = f32.run(st, packed.stream)) != EMBER_ERR_NOMEM) return rc;
    return run(g, st, packed.stream, packed);
}

int ember_linear_fwd_cached(const void *x, const void *w, const void *bias, void *qkv, void *k_cache, void *v_cache, int batch, int heads, int d,
                            int capacity, int pos, int dtype, void *stream)
{
    const LinearShape sh = {batch, 3 * heads * d, heads * d, dtype, 0, heads, 1, d};
    int rc = check_linear("ember_linear_fwd_cached", sh);
    if (rc) return rc;
    EMBER_REQUIRE(x && w && qkv && k_cache && v_cache, "ember_linear_fwd_cached: NULL tensor pointer");
    EMBER_REQUIRE(pos >= 0 && pos < capacity, "ember_linear_fwd_cached: row %d does not fit a cache of %d rows", pos, capacity);
    DeviceState *st = device_state();
    if (!st) return EMBER_ERR_CUDA;
    GemmArgs g = product_of(FORWARD, sh, x, w, qkv, nullptr);
    g.bias = bias;
    // (caches that the copy of rows or the decode kernels refuse take the two calls, which say so)
    if (d % 8 == 0 && (((uintptr_t)k_cache | (uintptr_t)v_cache) & 15) == 0 && sm100_skinny_gemm_supported(g) &&
        (!sm100_gemm_supported(g) || sm100_skinny_gemm_preferred(g))) {
        const CacheRows rows = {k_cache, v_cache, heads * d, heads, capacity, d, pos};
        g.cache = &rows;
        return sm100_skinny_gemm(g, st, pick_stream(stream, st));
    }
    if ((rc = ember_linear_fwd(x, w, bias, qkv, batch, sh.n, sh.k, dtype, 0, heads, 1, d, stream)) != EMBER_OK) return rc;
    const size_t part = (size_t)batch * heads * d * dtype_size(dtype);
    return ember_kv_cache_append(k_cache, v_cache, (const char *)qkv + part, (const char *)qkv + 2 * part, batch, heads, capacity, d, 1, pos, nullptr,
                                 nullptr, 0, 0, dtype, stream);
}

int ember_linear_bwd(const void *x, const void *w, const void *dy, void *dx, void *dw, void *db, long long m, int n,
                     int k, int dtype, int x_heads, int y_heads, int seq, int head_dim, void *stream)
{
    const LinearShape sh = {m, n, k, dtype, x_heads, y_heads, seq, head_dim};
    int rc = check_linear("ember_linear_bwd", sh);
    if (rc) return rc;
    EMBER_REQUIRE(x && w && dy, "ember_linear_bwd: NULL tensor pointer");
    EMBER_REQUIRE(dx || dw || db, "ember_linear_bwd: no gradient requested");
    EMBER_REQUIRE(m <= 0x7fffffffLL, "ember_linear_bwd: m=%lld does not fit the weight-gradient product", m);
    DeviceState *st = device_state();
    if (!st) return EMBER_ERR_CUDA;
    cudaStream_t s = pick_stream(stream, st);
    if (dtype == EMBER_F32 && dw && !x_heads && !y_heads && narrow_f32_bwd_supported(x, w, dy, dx, db, m, n, k)) {
        const size_t xs = (size_t)m * k * 4, ws = (size_t)k * n * 4, ys = (size_t)m * n * 4, bs = (size_t)n * 4;
        if (apart(dw, ws, x, xs) && apart(dw, ws, w, ws) && apart(dw, ws, dy, ys) &&
            (!dx || (apart(dx, xs, x, xs) && apart(dx, xs, w, ws) && apart(dx, xs, dy, ys) && apart(dx, xs, dw, ws))) &&
            (!db || (apart(db, bs, x, xs) && apart(db, bs, w, ws) && apart(db, bs, dy, ys) && apart(db, bs, dw, ws) && (!dx || apart(db, bs, dx, xs)))))
            return narrow_f32_backward(x, w, dy, dx, dw, db, m, n, k, st, s);
    }
    PackedOperands packed(s);
    GemmArgs gw = product_of(GRAD_W, sh, x, w, dy, dw), gx = product_of(GRAD_X, sh, x, w, dy, dx);
    F32Products f32;
    if (dtype == EMBER_F32 && dw) f32.add(gw);
    if (dtype == EMBER_F32 && dx) f32.add(gx);
    bool done = false;
    if (f32.preferred(st->sm_count)) {
        if ((rc = f32.run(st, s)) != EMBER_OK && rc != EMBER_ERR_NOMEM) return rc;
        done = rc == EMBER_OK;
    }
    // The products on the tile kernel: they and the bias gradient run side by side. The input gradient starts on the SMs that the weight
    // gradient's last round leaves idle, where that makes it end sooner, and the bias gradient's blocks fit beside a product's on its SM, whose
    // memory bandwidth the product leaves alone: beside the input gradient, or beside the weight gradient where the input gradient waits for
    // both. us, one after the other -> side by side (rows x inputs x outputs): 8192 x 2048 x 6144 323 -> 304, 8192 x 2048 x 2048 116 -> 102,
    // 4096 x 1536 x 4608 116 -> 92, 1000 x 512 x 1536 26.5 -> 18, 2048 x 128 x 32768 202 -> 177, 8192 x 2048 x 32768, which is bound by power,
    // 1612 -> 1593 (1633 with the bias gradient beside the input gradient). Weight and bias gradient alone: 42 x 2048 x 6144 21.8 -> 17.9, 8712 x 1024 x 1024
    // 54 -> 48.5, over 90 shapes 0.87.
    const size_t xs = (size_t)m * k * 2, ws = (size_t)k * n * 2, ys = (size_t)m * n * 2, bs = (size_t)n * 2;
    // Each result has to lie apart from what the other two read: dx from x and dy, dw from w and dy, db from all; and from one another.
    if (!done && dw && (dx || db) && on_tile_kernel(gw) && apart(dw, ws, dy, ys) &&
        (!dx || (on_tile_kernel(gx) && apart(dx, xs, x, xs) && apart(dx, xs, dy, ys) && apart(dx, xs, dw, ws) && apart(dw, ws, w, ws))) &&
        (!db || (apart(db, bs, x, xs) && apart(db, bs, w, ws) && apart(db, bs, dy, ys) && apart(db, bs, dw, ws) && (!dx || apart(db, bs, dx, xs))))) {
        gw.leaves_room = gx.leaves_room = db != nullptr;
        const bool gains = gw.held = dx && sm100_gemm_gains_beside(gw, gx, st);
        if (gains) gx.beside = &gw; else gx.leaves_room = false;
        if ((rc = sm100_gemm(gw, st, s)) != EMBER_OK) return rc;
        if (!gains && db && (rc = column_sums(gw.b, db, dtype, st, s, true)) != EMBER_OK) return rc;
        if (dx && (rc = sm100_gemm(gx, st, s)) != EMBER_OK) return rc;
        return gains && db ? column_sums(gw.b, db, dtype, st, s, true) : EMBER_OK;
    }
    if (!done && dw && (rc = run(gw, st, s, packed)) != EMBER_OK) return rc;
    if (db && (rc = column_sums(gw.b, db, dtype, st, s)) != EMBER_OK) return rc;  // grad_b = sum(dy, axis 0)
    if (!done && dx && (rc = run(gx, st, s, packed)) != EMBER_OK) return rc;
    return EMBER_OK;
}

const char *ember_linear_kernel_name(int product, long long m, int n, int k, int dtype, int x_heads, int y_heads,
                                     int seq, int head_dim)
{
    // Pointers do not matter for the answer except for their alignment; aligned stand-ins, one for each tensor.
    const void *at[4];
    for (int i = 0; i < 4; i++) at[i] = (const void *)(uintptr_t)(256 * (i + 1));
    const LinearShape sh = {m, n, k, dtype, x_heads, y_heads, seq, head_dim};
    const GemmArgs g = product_of(product, sh, at[0], at[1], at[2], at[3]);
    if (dtype == EMBER_F32) {
        int dev = 0, sms = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
            cudaGetLastError();
            sms = 148;
        }
        F32Products f32;
        if (product == FORWARD) {
            if (!skinny_f32_supported(g) && !narrow_f32_supported(g)) f32.add(g);
        } else if (x_heads || y_heads || !narrow_f32_bwd_supported(at[0], at[1], at[2], at[3], nullptr, m, n, k)) {
            f32.add(product_of(GRAD_W, sh, at[0], at[1], at[2], at[3]));
            f32.add(product_of(GRAD_X, sh, at[0], at[1], at[2], at[3]));
        }
        return f32.preferred(sms) ? "sm100_tcgen05" : "simt_f32";
    }
    return worth_packing(g) || sm100_skinny_gemm_supported(g) || sm100_gemm_supported(g) ? "sm100_tcgen05" : "simt_f32";
}

}  // extern "C"
