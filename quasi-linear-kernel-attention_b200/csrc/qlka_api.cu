// Host side of the C ABI declared in include/qlka.h: argument checks that mirror the
// reference's TORCH_CHECKs, workspace carving, launch plans, and the kernel sequences of the
// four operators. No allocation, no synchronisation, no torch types.
#include "../../include/qlka.h"
#include "qlka_common.cuh"
#include "dense_tiles.cuh"

#include <atomic>
#include <algorithm>
#include <climits>
#include <cmath>

namespace qlka {
cudaError_t launch_sort_rank_small(const SortArgs& a, cudaStream_t stream);
cudaError_t launch_sort_rank_large(const SortArgs& a, void* scratch, cudaStream_t stream);
size_t      sort_rank_large_scratch_bytes(int nseg, int N, int M);
cudaError_t launch_laplace_walk(const WalkArgs& a, int emit, int sms, cudaStream_t stream, cudaEvent_t mid);
cudaError_t launch_prefix_walk(const WalkArgs& a, int emit, int sms, cudaStream_t stream);
int         laplace_agg_stride(int C4);
int         prefix_agg_stride_host(int C4);
cudaError_t launch_split_rows(const float* x, const float* w, const float* b, void* out, long long rows, int K, float eps, cudaStream_t st);
cudaError_t launch_split_heads(const float* o, void* out, int B, int H, int S, int D, cudaStream_t st);
cudaError_t launch_linear_qkv(const void* a3, const void* w3, const float* bias, const float* table, float* q, float* k, float* v,
                              int B, int S, int H, int K, int sms, cudaStream_t st);
cudaError_t launch_linear_gelu(const void* a3, const void* w3, const float* bias, void* out3, int M, int N, int K, int sms, cudaStream_t st);
cudaError_t launch_linear_residual(const void* a3, const void* w3, const float* bias, float* x, int M, int N, int K, int sms, cudaStream_t st);
cudaError_t linear_error_word(int** host, int** device);
cudaError_t launch_colsum_d(const float* x, float* out, int P, int D, int L, cudaStream_t st);
cudaError_t launch_rowstat(const float* w, const float* s, float* wsum, float* swsum, float* ssum, int P, int R, int C4, cudaStream_t st);
cudaError_t launch_vecsum(const float* x, float* out, int P, int L, cudaStream_t st);
cudaError_t launch_abs_init(const float* ktot, const float* vsum, const float* qsum, const float* ksr,
                            float* out, float* out_u, int P, int M, int C4, int Nk, float A, float Bq, cudaStream_t st);
cudaError_t launch_pad_rows(const float* src, float* dst, long long rows, int C, int C4, cudaStream_t st);
cudaError_t launch_unpad_rows(const float* src, float* dst, long long rows, int C, int C4, cudaStream_t st);
cudaError_t launch_transpose_scale(const float* src, float* dst, const float* keep, float scale, int P, int S, int D, int H, cudaStream_t st);
cudaError_t launch_transpose_back(const float* src, float* dst, const float* keep, float scale, const float* qt, const float* dd, const float* n_pad,
                                  int P, int S, int D, int H, cudaStream_t st);
cudaError_t launch_attention_gradient_rows(const float* g, const float* out, const float* den, float* dn, float* dd, long long rows, int C, float clamp, cudaStream_t st);
cudaError_t launch_mask_rows(const float* src, float* dst, const float* keep, int P, int S, int C, int H, cudaStream_t st);
cudaError_t launch_npad(const float* keep, float* n_pad, int B, int S, cudaStream_t st);
cudaError_t launch_normalise(float* out, const float* out_u, const float* qt, const float* n_pad,
                             int P, int M, int D, int C, int H, float clamp, bool bump, float* den_out, cudaStream_t st);
cudaError_t launch_abscolsum_d(const float* x, float* out, int P, int D, int L, cudaStream_t st);
cudaError_t launch_riesz_epilogue(float* out, const float* out_u, const float* aq, const float* vsum, const float* akv,
                                  const float* aksum, const float* n_pad, int P, int M, int C, int H,
                                  float eps, float clamp, float* den_out, cudaStream_t st);
}  // namespace qlka

using namespace qlka;

namespace {

thread_local int g_last_cuda = 0;

constexpr int SMALL_MAX = 16384;     // longest segment the shared-memory sort handles
constexpr int LENGTH_MAX = 262144;   // the reference stops at 131072 (binding.cpp:78); the value-cut sort goes on
constexpr int EMIT_ROWS = 0, EMIT_DOT = 1, EMIT_BOTH = 2;

#define CU(expr)                                                   \
    do {                                                           \
        cudaError_t e_ = (expr);                                   \
        if (e_ != cudaSuccess) { g_last_cuda = (int)e_; return QLKA_ERR_CUDA; } \
    } while (0)

int check_dims(int P, int D, int N, int M, int C) {
    if (P <= 0 || D <= 0 || N <= 0 || M <= 0) return QLKA_ERR_BAD_SHAPE;
    if (C < 1 || C > 128) return QLKA_ERR_C_RANGE;
    if (N > LENGTH_MAX || M > LENGTH_MAX) return QLKA_ERR_LENGTH;
    const long long mx = N > M ? N : M;
    if ((long long)P * D * mx > (long long)INT_MAX) return QLKA_ERR_INT32;
    return QLKA_OK;
}

// bump allocator over the workspace; with base == nullptr it only measures
struct Bump {
    char*  base;
    size_t off = 0;
    explicit Bump(void* b) : base(static_cast<char*>(b)) {}
    template <class T> T* take(size_t n) {
        off = (off + 255) & ~size_t(255);
        T* p = base ? reinterpret_cast<T*>(base + off) : nullptr;
        off += n * sizeof(T);
        return p;
    }
};

// SM count of the current device, looked up once per device (racing first calls store the same value)
int sm_count() {
    constexpr int MAX_DEV = 64;
    static std::atomic<int> cached[MAX_DEV];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEV) return 148;      // B200; keeps workspace sizes defined without a device
    int n = cached[dev].load(std::memory_order_acquire);
    if (!n) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev].store(n, std::memory_order_release);
    }
    return n;
}

// How a walk over `nseg` segments of N keys is cut into streams and work items (eight streams). Streams are independent work units (the
// passes exchange their states through memory), so a segment may be cut into any number of them, as long as a stream keeps at least
// sixteen key blocks (a stream's start costs a few) - eight while there are fewer items than CTAs fit the GPU, four while there are fewer
// than a quarter of that (attention training, one head of 376 keys x 96 features 193 -> 168 us, of 2000 x 64 281 -> 245), with dots than a half: those
// streams share a warp, so the few of a head or two leave SMs idle (Laplace gradients, heads x features x keys x channels, four instead of eight
// at a half: 4 x 16 x 3000 x 16 187 -> 161 us, 1 x 64 x 3000 x 33 215 -> 189, 2 x 64 x 1024 x 64 123 -> 107; abs 158 -> 145, 194 -> 175, 122 -> 110). The streams of a head are
// neighbours, so the more of them, the fewer heads' rows are in use at a time and the better the L2 keeps them; against that, each leaves
// aggregates to write, fold and read. Items per CTA of 256 threads, ms:        4      8      16     32
//   Laplace sum, 4 x 12 heads x 16384 keys x 64 channels                       5.23   4.88   4.83   4.89
//   abs training step, 8 x 12 x 4096 x 64                                      7.84   6.85   6.72   6.82
//   abs sum, 16 x 262144 x 64                                                  38.2   36.4   35.4   35.9
//   Laplace gradients, 48 x 4096 x 64 / 16 x 8192 x 128                        3.49   3.46   3.55   3.55 / 3.82   3.78   3.95   3.95
//   Laplace sum, 16 x 8191 keys x 1030 queries x 128                           0.93   0.93   0.97   0.97
//   abs sum / Laplace sum, 48 x 4096 x 32                                             0.95 / 1.02   0.98 / 1.04
//   abs sum / Laplace sum, 16 x 16384 x 32                                            1.32 / 1.34   1.34 / 1.40
// hence sixteen for row walks of 33 to 64 channels, else eight. The prefix walks need no first pass with one stream per segment, which
// pays as soon as whole segments alone give every CTA a few items.
struct WalkPlan { int sps, nitems; };

// lean: as few streams as serve, for scratch that the usual number of aggregates would not fit
WalkPlan plan_walk(int nseg, int N, int C4, bool laplace, bool dots, bool lean = false) {
    constexpr int streams = 8;
    // resident CTAs, about (above 64 channels two per SM; planned for four, Laplace at 16 heads x 8191 keys x 1030 queries took 1.08
    // instead of 1.03 ms, its backward at 16 x 8192 4.71 instead of 4.45 ms)
    const int cap = sm_count() * (C4 > 64 ? 2 : 4), per_cta = dots || lean || C4 <= 32 || C4 > 64 ? 8 : 16;
    const int nbk = nblocks(N);
    auto items = [&](long long sps) { return (long long)(((long long)nseg * sps + streams - 1) / streams); };
    int sps = 1;
    if (laplace || items(1) < 2LL * cap)
        while (items(sps) < (long long)per_cta * cap && nbk / (sps * 2) >= (items(sps) < cap / (dots ? 2 : 4) && !lean ? 4 : items(sps) < cap ? 8 : 16) && sps < 4096) sps *= 2;
    return {sps, (int)items(sps)};
}

// per-stream aggregate table and (Laplace) per-segment checkpoint arrays of a planned walk
size_t walk_agg_floats(const WalkPlan& w, int nseg, int C4, bool laplace) {
    return (size_t)nseg * w.sps * (laplace ? laplace_agg_stride(C4) : prefix_agg_stride_host(C4));
}

// scratch of sort/rank runs over nseg segments
struct Records {
    uint32_t* xperm; float* xval; uint4* yrec; uint32_t* mstart; float* su0; float* su1;
    uint32_t* eidx; float2* esc;      // the event list, where one is wanted
    void* large; size_t large_bytes;  // extra scratch of the value-cut sort, only when max(N, M) > SMALL_MAX
    // for the row walks: N keys, the records of M queries
    void carve(Bump& b, int nseg, int N, int M) {
        carve_large(b, nseg, N, M, false);
        carve_keys(b, nseg, N);
        yrec = b.take<uint4>((size_t)nseg * (M + 1));
        eidx = nullptr; esc = nullptr;
        carve_scans(b, nseg, N);
    }
    // for the walks with dots: the events of N keys and M queries, then of the other way round
    void carve_events(Bump& b, int nseg, int N, int M) {
        carve_large(b, nseg, N, M, true);
        carve_keys(b, nseg, std::max(N, M));
        yrec = nullptr;
        eidx = b.take<uint32_t>((size_t)nseg * estride(N, M));
        esc  = b.take<float2>((size_t)nseg * estride(N, M));
        carve_scans(b, nseg, std::max(N, M));
    }
    // (its layout is neither symmetric in N and M nor bounded by that of the longer side twice: parts are cut by queries too where there are more of them)
    void carve_large(Bump& b, int nseg, int N, int M, bool both) {
        large_bytes = N > SMALL_MAX || M > SMALL_MAX ? sort_rank_large_scratch_bytes(nseg, N, M) : 0;
        if (large_bytes && both) large_bytes = std::max(large_bytes, sort_rank_large_scratch_bytes(nseg, M, N));
        large = large_bytes ? b.take<unsigned char>(large_bytes) : nullptr;
    }
private:
    void carve_keys(Bump& b, int nseg, int N) {
        xperm = b.take<uint32_t>((size_t)nseg * npad(N));
        xval  = b.take<float>((size_t)nseg * xstride(N));
    }
    void carve_scans(Bump& b, int nseg, int N) {
        mstart = b.take<uint32_t>((size_t)nseg * mstride(N));
        su0    = b.take<float>((size_t)nseg * (N + 1));
        su1    = b.take<float>((size_t)nseg * (N + 1));
    }
};

SortArgs sort_args(const Records& r, const float* x, const float* y, int nseg, int D, int N, int M, int mode, int scal) {
    SortArgs s{};
    s.x = x; s.y = y;
    s.xperm = r.xperm; s.xval = r.xval; s.yrec = r.yrec; s.eidx = r.eidx; s.esc = r.esc; s.mstart = r.mstart; s.su0 = r.su0; s.su1 = r.su1;
    s.nseg = nseg; s.D = D; s.N = N; s.M = M; s.mode = mode; s.scal = scal;
    return s;
}

// the sort/rank stage: shared-memory kernel up to SMALL_MAX elements per segment, cut by value into its parts above
cudaError_t launch_sort_rank(const SortArgs& s, const Records& r, cudaStream_t stream) {
    if (s.N <= SMALL_MAX && s.M <= SMALL_MAX) return launch_sort_rank_small(s, stream);
    if (sort_rank_large_scratch_bytes(s.nseg, s.N, s.M) > r.large_bytes) return cudaErrorInvalidValue;
    return launch_sort_rank_large(s, r.large, stream);
}

WalkArgs walk_args(const Records& r, const float* rows, int nseg, int D, int N, int M, int C4) {
    WalkArgs a{};
    a.rows = rows; a.xperm = r.xperm; a.xval = r.xval; a.yrec = r.yrec; a.mstart = r.mstart; a.eidx = r.eidx; a.esc = r.esc;
    a.nseg = nseg; a.D = D; a.N = N; a.M = M; a.C4 = C4;
    a.sign = 1.0f;
    a.Mrows = M;
    return a;
}

// channels as the kernels see them: padded to the lane granularity of the walk
inline int round4(int C) { return (C + 3) & ~3; }

// The row matrices (v, g_w, g, out_w, grad_v, the attention output) are read and written with 16-byte copies,
// loads and vector reductions: a pointer off that boundary would fault on the device, so it is refused here.
template <class... Ptr>
bool aligned16(Ptr... p) { return ((reinterpret_cast<uintptr_t>(p) | ...) & 15) == 0; }

bool ws_ok(const void* ws, size_t have, size_t need) {
    return need == 0 || (ws != nullptr && (reinterpret_cast<uintptr_t>(ws) & 255) == 0 && have >= need);
}

// ------------------------------------------------------------------ gradients, piece by piece
// The gradients' records and checkpoints grow with the batch, to several times the inputs. So a gradient can go over its heads in pieces, and over
// the features of one head: whole while that takes no more than PIECE_BUDGET, in halves and so on where it takes more, or where
// the caller's workspace is smaller. Pieces cost launches and tails (48 heads x 4096 keys, Laplace: 1.4 GB and 3.36 ms whole, 0.7 and 3.62 in
// two; abs 2.28, 2.51), above the budget nothing (48 x 16384, Laplace: 5.4 GB and 14.5 ms whole, 2.8 and 14.4 in two).
constexpr size_t PIECE_BUDGET = size_t(4) << 30;
constexpr size_t ANY_SIZE = ~size_t(0);

struct Piece {
    int heads, features;                    // features: all of them but where heads is 1
    Piece half() const { return heads > 1 ? Piece{(heads + 1) / 2, features} : Piece{1, (features + 1) / 2}; }
    bool  least() const { return heads == 1 && features == 1; }
};

// the sizes that the pieces of P heads with D features come in
struct PieceSizes {
    Piece p[3]; int n = 0;
    PieceSizes(int P, int D, const Piece& piece) {
        for (const Piece& c : {piece, Piece{P % piece.heads, piece.features}, Piece{piece.heads, D % piece.features}})
            if (c.heads && c.features) p[n++] = c;
    }
    const Piece* begin() const { return p; }
    const Piece* end() const { return p + n; }
};

// the workspace of the largest pieces that suit the budget (whole heads) and `have` bytes, as far as there are such
template <class Ws>
Ws in_pieces(void* base, size_t have, int P, int D, int N, int M, int C) {
    Piece piece{P, D};
    while (piece.heads > 1 && Ws(nullptr, P, D, N, M, C, piece).bytes > PIECE_BUDGET) piece = piece.half();
    while (!piece.least() && Ws(nullptr, P, D, N, M, C, piece).bytes > have) piece = piece.half();
    return Ws(base, P, D, N, M, C, piece);
}

// run(p0, pc, d0, dc): features d0 .. d0 + dc - 1 of heads p0 .. p0 + pc - 1
template <class Run>
int for_pieces(int P, int D, const Piece& piece, Run run) {
    for (int p0 = 0; p0 < P; p0 += piece.heads)
        for (int d0 = 0; d0 < D; d0 += piece.features)
            if (int st = run(p0, std::min(piece.heads, P - p0), d0, std::min(piece.features, D - d0))) return st;
    return QLKA_OK;
}

// ------------------------------------------------------------------ walks, a few heads at a time
// A walk gathers the rows of a head in 64 different orders and adds into its output rows; once the heads in flight no
// longer fit the L2 (long sequences) it pays to finish a few heads before starting the next ones, so every walk runs over
// chunks of whole heads whose row matrix stays under ROWS_BUDGET (one chunk up to B=4,H=12,N=16384,C=64 and well beyond;
// 15 heads at N=65536, 3 at N=262144 with 64 channels).
constexpr size_t ROWS_BUDGET = size_t(256) << 20;

int walk_chunk_heads(int P, int N, int C4) {
    size_t h = ROWS_BUDGET / ((size_t)N * C4 * sizeof(float));
    if (h < 1) h = 1;
    return (int)(h < (size_t)P ? h : (size_t)P);
}

// aggregate table of a prefix walk over P heads in chunks (the larger of the two chunk sizes that occur)
size_t prefix_agg_floats(int P, int D, int N, int C4, bool dots, bool lean = false) {
    const int heads = walk_chunk_heads(P, N, C4);
    size_t a = 0;
    for (const int h : {heads, P % heads})
        if (h) a = std::max(a, walk_agg_floats(plan_walk(h * D, N, C4, false, dots, lean), h * D, C4, false));
    return a;
}

// `w` describes the whole problem (pointers of head 0, nseg = P * D); every chunk gets its own plan
cudaError_t prefix_walk_chunked(WalkArgs w, int emit, int P, cudaStream_t stream, bool lean = false)
{
    const int heads = walk_chunk_heads(P, w.N, w.C4);
    const WalkArgs all = w;
    for (int p0 = 0; p0 < P; p0 += heads) {
        const int       pc = heads < P - p0 ? heads : P - p0;
        const long long s0 = (long long)p0 * all.D;
        const WalkPlan  plan = plan_walk(pc * all.D, all.N, all.C4, false, emit != EMIT_ROWS, lean);
        w.rows   = all.rows + (size_t)p0 * all.N * all.C4;
        w.xperm  = all.xperm + s0 * npad(all.N);
        w.xval   = all.xval + s0 * xstride(all.N);
        w.yrec   = all.yrec ? all.yrec + s0 * (all.M + 1) : nullptr;
        w.eidx   = all.eidx ? all.eidx + s0 * estride(all.N, all.M) : nullptr;
        w.esc    = all.esc ? all.esc + s0 * estride(all.N, all.M) : nullptr;
        w.mstart = all.mstart + s0 * mstride(all.N);
        w.out    = all.out ? all.out + (size_t)p0 * all.Mrows * all.C4 : nullptr;
        w.g      = all.g ? all.g + (size_t)p0 * all.M * all.C4 : nullptr;
        w.wtotal = all.wtotal ? all.wtotal + (size_t)p0 * all.C4 : nullptr;
        w.out_s  = all.out_s ? all.out_s + s0 * all.M : nullptr;
        w.nseg = pc * all.D; w.sps = plan.sps; w.nitems = plan.nitems;
        cudaError_t e = launch_prefix_walk(w, emit, sm_count(), stream);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// The first walk pass leaves one suffix checkpoint per block and segment for the second pass: D / 8 times the size of the row matrix for
// blocks of 8 keys, about twice that for blocks of 8 events (the walks with dots). So that this scratch does not grow with the batch, a chunk's
// checkpoints also stay under CKPT_BUDGET (the same chunks as the rows rule at D = 64), twice that with dots.
constexpr size_t CKPT_BUDGET = size_t(2) << 30;

long long ckpt_blocks(int N, int M, bool dots) { return dots ? estride(N, M) / EB : nblocks(N); }

int laplace_chunk_heads(int P, int D, int N, int M, int C4, bool dots) {
    const size_t per_head = (size_t)D * ckpt_blocks(N, M, dots) * C4 * sizeof(float);
    size_t h = (dots ? 2 : 1) * CKPT_BUDGET / per_head;
    if (h < 1) h = 1;
    const int by_rows = walk_chunk_heads(P, N > M || !dots ? N : M, C4);
    return (int)(h < (size_t)by_rows ? h : (size_t)by_rows);
}

struct LapWalkScratch {
    float *ckpt, *wck, *agg; int heads; bool lean;
    // dots: for the streams of either side, N keys and M queries or the other way round. sizes: heads and features of the walks to come
    void carve(Bump& b, const PieceSizes& sizes, int N, int M, int C4, bool dots, bool lean_ = false) {
        lean  = lean_;
        heads = laplace_chunk_heads(sizes.p[0].heads, sizes.p[0].features, N, M, C4, dots);
        const int nseg_c = heads * sizes.p[0].features;
        ckpt = b.take<float>((size_t)nseg_c * ckpt_blocks(N, M, dots) * C4);
        wck  = b.take<float>((size_t)nseg_c * ckpt_blocks(N, M, dots) * (dots ? 2 : 1));
        // the aggregate table of the largest of the chunks that occur (full chunks and the remainder)
        size_t a = 0;
        for (const Piece& size : sizes)
            for (const int h : {std::min(heads, size.heads), size.heads % heads})
                for (const int keys : {N, dots ? M : N})
                    if (h) a = std::max(a, walk_agg_floats(plan_walk(h * size.features, keys, C4, true, dots, lean), h * size.features, C4, true));
        agg = b.take<float>(a);
    }
};

// rows (P, N, C4): the stream's rows; out (P, Mrows, C4) / g (P, M, C4) / out_s (P*D, M) as the emission needs them;
// mid: optional event between the passes of the first chunk (the stage timing of a single-chunk call)
cudaError_t laplace_walk_chunked(const Records& r, const LapWalkScratch& sc, const float* rows, float* out, const float* g, float* out_s,
                                 int emit, int P, int D, int N, int M, int C4, cudaStream_t stream, cudaEvent_t mid)
{
    for (int p0 = 0; p0 < P; p0 += sc.heads) {
        const int       pc = sc.heads < P - p0 ? sc.heads : P - p0, nseg = pc * D;
        const long long s0 = (long long)p0 * D;
        const WalkPlan  plan = plan_walk(nseg, N, C4, true, emit != EMIT_ROWS, sc.lean);
        WalkArgs a{};
        a.rows = rows + (size_t)p0 * N * C4;
        a.xperm = r.xperm + s0 * npad(N); a.xval = r.xval + s0 * xstride(N);
        if (emit == EMIT_ROWS) a.yrec = r.yrec + s0 * (M + 1);
        else { a.eidx = r.eidx + s0 * estride(N, M); a.esc = r.esc + s0 * estride(N, M); }
        a.mstart = r.mstart + s0 * mstride(N);
        a.ckpt = sc.ckpt; a.wck = sc.wck; a.agg = sc.agg;
        a.out   = out ? out + (size_t)p0 * M * C4 : nullptr;
        a.g     = g ? g + (size_t)p0 * M * C4 : nullptr;
        a.out_s = out_s ? out_s + s0 * M : nullptr;
        a.nseg = nseg; a.D = D; a.N = N; a.M = M; a.C4 = C4; a.sps = plan.sps; a.nitems = plan.nitems;
        a.sign = 1.0f; a.Mrows = M;
        cudaError_t e = launch_laplace_walk(a, emit, sm_count(), stream, p0 == 0 ? mid : nullptr);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// ------------------------------------------------------------------ short sequences: pair by pair
// Whether the pairwise kernels beat the sorted walk, from two cost estimates fitted to measurements on a B200 (1 to 256 heads,
// 64 to 4096 keys, 32 and 64 features, 32 to 128 channels). The pairwise one is good to a tenth. The sorted one was fitted to slower walks
// and lies 43 to 68 % above what they take now (64 features and channels, estimate / measured in us: Laplace sum of 96 heads x 256 keys 473 / 285,
// 96 x 777 918 / 576, 48 x 1024 599 / 372, 48 x 4096 1911 / 1250; riesz 327, 615, 420, 1314; bump of 48 x 1024 1505 / 897), so near the line some calls
// run pair by pair that would be up to a third faster sorted (Laplace 96 x 777 873 / 576, abs 542 / 566, riesz 546 / 615). The sorted forward sums
// round no more (2-norm against float64, sorted / pairwise, 96 x 777: Laplace 1.3e-7 / 4.9e-7, abs 1.4e-7 / 4.9e-7, riesz 5.7e-7 / 5.7e-7, bump 4.1e-7 /
// 4.9e-7): accuracy is no reason for where this line lies, as it is for the Laplace gradients below.
double dense_us(int kind, double P, int D, int N, int M, int C) {
    // picoseconds per pair and feature, and per pair and channel, with three CTAs on every SM
    const double per_d = kind == DENSE_LAPLACE ? 0.155 : kind == DENSE_BUMP ? 0.115 : 0.090, per_c = 0.027;
    const int    sms = sm_count();
    const double tile = 4096e-6 * sms * (D * per_d + (C <= 32 ? 32 : C <= 64 ? 64 : 128) * per_c);     // us of one SM per 64 x 64 pairs
    const int    nt = (N + 63) / 64;
    const long long ctas = (long long)P * ((M + 63) / 64);
    const int split = dense_split(ctas, nt, sms);
    const double per_sm = std::ceil((double)ctas * split / sms), alone = per_sm < 2 ? 2.2 : per_sm < 3 ? 1.25 : 1.0;
    const double best = per_sm * alone * ((nt + split - 1) / split + 0.5) * tile;
    return 8.0 + best;
}
double sorted_us(int kind, double P, int D, int N, int M, int C) {
    const double segs = P * D, wide = C <= 32 ? 0.6 : C <= 64 ? 1.0 : 1.4;      // the walks move rows of 32, 64 or 128 channels
    const double keys = N * (0.022 + 0.045 * wide), queries = M * (0.022 + 0.050 * wide) * (kind == DENSE_BUMP ? 5.0 : 1.0);
    return 70.0 + segs * (30.0 + keys + queries) * 1e-3;               // (launches and tails; nanoseconds per segment)
}
// What a key mask does to either path is in its values, which are on the device; the factors are for the masks met in earnest. Measured at
// 96 heads x 256 and 777 keys, 48 x 1024, 2048 and 4096 (64 features and channels) and 8 x 1500 (32), masked against unmasked:
//   pairwise, texts padded to the longest (kept lengths N / 2 to N): forward 0.62 to 0.92, gradients 0.64 to 1.00 (tiles of padding are skipped);
//     masked keys scattered, or 20 at the end: 0.91 to 1.06
//   sorted (masked keys are zeros, too many in one bucket, so their segments take the radix sort), padded or scattered: Laplace and riesz
//     forward 1.22 to 1.52, bump 1.13 to 1.50, Laplace gradients 1.14 to 1.94; 20 at the end: 1.03 to 1.13
// 0.85 and 1.25 suit padded batches. They cost a call whose batch is hardly masked: 48 heads x 1024 keys, Laplace, 20 masked keys, runs
// pair by pair in 711 us where the sorted path takes 493.
bool dense_pays(int kind, long long P, int D, int N, int M, int C, bool masked = false) {
    if (D > DENSE_MAX_D) return false;
    return dense_us(kind, (double)P, D, N, M, C) * (masked ? 0.85 : 1.0) < sorted_us(kind, (double)P, D, N, M, C) * (masked ? 1.25 : 1.0);
}

// The same for the gradients: three kernels of the same tiling against two sorts and three walks. The abs estimate is fitted to the present
// walks (within a tenth; pairwise / sorted in us: 48 heads x 300 keys 227 / 316, x 450 490 / 401, x 600 759 / 512, 8 x 800 300 / 172,
// 48 x 600 with 32 features and channels 584 / 212), which are no less accurate (2-norm against float64, grad_q and grad_v at 600 keys: 1.3e-7 and
// 2.0e-7 pairwise, 1.2e-7 and 1.3e-7 sorted). The Laplace one lies 70 % above the walks (48 x 1024 1647 / 957 us): the sorted sums
// round more (grad_q at 900 keys 5.0e-7 against 1.6e-7 pairwise), so calls stay where they were. (The bump's are three abs
// gradients put together op by op, and so is the sorted riesz.)
bool dense_gradient_pays(int kind, long long P, int D, int N, int M, int C, bool masked = false) {
    if (D > DENSE_MAX_D) return false;
    const double grad_d = kind == DENSE_LAPLACE ? 0.50 : kind == DENSE_BUMP ? 0.68 : 0.26, grad_c = 0.054;
    const int    cw = C <= 32 ? 32 : C <= 64 ? 64 : 128;
    const double tile = 4096e-6 * sm_count() * (D * grad_d + cw * grad_c);
    const double per_sm = std::ceil((double)P * ((M + N + 127) / 128) / sm_count());
    const double dense = 20.0 + std::max(per_sm, 1.0) * ((M + N + 127) / 128) * tile * (per_sm < 2 ? 0.5 : 1.0) + dense_us(kind, (double)P, D, M, N, C);
    if (kind == DENSE_ABS) return dense < 100.0 + (double)P * D * (15.0 + 0.19 * (C <= 32 ? 0.55 : C <= 64 ? 1.0 : 1.6) * 0.5 * (N + M)) * 1e-3;
    const double wide = C <= 32 ? 0.8 : C <= 64 ? 1.0 : 1.4, pair = kind == DENSE_LAPLACE ? 0.43 : kind == DENSE_BUMP ? 1.45 : 0.30;
    const double sorted = (kind == DENSE_BUMP ? 250.0 : 110.0) + (double)P * D * (60.0 + pair * wide * 0.5 * (N + M)) * 1e-3;
    return dense * (masked ? 0.85 : 1.0) < sorted * (masked ? 1.25 : 1.0);
}

// scratch of the pairwise kernels where they are the ones to run
size_t dense_bytes(int kind, int P, int D, int N, int M, int C, bool masked = false) {
    return dense_pays(kind, P, D, N, M, C, masked) ? dense_workspace_bytes(kind, P, D, N, M) : 0;
}

DenseArgs dense_args(const float* q, const float* k, const float* v, float* out, float* out_u, void* ws, int P, int D, int N, int M, int C) {
    DenseArgs a{};
    a.q = q; a.k = k; a.v = v; a.out = out; a.out_u = out_u;
    a.P = P; a.H = 1; a.D = D; a.N = N; a.M = M; a.C = C;
    a.scale = 1.0f;
    a.staged = static_cast<float*>(ws);
    return a;
}

size_t dense_gradient_bytes(int kind, int P, int D, int N, int M, int C, bool attention) {
    return dense_gradient_pays(kind, P, D, N, M, C) ? dense_gradient_workspace_bytes(kind, P, D, N, M, C, attention) : 0;
}

DenseGradArgs dense_grad_args(const float* q, const float* k, const float* v, const float* g_w, const float* g_u,
                              float* grad_q, float* grad_k, float* grad_v, void* ws, int P, int D, int N, int M, int C) {
    DenseGradArgs g{};
    g.q = q; g.k = k; g.v = v; g.a = g_w; g.s = g_u;
    g.grad_q = grad_q; g.grad_k = grad_k; g.grad_v = grad_v;
    g.staged = static_cast<float*>(ws);
    g.P = P; g.H = 1; g.D = D; g.N = N; g.M = M; g.C = C;
    g.scale = 1.0f;
    return g;
}

// the attention entry points: (B, H, S, D) rows, scaled, masked, normalised
DenseArgs dense_attention_args(const float* q, const float* k, const float* v, const float* keep, float* out, float* den, float tau, void* ws,
                               int P, int H, int S, int D, int C) {
    DenseArgs a = dense_args(q, k, v, out, den, ws, P, D, S, S, C);
    a.keep = keep; a.H = H; a.scale = 1.0f / tau; a.eps = 1e-3f; a.clamp = 1e-6f; a.rows_layout = true; a.normalise = true;
    return a;
}

// ------------------------------------------------------------------ Laplace forward
struct LaplaceWs {
    float* vpad; float* opad; Records rec; LapWalkScratch walk; size_t bytes;
    LaplaceWs(void* base, int P, int D, int N, int M, int C, bool lean = false) {
        Bump b(base);
        const int C4 = round4(C), nseg = P * D;
        vpad = C4 != C ? b.take<float>((size_t)P * N * C4) : nullptr;
        opad = C4 != C ? b.take<float>((size_t)P * M * C4) : nullptr;
        rec.carve(b, nseg, N, M);
        walk.carve(b, PieceSizes(P, D, Piece{P, D}), N, M, C4, false, lean);
        bytes = (b.off + 255) & ~size_t(255);
    }
};

// ------------------------------------------------------------------ Laplace backward
struct LaplaceBwdWs {
    float *vpad, *gpad, *gvpad; Records rec; LapWalkScratch walk; Piece piece; size_t bytes;
    LaplaceBwdWs(void* base, int P, int D, int N, int M, int C, const Piece& piece_) : piece(piece_) {
        Bump b(base);
        const int C4 = round4(C), nseg = piece.heads * piece.features;
        vpad  = C4 != C ? b.take<float>((size_t)P * N * C4) : nullptr;
        gpad  = C4 != C ? b.take<float>((size_t)P * M * C4) : nullptr;
        gvpad = C4 != C ? b.take<float>((size_t)P * N * C4) : nullptr;
        rec.carve_events(b, nseg, N, M);
        walk.carve(b, PieceSizes(P, D, piece), N, M, C4, true);     // one scratch for both walks (stream of keys k, then stream of keys q)
        bytes = (b.off + 255) & ~size_t(255);
    }
};

// ------------------------------------------------------------------ abs forward
struct AbsFwdWs {
    float* vpad; float* opad; Records rec; float *qsum, *ksumd, *vsum, *ktot, *ksr, *agg; bool lean; size_t bytes;
    AbsFwdWs(void* base, int P, int D, int N, int M, int C, bool lean_ = false) : lean(lean_) {
        Bump b(base);
        const int C4 = round4(C), nseg = P * D;
        vpad = C4 != C ? b.take<float>((size_t)P * N * C4) : nullptr;
        opad = C4 != C ? b.take<float>((size_t)P * M * C4) : nullptr;
        rec.carve(b, nseg, N, M);
        qsum  = b.take<float>((size_t)P * M);
        ksumd = b.take<float>((size_t)P * N);
        vsum  = b.take<float>((size_t)P * C4 * 2 + P);     // vsum | ktot | ksr, zeroed together
        ktot  = vsum ? vsum + (size_t)P * C4 : nullptr;
        ksr   = vsum ? ktot + (size_t)P * C4 : nullptr;
        agg   = b.take<float>(prefix_agg_floats(P, D, N, C4, false, lean));
        bytes = (b.off + 255) & ~size_t(255);
    }
};

// ------------------------------------------------------------------ abs backward / sgn
struct AbsBwdWs {
    float *vpad, *gpad, *gvpad; Records rec;
    float *qsumd, *sums /* vsum | gwsum | qtotg | gu_total */, *agg;
    Piece piece; size_t bytes;
    AbsBwdWs(void* base, int P, int D, int N, int M, int C, const Piece& piece_) : piece(piece_) {
        Bump b(base);
        const int C4 = round4(C), nseg = piece.heads * piece.features;
        vpad  = C4 != C ? b.take<float>((size_t)P * N * C4) : nullptr;
        gpad  = C4 != C ? b.take<float>((size_t)P * M * C4) : nullptr;
        gvpad = C4 != C ? b.take<float>((size_t)P * N * C4) : nullptr;
        rec.carve_events(b, nseg, N, M);
        qsumd = b.take<float>((size_t)P * M);
        sums  = b.take<float>((size_t)P * C4 * 3 + P);
        size_t a = 0;
        for (const Piece& size : PieceSizes(P, D, piece))
            for (const int keys : {N, M}) a = std::max(a, prefix_agg_floats(size.heads, size.features, keys, C4, true));
        agg   = b.take<float>(a);
        bytes = (b.off + 255) & ~size_t(255);
    }
};

}  // namespace

extern "C" {

const char* qlka_status_string(int status) {
    switch (status) {
        case QLKA_OK:                    return "ok";
        case QLKA_ERR_BAD_SHAPE:         return "N, M and D must be > 0";
        case QLKA_ERR_C_RANGE:           return "C (v.size(2)) must be in [1, 128]";
        case QLKA_ERR_LENGTH:            return "N and M must be <= 262144 (the reference: <= 131072)";
        case QLKA_ERR_INT32:             return "P*D*max(N,M) must fit int32 (cub sort offsets)";
        case QLKA_ERR_PATH:              return "path must be -1 (auto), 0 (global) or 1 (fused)";
        case QLKA_ERR_FUSED_UNAVAILABLE: return "fused path pinned but unavailable: needs max(N,M) <= 4096 and the bucket's shared memory to fit this device";
        case QLKA_ERR_NULL:              return "a required pointer is NULL";
        case QLKA_ERR_WORKSPACE:         return "workspace too small or not 256-byte aligned";
        case QLKA_ERR_CUDA:              return "a CUDA runtime call failed";
        case QLKA_ERR_UNSUPPORTED:       return "no kernel in this build for these sizes (shifted abs sum: N and n_shifts * M must be <= 16384)";
        case QLKA_ERR_NO_ALLOC_LIMIT:    return "problem needs more scratch than the fixed 32 MiB of the no-allocation entry point; use the workspace variant";
        case QLKA_ERR_ALIGNMENT:         return "v, g_w, g, out_w, grad_v and the attention output must be 16-byte aligned";
        case QLKA_ERR_GAVE_UP:           return "an earlier linear layer gave up on a barrier wait: what it wrote is NaN";
        default:                         return "unknown status";
    }
}

int qlka_last_cuda_error(void) { return g_last_cuda; }

// ---------------------------------------------------------------- Laplace
int qlka_laplace_forward_workspace_bytes(int P, int D, int N, int M, int C, size_t* bytes) {
    if (!bytes) return QLKA_ERR_NULL;
    int st = check_dims(P, D, N, M, C);
    if (st) return st;
    *bytes = std::max(LaplaceWs(nullptr, P, D, N, M, C).bytes, dense_bytes(DENSE_LAPLACE, P, D, N, M, C));
    return QLKA_OK;
}

static int laplace_forward_impl(const float* q, const float* k, const float* v,
                                float* out_w, float* out_u, void* workspace, size_t workspace_bytes,
                                int P, int D, int N, int M, int C, cudaStream_t stream, cudaEvent_t* ev)
{
    int st = check_dims(P, D, N, M, C);
    if (st) return st;
    if (!q || !k || !v || !out_w || !out_u) return QLKA_ERR_NULL;
    if (!aligned16(v, out_w)) return QLKA_ERR_ALIGNMENT;
    if (dense_pays(DENSE_LAPLACE, P, D, N, M, C) && ws_ok(workspace, workspace_bytes, dense_workspace_bytes(DENSE_LAPLACE, P, D, N, M))) {
        if (ev) for (int i = 0; i < 3; i++) CU(cudaEventRecord(ev[i], stream));
        CU(launch_dense_forward(dense_args(q, k, v, out_w, out_u, workspace, P, D, N, M, C), DENSE_LAPLACE, sm_count(), stream));
        if (ev) CU(cudaEventRecord(ev[3], stream));
        return QLKA_OK;
    }
    LaplaceWs ws(workspace, P, D, N, M, C);
    if (!ws_ok(workspace, workspace_bytes, ws.bytes)) {
        ws = LaplaceWs(workspace, P, D, N, M, C, true);
        if (!ws_ok(workspace, workspace_bytes, ws.bytes)) return QLKA_ERR_WORKSPACE;
    }
    const int C4 = round4(C), nseg = P * D;

    const float* rows = v;
    float*       out  = out_w;
    if (C4 != C) {
        CU(launch_pad_rows(v, ws.vpad, (long long)P * N, C, C4, stream));
        rows = ws.vpad; out = ws.opad;
    }
    CU(cudaMemsetAsync(out, 0, sizeof(float) * (size_t)P * M * C4, stream));
    CU(cudaMemsetAsync(out_u, 0, sizeof(float) * (size_t)P * M, stream));
    if (ev) CU(cudaEventRecord(ev[0], stream));

    SortArgs s = sort_args(ws.rec, k, q, nseg, D, N, M, MODE_LAPLACE, SCAL_UNIT);
    s.out_u = out_u;
    CU(launch_sort_rank(s, ws.rec, stream));
    if (ev) CU(cudaEventRecord(ev[1], stream));

    CU(laplace_walk_chunked(ws.rec, ws.walk, rows, out, nullptr, nullptr, EMIT_ROWS, P, D, N, M, C4, stream, ev ? ev[2] : nullptr));
    if (ev) CU(cudaEventRecord(ev[3], stream));

    if (C4 != C) CU(launch_unpad_rows(out, out_w, (long long)P * M, C, C4, stream));
    return QLKA_OK;
}

int qlka_weighted_laplace_sum_forward(const float* q, const float* k, const float* v,
                                      float* out_w, float* out_u, void* workspace, size_t workspace_bytes,
                                      int P, int D, int N, int M, int C, qlka_stream_t stream_)
{
    return laplace_forward_impl(q, k, v, out_w, out_u, workspace, workspace_bytes, P, D, N, M, C,
                                reinterpret_cast<cudaStream_t>(stream_), nullptr);
}

int qlka_laplace_forward_stage_ms(const float* q, const float* k, const float* v,
                                  float* out_w, float* out_u, void* workspace, size_t workspace_bytes,
                                  int P, int D, int N, int M, int C, qlka_stream_t stream_,
                                  float* sort_ms, float* pass1_ms, float* pass2_ms)
{
    if (!sort_ms || !pass1_ms || !pass2_ms) return QLKA_ERR_NULL;
    cudaEvent_t ev[4];
    for (int i = 0; i < 4; i++) CU(cudaEventCreate(&ev[i]));
    int st = laplace_forward_impl(q, k, v, out_w, out_u, workspace, workspace_bytes, P, D, N, M, C,
                                  reinterpret_cast<cudaStream_t>(stream_), ev);
    if (st == QLKA_OK) {
        cudaError_t e = cudaEventSynchronize(ev[3]);
        if (e == cudaSuccess) e = cudaEventElapsedTime(sort_ms, ev[0], ev[1]);
        if (e == cudaSuccess) e = cudaEventElapsedTime(pass1_ms, ev[1], ev[2]);
        if (e == cudaSuccess) e = cudaEventElapsedTime(pass2_ms, ev[2], ev[3]);
        if (e != cudaSuccess) { g_last_cuda = (int)e; st = QLKA_ERR_CUDA; }
    }
    for (int i = 0; i < 4; i++) cudaEventDestroy(ev[i]);
    return st;
}

// ---------------------------------------------------------------- Laplace backward
int qlka_laplace_backward_workspace_bytes(int P, int D, int N, int M, int C, size_t* bytes) {
    if (!bytes) return QLKA_ERR_NULL;
    int st = check_dims(P, D, N, M, C);
    if (st) return st;
    *bytes = std::max(in_pieces<LaplaceBwdWs>(nullptr, ANY_SIZE, P, D, N, M, C).bytes, dense_gradient_bytes(DENSE_LAPLACE, P, D, N, M, C, false));
    return QLKA_OK;
}

int qlka_weighted_laplace_sum_backward(const float* q, const float* k, const float* v,
                                       const float* g_w, const float* g_u,
                                       float* grad_q, float* grad_k, float* grad_v,
                                       void* workspace, size_t workspace_bytes,
                                       int P, int D, int N, int M, int C, qlka_stream_t stream_)
{
    int st = check_dims(P, D, N, M, C);
    if (st) return st;
    if (!q || !k || !v || !g_w || !grad_q || !grad_k || !grad_v) return QLKA_ERR_NULL;
    if (!aligned16(v, g_w, grad_v)) return QLKA_ERR_ALIGNMENT;
    if (dense_gradient_pays(DENSE_LAPLACE, P, D, N, M, C)) {
        if (!ws_ok(workspace, workspace_bytes, dense_gradient_workspace_bytes(DENSE_LAPLACE, P, D, N, M, C, false))) return QLKA_ERR_WORKSPACE;
        CU(launch_dense_gradient(dense_grad_args(q, k, v, g_w, g_u, grad_q, grad_k, grad_v, workspace, P, D, N, M, C), DENSE_LAPLACE, sm_count(),
                                 reinterpret_cast<cudaStream_t>(stream_)));
        return QLKA_OK;
    }
    const LaplaceBwdWs ws = in_pieces<LaplaceBwdWs>(workspace, workspace_bytes, P, D, N, M, C);
    if (!ws_ok(workspace, workspace_bytes, ws.bytes)) return QLKA_ERR_WORKSPACE;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    const int C4 = round4(C), nseg = P * D;
    const bool full = g_u != nullptr;

    const float* vrows = v;
    const float* grows = g_w;
    float*       gv    = grad_v;
    if (C4 != C) {
        CU(launch_pad_rows(v, ws.vpad, (long long)P * N, C, C4, stream));
        CU(launch_pad_rows(g_w, ws.gpad, (long long)P * M, C, C4, stream));
        vrows = ws.vpad; grows = ws.gpad; gv = ws.gvpad;
    }
    CU(cudaMemsetAsync(gv, 0, sizeof(float) * (size_t)P * N * C4, stream));
    if (!full) {    // the walks add to grad_q and grad_k; with g_u the sort/rank kernel stores its term there first
        CU(cudaMemsetAsync(grad_q, 0, sizeof(float) * (size_t)nseg * M, stream));
        CU(cudaMemsetAsync(grad_k, 0, sizeof(float) * (size_t)nseg * N, stream));
    }
    st = for_pieces(P, D, ws.piece, [&](const int p0, const int pc, const int d0, const int dc) -> int {
        const size_t s0 = (size_t)p0 * D + d0;
        const float *qp = q + s0 * M, *kp = k + s0 * N, *vp = vrows + (size_t)p0 * N * C4, *gp = grows + (size_t)p0 * M * C4, *up = full ? g_u + (size_t)p0 * M : nullptr;
        {   // grad_q[d, m] = <g_w[m], e1 R_r - e0 L_{r-1}> + g_u[m] (e1 Ru_r - e0 Lu_{r-1}): queries q walk the key stream k
            SortArgs s = sort_args(ws.rec, kp, qp, pc * dc, dc, N, M, MODE_LAPLACE, full ? SCAL_SIGNED : SCAL_NONE);
            s.uq = up; s.out_s = grad_q + s0 * M;
            CU(launch_sort_rank(s, ws.rec, stream));
            CU(laplace_walk_chunked(ws.rec, ws.walk, vp, nullptr, gp, grad_q + s0 * M, EMIT_DOT, pc, dc, N, M, C4, stream, nullptr));
        }
        {   // roles swapped: queries k walk the stream q whose rows are g_w (and whose per-key scalar is g_u);
            // the row emission is grad_v, the dot with the v rows is grad_k
            SortArgs s = sort_args(ws.rec, qp, kp, pc * dc, dc, M, N, MODE_LAPLACE, full ? SCAL_SIGNED : SCAL_NONE);
            s.us = up; s.out_s = grad_k + s0 * N;
            CU(launch_sort_rank(s, ws.rec, stream));
            CU(laplace_walk_chunked(ws.rec, ws.walk, gp, gv + (size_t)p0 * N * C4, vp, grad_k + s0 * N, EMIT_BOTH, pc, dc, M, N, C4, stream, nullptr));
        }
        return QLKA_OK;
    });
    if (st) return st;
    if (C4 != C) CU(launch_unpad_rows(gv, grad_v, (long long)P * N, C, C4, stream));
    return QLKA_OK;
}

// ---------------------------------------------------------------- add_laplace attention on (B, H, S, D)
namespace {
struct LaplaceAttnWs {
    float *qt, *kt, *vm, *out_u, *n_pad; void* inner; size_t fixed, bytes, least;      // inner: what lies beyond `fixed`
    LaplaceAttnWs(void* base, int B, int H, int S, int D, int C, bool masked) {
        Bump b(base);
        const size_t P = (size_t)B * H;
        qt    = b.take<float>(P * D * S);
        kt    = b.take<float>(P * D * S);
        vm    = masked ? b.take<float>(P * S * C) : nullptr;
        out_u = b.take<float>(P * S);
        n_pad = masked ? b.take<float>((size_t)B) : nullptr;
        inner = b.take<unsigned char>(0);
        fixed = b.off;
        bytes = fixed + LaplaceWs(nullptr, (int)P, D, S, S, C).bytes;
        least = fixed + LaplaceWs(nullptr, (int)P, D, S, S, C, true).bytes;
    }
};
}  // namespace

static int attn_check(int B, int H, int S, int D, int C) {
    if (B <= 0 || H <= 0) return QLKA_ERR_BAD_SHAPE;
    if ((long long)B * H > INT_MAX || D > 32 * 65535) return QLKA_ERR_INT32;
    return check_dims(B * H, D, S, S, C);
}

int qlka_laplace_attention_workspace_bytes(int B, int H, int S, int D, int Dv, int masked, size_t* bytes) {
    if (!bytes) return QLKA_ERR_NULL;
    int st = attn_check(B, H, S, D, Dv);
    if (st) return st;
    *bytes = std::max(LaplaceAttnWs(nullptr, B, H, S, D, Dv, masked != 0).bytes, dense_bytes(DENSE_LAPLACE, B * H, D, S, S, Dv, masked != 0));
    return QLKA_OK;
}

// den: row sums (before the floor) for the backward pass, or null
static int laplace_attention_impl(const float* q, const float* k, const float* v, const float* keep, float tau,
                                  float* out, float* den, void* workspace, size_t workspace_bytes,
                                  int B, int H, int S, int D, int Dv, cudaStream_t stream)
{
    int st = attn_check(B, H, S, D, Dv);
    if (st) return st;
    if (!q || !k || !v || !out) return QLKA_ERR_NULL;
    if (!aligned16(v, out)) return QLKA_ERR_ALIGNMENT;
    if (!(tau > 0.0f)) return QLKA_ERR_BAD_SHAPE;
    if (dense_pays(DENSE_LAPLACE, (long long)B * H, D, S, S, Dv, keep != nullptr)) {
        if (!ws_ok(workspace, workspace_bytes, dense_workspace_bytes(DENSE_LAPLACE, B * H, D, S, S))) return QLKA_ERR_WORKSPACE;
        CU(launch_dense_forward(dense_attention_args(q, k, v, keep, out, den, tau, workspace, B * H, H, S, D, Dv), DENSE_LAPLACE, sm_count(), stream));
        return QLKA_OK;
    }
    const bool masked = keep != nullptr;
    LaplaceAttnWs ws(workspace, B, H, S, D, Dv, masked);
    if (!ws_ok(workspace, workspace_bytes, ws.least)) return QLKA_ERR_WORKSPACE;
    const int P = B * H;

    CU(launch_transpose_scale(q, ws.qt, nullptr, 1.0f / tau, P, S, D, H, stream));
    CU(launch_transpose_scale(k, ws.kt, keep, 1.0f / tau, P, S, D, H, stream));
    const float* rows = v;
    if (masked) {
        CU(launch_mask_rows(v, ws.vm, keep, P, S, Dv, H, stream));
        CU(launch_npad(keep, ws.n_pad, B, S, stream));
        rows = ws.vm;
    }
    st = laplace_forward_impl(ws.qt, ws.kt, rows, out, ws.out_u, ws.inner, workspace_bytes - ws.fixed, P, D, S, S, Dv, stream, nullptr);
    if (st) return st;
    CU(launch_normalise(out, ws.out_u, ws.qt, ws.n_pad, P, S, D, Dv, H, 1e-6f, false, den, stream));
    return QLKA_OK;
}

int qlka_laplace_attention_forward(const float* q, const float* k, const float* v, const float* keep, float tau,
                                   float* out, void* workspace, size_t workspace_bytes,
                                   int B, int H, int S, int D, int Dv, qlka_stream_t stream_)
{
    return laplace_attention_impl(q, k, v, keep, tau, out, nullptr, workspace, workspace_bytes, B, H, S, D, Dv, reinterpret_cast<cudaStream_t>(stream_));
}

// ---------------------------------------------------------------- add_riesz / add_bump attention on (B, H, S, D)
static int abs_forward_impl(const float* q, const float* k, const float* v, float* out_w, float* out_u,
                            void* workspace, size_t workspace_bytes, int P, int D, int N, int M, int C,
                            int ns, const float* shifts, const float* weights, cudaStream_t stream, bool walk = false);
namespace {
constexpr float BUMP_SHIFTS[3]  = {0.0f, 1.0f, -1.0f};     // max(0, 1 - |x|) = |x + 1| / 2 + |x - 1| / 2 - |x|
constexpr float BUMP_WEIGHTS[3] = {-1.0f, 0.5f, 0.5f};
struct AbsAttnWs {
    float *qt, *kt, *vm, *out_u, *n_pad, *aq, *ak, *sums /* vsum | akv | aksum */; void* inner; size_t fixed, bytes, least;
    AbsAttnWs(void* base, int B, int H, int S, int D, int C, bool masked, bool bump) {
        Bump b(base);
        const size_t P = (size_t)B * H;
        qt    = b.take<float>(P * D * S);
        kt    = b.take<float>(P * D * S);
        vm    = masked ? b.take<float>(P * S * C) : nullptr;
        out_u = b.take<float>(P * S);
        n_pad = masked ? b.take<float>((size_t)B) : nullptr;
        aq    = bump ? nullptr : b.take<float>(P * S);
        ak    = bump ? nullptr : b.take<float>(P * S);
        sums  = bump ? nullptr : b.take<float>(P * C * 2 + P);
        inner = b.take<unsigned char>(0);
        fixed = b.off;
        bytes = fixed + AbsFwdWs(nullptr, (int)P, D, S, bump ? 3 * S : S, C).bytes;
        least = fixed + AbsFwdWs(nullptr, (int)P, D, S, bump ? 3 * S : S, C, true).bytes;
    }
};
}  // namespace

static int abs_attn_check(int kind, int B, int H, int S, int D, int C) {
    if (kind != 0 && kind != 1) return QLKA_ERR_PATH;
    int st = attn_check(B, H, S, D, C);
    if (st) return st;
    if (kind == 1 && 3LL * S > SMALL_MAX) return QLKA_ERR_UNSUPPORTED;     // the three shifted query copies share one shared-memory sort
    return QLKA_OK;
}

int qlka_abs_attention_workspace_bytes(int kind, int B, int H, int S, int D, int Dv, int masked, size_t* bytes) {
    if (!bytes) return QLKA_ERR_NULL;
    int st = abs_attn_check(kind, B, H, S, D, Dv);
    if (st) return st;
    *bytes = std::max(AbsAttnWs(nullptr, B, H, S, D, Dv, masked != 0, kind == 1).bytes, dense_bytes(kind == 1 ? DENSE_BUMP : DENSE_RIESZ, B * H, D, S, S, Dv, masked != 0));
    return QLKA_OK;
}

static int abs_attention_impl(int kind, const float* q, const float* k, const float* v, const float* keep, float tau,
                              float* out, float* den, void* workspace, size_t workspace_bytes,
                              int B, int H, int S, int D, int Dv, cudaStream_t stream)
{
    int st = abs_attn_check(kind, B, H, S, D, Dv);
    if (st) return st;
    if (!q || !k || !v || !out) return QLKA_ERR_NULL;
    if (!aligned16(v, out)) return QLKA_ERR_ALIGNMENT;
    if (!(tau > 0.0f)) return QLKA_ERR_BAD_SHAPE;
    const bool masked = keep != nullptr, bump = kind == 1;
    if (const int dk = bump ? DENSE_BUMP : DENSE_RIESZ; dense_pays(dk, (long long)B * H, D, S, S, Dv, masked)) {
        if (!ws_ok(workspace, workspace_bytes, dense_workspace_bytes(dk, B * H, D, S, S))) return QLKA_ERR_WORKSPACE;
        CU(launch_dense_forward(dense_attention_args(q, k, v, keep, out, den, tau, workspace, B * H, H, S, D, Dv), dk, sm_count(), stream));
        return QLKA_OK;
    }
    AbsAttnWs ws(workspace, B, H, S, D, Dv, masked, bump);
    if (!ws_ok(workspace, workspace_bytes, ws.least)) return QLKA_ERR_WORKSPACE;
    const int P = B * H;

    CU(launch_transpose_scale(q, ws.qt, nullptr, 1.0f / tau, P, S, D, H, stream));
    CU(launch_transpose_scale(k, ws.kt, keep, 1.0f / tau, P, S, D, H, stream));
    const float* rows = v;
    if (masked) {
        CU(launch_mask_rows(v, ws.vm, keep, P, S, Dv, H, stream));
        CU(launch_npad(keep, ws.n_pad, B, S, stream));
        rows = ws.vm;
    }
    if (bump) {
        // numerator and row sum of the three shifted abs sums from one sort, then the row normalisation
        st = abs_forward_impl(ws.qt, ws.kt, rows, out, ws.out_u, ws.inner, workspace_bytes - ws.fixed, P, D, S, S, Dv, 3, BUMP_SHIFTS, BUMP_WEIGHTS, stream);
        if (st) return st;
        CU(launch_normalise(out, ws.out_u, ws.qt, ws.n_pad, P, S, D, Dv, H, 1e-6f, true, den, stream));
    } else {
        // A_ij = |q_i|_1 + |k_j|_1 - |q_i - k_j|_1 + eps: rank-1 terms from column and row statistics, the abs sum from the walk
        float* vsum  = ws.sums;
        float* akv   = vsum + (size_t)P * Dv;
        float* aksum = akv + (size_t)P * Dv;
        CU(launch_abscolsum_d(ws.qt, ws.aq, P, D, S, stream));
        CU(launch_abscolsum_d(ws.kt, ws.ak, P, D, S, stream));
        CU(cudaMemsetAsync(ws.sums, 0, sizeof(float) * ((size_t)P * Dv * 2 + P), stream));
        CU(launch_rowstat(rows, ws.ak, vsum, akv, aksum, P, S, Dv, stream));
        st = abs_forward_impl(ws.qt, ws.kt, rows, out, ws.out_u, ws.inner, workspace_bytes - ws.fixed, P, D, S, S, Dv, 0, nullptr, nullptr, stream, true);
        if (st) return st;
        CU(launch_riesz_epilogue(out, ws.out_u, ws.aq, vsum, akv, aksum, ws.n_pad, P, S, Dv, H, 1e-3f, 1e-6f, den, stream));
    }
    return QLKA_OK;
}

int qlka_abs_attention_forward(int kind, const float* q, const float* k, const float* v, const float* keep, float tau,
                               float* out, void* workspace, size_t workspace_bytes,
                               int B, int H, int S, int D, int Dv, qlka_stream_t stream_)
{
    return abs_attention_impl(kind, q, k, v, keep, tau, out, nullptr, workspace, workspace_bytes, B, H, S, D, Dv, reinterpret_cast<cudaStream_t>(stream_));
}

// ---------------------------------------------------------------- attention, training: row sums kept, backward
namespace {
constexpr int ATTN_LAPLACE = 2;
int dense_kind_of(int kind) { return kind == ATTN_LAPLACE ? DENSE_LAPLACE : kind == 1 ? DENSE_BUMP : DENSE_RIESZ; }

struct LaplaceAttnBwdWs {
    float *qt, *kt, *vm, *dn, *dd, *gqt, *gkt, *n_pad; void* inner; size_t fixed, bytes, least;
    LaplaceAttnBwdWs(void* base, int B, int H, int S, int D, int C, bool masked) {
        Bump b(base);
        const size_t P = (size_t)B * H;
        qt    = b.take<float>(P * D * S);
        kt    = b.take<float>(P * D * S);
        gqt   = b.take<float>(P * D * S);
        gkt   = b.take<float>(P * D * S);
        vm    = masked ? b.take<float>(P * S * C) : nullptr;
        dn    = b.take<float>(P * S * C);
        dd    = b.take<float>(P * S);
        n_pad = masked ? b.take<float>((size_t)B) : nullptr;
        inner = b.take<unsigned char>(0);
        fixed = b.off;
        bytes = fixed + in_pieces<LaplaceBwdWs>(nullptr, ANY_SIZE, (int)P, D, S, S, C).bytes;
        least = fixed + in_pieces<LaplaceBwdWs>(nullptr, 0, (int)P, D, S, S, C).bytes;
    }
};
}  // namespace

int qlka_attention_forward(int kind, const float* q, const float* k, const float* v, const float* keep, float tau,
                           float* out, float* den, void* workspace, size_t workspace_bytes,
                           int B, int H, int S, int D, int Dv, qlka_stream_t stream_)
{
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (kind == ATTN_LAPLACE) return laplace_attention_impl(q, k, v, keep, tau, out, den, workspace, workspace_bytes, B, H, S, D, Dv, stream);
    return abs_attention_impl(kind, q, k, v, keep, tau, out, den, workspace, workspace_bytes, B, H, S, D, Dv, stream);
}

int qlka_attention_workspace_bytes(int kind, int B, int H, int S, int D, int Dv, int masked, size_t* bytes) {
    if (kind == ATTN_LAPLACE) return qlka_laplace_attention_workspace_bytes(B, H, S, D, Dv, masked, bytes);
    return qlka_abs_attention_workspace_bytes(kind, B, H, S, D, Dv, masked, bytes);
}

int qlka_attention_backward_workspace_bytes(int kind, int B, int H, int S, int D, int Dv, int masked, size_t* bytes) {
    if (!bytes) return QLKA_ERR_NULL;
    int st = kind == ATTN_LAPLACE ? attn_check(B, H, S, D, Dv) : abs_attn_check(kind, B, H, S, D, Dv);
    if (st) return st;
    const int dk = dense_kind_of(kind);
    if (dense_gradient_pays(dk, (long long)B * H, D, S, S, Dv, masked != 0)) *bytes = dense_gradient_workspace_bytes(dk, B * H, D, S, S, Dv, true);
    else if (kind == ATTN_LAPLACE)                              *bytes = LaplaceAttnBwdWs(nullptr, B, H, S, D, Dv, masked != 0).bytes;
    else                                                        return QLKA_ERR_UNSUPPORTED;
    return QLKA_OK;
}

int qlka_attention_backward(int kind, const float* q, const float* k, const float* v, const float* keep, float tau,
                            const float* out, const float* den, const float* grad_out,
                            float* grad_q, float* grad_k, float* grad_v, void* workspace, size_t workspace_bytes,
                            int B, int H, int S, int D, int Dv, qlka_stream_t stream_)
{
    const bool masked = keep != nullptr;
    size_t need = 0;
    int st = qlka_attention_backward_workspace_bytes(kind, B, H, S, D, Dv, masked, &need);
    if (st) return st;
    if (!q || !k || !v || !out || !den || !grad_out || !grad_q || !grad_k || !grad_v) return QLKA_ERR_NULL;
    if (!aligned16(v, out, grad_out, grad_v)) return QLKA_ERR_ALIGNMENT;
    if (!(tau > 0.0f)) return QLKA_ERR_BAD_SHAPE;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    const int P = B * H, dk = dense_kind_of(kind);
    if (dense_gradient_pays(dk, P, D, S, S, Dv, masked)) {
        if (!ws_ok(workspace, workspace_bytes, need)) return QLKA_ERR_WORKSPACE;
        DenseGradArgs g = dense_grad_args(q, k, v, grad_out, nullptr, grad_q, grad_k, grad_v, workspace, P, D, S, S, Dv);
        g.attention = true; g.H = H; g.scale = 1.0f / tau; g.eps = 1e-3f; g.clamp = 1e-6f; g.keep = keep; g.out = out; g.den = den;
        CU(launch_dense_gradient(g, dk, sm_count(), stream));
        return QLKA_OK;
    }
    LaplaceAttnBwdWs ws(workspace, B, H, S, D, Dv, masked);
    if (!ws_ok(workspace, workspace_bytes, ws.least)) return QLKA_ERR_WORKSPACE;
    CU(launch_transpose_scale(q, ws.qt, nullptr, 1.0f / tau, P, S, D, H, stream));
    CU(launch_transpose_scale(k, ws.kt, keep, 1.0f / tau, P, S, D, H, stream));
    const float* rows = v;
    if (masked) {
        CU(launch_mask_rows(v, ws.vm, keep, P, S, Dv, H, stream));
        CU(launch_npad(keep, ws.n_pad, B, S, stream));
        rows = ws.vm;
    }
    CU(launch_attention_gradient_rows(grad_out, out, den, ws.dn, ws.dd, (long long)P * S, Dv, 1e-6f, stream));
    st = qlka_weighted_laplace_sum_backward(ws.qt, ws.kt, rows, ws.dn, ws.dd, ws.gqt, ws.gkt, grad_v, ws.inner, workspace_bytes - ws.fixed, P, D, S, S, Dv, stream_);
    if (st) return st;
    CU(launch_transpose_back(ws.gqt, grad_q, nullptr, 1.0f / tau, masked ? ws.qt : nullptr, ws.dd, ws.n_pad, P, S, D, H, stream));
    CU(launch_transpose_back(ws.gkt, grad_k, keep, 1.0f / tau, nullptr, nullptr, nullptr, P, S, D, H, stream));
    if (masked) CU(launch_mask_rows(grad_v, grad_v, keep, P, S, Dv, H, stream));
    return QLKA_OK;
}

// ---------------------------------------------------------------- Laplace, fixed scratch
// Scratch for qlka_weighted_laplace_sum_forward_noalloc: lives in the library image, so every
// device that loads the library reserves QLKA_NOALLOC_SCRATCH_BYTES for as long as the process runs.
constexpr size_t QLKA_NOALLOC_SCRATCH_BYTES = size_t(32) << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[QLKA_NOALLOC_SCRATCH_BYTES];

// In host code `g_noalloc_scratch` is only a handle for the runtime, not an address a kernel could
// use: the device address is looked up once per device (with that device current) and cached.
static int noalloc_scratch(void** out) {
    constexpr int MAX_DEV = 64;
    static std::atomic<void*> cached[MAX_DEV];
    int dev = 0;
    CU(cudaGetDevice(&dev));
    if (dev < 0 || dev >= MAX_DEV) return QLKA_ERR_UNSUPPORTED;
    void* ptr = cached[dev].load(std::memory_order_acquire);
    if (!ptr) {
        CU(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
        cached[dev].store(ptr, std::memory_order_release);      // racing first calls store the same value
    }
    *out = ptr;
    return QLKA_OK;
}

size_t qlka_noalloc_scratch_bytes(void) { return QLKA_NOALLOC_SCRATCH_BYTES; }

int qlka_weighted_laplace_sum_forward_noalloc(const float* q, const float* k, const float* v,
                                              float* out_w, float* out_u,
                                              int P, int D, int N, int M, int C, qlka_stream_t stream_)
{
    int st = check_dims(P, D, N, M, C);
    if (st) return st;
    if (!q || !k || !v || !out_w || !out_u) return QLKA_ERR_NULL;
    if (!aligned16(v, out_w)) return QLKA_ERR_ALIGNMENT;
    if (LaplaceWs(nullptr, P, D, N, M, C, true).bytes > QLKA_NOALLOC_SCRATCH_BYTES) return QLKA_ERR_NO_ALLOC_LIMIT;
    void* scratch = nullptr;
    st = noalloc_scratch(&scratch);
    if (st) return st;
    // every byte of scratch that the kernels read is written earlier in the same call, and the
    // outputs are zeroed by the call itself, so what a previous call left behind is never seen
    return laplace_forward_impl(q, k, v, out_w, out_u, scratch, QLKA_NOALLOC_SCRATCH_BYTES, P, D, N, M, C,
                                reinterpret_cast<cudaStream_t>(stream_), nullptr);
}

// ---------------------------------------------------------------- abs forward
int qlka_abs_forward_workspace_bytes(int P, int D, int N, int M, int C, size_t* bytes) {
    if (!bytes) return QLKA_ERR_NULL;
    int st = check_dims(P, D, N, M, C);
    if (st) return st;
    *bytes = std::max(AbsFwdWs(nullptr, P, D, N, M, C).bytes, dense_bytes(DENSE_ABS, P, D, N, M, C));
    return QLKA_OK;
}

// ns == 0: the plain abs sum. ns >= 1: sum_s weights[s] * abs_sum(q + shifts[s]) from one sort of the keys. walk: by the sorted walk
// whatever the size.
static int abs_forward_impl(const float* q, const float* k, const float* v, float* out_w, float* out_u,
                            void* workspace, size_t workspace_bytes, int P, int D, int N, int M, int C,
                            int ns, const float* shifts, const float* weights, cudaStream_t stream, bool walk)
{
    if (!ns && !walk && dense_pays(DENSE_ABS, P, D, N, M, C)) {
        if (!ws_ok(workspace, workspace_bytes, dense_workspace_bytes(DENSE_ABS, P, D, N, M))) return QLKA_ERR_WORKSPACE;
        CU(launch_dense_forward(dense_args(q, k, v, out_w, out_u, workspace, P, D, N, M, C), DENSE_ABS, sm_count(), stream));
        return QLKA_OK;
    }
    const int MQ = ns ? ns * M : M;                 // queries per segment
    AbsFwdWs ws(workspace, P, D, N, MQ, C);
    if (!ws_ok(workspace, workspace_bytes, ws.bytes)) {
        ws = AbsFwdWs(workspace, P, D, N, MQ, C, true);
        if (!ws_ok(workspace, workspace_bytes, ws.bytes)) return QLKA_ERR_WORKSPACE;
    }
    const int C4 = round4(C), nseg = P * D;
    const bool full = out_u != nullptr;
    float A = 1.0f, Bq = 0.0f;
    if (ns) { A = 0.0f; for (int s = 0; s < ns; s++) { A += weights[s]; Bq += weights[s] * shifts[s] * (float)D; } }

    const float* rows = v;
    float*       out  = out_w;
    if (C4 != C) {
        CU(launch_pad_rows(v, ws.vpad, (long long)P * N, C, C4, stream));
        rows = ws.vpad; out = ws.opad;
    }
    // rank-1 part: out = k_total - qsum * vsum, out_u = ksum_raw - N * qsum (weighted over the shifts when folded)
    CU(launch_colsum_d(q, ws.qsum, P, D, M, stream));
    CU(launch_colsum_d(k, ws.ksumd, P, D, N, stream));
    CU(cudaMemsetAsync(ws.vsum, 0, sizeof(float) * ((size_t)P * C4 * 2 + P), stream));
    CU(launch_rowstat(rows, ws.ksumd, ws.vsum, ws.ktot, ws.ksr, P, N, C4, stream));
    CU(launch_abs_init(ws.ktot, ws.vsum, ws.qsum, ws.ksr, out, out_u, P, M, C4, N, A, Bq, stream));

    SortArgs s = sort_args(ws.rec, k, q, nseg, D, N, MQ, MODE_ABS, full ? SCAL_UNIT : SCAL_NONE);
    s.out_u = out_u; s.rows_coef = 1;
    if (ns) { s.fold = M; for (int i = 0; i < ns; i++) { s.shift[i] = shifts[i]; s.wgt[i] = weights[i]; } }
    CU(launch_sort_rank(s, ws.rec, stream));

    WalkArgs w = walk_args(ws.rec, rows, nseg, D, N, MQ, C4);
    w.out = out; w.Mrows = M; w.agg = ws.agg;
    CU(prefix_walk_chunked(w, EMIT_ROWS, P, stream, ws.lean));

    if (C4 != C) CU(launch_unpad_rows(out, out_w, (long long)P * M, C, C4, stream));
    return QLKA_OK;
}

int qlka_weighted_abs_sum_forward(const float* q, const float* k, const float* v,
                                  float* out_w, float* out_u, void* workspace, size_t workspace_bytes,
                                  int P, int D, int N, int M, int C, int path, qlka_stream_t stream_)
{
    int st = check_dims(P, D, N, M, C);
    if (st) return st;
    if (path < -1 || path > 1) return QLKA_ERR_PATH;
    if (path == 1 && (N > 4096 || M > 4096)) return QLKA_ERR_FUSED_UNAVAILABLE;
    if (!q || !k || !v || !out_w) return QLKA_ERR_NULL;
    if (!aligned16(v, out_w)) return QLKA_ERR_ALIGNMENT;
    return abs_forward_impl(q, k, v, out_w, out_u, workspace, workspace_bytes, P, D, N, M, C, 0, nullptr, nullptr,
                            reinterpret_cast<cudaStream_t>(stream_), path == 0);
}

int qlka_abs_shifted_forward_workspace_bytes(int P, int D, int N, int M, int C, int n_shifts, size_t* bytes) {
    if (!bytes) return QLKA_ERR_NULL;
    if (n_shifts < 1 || n_shifts > 4) return QLKA_ERR_BAD_SHAPE;
    int st = check_dims(P, D, N, M, C);
    if (st) return st;
    if ((long long)n_shifts * M > SMALL_MAX || N > SMALL_MAX) return QLKA_ERR_UNSUPPORTED;
    *bytes = AbsFwdWs(nullptr, P, D, N, n_shifts * M, C).bytes;
    return QLKA_OK;
}

int qlka_weighted_abs_sum_shifted_forward(const float* q, const float* k, const float* v,
                                          float* out_w, float* out_u, const float* shifts, const float* weights, int n_shifts,
                                          void* workspace, size_t workspace_bytes,
                                          int P, int D, int N, int M, int C, qlka_stream_t stream_)
{
    if (n_shifts < 1 || n_shifts > 4) return QLKA_ERR_BAD_SHAPE;
    int st = check_dims(P, D, N, M, C);
    if (st) return st;
    if ((long long)n_shifts * M > SMALL_MAX || N > SMALL_MAX) return QLKA_ERR_UNSUPPORTED;
    if (!q || !k || !v || !out_w || !shifts || !weights) return QLKA_ERR_NULL;
    if (!aligned16(v, out_w)) return QLKA_ERR_ALIGNMENT;
    return abs_forward_impl(q, k, v, out_w, out_u, workspace, workspace_bytes, P, D, N, M, C, n_shifts, shifts, weights,
                            reinterpret_cast<cudaStream_t>(stream_));
}

// ---------------------------------------------------------------- abs backward
int qlka_abs_backward_workspace_bytes(int P, int D, int N, int M, int C, size_t* bytes) {
    if (!bytes) return QLKA_ERR_NULL;
    int st = check_dims(P, D, N, M, C);
    if (st) return st;
    *bytes = std::max(in_pieces<AbsBwdWs>(nullptr, ANY_SIZE, P, D, N, M, C).bytes, dense_gradient_bytes(DENSE_ABS, P, D, N, M, C, false));
    return QLKA_OK;
}

int qlka_weighted_abs_sum_backward(const float* q, const float* k, const float* v,
                                   const float* g_w, const float* g_u,
                                   float* grad_q, float* grad_k, float* grad_v,
                                   void* workspace, size_t workspace_bytes,
                                   int P, int D, int N, int M, int C, qlka_stream_t stream_)
{
    int st = check_dims(P, D, N, M, C);
    if (st) return st;
    if (!q || !k || !v || !g_w || !grad_q || !grad_k || !grad_v) return QLKA_ERR_NULL;
    if (!aligned16(v, g_w, grad_v)) return QLKA_ERR_ALIGNMENT;
    if (dense_gradient_pays(DENSE_ABS, P, D, N, M, C)) {
        if (!ws_ok(workspace, workspace_bytes, dense_gradient_workspace_bytes(DENSE_ABS, P, D, N, M, C, false))) return QLKA_ERR_WORKSPACE;
        CU(launch_dense_gradient(dense_grad_args(q, k, v, g_w, g_u, grad_q, grad_k, grad_v, workspace, P, D, N, M, C), DENSE_ABS, sm_count(),
                                 reinterpret_cast<cudaStream_t>(stream_)));
        return QLKA_OK;
    }
    const AbsBwdWs ws = in_pieces<AbsBwdWs>(workspace, workspace_bytes, P, D, N, M, C);
    if (!ws_ok(workspace, workspace_bytes, ws.bytes)) return QLKA_ERR_WORKSPACE;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    const int C4 = round4(C);
    const bool full = g_u != nullptr;

    const float* vrows = v;
    const float* grows = g_w;
    float*       gv    = grad_v;
    if (C4 != C) {
        CU(launch_pad_rows(v, ws.vpad, (long long)P * N, C, C4, stream));
        CU(launch_pad_rows(g_w, ws.gpad, (long long)P * M, C, C4, stream));
        vrows = ws.vpad; grows = ws.gpad; gv = ws.gvpad;
    }
    float* vsum     = ws.sums;
    float* gwsum    = vsum + (size_t)P * C4;
    float* qtotg    = gwsum + (size_t)P * C4;
    float* gu_total = qtotg + (size_t)P * C4;
    CU(launch_colsum_d(q, ws.qsumd, P, D, M, stream));
    CU(cudaMemsetAsync(ws.sums, 0, sizeof(float) * ((size_t)P * C4 * 3 + P), stream));
    CU(launch_rowstat(vrows, nullptr, vsum, nullptr, nullptr, P, N, C4, stream));
    CU(launch_rowstat(grows, ws.qsumd, gwsum, qtotg, nullptr, P, M, C4, stream));
    if (full) CU(launch_vecsum(g_u, gu_total, P, M, stream));

    // grad_v starts from a constant row per head
    CU(launch_abs_init(qtotg, gwsum, nullptr, nullptr, gv, nullptr, P, N, C4, M, 1.0f, 0.0f, stream));
    st = for_pieces(P, D, ws.piece, [&](const int p0, const int pc, const int d0, const int dc) -> int {
        const size_t s0 = (size_t)p0 * D + d0;
        const float *qp = q + s0 * M, *kp = k + s0 * N, *vp = vrows + (size_t)p0 * N * C4, *gp = grows + (size_t)p0 * M * C4, *up = full ? g_u + (size_t)p0 * M : nullptr;
        {   // grad_q: queries q walk the key stream k; prefix of v rows contracted with g_w rows
            SortArgs s = sort_args(ws.rec, kp, qp, pc * dc, dc, N, M, MODE_SGN, full ? SCAL_RANK : SCAL_NONE);
            s.uq = up;
            CU(launch_sort_rank(s, ws.rec, stream));
            WalkArgs w = walk_args(ws.rec, vp, pc * dc, dc, N, M, C4);
            w.g = gp; w.wtotal = vsum + (size_t)p0 * C4; w.out_s = grad_q + s0 * M; w.agg = ws.agg;
            CU(prefix_walk_chunked(w, EMIT_DOT, pc, stream));
        }
        {   // roles swapped: queries k walk the stream q whose rows are g_w. One walk for both: grad_v = abs sum with keys q, weights
            // g_w, evaluated at the keys k (row reductions); grad_k = prefix of g_w rows contracted with v rows (+ the g_u term in e1)
            SortArgs s = sort_args(ws.rec, qp, kp, pc * dc, dc, M, N, MODE_ABS, full ? SCAL_PREFIX : SCAL_NONE);
            s.us = up; s.us_total = gu_total + p0;
            CU(launch_sort_rank(s, ws.rec, stream));
            WalkArgs w = walk_args(ws.rec, gp, pc * dc, dc, M, N, C4);
            w.g = vp; w.wtotal = gwsum + (size_t)p0 * C4; w.out_s = grad_k + s0 * N; w.out = gv + (size_t)p0 * N * C4; w.agg = ws.agg;
            CU(prefix_walk_chunked(w, EMIT_BOTH, pc, stream));
        }
        return QLKA_OK;
    });
    if (st) return st;
    if (C4 != C) CU(launch_unpad_rows(gv, grad_v, (long long)P * N, C, C4, stream));
    return QLKA_OK;
}

// ---------------------------------------------------------------- sgn
int qlka_sgn_forward_workspace_bytes(int P, int D, int N, int M, int C, size_t* bytes) {
    return qlka_abs_backward_workspace_bytes(P, D, N, M, C, bytes);
}

int qlka_weighted_sgn_sum_forward(const float* q, const float* k, const float* v, const float* g,
                                  float* out, void* workspace, size_t workspace_bytes,
                                  int P, int D, int N, int M, int C, qlka_stream_t stream_)
{
    int st = check_dims(P, D, N, M, C);
    if (st) return st;
    if (!q || !k || !v || !g || !out) return QLKA_ERR_NULL;
    if (!aligned16(v, g)) return QLKA_ERR_ALIGNMENT;
    const AbsBwdWs ws = in_pieces<AbsBwdWs>(workspace, workspace_bytes, P, D, N, M, C);
    if (!ws_ok(workspace, workspace_bytes, ws.bytes)) return QLKA_ERR_WORKSPACE;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    const int C4 = round4(C);

    const float* vrows = v;
    const float* grows = g;
    if (C4 != C) {
        CU(launch_pad_rows(v, ws.vpad, (long long)P * N, C, C4, stream));
        CU(launch_pad_rows(g, ws.gpad, (long long)P * M, C, C4, stream));
        vrows = ws.vpad; grows = ws.gpad;
    }
    float* vsum = ws.sums;
    CU(cudaMemsetAsync(vsum, 0, sizeof(float) * (size_t)P * C4, stream));
    CU(launch_rowstat(vrows, nullptr, vsum, nullptr, nullptr, P, N, C4, stream));

    return for_pieces(P, D, ws.piece, [&](const int p0, const int pc, const int d0, const int dc) -> int {
        const size_t s0 = (size_t)p0 * D + d0;
        SortArgs s = sort_args(ws.rec, k + s0 * N, q + s0 * M, pc * dc, dc, N, M, MODE_SGN, SCAL_NONE);
        CU(launch_sort_rank(s, ws.rec, stream));
        WalkArgs w = walk_args(ws.rec, vrows + (size_t)p0 * N * C4, pc * dc, dc, N, M, C4);
        w.g = grows + (size_t)p0 * M * C4; w.wtotal = vsum + (size_t)p0 * C4; w.out_s = out + s0 * M; w.sign = -1.0f; w.agg = ws.agg;
        CU(prefix_walk_chunked(w, EMIT_DOT, pc, stream));
        return QLKA_OK;
    });
}

// ---------------------------------------------------------------- linear layers of the encoder
int qlka_split_rows(const float* x, const float* ln_weight, const float* ln_bias, float eps, void* parts, int rows, int K, qlka_stream_t stream) {
    if (rows <= 0 || K <= 0) return QLKA_ERR_BAD_SHAPE;
    if (!x || !parts || !ln_weight != !ln_bias) return QLKA_ERR_NULL;
    if (K % 4) return QLKA_ERR_UNSUPPORTED;
    if (!aligned16(x, parts, ln_weight, ln_bias)) return QLKA_ERR_ALIGNMENT;
    CU(launch_split_rows(x, ln_weight, ln_bias, parts, rows, K, eps, reinterpret_cast<cudaStream_t>(stream)));
    return QLKA_OK;
}

int qlka_split_heads(const float* o, void* parts, int B, int H, int S, int D, qlka_stream_t stream) {
    if (B <= 0 || H <= 0 || S <= 0 || D <= 0) return QLKA_ERR_BAD_SHAPE;
    if (!o || !parts) return QLKA_ERR_NULL;
    if (D % 4) return QLKA_ERR_UNSUPPORTED;
    if (!aligned16(o, parts)) return QLKA_ERR_ALIGNMENT;
    CU(launch_split_heads(o, parts, B, H, S, D, reinterpret_cast<cudaStream_t>(stream)));
    return QLKA_OK;
}

size_t qlka_linear_workspace_bytes(int N, int K) { return (size_t)6 * N * K; }

// the checks shared by the three layers, and the weight's parts in the workspace
static int linear_begin(const void* parts, const float* weight, const float* bias, void* workspace, size_t workspace_bytes, int M, int N, int K, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || K <= 0) return QLKA_ERR_BAD_SHAPE;
    if (!parts || !weight || !bias) return QLKA_ERR_NULL;
    if (K % 32 || N % 32) return QLKA_ERR_UNSUPPORTED;
    if (!aligned16(parts, weight, bias)) return QLKA_ERR_ALIGNMENT;
    if (!ws_ok(workspace, workspace_bytes, qlka_linear_workspace_bytes(N, K))) return QLKA_ERR_WORKSPACE;
    volatile int* word = nullptr;
    if (int st = qlka_linear_error_word(&word)) return st;
    if (*word) { *word = 0; return QLKA_ERR_GAVE_UP; }        // an earlier call's kernel: reported once
    CU(launch_split_rows(weight, nullptr, nullptr, workspace, N, K, 0.0f, stream));
    return QLKA_OK;
}

int qlka_linear_qkv(const void* parts, const float* weight, const float* bias, const float* table, float* q, float* k, float* v,
                    void* workspace, size_t workspace_bytes, int B, int S, int H, int K, qlka_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (B <= 0 || S <= 0 || H <= 0) return QLKA_ERR_BAD_SHAPE;
    if ((long long)B * S > INT_MAX || (long long)H * 192 > INT_MAX) return QLKA_ERR_INT32;
    if (!table || !q || !k || !v) return QLKA_ERR_NULL;
    if (!aligned16(table, q, k, v)) return QLKA_ERR_ALIGNMENT;
    int st = linear_begin(parts, weight, bias, workspace, workspace_bytes, B * S, 3 * H * 64, K, stream);
    if (st) return st;
    CU(launch_linear_qkv(parts, workspace, bias, table, q, k, v, B, S, H, K, sm_count(), stream));
    return QLKA_OK;
}

int qlka_linear_gelu(const void* parts, const float* weight, const float* bias, void* out_parts, void* workspace, size_t workspace_bytes,
                     int M, int N, int K, qlka_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (!out_parts) return QLKA_ERR_NULL;
    if (!aligned16(out_parts)) return QLKA_ERR_ALIGNMENT;
    int st = linear_begin(parts, weight, bias, workspace, workspace_bytes, M, N, K, stream);
    if (st) return st;
    CU(launch_linear_gelu(parts, workspace, bias, out_parts, M, N, K, sm_count(), stream));
    return QLKA_OK;
}

int qlka_linear_residual(const void* parts, const float* weight, const float* bias, float* x, void* workspace, size_t workspace_bytes,
                         int M, int N, int K, qlka_stream_t stream_) {
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (!x) return QLKA_ERR_NULL;
    if (!aligned16(x)) return QLKA_ERR_ALIGNMENT;
    int st = linear_begin(parts, weight, bias, workspace, workspace_bytes, M, N, K, stream);
    if (st) return st;
    CU(launch_linear_residual(parts, workspace, bias, x, M, N, K, sm_count(), stream));
    return QLKA_OK;
}

int qlka_linear_error_word(volatile int** word) {
    if (!word) return QLKA_ERR_NULL;
    int *host = nullptr, *device = nullptr;
    CU(linear_error_word(&host, &device));
    *word = host;
    return QLKA_OK;
}

int qlka_linear_error(int* error) {
    if (!error) return QLKA_ERR_NULL;
    CU(cudaDeviceSynchronize());
    volatile int* word = nullptr;
    int st = qlka_linear_error_word(&word);
    if (st) return st;
    *error = *word;
    *word = 0;
    return QLKA_OK;
}

// ---------------------------------------------------------------- diagnostic
int qlka_sort_rank_workspace_bytes(int P, int D, int N, int M, size_t* bytes) {
    if (!bytes) return QLKA_ERR_NULL;
    int st = check_dims(P, D, N, M, 1);
    if (st) return st;
    *bytes = sizeof(float) * 2 * (size_t)P * D * (N + 1) + 1024
           + ((N > SMALL_MAX || M > SMALL_MAX) ? sort_rank_large_scratch_bytes(P * D, N, M) : 0);
    return QLKA_OK;
}

// r: the output arrays, either of queries' records or of events
static int sort_rank_diagnostic(const float* x, const float* y, Records r, void* workspace, size_t workspace_bytes,
                                int P, int D, int N, int M, int mode, qlka_stream_t stream)
{
    int st = check_dims(P, D, N, M, 1);
    if (st) return st;
    if (!x || !y || !r.xperm || !r.xval || !r.mstart) return QLKA_ERR_NULL;
    if (mode != MODE_LAPLACE && mode != MODE_ABS) return QLKA_ERR_PATH;
    size_t need = 0;
    qlka_sort_rank_workspace_bytes(P, D, N, M, &need);
    if (!ws_ok(workspace, workspace_bytes, need)) return QLKA_ERR_WORKSPACE;
    Bump b(workspace);
    r.su0 = b.take<float>((size_t)P * D * (N + 1));
    r.su1 = b.take<float>((size_t)P * D * (N + 1));
    r.carve_large(b, P * D, N, M, false);
    SortArgs s = sort_args(r, x, y, P * D, D, N, M, mode, SCAL_NONE);
    CU(launch_sort_rank(s, r, reinterpret_cast<cudaStream_t>(stream)));
    return QLKA_OK;
}

int qlka_sort_rank_records(const float* x, const float* y,
                           uint32_t* xperm, float* xval, uint32_t* yrec, uint32_t* mstart,
                           void* workspace, size_t workspace_bytes,
                           int P, int D, int N, int M, int mode, qlka_stream_t stream)
{
    Records r{};
    r.xperm = xperm; r.xval = xval; r.yrec = reinterpret_cast<uint4*>(yrec); r.mstart = mstart;
    int st = check_dims(P, D, N, M, 1);
    if (st) return st;
    if (!yrec) return QLKA_ERR_NULL;
    return sort_rank_diagnostic(x, y, r, workspace, workspace_bytes, P, D, N, M, mode, stream);
}

int qlka_sort_rank_events(const float* x, const float* y,
                          uint32_t* xperm, float* xval, uint32_t* eidx, float* esc, uint32_t* mstart,
                          void* workspace, size_t workspace_bytes,
                          int P, int D, int N, int M, int mode, qlka_stream_t stream)
{
    Records r{};
    r.xperm = xperm; r.xval = xval; r.eidx = eidx; r.esc = reinterpret_cast<float2*>(esc); r.mstart = mstart;
    int st = check_dims(P, D, N, M, 1);
    if (st) return st;
    if (!eidx || !esc) return QLKA_ERR_NULL;
    return sort_rank_diagnostic(x, y, r, workspace, workspace_bytes, P, D, N, M, mode, stream);
}

}  // extern "C"
