// Sort/rank for segments longer than the shared-memory kernel holds (max(N, M) > 16384, up to 262144): the segment is cut by
// value into parts of at most PART_CAP keys, and every part goes through the shared-memory kernel of sort_rank.cu. The work of a
// segment is spread over as many CTAs as it has tiles and parts, whatever the number of segments.
//
//   sample_splitters  per segment: a stratified random sample of the keys is sorted; every SAMPLES_PER_BIN-th sample starts a
//                     bin (32 to 256 bins, some five hundred to a thousand keys each). Bins are intervals of (value,
//                     index), so ties cannot make a bin crowded.
//   count_bins        per tile of 4096 keys or queries: the bin of every element (binary search over the splitters), kept as
//                     a byte; counts per bin. A query's bin is chosen so that every key below it lies in its own bin or an
//                     earlier one and every key of a later bin is not below it.
//   merge_bins        per segment: consecutive bins are merged into parts while they stay within PART_CAP keys (and as many queries,
//                     where there are more queries than keys); starts.
//   scatter_parts     per tile: elements to their parts, through shared memory so that the lists are written in runs.
//   part_stats        per part: smallest and largest key and the part's own scalar sums; the last CTA of a segment chains them
//                     into what enters each part from below and from above.
//   sort_rank_small<..., PART>   the parts.
//   mark_part_starts  Laplace events: the marks of the parts' first keys.
//
// An exact bin count is what bounds a part, not the sample: a part overflows only if a single bin does, that is if more than
// PART_CAP consecutive keys held no more than SAMPLES_PER_BIN of the samples although 64 or more are expected (below 1e-16
// per segment); such a part would be cut short, never written past its end.
//
// Streaming and shared-memory bound: about 90 bytes per key and query through L2 and DRAM outside the last kernel. Four
// global radix passes, a global rank search and scattered records (the kernels this replaces) took 5.7 ms of the 11.4 ms of a
// Laplace sum at B=1, H=16, N=65536, and one CTA per segment and pass, which left most of the GPU idle for a few segments.
#include "qlka_common.cuh"

namespace qlka {

cudaError_t launch_sort_rank_parts(const SortArgs& a, const PartArgs& pa, cudaStream_t stream);

namespace {

constexpr int MAX_BINS = 256, SAMPLES_PER_BIN = 8;
constexpr int TILE = 4096, TILE_THREADS = 256, TILE_E = TILE / TILE_THREADS;

// With more queries than keys, parts are cut by their queries as well, and the bins are made finer as far as there are samples: a part is
// one CTA's, and one that has more than PART_CAP queries ranks them twice, with a scattered record per thread and turn. Laplace sums
// with and without (ms): 1 head x 64 features, 8192 keys, 262144 queries 1.59 / 2.88; 16 heads, 8192 x 65536, 5.5 / 6.4; 130 features,
// 1000 x 262144, 5.28 / 5.55. Below 512 keys the parts get too few keys for what a CTA costs: 24 heads x 130 features, 300 x 32768, 9.3 / 8.7.
inline bool cut_by_queries(int N, int M) { return M > N && N >= 512; }
inline int bins_of(int N, int M) {
    int b = 32;
    while (b < MAX_BINS && (b * 512 < N || (cut_by_queries(N, M) && b * 512 < M && b * 2 * SAMPLES_PER_BIN <= N))) b *= 2;
    return b;
}
// two neighbouring parts hold more than PART_CAP keys, or queries
inline int max_parts(int N, int M) { return 2 * (N / PART_CAP) + (cut_by_queries(N, M) ? 2 * (M / PART_CAP) : 0) + 2; }
constexpr int MAX_PARTS = 4 * (262144 / PART_CAP) + 2;
static_assert(MAX_PARTS <= 256, "parts are bytes, and one thread each in part_stats");
__host__ __device__ inline int tiles_of(int n) { return (n + TILE - 1) / TILE; }

// key order with the two zeros equal, as the float comparisons of the rank search see them
__device__ __forceinline__ uint32_t order_key(const float x) { return f2key(x + 0.0f); }

struct Lists {
    unsigned long long* split;      // [seg][MAX_BINS] first (value, index) of every bin
    uint32_t *bin_keys, *bin_queries;            // [seg][MAX_BINS]
    uint8_t  *kbin, *qbin;          // [seg][N], [seg][M]
    uint8_t  *part_of;              // [seg][MAX_BINS]
    uint32_t *cursor;               // [seg][maxparts][2] where the next keys / queries of a part go
    uint32_t *kkey, *kidx, *qidx;
    float    *qval;
    PartInfo *info;                 // [seg][maxparts]
    float4   *stats;                // [seg][maxparts] smallest key, largest key, sum seen from the largest, sum seen from the smallest
    uint32_t *done;                 // [seg] parts whose stats are written
    size_t   bytes;
    int      bins, mp, qcap;        // bins and (at most) parts per segment, queries that a part may collect
    Lists(void* base, int nseg, int N, int M) : bins(bins_of(N, M)), mp(max_parts(N, M)), qcap(cut_by_queries(N, M) ? PART_CAP : M) {
        char*  b = static_cast<char*>(base);
        size_t off = 0;
        auto take = [&](size_t n) { char* p = b ? b + off : nullptr; off += (n + 255) & ~size_t(255); return p; };
        const size_t s = nseg, mp = this->mp;
        bin_keys    = reinterpret_cast<uint32_t*>(take(s * MAX_BINS * 4));        // zeroed together: bin_keys, bin_queries, done
        bin_queries = reinterpret_cast<uint32_t*>(take(s * MAX_BINS * 4));
        done        = reinterpret_cast<uint32_t*>(take(s * 4));
        zeroed      = off;
        split  = reinterpret_cast<unsigned long long*>(take(s * MAX_BINS * 8));
        kbin   = reinterpret_cast<uint8_t*>(take(s * N));
        qbin   = reinterpret_cast<uint8_t*>(take(s * M));
        part_of = reinterpret_cast<uint8_t*>(take(s * MAX_BINS));
        cursor = reinterpret_cast<uint32_t*>(take(s * mp * 8));
        kkey   = reinterpret_cast<uint32_t*>(take(s * N * 4));
        kidx   = reinterpret_cast<uint32_t*>(take(s * N * 4));
        qval   = reinterpret_cast<float*>(take(s * M * 4));
        qidx   = reinterpret_cast<uint32_t*>(take(s * M * 4));
        info   = reinterpret_cast<PartInfo*>(take(s * mp * sizeof(PartInfo)));
        stats  = reinterpret_cast<float4*>(take(s * mp * sizeof(float4)));
        bytes  = off;
    }
    size_t zeroed;
};

// The published integer hash "lowbias32" (Chris Wellons, found by search over xor-shift-multiply hashes for low bias; public domain).
__device__ __forceinline__ uint32_t mix(uint32_t x) {
    x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; return x ^ (x >> 16);
}

__global__ void __launch_bounds__(512) sample_splitters(const SortArgs a, const Lists l)
{
    __shared__ unsigned long long s[MAX_BINS * SAMPLES_PER_BIN];
    const int N = a.N, bins = l.bins, n = bins * SAMPLES_PER_BIN;
    const long long seg = blockIdx.x;
    const float* x = a.x + seg * N;
    for (int i = threadIdx.x; i < n; i += 512) {
        const uint32_t lo = (uint32_t)((long long)i * N / n), hi = (uint32_t)((long long)(i + 1) * N / n);      // one sample from each stratum
        const uint32_t at = lo + (hi > lo ? mix((uint32_t)seg * 0x9e3779b9u + i) % (hi - lo) : 0u);
        s[i] = (unsigned long long)order_key(x[at]) << 32 | at;
    }
    for (int k = 2; k <= n; k *= 2) {
        for (int j = k / 2; j > 0; j /= 2) {
            __syncthreads();
            for (int i = threadIdx.x; i < n / 2; i += 512) {
                const int p = 2 * i - (i & (j - 1)), q = p + j;
                const unsigned long long u = s[p], v = s[q];
                if ((u > v) == ((p & k) == 0)) { s[p] = v; s[q] = u; }
            }
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < bins; b += 512) l.split[seg * MAX_BINS + b] = b ? s[b * SAMPLES_PER_BIN] : 0ull;
}

// blocks of a tile kernel: the segment's key tiles, then its query tiles
struct Tile {
    long long seg; bool keys; int t0, n;
    __device__ Tile(const SortArgs& a) {
        const int kt = tiles_of(a.N), qt = tiles_of(a.M);
        seg = blockIdx.x / (kt + qt);
        const int t = blockIdx.x % (kt + qt);
        keys = t < kt;
        t0 = (keys ? t : t - kt) * TILE;
        n  = min(TILE, (keys ? a.N : a.M) - t0);
    }
};

// Shared-memory bound. The splitters are searched as a tree in breadth-first order: the nodes of a level are neighbours, so the lanes
// of a warp, at different nodes of one level, meet in a bank only on the two last levels. In the sorted array, whose level with
// step s has its entries 2 s words apart, the last five levels cost 4 to 8 passes each: 0.34 ms for 128 segments of
// 262144 keys and queries.
__global__ void __launch_bounds__(TILE_THREADS, 8) count_bins(const SortArgs a, const Lists l)
{
    __shared__ uint32_t value[MAX_BINS], index[MAX_BINS];          // first (value, index) of every bin
    __shared__ uint32_t count[MAX_BINS], tree[MAX_BINS];           // node j's children are 2 j and 2 j + 1, the root is 1
    const Tile t(a);
    const int  bins = l.bins, tid = threadIdx.x;
    for (int b = tid; b < bins; b += TILE_THREADS) {
        const unsigned long long c = l.split[t.seg * MAX_BINS + b];
        value[b] = (uint32_t)(c >> 32); index[b] = (uint32_t)c; count[b] = 0;
        if (b > 0) {                               // 2^z times an odd number: z levels above the last one
            const int z = __ffs(b) - 1;
            tree[((bins >> 1) + (b >> 1)) >> z] = value[b];
        }
    }
    const float* src = t.keys ? a.x + t.seg * a.N + t.t0 : a.y + t.seg * a.M + t.t0;
    uint8_t*     dst = t.keys ? l.kbin + t.seg * a.N + t.t0 : l.qbin + t.seg * a.M + t.t0;
    float x[TILE_E];
    #pragma unroll
    for (int s = 0; s < TILE_E; s++) { const int i = s * TILE_THREADS + tid; x[s] = i < t.n ? src[i] : 0.0f; }
    __syncthreads();
    #pragma unroll
    for (int s0 = 0; s0 < TILE_E; s0 += 4) {
        // by value: bins that start at or below a key, below a query
        uint32_t c[4];
        int at[4];
        #pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t k = order_key(x[s0 + u]);
            c[u]  = t.keys || k == 0 ? k : k - 1;
            at[u] = 1;
        }
        for (int level = 1; level < bins; level *= 2) {
            #pragma unroll
            for (int u = 0; u < 4; u++) at[u] = 2 * at[u] + (tree[at[u]] <= c[u] ? 1 : 0);
        }
        #pragma unroll
        for (int u = 0; u < 4; u++) at[u] -= bins;
        #pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = (s0 + u) * TILE_THREADS + tid;
            if (t.keys)                                            // a key equal to the start of its bin: the index decides
                while (at[u] > 0 && value[at[u]] == c[u] && index[at[u]] > (uint32_t)(t.t0 + i)) at[u]--;
            if (i < t.n) { atomicAdd(&count[at[u]], 1u); dst[i] = (uint8_t)at[u]; }
        }
    }
    __syncthreads();
    uint32_t* total = (t.keys ? l.bin_keys : l.bin_queries) + t.seg * MAX_BINS;
    for (int b = tid; b < bins; b += TILE_THREADS) if (count[b]) atomicAdd(total + b, count[b]);
}

__global__ void __launch_bounds__(MAX_BINS) merge_bins(const SortArgs a, const Lists l)
{
    __shared__ uint32_t nk[MAX_BINS], nq[MAX_BINS];
    __shared__ uint8_t  part[MAX_BINS];
    const long long seg = blockIdx.x;
    const int bins = l.bins, mp = l.mp, tid = threadIdx.x;
    if (tid < bins) { nk[tid] = l.bin_keys[seg * MAX_BINS + tid]; nq[tid] = l.bin_queries[seg * MAX_BINS + tid]; }
    for (int i = tid; i < mp; i += MAX_BINS) l.info[seg * mp + i].n = 0;
    __syncthreads();
    if (tid == 0) {
        PartInfo* info = l.info + seg * mp;
        uint32_t* cur  = l.cursor + seg * mp * 2;
        int np = 0, ks = 0, qs = 0, k = 0, q = 0;
        auto close = [&]() {
            if (np < mp) {
                info[np].ks = ks; info[np].n = min(k, PART_CAP); info[np].qs = qs; info[np].m = q;
                cur[2 * np] = ks; cur[2 * np + 1] = qs;
            }
            np++; ks += k; qs += q; k = q = 0;
        };
        for (int b = 0; b < bins; b++) {
            if (k > 0 && nk[b] > 0 && (k + (int)nk[b] > PART_CAP || q + (int)nq[b] > l.qcap)) close();       // (every part has keys)
            part[b] = (uint8_t)np;
            k += nk[b]; q += nq[b];
        }
        close();
    }
    __syncthreads();
    if (tid < bins) l.part_of[seg * MAX_BINS + tid] = part[tid];
}

__global__ void __launch_bounds__(TILE_THREADS) scatter_parts(const SortArgs a, const Lists l)
{
    __shared__ uint32_t sval[TILE], sidx[TILE];
    __shared__ uint8_t  spart[TILE], part_of[MAX_BINS];
    __shared__ uint32_t count[MAX_PARTS], start[MAX_PARTS], gofs[MAX_PARTS];
    const Tile t(a);
    const int  tid = threadIdx.x, mp = l.mp, lane = tid & 31;
    const float*   src = t.keys ? a.x + t.seg * a.N + t.t0 : a.y + t.seg * a.M + t.t0;
    const uint8_t* bin = t.keys ? l.kbin + t.seg * a.N + t.t0 : l.qbin + t.seg * a.M + t.t0;
    float    x[TILE_E];
    uint32_t pr[TILE_E];                                // bin, then part << 16 | place among the tile's elements of the part
    #pragma unroll
    for (int s = 0; s < TILE_E; s++) {
        const int i = s * TILE_THREADS + tid;
        x[s]  = i < t.n ? src[i] : 0.0f;
        pr[s] = i < t.n ? bin[i] : 0u;
    }
    part_of[tid] = tid < l.bins ? l.part_of[t.seg * MAX_BINS + tid] : 0;
    if (tid < mp) count[tid] = 0;
    __syncthreads();
    #pragma unroll
    for (int s = 0; s < TILE_E; s++) {
        const int i = s * TILE_THREADS + tid;
        if (i < t.n) { const uint32_t p = part_of[pr[s]]; pr[s] = p << 16 | atomicAdd(&count[p], 1u); }
    }
    __syncthreads();
    if (tid < 32) {                                     // exclusive scan of the counts; room in the part lists
        uint32_t carry = 0;
        for (int p0 = 0; p0 < mp; p0 += 32) {
            const int p = p0 + lane;
            const uint32_t c = p < mp ? count[p] : 0u;
            uint32_t incl = c;
            #pragma unroll
            for (int off = 1; off < 32; off <<= 1) { const uint32_t u = __shfl_up_sync(FULL, incl, off); if (lane >= off) incl += u; }
            if (p < mp) {
                start[p] = carry + incl - c;
                gofs[p]  = c ? atomicAdd(l.cursor + (t.seg * mp + p) * 2 + (t.keys ? 0 : 1), c) : 0u;
            }
            carry += __shfl_sync(FULL, incl, 31);
        }
    }
    __syncthreads();
    #pragma unroll
    for (int s = 0; s < TILE_E; s++) {
        const int i = s * TILE_THREADS + tid;
        if (i < t.n) {
            const uint32_t p = pr[s] >> 16, at = start[p] + (pr[s] & 0xffffu);
            sval[at]  = t.keys ? order_key(x[s]) : __float_as_uint(x[s]);
            sidx[at]  = (uint32_t)(t.t0 + i);
            spart[at] = (uint8_t)p;
        }
    }
    __syncthreads();
    uint32_t* val = t.keys ? l.kkey + t.seg * a.N : reinterpret_cast<uint32_t*>(l.qval) + t.seg * a.M;
    uint32_t* idx = t.keys ? l.kidx + t.seg * a.N : l.qidx + t.seg * a.M;
    #pragma unroll 4
    for (int i = tid; i < t.n; i += TILE_THREADS) {
        const uint32_t p = spart[i], dst = gofs[p] + (uint32_t)i - start[p];
        val[dst] = sval[i];
        idx[dst] = sidx[i];
    }
}

__device__ __forceinline__ float block_reduce(float v, float* red, const int op)       // op 0: sum, 1: min, 2: max; 256 threads
{
    auto join = [&](const float x, const float y) -> float { return op == 0 ? x + y : op == 1 ? fminf(x, y) : fmaxf(x, y); };
    #pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = join(v, __shfl_xor_sync(FULL, v, off));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[0];
    for (int w = 1; w < 8; w++) v = join(v, red[w]);
    return v;
}

// The scalar sums of one part as sort_rank_small forms them: Laplace, u weighted, decayed to the part's largest key and to its
// smallest; abs: sum of the keys, or of the per-key scalar.
__global__ void __launch_bounds__(256) part_stats(const SortArgs a, const Lists l)
{
    __shared__ float  red[8];
    __shared__ float4 st[MAX_PARTS];
    __shared__ bool   finish;
    const int mp = l.mp, tid = threadIdx.x, N = a.N;
    const long long seg = blockIdx.x / mp;
    const int part = blockIdx.x % mp;
    const PartInfo pi = l.info[seg * mp + part];
    if (pi.n > 0) {
        const int p = (int)(seg / a.D);
        const uint32_t* kkey = l.kkey + seg * N + pi.ks;
        const uint32_t* kidx = l.kidx + seg * N + pi.ks;
        constexpr int U = PART_CAP / 256;
        float x[U], lo = INFINITY, hi = -INFINITY;
        #pragma unroll
        for (int u = 0; u < U; u++) {
            const int j = u * 256 + tid;
            x[u] = j < pi.n ? key2f(__ldg(kkey + j)) : 0.0f;
            if (j < pi.n) { lo = fminf(lo, x[u]); hi = fmaxf(hi, x[u]); }
        }
        lo = block_reduce(lo, red, 1);
        hi = block_reduce(hi, red, 2);
        float up = 0.0f, down = 0.0f;
        const bool lap = a.mode == MODE_LAPLACE;
        if (a.scal == SCAL_UNIT || a.scal == SCAL_PREFIX || a.scal == SCAL_SIGNED) {
            const float* us = (a.scal == SCAL_PREFIX || a.scal == SCAL_SIGNED) && a.us ? a.us + (long long)p * N : nullptr;
            #pragma unroll 8
            for (int u = 0; u < U; u++) {
                const int j = u * 256 + tid;
                if (j >= pi.n) break;
                const float w = us ? __ldg(us + __ldg(kidx + j)) : 1.0f;
                if (lap) { up = fmaf(w, expf(x[u] - hi), up); down = fmaf(w, expf(lo - x[u]), down); }
                else     up += us ? w : x[u];
            }
            up   = block_reduce(up, red, 0);
            down = block_reduce(down, red, 0);
        }
        if (tid == 0) l.stats[seg * mp + part] = make_float4(lo, hi, up, down);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) finish = atomicAdd(l.done + seg, 1u) == (uint32_t)mp - 1;
    __syncthreads();
    if (!finish) return;
    __threadfence();
    if (tid < mp) st[tid] = __ldcg(l.stats + seg * mp + tid);
    __syncthreads();
    if (tid > 1) return;
    PartInfo* info = l.info + seg * mp;
    int np = 0;
    while (np < mp && info[np].n > 0) np++;
    const bool lap = a.mode == MODE_LAPLACE;
    if (tid == 0) {                                     // from below
        float state = 0.0f, at = 0.0f;
        for (int i = 0; i < np; i++) {
            info[i].prevmax = at; info[i].lin = state;
            state = lap ? fmaf(i ? expf(at - st[i].y) : 0.0f, state, st[i].z) : state + st[i].z;
            at = st[i].y;
        }
    } else {                                            // from above
        float state = 0.0f, at = 0.0f;
        for (int i = np - 1; i >= 0; i--) {
            info[i].nextmin = at; info[i].rin = state;
            state = fmaf(i + 1 < np ? expf(st[i].x - at) : 0.0f, state, st[i].w);
            at = st[i].x;
        }
    }
}

// The marks of the first keys of a segment's parts but the first: the key before is as many events before the part as the part before
// has queries above its largest key. A thread per part.
__global__ void __launch_bounds__(256) mark_part_starts(const SortArgs a, const PartArgs pa)
{
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= (long long)a.nseg * pa.maxparts || i % pa.maxparts == 0 || pa.info[i].n == 0) return;
    const int ks = pa.info[i].ks;
    const uint32_t at = (uint32_t)(ks + pa.info[i].qs);
    a.xperm[i / pa.maxparts * npad(a.N) + ks] |= key_marks(at - pa.ends[i - 1].y, at + pa.ends[i].x);
}

}  // namespace

size_t sort_rank_large_scratch_bytes(int nseg, int N, int M) { return Lists(nullptr, nseg, N, M).bytes; }

cudaError_t launch_sort_rank_large(const SortArgs& a, void* scratch, cudaStream_t stream)
{
    const Lists l(scratch, a.nseg, a.N, a.M);
    cudaError_t e = cudaMemsetAsync(scratch, 0, l.zeroed, stream);
    if (e != cudaSuccess) return e;
    const unsigned tiles = (unsigned)a.nseg * (unsigned)(tiles_of(a.N) + tiles_of(a.M)), parts = (unsigned)a.nseg * (unsigned)l.mp;
    sample_splitters<<<a.nseg, 512, 0, stream>>>(a, l);
    count_bins<<<tiles, TILE_THREADS, 0, stream>>>(a, l);
    merge_bins<<<a.nseg, MAX_BINS, 0, stream>>>(a, l);
    scatter_parts<<<tiles, TILE_THREADS, 0, stream>>>(a, l);
    part_stats<<<parts, 256, 0, stream>>>(a, l);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    PartArgs pa{};
    pa.kkey = l.kkey; pa.kidx = l.kidx; pa.qval = l.qval; pa.qidx = l.qidx; pa.info = l.info; pa.maxparts = l.mp;
    pa.ends = reinterpret_cast<uint2*>(l.stats);            // (chained into info by now)
    e = launch_sort_rank_parts(a, pa, stream);
    if (e != cudaSuccess || !a.eidx || a.mode != MODE_LAPLACE) return e;
    mark_part_starts<<<(parts + 255) / 256, 256, 0, stream>>>(a, pa);
    return cudaGetLastError();
}

}  // namespace qlka
