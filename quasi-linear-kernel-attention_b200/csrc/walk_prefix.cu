// Prefix walk: for every query m of every segment, with r its rank among the sorted keys,
// PV = sum of the rows of the r keys below it and PK = sum of key * row over the same keys:
//
//   EMIT_ROWS  out[p, row_m, :] += e0_m * PV + e1_m * PK       (vector reductions)
//              with e0 = 2 * query and e1 = -2 this is the walk term 2 (q PV - PK) of the abs sum; folded
//              queries (shifted, weighted copies that share a row) scale both by their weight
//              (Weighted_Abs_Sum/csrc/abs_kernels.cu:9-18; abs_chunk :78-199, abs_prefix :202-405)
//
// EMIT_DOT and EMIT_BOTH (the walks of the gradients) share the first launch and the fold; their emission is in walk_events.cu.
//
// Same mapping and staging as the Laplace walk (walk_ring.cuh; SPS independent streams per
// segment numbered over all segments). The first launch sums each stream's rows into an aggregate
// table, a small kernel turns the table into exclusive prefix sums over each segment's streams, the last launch walks
// every stream forward from its incoming prefix and emits. With one stream per segment only the last one runs.
#include "walk_ring.cuh"

namespace qlka {

cudaError_t launch_prefix_events(const WalkArgs& a, bool rows, cudaStream_t stream);      // walk_events.cu

enum { EMIT_ROWS = 0, EMIT_DOT = 1, EMIT_BOTH = 2 };

// resident CTAs per SM that the passes are compiled for, and blocks in the emitting pass's rings (as in the Laplace walk)
constexpr int PREFIX_CTAS_ROWS = 8;
__host__ __device__ constexpr int prefix_ctas2(int cpl) { return cpl == 4 ? 2 : 4; }
constexpr int PREFIX_DEPTH2 = 3;

// floats per stream in the aggregate table: sum of the stream's rows | sum of key * row
__host__ __device__ inline int prefix_agg_stride(int C4) { return 2 * C4; }

// First launch (only with more than one stream per segment): every stream sums its rows (and key * row).
template <int LPS, int CPL, bool WITH_K>
__global__ void __launch_bounds__(KEY_THREADS, KEY_CTAS) prefix_pass1(const WalkArgs a)
{
    using F = KeyFeeder<LPS, CPL, WITH_K, 1>;
    __shared__ __align__(16) unsigned char smem[F::SMEM];
    const int C4 = a.C4, NBK = nblocks(a.N);
    F f;
    f.init(smem_u32(smem), a.N, C4);
    const StreamOf st(a, blockIdx.x, threadIdx.x / LPS, NBK, F::STREAMS);
    Vec<CPL> PV, PK;
    PV.zero(); PK.zero();
    Vec<CPL> x[KB];
    f.start(a, st, x);
    const int steps = __reduce_max_sync(FULL, f.nblk);
    for (int t = 0; t < steps; t++) {
        f.step(t, x);
        uint32_t n[KB];
        float    kv[KB];
        if (WITH_K) f.scalars(kv);
        f.read_index(f.next, n);
        if (t >= f.nblk) continue;                 // (the warp's other streams may be a block longer)
        #pragma unroll
        for (int h = 0; h < KB; h += 4) {
            #pragma unroll
            for (int i = h; i < h + 4; i++) {
                vadd(PV, x[i]);
                if (WITH_K) axpy8(PK, kv[i], x[i], PK);
            }
            if (t + 1 < f.nblk) {
                #pragma unroll
                for (int i = h; i < h + 4; i++) x[i] = f.row(n[i]);
            }
        }
    }
    cp_async_wait<0>();
    if (st.on) {
        float* ag = a.agg + st.g * prefix_agg_stride(C4);
        #pragma unroll
        for (int q = 0; q < F::Q; q++) {
            if (!f.on[q]) continue;
            *reinterpret_cast<float4*>(ag + f.channel(q)) = make_float4(PV.x[4 * q], PV.x[4 * q + 1], PV.x[4 * q + 2], PV.x[4 * q + 3]);
            if (WITH_K) *reinterpret_cast<float4*>(ag + C4 + f.channel(q)) = make_float4(PK.x[4 * q], PK.x[4 * q + 1], PK.x[4 * q + 2], PK.x[4 * q + 3]);
        }
    }
}

// Between the launches: per segment and channel, exclusive prefix sums of the stream aggregates, in place.
__global__ void __launch_bounds__(32 * FOLD_WARPS) prefix_fold(float* __restrict__ agg, const int nseg, const int SPS, const int C4, const int warps, const int with_k)
{
    __shared__ float total[2][FOLD_WARPS][32];
    const FoldOf f(nseg, SPS, C4, warps);
    const int lane = threadIdx.x & 31, c = f.c, first = f.first, last = f.last, AGS = prefix_agg_stride(C4);
    float* ag = agg + f.sg * SPS * AGS;
    float pv = 0.0f, pk = 0.0f;
    if (warps > 1) {
        #pragma unroll FOLD_CHUNK
        for (int t = first; t < last; t++) {
            pv += ag[(long long)t * AGS + c];
            if (with_k) pk += ag[(long long)t * AGS + C4 + c];
        }
        total[0][threadIdx.x >> 5][lane] = pv;
        total[1][threadIdx.x >> 5][lane] = pk;
        __syncthreads();
        pv = pk = 0.0f;
        for (int u = f.group; u < f.group + f.share; u++) { pv += total[0][u][lane]; pk += total[1][u][lane]; }
    }
    if (!f.on) return;
    for (int t0 = first; t0 < last; t0 += FOLD_CHUNK) {
        float v[FOLD_CHUNK], k[FOLD_CHUNK];
        #pragma unroll
        for (int j = 0; j < FOLD_CHUNK; j++) {
            const float* at = ag + (long long)min(t0 + j, last - 1) * AGS;
            v[j] = at[c]; k[j] = with_k ? at[C4 + c] : 0.0f;
        }
        #pragma unroll
        for (int j = 0; j < FOLD_CHUNK; j++) {
            if (t0 + j < last) {
                float* at = ag + (long long)(t0 + j) * AGS;
                at[c] = pv; pv += v[j];
                if (with_k) { at[C4 + c] = pk; pk += k[j]; }
            }
        }
    }
}

// Last launch: the walk with row emission, every stream starting from its incoming prefix sums, one stream per warp.
template <int CPL>
__global__ void __launch_bounds__(WALK_THREADS, prefix_ctas2(CPL)) prefix_pass2(const WalkArgs a)
{
    using F2 = Feeder<CPL, true, PREFIX_DEPTH2>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = warp_index(), c0 = lane * CPL;
    const int N = a.N, C4 = a.C4, NBK = nblocks(N);
    const bool lane_on = c0 < C4;
    const int  c0l     = lane_on ? c0 : 0;         // idle lanes shadow lane 0's loads and store nothing

    F2 f;
    f.init(smem_u32(smem) + warp * warp_bytes<CPL, PREFIX_DEPTH2>(), lane, N, C4);

    // static round-robin over the work items (an atomic work counter was measured 10 % slower)
    for (int item = blockIdx.x; item < a.nitems; item += gridDim.x) {
        const StreamOf st(a, item, warp, NBK);
        if (!st.on) break;
        f.start(a, st.sg, st.p, st.b0);
        char* out = reinterpret_cast<char*>(a.out + (long long)st.p * a.Mrows * C4 + c0l);

        Vec<CPL> PV, PK;
        PV.zero(); PK.zero();
        if (a.sps > 1) {        // incoming prefix sums (prefix_fold left them in the aggregate table)
            const float* ag = a.agg + st.g * prefix_agg_stride(C4) + c0l;
            PV = vload<CPL>(ag);
            PK = vload<CPL>(ag + C4);
        }

        __syncwarp();                              // every lane has left the previous item's slots
        f.prologue(st.nblk);
        int cur = 0, j0 = st.b0 * KB;
        for (int t = 0; t < st.nblk; t++, j0 += KB, cur = F2::next_slot(cur)) {
            f.advance_range();
            __syncwarp();
            f.step_issue(t, cur, st.nblk);
            cp_async_wait<F2::AHEAD>();
            __syncwarp();
            float kv[KB + 1];
            f.read_scalars(cur, kv);
            Vec<CPL> v[KB], kb[KB];
            f.read_rows(cur, j0, v);
            // prefix states before each key, in place of the rows
            #pragma unroll
            for (int i = 0; i < KB; i++) {
                const Vec<CPL> row = v[i];
                v[i]  = PV;
                kb[i] = PK;
                vadd(PV, row);
                axpy(PK, kv[i], row, PK);
            }
            for_queries(f, cur, j0, [&](const int i, const uint4& rec) {
                Vec<CPL> r;
                scale(r, __uint_as_float(rec.y), kb[i]);
                axpy(r, __uint_as_float(rec.x), v[i], r);
                if (lane_on) vred(reinterpret_cast<float*>(out + (unsigned long long)rec.z * f.row_bytes), r);
            });
        }
        cp_async_wait<0>();
    }
}

// Row emission with 4 channels per lane (RowFeeder; walk_ring.cuh's rows_by_quads says when)
template <int LPS>
__global__ void __launch_bounds__(ROW_THREADS, PREFIX_CTAS_ROWS) prefix_rows(const WalkArgs a)
{
    constexpr int STREAMS = ROW_THREADS / LPS;
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, ln = tid % LPS, c0 = ln * 4;
    const int N = a.N, C4 = a.C4, NBK = nblocks(N);
    const bool lane_on = c0 < C4;
    const int  c0l     = lane_on ? c0 : 0;
    const unsigned gmask = LPS == 32 ? FULL : (((1u << (LPS & 31)) - 1u) << ((tid & 31) & ~(LPS - 1)));

    RowFeeder<LPS> f;
    f.init(smem_u32(smem), N, a.M, C4);

    const StreamOf st(a, blockIdx.x, tid / LPS, NBK, STREAMS);
    f.start(a, st.sg, st.p, st.b0);
    char* out = reinterpret_cast<char*>(a.out + (long long)st.p * a.Mrows * C4 + c0l);
    Vec<4> PV, PK;
    PV.zero(); PK.zero();
    if (a.sps > 1) {        // incoming prefix sums (prefix_fold left them in the aggregate table)
        const float* ag = a.agg + (st.on ? st.g : 0) * prefix_agg_stride(C4) + c0l;
        PV = vload<4>(ag);
        PK = vload<4>(ag + C4);
    }
    f.prologue(st.nblk);
    int cur = 0, j0 = st.b0 * KB;
    for (int t = 0; t < st.nblk; t++, j0 += KB, cur ^= 1) {
        __syncwarp(gmask);                     // every lane is done with the slot refilled below
        f.step(t, cur, st.nblk);
        __syncwarp(gmask);
        float kv[KB + 1];
        f.read_scalars(cur, kv);
        Vec<4> v[KB], kb[KB];
        f.read_rows(cur, j0, v);
        // prefix states before each key, in place of the rows
        #pragma unroll
        for (int i = 0; i < KB; i++) {
            const Vec<4> row = v[i];
            v[i]  = PV;
            kb[i] = PK;
            vadd(PV, row);
            axpy(PK, kv[i], row, PK);
        }
        f.for_queries(cur, j0, [&](const int i, const uint4& rec) {
            Vec<4> r;
            scale(r, __uint_as_float(rec.y), kb[i]);
            axpy(r, __uint_as_float(rec.x), v[i], r);
            if (lane_on) vred(reinterpret_cast<float*>(out + (unsigned long long)rec.z * f.row_bytes), r);
        });
    }
    cp_async_wait<0>();
}

template <int LPS>
static cudaError_t launch_rows(const WalkArgs& a, cudaStream_t stream) {
    constexpr int smem = row_smem_bytes<LPS>();
    cudaError_t e = cudaFuncSetAttribute(prefix_rows<LPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const long long items = ((long long)a.nseg * a.sps * LPS + ROW_THREADS - 1) / ROW_THREADS;
    prefix_rows<LPS><<<(unsigned)items, ROW_THREADS, smem, stream>>>(a);
    return cudaGetLastError();
}

template <int CPL>
static cudaError_t launch_pass2(const WalkArgs& a, int sms, cudaStream_t stream) {
    auto k2 = prefix_pass2<CPL>;
    constexpr int smem2 = WALK_STREAMS * warp_bytes<CPL, PREFIX_DEPTH2>();
    const int cap2 = sms * prefix_ctas2(CPL);
    cudaError_t e = cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, smem2);
    if (e != cudaSuccess) return e;
    k2<<<a.nitems < cap2 ? a.nitems : cap2, WALK_THREADS, smem2, stream>>>(a);
    return cudaGetLastError();
}

template <int LPS, int CPL, bool WITH_K>
static cudaError_t launch_pass1(const WalkArgs& a, cudaStream_t stream) {
    constexpr int streams = KEY_THREADS / LPS;
    prefix_pass1<LPS, CPL, WITH_K><<<(unsigned)(((long long)a.nseg * a.sps + streams - 1) / streams), KEY_THREADS, 0, stream>>>(a);
    prefix_fold<<<fold_grid(a), 32 * FOLD_WARPS, 0, stream>>>(a.agg, a.nseg, a.sps, a.C4, fold_share_warps(a), WITH_K ? 1 : 0);
    return cudaGetLastError();
}

template <int LPS, int CPL>
static cudaError_t launch_pw(const WalkArgs& a, int emit, int sms, cudaStream_t stream) {
    if (a.sps > 1) {                                                   // (a lone stream per segment has nothing before it)
        constexpr int L = LPS < 32 ? 8 : 16, W = LPS == 8 ? 4 : 8;         // lanes of a stream and channels of each in the first launch
        cudaError_t e = emit == EMIT_DOT ? launch_pass1<L, W, false>(a, stream) : launch_pass1<L, W, true>(a, stream);
        if (e != cudaSuccess) return e;
    }
    if (emit != EMIT_ROWS) return launch_prefix_events(a, emit == EMIT_BOTH, stream);
    if (CPL == 4 || rows_by_quads(a)) return launch_rows<LPS>(a, stream);
    if constexpr (CPL < 4) return launch_pass2<CPL>(a, sms, stream);
}

int prefix_agg_stride_host(int C4) { return prefix_agg_stride(C4); }

// emit: EMIT_ROWS, EMIT_DOT or EMIT_BOTH
cudaError_t launch_prefix_walk(const WalkArgs& a, int emit, int sms, cudaStream_t stream) {
    if (emit != EMIT_ROWS && emit != EMIT_DOT && emit != EMIT_BOTH) return cudaErrorInvalidValue;
    if (a.C4 <= 32)  return launch_pw<8, 1>(a, emit, sms, stream);
    if (a.C4 <= 64)  return launch_pw<16, 2>(a, emit, sms, stream);
    if (a.C4 <= 128) return launch_pw<32, 4>(a, emit, sms, stream);
    return cudaErrorInvalidValue;
}

}  // namespace qlka
