// Laplace walk: out[p, row_m, :] += e0_m * L_{r-1} + e1_m * R_r for every query m of every
// segment, where r is the query's rank, L the decayed prefix sum of the gathered rows and R
// the decayed suffix sum (recurrences of Weighted_Laplace_Sum/csrc/laplace_kernels.cu:5-13).
// LAP_DOT and LAP_BOTH, the walks of the gradients of the sum, share the fold between the passes; their passes are in walk_events.cu.
// (The reference's training route is the chunked PyTorch path, Experiments/kernel_attention/attention.py:110-115.)
//
// Replaces the reference's laplace_chunk / laplace_scan / laplace_walk trio
// (laplace_kernels.cu:65-127, 134-188, 219-409) with two launches over independent work units:
//   * a "stream" is a contiguous run of key blocks of one segment; a segment is cut into SPS of them
//     (any number: the host picks it so that every SM gets its share) and the streams of all
//     segments are numbered consecutively (walk_ring.cuh: how lanes share a stream); nothing couples the
//     streams of a CTA.
//   * laplace_pass1 walks every stream backwards once: the local suffix state at every block start goes
//     to the segment's checkpoint array, the stream's forward and backward aggregates and the decay
//     across it to the aggregate table.
//   * laplace_fold turns the aggregates of a segment's streams into the prefix state entering each stream
//     and the suffix state entering it from above (serial over the streams, parallel over channels).
//   * laplace_rows or laplace_pass2 (persistent CTAs) walks every stream forward from those states: per
//     block of 8 keys the suffix states are rebuilt in registers from the next checkpoint, the prefix
//     states overwrite the row registers, and the block's queries are emitted in rank order.
// The rows are therefore gathered twice (the reference gathers them three times) and every
// exponential was already taken by the sort/rank kernel.
#include "walk_ring.cuh"

namespace qlka {

cudaError_t launch_laplace_events(const WalkArgs& a, bool rows, cudaStream_t stream);      // walk_events.cu

enum { LAP_ROWS = 0, LAP_DOT = 1, LAP_BOTH = 2 };

// resident CTAs per SM that the emitting pass is compiled for, and blocks in its rings: three CTAs with one stream per warp (two: 3.34
// instead of 3.02 ms at 48 heads x 16384 keys; four leave 64 registers: 4.1 ms)
constexpr int LAP_CTAS_ROWS = 8;
__host__ __device__ constexpr int lap_ctas2(int cpl) { return cpl == 4 ? 2 : 3; }
constexpr int LAP_DEPTH2 = 3;

// floats per stream in the aggregate table: forward aggregate | backward aggregate | decay forward, decay backward, checkpoints (an int), pad
__host__ __device__ inline int lap_agg_stride(int C4) { return 2 * C4 + 4; }

// MARKS: for a walk over events, which wants the state at the first key of every block of events but a stream's first. These checkpoints of a stream
// take the places of its last blocks, and their number goes to the aggregate table; each with {the decay from the key to the next
// stream's first, the key's own}. (A first pass over events has queries to step over: Laplace gradients of
// 48 heads x 1024 x 64 channels 1003 instead of 957 us, of 8 heads, 1000 keys x 9000 queries 1026 instead of 948.)
template <int LPS, int CPL, bool MARKS>
__global__ void __launch_bounds__(KEY_THREADS, KEY_CTAS) laplace_pass1(const WalkArgs a)
{
    using F = KeyFeeder<LPS, CPL, true, -1>;
    __shared__ __align__(16) unsigned char smem[F::SMEM];
    const int C4 = a.C4, NBK = nblocks(a.N);
    F f;
    f.init(smem_u32(smem), a.N, C4);
    const StreamOf st(a, blockIdx.x, threadIdx.x / LPS, NBK, F::STREAMS);
    long long at = (long long)st.sg * NBK + st.b1 - 1;         // checkpoint of the block in use; with marks, of the next key marked
    if (MARKS) at = (events_end(a, st.sg, st.b1) - 1) / EB;
    const long long at0 = at;
    Vec<CPL> A, R;                                 // the stream's forward aggregate, its suffix state
    A.zero(); R.zero();
    float w = 1.0f, wr = 1.0f;                     // decay from the last key visited to the stream's last one, to the next stream's first
    float anext = st.b1 < NBK ? __ldg(a.xval + (long long)st.sg * xstride(a.N) + st.b1 * KB) : 0.0f;
    Vec<CPL> x[KB];
    f.start(a, st, x);
    const int steps = __reduce_max_sync(FULL, f.nblk);
    for (int t = 0; t < steps; t++) {
        f.step(t, x);
        uint32_t n[KB], own[KB];
        float    av[KB];
        f.scalars(av);
        f.read_index(f.next, n);
        if (MARKS) f.read_index(f.rec, own);
        if (t >= f.nblk) continue;                 // (the warp's other streams may be a block longer)
        #pragma unroll
        for (int h = KB - 4; h >= 0; h -= 4) {
            #pragma unroll
            for (int i = h + 3; i >= h; i--) {
                axpy8(A, w, x[i], A);
                axpy8(R, anext, R, x[i]);
                wr *= anext; w *= av[i]; anext = av[i];
                if (MARKS && (own[i] & (i == 0 && t == f.nblk - 1 ? KEY_LATER : KEY_FIRST))) {
                    #pragma unroll
                    for (int q = 0; q < F::Q; q++)
                        if (f.on[q]) __stcs(reinterpret_cast<float4*>(a.ckpt + at * C4 + f.channel(q)), make_float4(R.x[4 * q], R.x[4 * q + 1], R.x[4 * q + 2], R.x[4 * q + 3]));
                    if (f.ln == 0) *reinterpret_cast<float2*>(a.wck + 2 * at) = make_float2(wr, av[i]);
                    at--;
                }
            }
            if (t + 1 < f.nblk) {
                #pragma unroll
                for (int i = h; i < h + 4; i++) x[i] = f.row(n[i]);
            }
        }
        if (!MARKS) {                              // (streaming: the second pass reads them long after, once)
            #pragma unroll
            for (int q = 0; q < F::Q; q++)
                if (f.on[q]) __stcs(reinterpret_cast<float4*>(a.ckpt + at * C4 + f.channel(q)), make_float4(R.x[4 * q], R.x[4 * q + 1], R.x[4 * q + 2], R.x[4 * q + 3]));
            if (f.ln == 0) a.wck[at] = wr;
            at--;
        }
    }
    cp_async_wait<0>();
    if (st.on) {
        float* ag = a.agg + st.g * lap_agg_stride(C4);
        #pragma unroll
        for (int q = 0; q < F::Q; q++) {
            if (!f.on[q]) continue;
            *reinterpret_cast<float4*>(ag + f.channel(q))      = make_float4(A.x[4 * q], A.x[4 * q + 1], A.x[4 * q + 2], A.x[4 * q + 3]);
            *reinterpret_cast<float4*>(ag + C4 + f.channel(q)) = make_float4(R.x[4 * q], R.x[4 * q + 1], R.x[4 * q + 2], R.x[4 * q + 3]);
        }
        if (f.ln == 0) { ag[2 * C4] = w; ag[2 * C4 + 1] = wr; ag[2 * C4 + 2] = __int_as_float((int)(at0 - at)); }
    }
}

// Between the passes: per segment and channel, the aggregates of the SPS streams become the states entering each
// stream - in place, forward aggregate -> prefix state before the stream (L = decay * L + aggregate over the earlier
// streams), backward aggregate -> suffix state after it. A warp's share of the streams is one such step itself: its aggregate and the
// product of its decays. Bound by latency: with the share in registers, read once and at once, 26 -> 12 us for 24576 streams of 64 channels
// (48 heads x 1024 keys).
__global__ void __launch_bounds__(32 * FOLD_WARPS) laplace_fold(float* __restrict__ agg, const int nseg, const int SPS, const int C4, const int warps)
{
    __shared__ float4 total[FOLD_WARPS][32];       // forward and backward aggregate, forward and backward decay of a share
    const FoldOf f(nseg, SPS, C4, warps);
    const int lane = threadIdx.x & 31, c = f.c, first = f.first, last = f.last, AGS = lap_agg_stride(C4);
    float* ag = agg + f.sg * SPS * AGS;
    float L = 0.0f, R = 0.0f;
    if ((SPS + warps - 1) / warps <= FOLD_CHUNK) {         // the share fits registers: read once, everything in flight together
        float fv[FOLD_CHUNK], bv[FOLD_CHUNK], af[FOLD_CHUNK], ab[FOLD_CHUNK];
        #pragma unroll
        for (int k = 0; k < FOLD_CHUNK; k++) {
            fv[k] = bv[k] = 0.0f; af[k] = ab[k] = 1.0f;
            if (first + k < last) {
                const float* at = ag + (long long)(first + k) * AGS;
                fv[k] = at[c]; bv[k] = at[C4 + c];
                const float2 d = *reinterpret_cast<const float2*>(at + 2 * C4);
                af[k] = d.x; ab[k] = d.y;
            }
        }
        if (warps > 1) {
            float dl = 1.0f, dr = 1.0f;
            #pragma unroll
            for (int k = 0; k < FOLD_CHUNK; k++) {
                L = fmaf(af[k], L, fv[k]);
                R = fmaf(dr, bv[k], R);
                dl *= af[k]; dr *= ab[k];
            }
            total[threadIdx.x >> 5][lane] = make_float4(L, R, dl, dr);
            __syncthreads();
            L = R = 0.0f;
            for (int u = f.group; u < f.group + f.share; u++)             { const float4 t = total[u][lane]; L = fmaf(t.z, L, t.x); }
            for (int u = f.group + warps - 1; u > f.group + f.share; u--) { const float4 t = total[u][lane]; R = fmaf(t.w, R, t.y); }
        }
        if (!f.on) return;
        #pragma unroll
        for (int k = 0; k < FOLD_CHUNK; k++)
            if (first + k < last) { ag[(long long)(first + k) * AGS + c] = L; L = fmaf(af[k], L, fv[k]); }
        #pragma unroll
        for (int k = FOLD_CHUNK - 1; k >= 0; k--)
            if (first + k < last) { ag[(long long)(first + k) * AGS + C4 + c] = R; R = fmaf(ab[k], R, bv[k]); }
        return;
    }
    if (warps > 1) {
        float dl = 1.0f, dr = 1.0f;
        #pragma unroll FOLD_CHUNK
        for (int t = first; t < last; t++) {           // (the backward aggregates forwards: R = b + d * (next b + next d * (...)))
            const float* at = ag + (long long)t * AGS;
            const float  af = at[2 * C4], ab = at[2 * C4 + 1];
            L = fmaf(af, L, at[c]);
            R = fmaf(dr, at[C4 + c], R);
            dl *= af; dr *= ab;
        }
        total[threadIdx.x >> 5][lane] = make_float4(L, R, dl, dr);
        __syncthreads();
        L = R = 0.0f;
        for (int u = f.group; u < f.group + f.share; u++)             { const float4 t = total[u][lane]; L = fmaf(t.z, L, t.x); }
        for (int u = f.group + warps - 1; u > f.group + f.share; u--) { const float4 t = total[u][lane]; R = fmaf(t.w, R, t.y); }
    }
    if (!f.on) return;
    for (int t0 = first; t0 < last; t0 += FOLD_CHUNK) {
        float fv[FOLD_CHUNK], af[FOLD_CHUNK];
        #pragma unroll
        for (int k = 0; k < FOLD_CHUNK; k++) {
            const float* at = ag + (long long)min(t0 + k, last - 1) * AGS;
            fv[k] = at[c]; af[k] = at[2 * C4];
        }
        #pragma unroll
        for (int k = 0; k < FOLD_CHUNK; k++) {
            if (t0 + k < last) { ag[(long long)(t0 + k) * AGS + c] = L; L = fmaf(af[k], L, fv[k]); }
        }
    }
    for (int t0 = last - 1; t0 >= first; t0 -= FOLD_CHUNK) {
        float bv[FOLD_CHUNK], ab[FOLD_CHUNK];
        #pragma unroll
        for (int k = 0; k < FOLD_CHUNK; k++) {
            const float* at = ag + (long long)max(t0 - k, first) * AGS;
            bv[k] = at[C4 + c]; ab[k] = at[2 * C4 + 1];
        }
        #pragma unroll
        for (int k = 0; k < FOLD_CHUNK; k++) {
            if (t0 - k >= first) { ag[(long long)(t0 - k) * AGS + C4 + c] = R; R = fmaf(ab[k], R, bv[k]); }
        }
    }
}

// The second pass with a warp per stream
template <int CPL>
__global__ void __launch_bounds__(WALK_THREADS, lap_ctas2(CPL)) laplace_pass2(const WalkArgs a)
{
    using F2 = Feeder<CPL, true, LAP_DEPTH2>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = warp_index(), c0 = lane * CPL;
    const int N = a.N, C4 = a.C4, NBK = nblocks(N);
    const bool lane_on = c0 < C4;
    const int  c0l     = lane_on ? c0 : 0;         // idle lanes shadow lane 0's loads and store nothing
    const int  AGS     = lap_agg_stride(C4);

    F2 f;
    f.init(smem_u32(smem) + warp * warp_bytes<CPL, LAP_DEPTH2>(), lane, N, C4);

    // static round-robin over the work items (an atomic work counter was measured 10 % slower)
    for (int item = blockIdx.x; item < a.nitems; item += gridDim.x) {
        const StreamOf st(a, item, warp, NBK);
        if (!st.on) break;
        const int b0 = st.b0, nblk = st.nblk;
        f.start(a, st.sg, st.p, b0);
        char* out = reinterpret_cast<char*>(a.out + (long long)st.p * a.Mrows * C4 + c0l);
        const float* ck = a.ckpt + ((long long)st.sg * NBK + b0 + 1) * C4 + c0l;      // of the next block to fetch
        const float* wk = a.wck + (long long)st.sg * NBK + b0 + 1;

        // incoming prefix and suffix state (laplace_fold left them in the aggregate table)
        Vec<CPL> L = vload<CPL>(a.agg + st.g * AGS + c0l), Rin = vload<CPL>(a.agg + st.g * AGS + C4 + c0l);

        __syncwarp();                              // every lane has left the previous item's slots
        f.prologue(nblk);
        // checkpoint of the block after the current one, fetched one iteration early
        Vec<CPL> cnext; cnext.zero();
        float    wnext = 0.0f;
        auto load_ckpt = [&]() { wnext = *wk++; cnext = vload_once<CPL>(ck); ck += C4; };
        if (nblk > 1) load_ckpt();

        int cur = 0, j0 = b0 * KB;
        for (int t = 0; t < nblk; t++, j0 += KB, cur = F2::next_slot(cur)) {
            f.advance_range();
            __syncwarp();
            // suffix state entering the block from above: corrected checkpoint, or the stream's incoming state
            Vec<CPL> Rn = Rin;
            if (t + 1 < nblk) axpy(Rn, wnext, Rin, cnext);
            if (t + 2 < nblk) load_ckpt();
            f.step_issue(t, cur, nblk);
            cp_async_wait<F2::AHEAD>();
            __syncwarp();
            float av[KB + 1];
            f.read_scalars(cur, av);
            Vec<CPL> v[KB], Rb[KB];
            f.read_rows(cur, j0, v);
            #pragma unroll
            for (int i = KB - 1; i >= 0; i--) {
                axpy(Rn, av[i + 1], Rn, v[i]);
                Rb[i] = Rn;
            }
            // prefix state before each key, in place of the rows
            #pragma unroll
            for (int i = 0; i < KB; i++) {
                const Vec<CPL> row = v[i];
                v[i] = L;
                axpy(L, av[i], L, row);
            }
            for_queries(f, cur, j0, [&](const int i, const uint4& rec) {
                Vec<CPL> r;
                scale(r, __uint_as_float(rec.y), Rb[i]);
                axpy(r, __uint_as_float(rec.x), v[i], r);
                if (lane_on) vred(reinterpret_cast<float*>(out + (unsigned long long)rec.z * f.row_bytes), r);
            });
        }
        cp_async_wait<0>();
    }
}

// The second pass's row emission with 4 channels per lane (RowFeeder; rows_by_quads says when). A CTA per item, eight of them (16 warps) on an
// SM: its state takes some 120 registers. Bound by the L2 traffic of one row gathered and one row reduced per key and query (2.38 of its 2.64 ms
// at 48 heads x 16384 keys and queries; with one stream per warp it took 3.0).
template <int LPS>
__global__ void __launch_bounds__(ROW_THREADS, LAP_CTAS_ROWS) laplace_rows(const WalkArgs a)
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
    const int nblk = st.nblk;
    f.start(a, st.sg, st.p, st.b0);
    char* out = reinterpret_cast<char*>(a.out + (long long)st.p * a.Mrows * C4 + c0l);
    const float* ck = a.ckpt + ((long long)st.sg * NBK + st.b0 + 1) * C4 + c0l;      // of the next block to fetch
    const float* wk = a.wck + (long long)st.sg * NBK + st.b0 + 1;
    const float* ag = a.agg + (st.on ? st.g : 0) * lap_agg_stride(C4) + c0l;
    Vec<4> L = vload<4>(ag), Rin = vload<4>(ag + C4);

    f.prologue(nblk);
    Vec<4> cnext; cnext.zero();
    float  wnext = 0.0f;
    auto load_ckpt = [&]() { wnext = *wk++; cnext = vload_once<4>(ck); ck += C4; };
    if (nblk > 1) load_ckpt();
    int cur = 0, j0 = st.b0 * KB;
    for (int t = 0; t < nblk; t++, j0 += KB, cur ^= 1) {
        __syncwarp(gmask);                     // every lane is done with the slot refilled below
        // suffix state entering the block from above: corrected checkpoint, or the stream's incoming state
        Vec<4> Rn = Rin;
        if (t + 1 < nblk) axpy(Rn, wnext, Rin, cnext);
        if (t + 2 < nblk) load_ckpt();
        f.step(t, cur, nblk);
        __syncwarp(gmask);
        float av[KB + 1];
        f.read_scalars(cur, av);
        Vec<4> v[KB], Rb[KB];
        f.read_rows(cur, j0, v);
        #pragma unroll
        for (int i = KB - 1; i >= 0; i--) {
            axpy(Rn, av[i + 1], Rn, v[i]);
            Rb[i] = Rn;
        }
        // prefix state before each key, in place of the rows
        #pragma unroll
        for (int i = 0; i < KB; i++) {
            const Vec<4> row = v[i];
            v[i] = L;
            axpy(L, av[i], L, row);
        }
        f.for_queries(cur, j0, [&](const int i, const uint4& rec) {
            Vec<4> r;
            scale(r, __uint_as_float(rec.y), Rb[i]);
            axpy(r, __uint_as_float(rec.x), v[i], r);
            if (lane_on) vred(reinterpret_cast<float*>(out + (unsigned long long)rec.z * f.row_bytes), r);
        });
    }
    cp_async_wait<0>();
}

template <int LPS>
static cudaError_t launch_lap_rows(const WalkArgs& a, cudaStream_t stream) {
    constexpr int smem = row_smem_bytes<LPS>();
    cudaError_t e = cudaFuncSetAttribute(laplace_rows<LPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const long long items = ((long long)a.nseg * a.sps * LPS + ROW_THREADS - 1) / ROW_THREADS;
    laplace_rows<LPS><<<(unsigned)items, ROW_THREADS, smem, stream>>>(a);
    return cudaGetLastError();
}

template <int CPL>
static cudaError_t launch_lap_pass2(const WalkArgs& a, int sms, cudaStream_t stream) {
    constexpr int smem = WALK_STREAMS * warp_bytes<CPL, LAP_DEPTH2>();
    cudaError_t e = cudaFuncSetAttribute(laplace_pass2<CPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const int cap = sms * lap_ctas2(CPL);
    laplace_pass2<CPL><<<a.nitems < cap ? a.nitems : cap, WALK_THREADS, smem, stream>>>(a);
    return cudaGetLastError();
}

template <int LPS, int CPL, bool MARKS>
static cudaError_t launch_lap_pass1(const WalkArgs& a, cudaStream_t stream) {
    constexpr int streams = KEY_THREADS / LPS;
    laplace_pass1<LPS, CPL, MARKS><<<(unsigned)(((long long)a.nseg * a.sps + streams - 1) / streams), KEY_THREADS, 0, stream>>>(a);
    return cudaGetLastError();
}

template <int LPS, int CPL>
static cudaError_t launch_lap(const WalkArgs& a, int emit, int sms, cudaStream_t stream, cudaEvent_t mid) {
    constexpr int L = LPS < 32 ? 8 : 16, W = LPS == 8 ? 4 : 8;         // lanes of a stream and channels of each in the first pass
    cudaError_t e = emit == LAP_ROWS ? launch_lap_pass1<L, W, false>(a, stream) : launch_lap_pass1<L, W, true>(a, stream);
    if (e != cudaSuccess) return e;
    laplace_fold<<<fold_grid(a), 32 * FOLD_WARPS, 0, stream>>>(a.agg, a.nseg, a.sps, a.C4, fold_share_warps(a));
    e = cudaGetLastError();
    if (e == cudaSuccess && mid) e = cudaEventRecord(mid, stream);
    if (e != cudaSuccess) return e;
    if (emit != LAP_ROWS) return launch_laplace_events(a, emit == LAP_BOTH, stream);
    if (CPL == 4 || rows_by_quads(a)) return launch_lap_rows<LPS>(a, stream);
    if constexpr (CPL < 4) return launch_lap_pass2<CPL>(a, sms, stream);
}

int laplace_agg_stride(int C4) { return lap_agg_stride(C4); }

// emit: 0 = row reductions (the forward sum), 1 = dot, 2 = both;
// mid: optional event recorded between the first pass (with the fold) and the second
cudaError_t launch_laplace_walk(const WalkArgs& a, int emit, int sms, cudaStream_t stream, cudaEvent_t mid) {
    if (a.C4 <= 32)  return launch_lap<8, 1>(a, emit, sms, stream, mid);
    if (a.C4 <= 64)  return launch_lap<16, 2>(a, emit, sms, stream, mid);
    if (a.C4 <= 128) return launch_lap<32, 4>(a, emit, sms, stream, mid);
    return cudaErrorInvalidValue;
}

}  // namespace qlka
