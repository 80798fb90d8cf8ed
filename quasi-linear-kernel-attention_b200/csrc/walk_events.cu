// Walks that need a row per query as well as per key: the dot emissions of the gradients and of the public sgn op.
//
//   prefix_events   out_s[seg, row_m] = sign * (2 <g[p, row_m, :], PV - wtotal[p, :] / 2> + e1_m), PV = sum of the rows of the keys below
//                   query m: the signed-rank walk behind grad_q, grad_k and the sgn op (Weighted_Abs_Sum/csrc/sgn_kernels.cu:8-15,
//                   sgn_prefix :17-192); with ROWS also out[p, row_m, :] += e0_m (PV - wtotal[p, :] / 2) - 2 PK, PK = sum of
//                   key * row (grad_v and grad_k from one walk)
//   laplace_events  out_s[seg, row_m] += <g[p, row_m, :], e1_m R_r - e0_m L_{r-1}>, R and L the decayed suffix and prefix sums around the
//                   query (d/dquery of the Laplace sum, contracted with the upstream gradient); with ROWS also
//                   out[p, row_m, :] += e0_m L_{r-1} + e1_m R_r
//
// Keys and queries travel as one list of events in walk order (qlka_common.cuh), EB = 8 to a block, each with a row: of the stream's
// matrix for a key, of the contracted one for a query. A key adds its row to the state, a query contracts its row with it; which of the
// two an event is only predicates instructions, so nothing diverges and 2 or 4 streams share a warp with 8 (prefix) or 4 channels per
// lane. A loop over each key's queries, one stream per warp, with the queries' rows fetched once their records had arrived, took 60
// instructions per key and query where this takes 20 (dots) to 45. At 96 heads x 4096 keys x 64 features and channels: prefix dots
// 1.94 -> 0.78 ms, rows and dots 2.78 -> 1.69; Laplace at 24 heads x 4096, both passes: dots 0.79 -> 0.65, rows and dots 0.93 -> 0.79.
// A row gathered per event is 0.65 ms of the first at the L2's rate (a bare loop over the same gathers), with a row reduced 1.5 of the second.
// Rows go straight to registers, block t + 1's as soon as block t's are done with: through shared memory (cp.async) the load/store
// pipe moved every row twice and was 77 % busy (dots 1.20 ms); with L1::no_allocate on the loads the L2 did not keep them (7.4 instead of
// 0.9 GB from memory, 1.23 ms); bulk copies go at half the rate. 16 warps per SM: 24, with registers spilled, are slower.
// The events' indices and scalars are shared by the lanes of a stream and arrive in shared memory a block ahead of the rows they point at.
// A query's dot is a sum over the stream's lanes: each parks its part in shared memory, and after every block LPS / 8 lanes add up the
// parts of one event each (shuffles instead: a third more instructions, 1.40 against 1.20 ms).
#include "walk_ring.cuh"

#include <algorithm>

namespace qlka {

constexpr int EV_THREADS = 64, EV_CTAS = 8;            // small CTAs, one item each: they spread over the SMs however few streams there are
constexpr int EV_REC  = EB * 12;                       // indices and scalars of a block
constexpr int EV_GROUP = 4;                            // events between two rounds of loads
// a stream's lanes and the channels of each: quads ln, and with 8 channels LPS + ln, of the row's
template <int LPS, int CPL> struct Shape {
    static constexpr int STREAMS = EV_THREADS / LPS;
    static constexpr int PITCH = 128 + LPS * 2;        // between the parts of two events in a warp's area: no bank conflicts in either direction
    static constexpr int PARTS = EB * PITCH;
    static constexpr int SMEM = EV_THREADS / 32 * PARTS + STREAMS * 3 * EV_REC;
};

__device__ __forceinline__ float2 lds_f2(const uint32_t addr) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}
// two floats in one register pair
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(const float a, const float b) { f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpack2(const f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 mul2(const f2 a, const f2 b) { f2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f2 fma2(const f2 a, const f2 b, const f2 c) { f2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ bool is_query(const uint32_t e) { return (int)e < 0; }

// A stream's events: LPS lanes, block t = 0 .. nblk-1.
template <int LPS, int CPL>
struct EventFeeder {
    using S = Shape<LPS, CPL>;
    static constexpr int LPE = LPS / EB;       // lanes that add up an event's parts
    static constexpr int Q = CPL / 4;          // a lane's quads
    uint32_t           rec, next, after;       // shared addresses: the records of the block in use, the next one and the one after it
    uint32_t           part, sums;     // this lane's part of event 0, its share of the parts to add up
    int                ln, mine;       // mine: the event whose parts this lane adds up
    bool               on[Q];          // quad q lies inside the row (idle ones read the first)
    uint32_t           row_bytes;
    unsigned long long krows, qrows;   // matrix of the keys, of the queries: + p * rows * row_bytes + my first 16 bytes (- EVENT_QUERY rows)
    uint32_t           second;         // from there to the second 16
    const char*        aux;            // lanes 0, 1: the indices of the next block to copy; lanes 2 .. 5: the scalars, + my 16 bytes
    int                aux_step;
    int                ev0, ev1;       // the stream's events, counted from its first block in memory
    int                nblk, inner;    // its blocks; of this step on, the block is the last one of a stream of the warp, or beyond

    __device__ __forceinline__ int channel(const int q) const { return on[q] ? (q * LPS + ln) * 4 : 0; }
    __device__ __forceinline__ void init(const uint32_t smem, const int C4) {
        const int lane = threadIdx.x & 31;
        ln = threadIdx.x % LPS; mine = ln / LPE;
        const uint32_t area = smem + (threadIdx.x >> 5) * S::PARTS;
        part = area + lane * 4;
        sums = area + mine * S::PITCH + (lane - ln) * 4 + (ln % LPE) * 16;
        rec  = smem + EV_THREADS / 32 * S::PARTS + (threadIdx.x / LPS) * 3 * EV_REC;
        next = rec + EV_REC; after = next + EV_REC;
        #pragma unroll
        for (int q = 0; q < Q; q++) on[q] = (q * LPS + ln) * 4 < C4;
        second = Q > 1 && on[Q - 1] ? LPS * 16 : 0;
        row_bytes = (uint32_t)C4 * 4u;
    }
    // the events of key blocks [b0, b1) of segment sg (head p); returns the place in memory of the first block
    __device__ __forceinline__ long long start(const WalkArgs& a, const StreamOf& st, const int NBK) {
        const uint32_t* ms = a.mstart + (long long)st.sg * mstride(a.N);
        const int e0 = st.b0 * KB + (int)__ldg(ms + st.b0), e1 = min(st.b1 * KB, a.N) + (int)__ldg(ms + st.b1);
        const long long first = (long long)st.sg * estride(a.N, a.M) + e0 / EB * EB;
        ev0   = e0 % EB;
        ev1   = st.on ? ev0 + (e1 - e0) : 0;
        nblk  = st.on && e1 > e0 ? (ev1 + EB - 1) / EB : 0;
        inner = __reduce_min_sync(FULL, nblk) - 1;
        krows = (unsigned long long)__cvta_generic_to_global(a.rows + (long long)st.p * a.N * a.C4 + channel(0));
        qrows = (unsigned long long)__cvta_generic_to_global(a.g + (long long)st.p * a.M * a.C4 + channel(0)) - (unsigned long long)EVENT_QUERY * row_bytes;
        aux = ln < 2 ? reinterpret_cast<const char*>(a.eidx + first) + ln * 16 : reinterpret_cast<const char*>(a.esc + first) + (ln - 2) * 16;
        aux_step = EB * (ln < 2 ? 4 : 8);
        return first;
    }
    __device__ __forceinline__ bool has(const int t, const int i) const { const int at = t * EB + i; return t < nblk && at >= ev0 && at < ev1; }
    __device__ __forceinline__ bool edge(const int t) const { return t == 0 || t >= inner; }
    __device__ __forceinline__ void copy_records(const int t, const uint32_t dst) {
        if (t < nblk && ln < 6) { cp_async16(dst + ln * 16, aux); aux += aux_step; }
    }
    // Events before or after the stream in its first and last block become queries of row 0 that nobody writes: the loops need no bounds.
    __device__ __forceinline__ void trim(const int t, const uint32_t r) const {
        if (ln < EB && !has(t, ln)) asm volatile("st.shared.u32 [%0], %1;" :: "r"(r + ln * 4), "r"(EVENT_QUERY) : "memory");
        __syncwarp();
    }
    __device__ __forceinline__ void read_index(const uint32_t r, uint32_t (&e)[EB]) const {
        const uint4 a = lds128u(r), b = lds128u(r + 16);
        e[0] = a.x; e[1] = a.y; e[2] = a.z; e[3] = a.w; e[4] = b.x; e[5] = b.y; e[6] = b.z; e[7] = b.w;
    }
    __device__ __forceinline__ Vec<CPL> row(const uint32_t e) const {
        const unsigned long long at = (is_query(e) ? qrows : krows) + (unsigned long long)e * row_bytes;
        Vec<CPL> v;
        #pragma unroll
        for (int q = 0; q < Q; q++)
            asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v.x[4 * q]), "=f"(v.x[4 * q + 1]), "=f"(v.x[4 * q + 2]), "=f"(v.x[4 * q + 3]) : "l"(at + (q ? second : 0u)));
        return v;
    }
    // rows of block 0 under way, records of block 1 as well
    __device__ __forceinline__ void prologue(Vec<CPL> (&x)[EB], uint32_t (&e)[EB]) {
        copy_records(0, next);
        cp_async_commit();
        cp_async_wait<0>();
        __syncwarp();
        trim(0, next);
        copy_records(1, after);
        cp_async_commit();
        read_index(next, e);
        #pragma unroll
        for (int i = 0; i < EB; i++) x[i] = row(e[i]);
    }
    // block t becomes the block in use; the indices of block t + 1 are readable
    __device__ __forceinline__ void step(const int t) {
        const uint32_t r = rec;
        rec = next; next = after; after = r;
        cp_async_wait<0>();
        __syncwarp();                  // ... by every lane; and every lane has left block t - 1
        if (t + 1 >= inner) trim(t + 1, next);
        copy_records(t + 2, after);
        cp_async_commit();
    }
    // this lane's channels of a row of C4 floats that is read once
    __device__ __forceinline__ Vec<CPL> vector(const float* p) const {
        Vec<CPL> v;
        #pragma unroll
        for (int q = 0; q < Q; q++)
            asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x[4 * q]), "=f"(v.x[4 * q + 1]), "=f"(v.x[4 * q + 2]), "=f"(v.x[4 * q + 3]) : "l"(p + channel(q)));
        return v;
    }
    __device__ __forceinline__ float2 scalars(const int i) const { return lds_f2(rec + EB * 4 + i * 8); }
    // this lane's part of <x, s>; idle quads hold no rows
    __device__ __forceinline__ float dot(const Vec<CPL>& x, const Vec<CPL>& s) const {
        float r = 0.0f;
        #pragma unroll
        for (int q = 0; q < Q; q++) {
            float d = x.x[4 * q] * s.x[4 * q];
            #pragma unroll
            for (int c = 1; c < 4; c++) d = fmaf(x.x[4 * q + c], s.x[4 * q + c], d);
            d = on[q] ? d : 0.0f;
            r = q ? r + d : d;
        }
        return r;
    }
    __device__ __forceinline__ void park(const int i, const float v) const { sts32f(part + i * S::PITCH, v); }
    // done(sum, row, shared address of the scalars) for every query of block t, in one lane each
    template <class Done>
    __device__ __forceinline__ void finish(const int t, Done done) const {
        __syncwarp();
        const float4 a = lds128(sums), b = lds128(sums + LPS * 2);
        float s = ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
        #pragma unroll
        for (int off = 1; off < LPE; off <<= 1) s += __shfl_xor_sync(FULL, s, off);
        const uint32_t e = lds32u(rec + mine * 4);
        bool mark = ln % LPE == 0 && is_query(e);
        if (edge(t)) mark = mark && has(t, mine);
        if (mark) done(s, e & ~EVENT_QUERY, rec + EB * 4 + mine * 8);
    }
};

// a query's 16 bytes of its output row (`out` as qrows), if `on`
__device__ __forceinline__ void red_if_query(const bool on, const uint32_t e, const unsigned long long out, const uint32_t row_bytes, const float* r) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .u64 d;\n\tsetp.ne.s32 p, %3, 0;\n\tsetp.lt.and.s32 p, %0, 0, p;\n\tmad.wide.u32 d, %0, %2, %1;\n\t"
                 "@p red.global.add.v4.f32 [d], {%4, %5, %6, %7};\n\t}"
                 :: "r"(e), "l"(out), "r"(row_bytes), "r"((int)on), "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]) : "memory");
}

// The prefix walk with dots. The state is H = PV - wtotal / 2 and (with rows) T = -2 PK, so that a query costs one
// multiply-add per channel for its dot (doubled when it is written) and one for its row.
template <int LPS, int CPL, bool ROWS>
__global__ void __launch_bounds__(EV_THREADS, EV_CTAS) prefix_events(const WalkArgs a)
{
    using F = EventFeeder<LPS, CPL>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int C4 = a.C4, NBK = nblocks(a.N);
    F f;
    f.init(smem_u32(smem), C4);

    const StreamOf st(a, blockIdx.x, threadIdx.x / LPS, NBK, F::S::STREAMS);
    f.start(a, st, NBK);
    float* out_s = a.out_s + (long long)st.sg * a.M;
    const unsigned long long out = ROWS ? (unsigned long long)__cvta_generic_to_global(a.out + (long long)st.p * a.Mrows * C4 + f.channel(0)) - (unsigned long long)EVENT_QUERY * f.row_bytes : 0ull;
    Vec<CPL> H, T;
    H.zero(); T.zero();
    #pragma unroll
    for (int q = 0; q < F::Q; q++) {
        const int c = f.channel(q);
        if (a.sps > 1) {           // incoming prefix sums (prefix_fold left them in the aggregate table)
            const float* ag = a.agg + (st.on ? st.g : 0) * 2 * C4 + c;
            const float4 h = ldg4(ag);
            H.x[4 * q] = h.x; H.x[4 * q + 1] = h.y; H.x[4 * q + 2] = h.z; H.x[4 * q + 3] = h.w;
            if (ROWS) {
                const float4 u = ldg4(ag + C4);
                T.x[4 * q] = -2.0f * u.x; T.x[4 * q + 1] = -2.0f * u.y; T.x[4 * q + 2] = -2.0f * u.z; T.x[4 * q + 3] = -2.0f * u.w;
            }
        }
        const float4 w = ldg4(a.wtotal + (long long)st.p * C4 + c);
        H.x[4 * q] = fmaf(-0.5f, w.x, H.x[4 * q]);         H.x[4 * q + 1] = fmaf(-0.5f, w.y, H.x[4 * q + 1]);
        H.x[4 * q + 2] = fmaf(-0.5f, w.z, H.x[4 * q + 2]); H.x[4 * q + 3] = fmaf(-0.5f, w.w, H.x[4 * q + 3]);
    }
    Vec<CPL> x[EB];
    uint32_t e[EB];
    f.prologue(x, e);
    const int steps = __reduce_max_sync(FULL, f.nblk);
    for (int t = 0; t < steps; t++) {
        f.step(t);
        uint32_t n[EB];
        f.read_index(f.next, n);
        #pragma unroll
        for (int h = 0; h < EB; h += EV_GROUP) {
            #pragma unroll
            for (int i = h; i < h + EV_GROUP; i++) {
                const Vec<CPL> y = x[i];
                f.park(i, f.dot(y, H));
                const float s = ROWS ? f.scalars(i).x : 0.0f;
                if (ROWS) {
                    float r[CPL];
                    #pragma unroll
                    for (int c = 0; c < CPL; c++) r[c] = fmaf(s, H.x[c], T.x[c]);
                    const bool write = !f.edge(t) || f.has(t, i);
                    #pragma unroll
                    for (int q = 0; q < F::Q; q++) red_if_query(f.on[q] && write, e[i], out + (q ? f.second : 0u), f.row_bytes, r + 4 * q);
                }
                if (!is_query(e[i])) {
                    #pragma unroll
                    for (int c = 0; c < CPL; c++) { if (ROWS) T.x[c] = fmaf(s, y.x[c], T.x[c]); H.x[c] += y.x[c]; }
                }
            }
            // the next block's rows into the registers that are free now
            #pragma unroll
            for (int i = h; i < h + EV_GROUP; i++) x[i] = f.row(n[i]);
        }
        f.finish(t, [&](const float sum, const uint32_t row, const uint32_t sc) {
            out_s[row] = a.sign * fmaf(2.0f, sum, lds_f2(sc).y);
        });
        #pragma unroll
        for (int i = 0; i < EB; i++) e[i] = n[i];
    }
    cp_async_wait<0>();
}

template <int LPS, int CPL, bool ROWS>
static cudaError_t launch_prefix(const WalkArgs& a, cudaStream_t stream) {
    constexpr int smem = Shape<LPS, CPL>::SMEM;
    const long long items = ((long long)a.nseg * a.sps * LPS + EV_THREADS - 1) / EV_THREADS;
    prefix_events<LPS, CPL, ROWS><<<(unsigned)items, EV_THREADS, smem, stream>>>(a);
    return cudaGetLastError();
}

// dots, or rows and dots, of a prefix walk whose streams' incoming sums are in a.agg
cudaError_t launch_prefix_events(const WalkArgs& a, bool rows, cudaStream_t stream) {
    if (a.C4 <= 32)  return rows ? launch_prefix<8, 4, true>(a, stream) : launch_prefix<8, 4, false>(a, stream);
    if (a.C4 <= 64)  return rows ? launch_prefix<8, 8, true>(a, stream) : launch_prefix<8, 8, false>(a, stream);
    if (a.C4 <= 128) return rows ? launch_prefix<16, 8, true>(a, stream) : launch_prefix<16, 8, false>(a, stream);
    return cudaErrorInvalidValue;
}

// The Laplace walk with dots goes over its streams twice, as the row walk does: backwards over the keys (laplace_pass1, with marks), then
// forwards over the events. There a block is swept twice in registers: backwards with the suffix state, which the checkpoint of the
// first key after the block gives, forwards with the prefix state. (Dots with the stream's own suffix state in the first walk, corrected by
// the second with what comes from beyond, need no checkpoints but gather the queries' rows twice: 0.35 against 0.33 ms at 48 x 1024.)
template <int LPS, int CPL, bool ROWS>
__global__ void __launch_bounds__(EV_THREADS, EV_CTAS) laplace_events(const WalkArgs a)
{
    using F = EventFeeder<LPS, CPL>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int C4 = a.C4, NBK = nblocks(a.N);
    F f;
    f.init(smem_u32(smem), C4);

    const StreamOf st(a, blockIdx.x, threadIdx.x / LPS, NBK, F::S::STREAMS);
    const long long block0 = f.start(a, st, NBK) / EB;
    float* out_s = a.out_s + (long long)st.sg * a.M;
    const unsigned long long out = ROWS ? (unsigned long long)__cvta_generic_to_global(a.out + (long long)st.p * a.Mrows * C4 + f.channel(0)) - (unsigned long long)EVENT_QUERY * f.row_bytes : 0ull;
    const float* ag = a.agg + (st.on ? st.g : 0) * (2 * C4 + 4);       // incoming states (laplace_fold left them in the aggregate table)
    Vec<CPL> L = f.vector(ag);
    const float alast = st.on && st.b1 < NBK ? __ldg(a.xval + (long long)st.sg * xstride(a.N) + st.b1 * KB) : 0.0f;
    // checkpoints: of the first keys of the blocks after the first that have any, in the places of the stream's last blocks
    int       left = st.on ? __float_as_int(__ldg(ag + 2 * C4 + 2)) : 0;
    long long at   = block0 + f.nblk - left;
    // the checkpoint of the first key after the block in use, fetched one block early, into registers that the backward sweep leaves
    Vec<CPL> cnext;
    float2   wnext = make_float2(0.0f, 0.0f);
    cnext.zero();
    auto load_ckpt = [&]() { wnext = __ldg(reinterpret_cast<const float2*>(a.wck + 2 * at)); cnext = f.vector(a.ckpt + at * C4); };
    if (left > 0) load_ckpt();
    Vec<CPL> x[EB];
    uint32_t e[EB];
    f.prologue(x, e);
    const int steps = __reduce_max_sync(FULL, f.nblk);
    for (int t = 0; t < steps; t++) {
        f.step(t);
        // the state at the first key after the block, that key's decay
        Vec<CPL> R = f.vector(ag + C4);
        float anext = alast;
        if (left > 0) {
            #pragma unroll
            for (int c = 0; c < CPL; c++) R.x[c] = fmaf(wnext.x, R.x[c], cnext.x[c]);
            anext = wnext.y;
        }
        float dr[ROWS ? 1 : EB];                      // dots with the suffix state ...
        f2    r[ROWS ? EB : 1][CPL / 2];              // ... or that state, for rows and dots
        #pragma unroll
        for (int i = EB - 1; i >= 0; i--) {
            const float2 s = f.scalars(i);
            if (ROWS) {
                #pragma unroll
                for (int c = 0; c < CPL / 2; c++) r[ROWS ? i : 0][c] = mul2(pack2(s.y, s.y), pack2(R.x[2 * c], R.x[2 * c + 1]));
            } else {
                dr[ROWS ? 0 : i] = s.y * f.dot(x[i], R);
            }
            if (!is_query(e[i])) {
                #pragma unroll
                for (int c = 0; c < CPL; c++) R.x[c] = fmaf(anext, R.x[c], x[i].x[c]);
                anext = s.x;
            }
        }
        uint32_t n[EB];
        f.read_index(f.next, n);
        if (left > 0) {                               // (the last one read stays until its block comes)
            bool keys = false;
            #pragma unroll
            for (int i = 0; i < EB; i++) keys |= !is_query(n[i]);
            if (keys) { left--; at++; }
            if (left > 0) load_ckpt();
        }
        #pragma unroll
        for (int h = 0; h < EB; h += EV_GROUP) {
            #pragma unroll
            for (int i = h; i < h + EV_GROUP; i++) {
                const float s = f.scalars(i).x;
                if (ROWS) {
                    float row[CPL];
                    Vec<CPL> z;                       // e1 R - e0 L
                    #pragma unroll
                    for (int c = 0; c < CPL / 2; c++) {
                        const f2 l = pack2(L.x[2 * c], L.x[2 * c + 1]), suf = r[ROWS ? i : 0][c];
                        unpack2(fma2(pack2(s, s), l, suf), row[2 * c], row[2 * c + 1]);
                        unpack2(fma2(pack2(-s, -s), l, suf), z.x[2 * c], z.x[2 * c + 1]);
                    }
                    f.park(i, f.dot(x[i], z));
                    #pragma unroll
                    for (int q = 0; q < F::Q; q++) red_if_query(f.on[q] && (!f.edge(t) || f.has(t, i)), e[i], out + (q ? f.second : 0u), f.row_bytes, row + 4 * q);
                } else {
                    f.park(i, fmaf(-s, f.dot(x[i], L), dr[ROWS ? 0 : i]));
                }
                if (!is_query(e[i])) {
                    #pragma unroll
                    for (int c = 0; c < CPL; c++) L.x[c] = fmaf(s, L.x[c], x[i].x[c]);
                }
            }
            // the next block's rows into the registers that are free now
            #pragma unroll
            for (int i = h; i < h + EV_GROUP; i++) x[i] = f.row(n[i]);
        }
        f.finish(t, [&](const float sum, const uint32_t row, const uint32_t) { atomicAdd(out_s + row, sum); });
        #pragma unroll
        for (int i = 0; i < EB; i++) e[i] = n[i];
    }
    cp_async_wait<0>();
}

template <int LPS, int CPL, bool ROWS>
static cudaError_t launch_lap(const WalkArgs& a, cudaStream_t stream) {
    const long long items = ((long long)a.nseg * a.sps * LPS + EV_THREADS - 1) / EV_THREADS;
    laplace_events<LPS, CPL, ROWS><<<(unsigned)items, EV_THREADS, Shape<LPS, CPL>::SMEM, stream>>>(a);
    return cudaGetLastError();
}

// the second pass of the Laplace walk with dots, after laplace_pass1 and laplace_fold: dots, or rows and dots
cudaError_t launch_laplace_events(const WalkArgs& a, bool rows, cudaStream_t stream) {
    if (a.C4 <= 32)  return rows ? launch_lap<8, 4, true>(a, stream) : launch_lap<8, 4, false>(a, stream);
    if (a.C4 <= 64)  return rows ? launch_lap<16, 4, true>(a, stream) : launch_lap<16, 4, false>(a, stream);
    if (a.C4 <= 128) return rows ? launch_lap<32, 4, true>(a, stream) : launch_lap<32, 4, false>(a, stream);
    return cudaErrorInvalidValue;
}

}  // namespace qlka
