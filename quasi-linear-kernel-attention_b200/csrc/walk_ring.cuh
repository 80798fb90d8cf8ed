// Asynchronous staging shared by the walk kernels.
//
// Emitting passes (Feeder): one warp walks one stream (a contiguous run of key blocks of a segment). Lane l owns the CPL
// consecutive channels from l * CPL on, with CPL = 1, 2 or 4 for up to 32, 64 or 128 channels, so that every loop below is uniform
// over the warp.
// First passes (KeyFeeder), which have nothing that diverges, have 4 or 8 channels per lane and 2 or 4 streams per warp.
//
// Every warp owns a ring of DEPTH slots in shared memory; a slot holds the KB rows of one key block, the block's per-key
// scalars (12 floats of which 9 are used) and its first QCAP query records. All of it is fetched with cp.async (global ->
// shared, no registers, L2 only) DEPTH - 1 blocks ahead of its use, one commit group per block: 16 bytes per lane, so that
// 32 / (8 CPL) rows travel with one instruction. cp.async.wait_group and a warp barrier make the copies readable by every lane;
// a warp barrier at the top of the next iteration lets the slot be refilled. Blocks with QCAP queries or more read the further
// records into the same place. The blocks' query ranges travel in registers. Shared memory is addressed with 32-bit
// shared-window addresses throughout.
#pragma once
#include "qlka_common.cuh"

namespace qlka {

constexpr int WALK_THREADS = 256;
constexpr int WALK_STREAMS = WALK_THREADS / 32;      // streams per CTA
constexpr int SX_STRIDE    = 12;     // floats per staged scalar slot: 8 decays / keys and the next four
constexpr int QCAP         = 16;     // query records staged per block

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp_async16(const uint32_t dst, const void* gmem_src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

__device__ __forceinline__ float4 lds128(const uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds32u(const uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts32f(const uint32_t addr, const float v) {
    asm volatile("st.shared.f32 [%0], %1;" :: "r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ uint4 lds128u(const uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts128u(const uint32_t addr, const uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" :: "r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// ------------------------------------------------------------------ a lane's channels
template <int CPL>
struct Vec {
    float x[CPL];
    __device__ __forceinline__ void zero() {
        #pragma unroll
        for (int c = 0; c < CPL; c++) x[c] = 0.0f;
    }
};

// d = a * x + y. Two packed floats per instruction where a lane has 4 channels; with fewer, pairing the broadcast factor costs
// the instruction it saves.
template <int CPL>
__device__ __forceinline__ void axpy(Vec<CPL>& d, const float a, const Vec<CPL>& x, const Vec<CPL>& y) {
    if constexpr (CPL == 4) {
        #pragma unroll
        for (int c = 0; c < CPL; c += 2)
            asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
                "mov.b64 ra, {%2, %2};\n\tmov.b64 rb, {%3, %4};\n\tmov.b64 rc, {%5, %6};\n\t"
                "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
                : "=f"(d.x[c]), "=f"(d.x[c + 1]) : "f"(a), "f"(x.x[c]), "f"(x.x[c + 1]), "f"(y.x[c]), "f"(y.x[c + 1]));
    } else {
        #pragma unroll
        for (int c = 0; c < CPL; c++) d.x[c] = fmaf(a, x.x[c], y.x[c]);
    }
}
// d = a * x
template <int CPL>
__device__ __forceinline__ void scale(Vec<CPL>& d, const float a, const Vec<CPL>& x) {
    if constexpr (CPL == 4) {
        #pragma unroll
        for (int c = 0; c < CPL; c += 2)
            asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
                "mov.b64 ra, {%2, %2};\n\tmov.b64 rb, {%3, %4};\n\t"
                "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
                : "=f"(d.x[c]), "=f"(d.x[c + 1]) : "f"(a), "f"(x.x[c]), "f"(x.x[c + 1]));
    } else {
        #pragma unroll
        for (int c = 0; c < CPL; c++) d.x[c] = a * x.x[c];
    }
}
// the same where a lane has 4 or 8 channels
template <int CPL>
__device__ __forceinline__ void axpy8(Vec<CPL>& d, const float a, const Vec<CPL>& x, const Vec<CPL>& y) {
    #pragma unroll
    for (int c = 0; c < CPL; c += 2)
        asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
            "mov.b64 ra, {%2, %2};\n\tmov.b64 rb, {%3, %4};\n\tmov.b64 rc, {%5, %6};\n\t"
            "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
            : "=f"(d.x[c]), "=f"(d.x[c + 1]) : "f"(a), "f"(x.x[c]), "f"(x.x[c + 1]), "f"(y.x[c]), "f"(y.x[c + 1]));
}
// d += x
template <int CPL>
__device__ __forceinline__ void vadd(Vec<CPL>& d, const Vec<CPL>& x) {
    if constexpr (CPL >= 2) {
        #pragma unroll
        for (int c = 0; c < CPL; c += 2)
            asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
                "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
                "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
                : "=f"(d.x[c]), "=f"(d.x[c + 1]) : "f"(d.x[c]), "f"(d.x[c + 1]), "f"(x.x[c]), "f"(x.x[c + 1]));
    } else {
        d.x[0] += x.x[0];
    }
}

template <int CPL>
__device__ __forceinline__ Vec<CPL> vload_shared(const uint32_t addr) {
    Vec<CPL> v;
    if constexpr (CPL == 4)      { const float4 t = lds128(addr); v.x[0] = t.x; v.x[1] = t.y; v.x[2] = t.z; v.x[3] = t.w; }
    else if constexpr (CPL == 2) asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x[0]), "=f"(v.x[1]) : "r"(addr));
    else                         asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v.x[0]) : "r"(addr));
    return v;
}
template <int CPL>
__device__ __forceinline__ Vec<CPL> vload(const float* p) {
    Vec<CPL> v;
    if constexpr (CPL == 4)      { const float4 t = ldg4(p); v.x[0] = t.x; v.x[1] = t.y; v.x[2] = t.z; v.x[3] = t.w; }
    else if constexpr (CPL == 2) { const float2 t = __ldg(reinterpret_cast<const float2*>(p)); v.x[0] = t.x; v.x[1] = t.y; }
    else                         v.x[0] = __ldg(p);
    return v;
}
// loads of data that is used once, long after it was written
template <int CPL>
__device__ __forceinline__ Vec<CPL> vload_once(const float* p) {
    Vec<CPL> v;
    if constexpr (CPL == 4)      { const float4 t = __ldcs(reinterpret_cast<const float4*>(p)); v.x[0] = t.x; v.x[1] = t.y; v.x[2] = t.z; v.x[3] = t.w; }
    else if constexpr (CPL == 2) { const float2 t = __ldcs(reinterpret_cast<const float2*>(p)); v.x[0] = t.x; v.x[1] = t.y; }
    else                         v.x[0] = __ldcs(p);
    return v;
}
// vector reduction into global memory (no return value): a row of the output per warp
template <int CPL>
__device__ __forceinline__ void vred(float* p, const Vec<CPL>& v) {
    if constexpr (CPL == 4)      red_add4(p, v.x[0], v.x[1], v.x[2], v.x[3]);
    else if constexpr (CPL == 2) asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" :: "l"(p), "f"(v.x[0]), "f"(v.x[1]) : "memory");
    else                         asm volatile("red.global.add.f32 [%0], %1;" :: "l"(p), "f"(v.x[0]) : "memory");
}

// ------------------------------------------------------------------ shared memory of a warp
template <int CPL> __host__ __device__ constexpr int row_pitch()  { return 128 * CPL; }
template <int CPL> __host__ __device__ constexpr int slot_bytes() { return KB * row_pitch<CPL>(); }
// row slots | scalar slots | record slots, and one more: a read may look one ahead
template <int CPL, int DEPTH> __host__ __device__ constexpr int sx_offset()  { return DEPTH * slot_bytes<CPL>(); }
template <int CPL, int DEPTH> __host__ __device__ constexpr int rec_offset() { return sx_offset<CPL, DEPTH>() + DEPTH * SX_STRIDE * 4; }
template <int CPL, int DEPTH> __host__ __device__ constexpr int warp_bytes() { return rec_offset<CPL, DEPTH>() + (DEPTH * QCAP + 1) * 16; }

// the warp's index in its CTA, in a form the compiler knows to be uniform
__device__ __forceinline__ int warp_index() { return __shfl_sync(FULL, (int)(threadIdx.x >> 5), 0); }

// What a stream of an emitting pass needs to stage its blocks, in order. The pointers run along.
template <int CPL, bool WITH_X, int DEPTH>
struct Feeder {
    static constexpr int AHEAD = DEPTH - 1;
    static constexpr int LR = 8 * CPL, RPC = 32 / LR, NCP = KB / RPC;     // lanes per row, rows per copy instruction, copies per lane and block
    uint32_t        area;      // shared address of the warp's area
    uint32_t        copy_dst;  // + my first row and my 16 bytes of it
    uint32_t        row_bytes; // C4 * 4
    bool            copy_on;   // my 16 bytes lie inside the row
    int             lane, N, M;
    const char*     rows;      // + p * N * row_bytes + my 16 bytes
    const uint32_t* xperm;     // of the stream's first block, + my first row
    const uint32_t* mstart;    // of the stream's first block
    const char*     aux;       // lanes 0 .. 15: the segment's records; lanes 16 .. 18: the first block's scalars, + my 16 bytes
    uint32_t        aux_dst;   // shared address they go to in slot 0
    const uint4*    yrec;      // the segment's records
    // prefetched one block before its issue
    uint32_t idx[NCP], ms;
    // first query of the block in use and of the blocks in flight
    uint32_t m_lo, mq_lo[AHEAD];

    __device__ __forceinline__ void init(const uint32_t area_, const int lane_, const int N_, const int C4) {
        area = area_; lane = lane_; N = N_;
        row_bytes = (uint32_t)C4 * 4u;
        copy_on   = (uint32_t)(lane % LR) * 16u < row_bytes;
        copy_dst  = area + (lane / LR) * NCP * row_pitch<CPL>() + (lane % LR) * 16;
        aux_dst   = area + (lane < QCAP ? rec_offset<CPL, DEPTH>() + lane * 16 : sx_offset<CPL, DEPTH>() + (lane - QCAP) * 16);
    }
    // a stream of segment sg (head p) that starts at block b
    __device__ __forceinline__ void start(const WalkArgs& a, const int sg, const int p, const int b) {
        xperm  = a.xperm + (long long)sg * npad(a.N) + b * KB + (lane / LR) * NCP;
        rows   = reinterpret_cast<const char*>(a.rows + (long long)p * a.N * a.C4) + (lane % LR) * 16;
        mstart = a.mstart + (long long)sg * mstride(a.N) + b;
        yrec   = a.yrec + (long long)sg * (a.M + 1);
        M      = a.M;
        aux    = lane < QCAP ? reinterpret_cast<const char*>(yrec)
                             : reinterpret_cast<const char*>(WITH_X ? a.xval + (long long)sg * xstride(a.N) + b * KB + 4 * (lane - QCAP) : nullptr);
    }

    // t: the block's place in the stream
    __device__ __forceinline__ void prefetch_index(const uint32_t t) {
        const uint32_t* at = xperm + t * KB;
        if constexpr (NCP == 2) { const uint2 u = __ldg(reinterpret_cast<const uint2*>(at)); idx[0] = u.x; idx[1] = u.y; }
        else {
            #pragma unroll
            for (int i = 0; i < NCP; i += 4) {
                const uint4 u = __ldg(reinterpret_cast<const uint4*>(at + i));
                idx[i] = u.x; idx[i + 1] = u.y; idx[i + 2] = u.z; idx[i + 3] = u.w;
            }
        }
        ms = __ldg(mstart + t);
    }

    // start the copies of the block whose indices were prefetched last into `slot`; one commit group
    __device__ __forceinline__ void issue(const int slot, const int ahead, const uint32_t t) {
        mq_lo[ahead] = ms;
        const uint32_t dst = copy_dst + slot * slot_bytes<CPL>();
        if (copy_on) {                                 // (positions past the last key point at row 0; read_rows zeroes them)
            #pragma unroll
            for (int i = 0; i < NCP; i++) cp_async16(dst + i * row_pitch<CPL>(), rows + (unsigned long long)idx[i] * row_bytes);
        }
        // lanes 0..15 the first QCAP records from the block's first one on (past the segment's end: its sentinel, whose rank no block
        // has), lanes 16..18 the scalars (padded by KB floats)
        if (lane < (WITH_X ? QCAP + 3 : QCAP))
            cp_async16(aux_dst + slot * (lane < QCAP ? QCAP * 16 : SX_STRIDE * 4), aux + (unsigned long long)(lane < QCAP ? min(ms + lane, (uint32_t)M) * 16ull : t * (KB * 4ull)));
        cp_async_commit();
    }

    // Blocks are visited in steps t = 0 .. nblk-1; slot of step t = t mod DEPTH.
    __device__ __forceinline__ void prologue(const int nblk) {
        #pragma unroll
        for (int i = 0; i < AHEAD; i++) {
            if (i < nblk) { prefetch_index(i); issue(i, i, i); }
            else cp_async_commit();
        }
        if (AHEAD < nblk) prefetch_index(AHEAD);
    }
    // first thing of every step: the oldest block in flight becomes the block in use
    __device__ __forceinline__ void advance_range() {
        m_lo = mq_lo[0];
        #pragma unroll
        for (int i = 0; i + 1 < AHEAD; i++) mq_lo[i] = mq_lo[i + 1];
    }
    __device__ __forceinline__ void step_issue(const int t, const int cur, const int nblk) {
        if (t + AHEAD < nblk) issue(cur == 0 ? DEPTH - 1 : cur - 1, AHEAD - 1, t + AHEAD);
        else cp_async_commit();
        if (t + AHEAD + 1 < nblk) prefetch_index(t + AHEAD + 1);
    }
    __device__ __forceinline__ static int next_slot(const int cur) { return cur == DEPTH - 1 ? 0 : cur + 1; }

    // this lane's slice of the block's rows from `slot`; rows at positions >= N read as zero
    __device__ __forceinline__ void read_rows(const int slot, const int j0, Vec<CPL> (&v)[KB]) const {
        const uint32_t src = area + slot * slot_bytes<CPL>() + lane * (4 * CPL);
        #pragma unroll
        for (int i = 0; i < KB; i++) v[i] = vload_shared<CPL>(src + i * row_pitch<CPL>());
        if (j0 + KB > N) {
            #pragma unroll
            for (int i = 0; i < KB; i++) if (j0 + i >= N) v[i].zero();
        }
    }
    // the block's nine scalars, from `slot`
    __device__ __forceinline__ void read_scalars(const int slot, float (&av)[KB + 1]) const {
        const uint32_t sx = area + sx_offset<CPL, DEPTH>() + slot * SX_STRIDE * 4;
        const float4 a0 = lds128(sx), a1 = lds128(sx + 16), a2 = lds128(sx + 32);
        av[0] = a0.x; av[1] = a0.y; av[2] = a0.z; av[3] = a0.w;
        av[4] = a1.x; av[5] = a1.y; av[6] = a1.z; av[7] = a1.w;
        av[8] = a2.x;
    }

    __device__ __forceinline__ uint32_t records(const int slot) const { return area + rec_offset<CPL, DEPTH>() + slot * QCAP * 16; }
};

// The queries of the block of key j0, in rank order: emit(i, rec) for the queries that precede key i. The staged records are followed by one
// of a later block (or the segment's sentinel), so a record's rank alone says where the block ends; when the last staged record is
// still the block's, it goes QCAP - 1 queries at a time, with a terminator.
template <class F, class Emit>
__device__ __forceinline__ void for_queries(const F& f, const int slot, const int j0, Emit emit) {
    constexpr uint32_t BATCH = QCAP - 1;
    const uint32_t recs = f.records(slot);
    uint32_t at = f.m_lo;
    while (true) {
        const bool more = lds32u(recs + BATCH * 16 + 12) - (uint32_t)j0 < (uint32_t)KB;
        if (more) {
            __syncwarp();
            if (f.lane == 0) sts32f(recs + BATCH * 16 + 12, __uint_as_float(0xffffffffu));
            __syncwarp();
        }
        uint32_t qa  = recs;
        uint4    rec = lds128u(qa);
        #pragma unroll
        for (int i = 0; i < KB; i++) {
            while (rec.w - (uint32_t)j0 == (uint32_t)i) {
                qa += 16;
                emit(i, rec);
                rec = lds128u(qa);
            }
        }
        if (!more) break;
        at += BATCH;
        __syncwarp();
        if (f.lane < QCAP) sts128u(recs + f.lane * 16, __ldg(f.yrec + min(at + f.lane, (uint32_t)f.M)));
        __syncwarp();
    }
}

// Row emission by quads: LPS lanes per stream (8, 16 or 32 for up to 32, 64 or 128 channels), 4 channels per lane. Every lane
// copies its own 16 bytes of each row into a private ring of two slots, and reads only those; the block's scalars are shared by
// the lanes of the stream.
constexpr int ROW_THREADS = 64;      // one item each: with 256, persistent, a stream that meets more queries than others kept its CTA's share waiting
constexpr int SUM_SLOT_BYTES = KB * ROW_THREADS * 16;
template <int LPS> __host__ __device__ constexpr int sum_smem_bytes() { return 2 * SUM_SLOT_BYTES + (ROW_THREADS / LPS) * 2 * SX_STRIDE * 4; }

template <int LPS>
struct QuadFeeder {
    uint32_t        ring, sx;  // shared addresses: this lane's 16 bytes of row 0 of slot 0, the stream's scalar slots
    uint32_t        row_bytes;
    int             ln, N;
    bool            on;        // this lane's 16 bytes lie inside the row
    const char*     rows;      // + p * N * row_bytes + my 16 bytes
    const float*    xval;      // of the next block to start, + my 16 bytes (lanes 0 .. 2)
    const uint32_t* xperm;     // of the next block to prefetch
    uint4           p0, p1;    // prefetched one block before its issue

    __device__ __forceinline__ void init(const uint32_t smem, const int N_, const int C4) {
        ring = smem + threadIdx.x * 16;
        sx   = smem + 2 * SUM_SLOT_BYTES + (threadIdx.x / LPS) * 2 * SX_STRIDE * 4;
        ln   = threadIdx.x % LPS; N = N_;
        on   = ln * 4 < C4;
        row_bytes = (uint32_t)C4 * 4u;
    }
    __device__ __forceinline__ void start(const WalkArgs& a, const int sg, const int p, const int b) {
        xperm = a.xperm + (long long)sg * npad(a.N) + b * KB;
        xval = a.xval + (long long)sg * xstride(a.N) + b * KB + 4 * ln;
        rows = reinterpret_cast<const char*>(a.rows + (long long)p * a.N * a.C4) + ln * 16;
    }
    __device__ __forceinline__ void prefetch_index() {
        p0 = __ldg(reinterpret_cast<const uint4*>(xperm));
        p1 = __ldg(reinterpret_cast<const uint4*>(xperm + 4));
        xperm += KB;
    }
    __device__ __forceinline__ void issue(const int slot) {
        const uint32_t pr[KB] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
        if (on) {
            #pragma unroll
            for (int i = 0; i < KB; i++) cp_async16(ring + slot * SUM_SLOT_BYTES + i * ROW_THREADS * 16, rows + (unsigned long long)pr[i] * row_bytes);
        }
        if (ln < 3) cp_async16(sx + slot * SX_STRIDE * 4 + 16 * ln, xval);
        xval += KB;
        cp_async_commit();
    }
    __device__ __forceinline__ void read_rows(const int slot, const int j0, Vec<4> (&v)[KB]) const {
        #pragma unroll
        for (int i = 0; i < KB; i++) v[i] = vload_shared<4>(ring + slot * SUM_SLOT_BYTES + i * ROW_THREADS * 16);
        if (j0 + KB > N) {
            #pragma unroll
            for (int i = 0; i < KB; i++) if (j0 + i >= N) v[i].zero();
        }
    }
    __device__ __forceinline__ void read_scalars(const int slot, float (&av)[KB + 1]) const {
        const uint32_t s = sx + slot * SX_STRIDE * 4;
        const float4 a0 = lds128(s), a1 = lds128(s + 16), a2 = lds128(s + 32);
        av[0] = a0.x; av[1] = a0.y; av[2] = a0.z; av[3] = a0.w;
        av[4] = a1.x; av[5] = a1.y; av[6] = a1.z; av[7] = a1.w;
        av[8] = a2.x;
    }
};

// The same mapping with the queries' records, for row emission where queries are few beside the keys or the rows are wide: what a
// block costs besides its queries is then what counts, and 4 channels per lane halve (LPS = 16) or quarter (LPS = 8) it. The
// streams of a warp go through their queries side by side, each in its own loop.
template <int LPS> __host__ __device__ constexpr int row_smem_bytes() { return sum_smem_bytes<LPS>() + ROW_THREADS * 2 * 16; }

template <int LPS>
struct RowFeeder : QuadFeeder<LPS> {
    using Base = QuadFeeder<LPS>;
    uint32_t        recs;      // shared address of the stream's record slots [2][LPS]
    const uint4*    yrec;      // the segment's records
    const uint32_t* mstart;    // of the next block to prefetch
    uint32_t        ms, m_lo, m_next, M;     // first query: of the block prefetched, in use, in flight

    __device__ __forceinline__ void init(const uint32_t smem, const int N_, const int M_, const int C4) {
        Base::init(smem, N_, C4);
        recs = smem + sum_smem_bytes<LPS>() + (threadIdx.x / LPS) * 2 * LPS * 16;
        M = (uint32_t)M_;
    }
    __device__ __forceinline__ void start(const WalkArgs& a, const int sg, const int p, const int b) {
        Base::start(a, sg, p, b);
        yrec   = a.yrec + (long long)sg * (a.M + 1);
        mstart = a.mstart + (long long)sg * mstride(a.N) + b;
    }
    __device__ __forceinline__ void prefetch() { Base::prefetch_index(); ms = __ldg(mstart++); }
    // (a block with fewer than LPS queries finds all of them staged, followed by a record of a later block or the sentinel)
    __device__ __forceinline__ void issue_with_records(const int slot) {
        m_next = ms;
        cp_async16(recs + (slot * LPS + this->ln) * 16, yrec + min(ms + (uint32_t)this->ln, M));
        Base::issue(slot);
    }
    __device__ __forceinline__ void prologue(const int nblk) {
        if (nblk > 0) { prefetch(); issue_with_records(0); }
        if (nblk > 1) prefetch();
    }
    __device__ __forceinline__ void step(const int t, const int cur, const int nblk) {
        m_lo = m_next;
        if (t + 1 < nblk) issue_with_records(cur ^ 1);
        else cp_async_commit();
        if (t + 2 < nblk) prefetch();
        cp_async_wait<1>();
    }
    // emit(i, rec) for the queries of the block of key j0 that precede key i, in rank order
    template <class Emit>
    __device__ __forceinline__ void for_queries(const int slot, const int j0, Emit emit) const {
        uint32_t qa = recs + slot * LPS * 16;
        if (lds32u(qa + (LPS - 1) * 16 + 12) - (uint32_t)j0 >= (uint32_t)KB) {
            uint4 rec = lds128u(qa);
            #pragma unroll
            for (int i = 0; i < KB; i++) {
                while (rec.w == (uint32_t)(j0 + i)) {
                    qa += 16;
                    const uint4 next = lds128u(qa);
                    emit(i, rec);
                    rec = next;
                }
            }
        } else {                                       // more queries than the slot holds: read them from memory
            const uint4* yp  = yrec + m_lo;
            uint4        rec = __ldg(yp);
            #pragma unroll
            for (int i = 0; i < KB; i++) {
                while (rec.w == (uint32_t)(j0 + i)) {
                    const uint4 next = __ldg(++yp);    // at most the segment's sentinel
                    emit(i, rec);
                    rec = next;
                }
            }
        }
    }
};

// Which mapping emits rows: at 33 .. 64 channels a warp per stream is the faster one once queries outnumber keys (48 heads x 1024
// keys x 8192 queries 2.52 -> 1.70 ms; at equal numbers Laplace 5.47 -> 5.53 ms at 16384, abs 1.33 -> 1.37 ms at 4096; at 15847 keys
// x 2522 queries 3.88 -> 4.13 ms), at up to 32 from a quarter as many queries as keys on (4096 x 4096: 1.32 -> 1.05 ms, x 512
// queries: 0.68 -> 0.79 ms); wider rows leave one stream per warp either way, with shared-memory copies of its own in favour
// of this one (abs at 8192: 1.49 against 1.55 ms).
inline bool rows_by_quads(const WalkArgs& a) { return a.C4 > 64 || (a.C4 > 32 ? a.M <= a.N : 4LL * a.M <= a.N); }

// the key blocks [b0, b1) that stream s of the SPS streams of a segment owns (NBK blocks per segment)
__device__ __forceinline__ void stream_blocks(const int s, const int SPS, const int NBK, int& b0, int& b1) {
    b0 = (int)((long long)s * NBK / SPS);
    b1 = (int)((long long)(s + 1) * NBK / SPS);
}

// The kernels between the passes: a lane per segment and channel. From 32 streams per segment on, 2, 4 or 8 warps share a column:
// each folds its share of the streams, the totals go through shared memory, then each writes the states entering its
// streams. (One thread per column whatever the number: a serial chain through memory, 0.38 instead of 0.32 ms for a whole
// Laplace sum of 16 segments of 65536 keys; sharing fewer streams only reads them twice.)
constexpr int FOLD_WARPS = 8, FOLD_CHUNK = 16;     // warps per CTA; loads of FOLD_CHUNK streams are in flight together
inline int      fold_share_warps(const WalkArgs& a) { return a.sps < 32 ? 1 : a.sps < 64 ? 2 : a.sps < 128 ? 4 : FOLD_WARPS; }
inline unsigned fold_grid(const WalkArgs& a) {
    const int columns = 32 * FOLD_WARPS / fold_share_warps(a);                     // per CTA
    return (unsigned)(((long long)a.nseg * a.C4 + columns - 1) / columns);
}
// where a thread of a fold stands: segment and channel (the last column's for lanes past the end), its share [first, last) of the
// SPS streams, and which share of how many that is
struct FoldOf {
    bool on; long long sg; int c, first, last, share, group;      // group: first warp of the CTA that works on the column
    __device__ __forceinline__ FoldOf(const int nseg, const int SPS, const int C4, const int warps) {
        const int w = threadIdx.x >> 5;
        share = w % warps; group = w - share;
        const long long col = ((long long)blockIdx.x * (FOLD_WARPS / warps) + w / warps) * 32 + (threadIdx.x & 31), all = (long long)nseg * C4;
        on = col < all;
        const long long i = on ? col : all - 1;
        sg = i / C4; c = (int)(i - sg * C4);
        const int per = (SPS + warps - 1) / warps;
        first = min(share * per, SPS); last = min(first + per, SPS);
    }
};

// the stream of a warp: segment, block range
struct StreamOf {
    long long g; bool on; int sg, p, b0, b1, nblk;
    // stream `i` of the `streams` of work item `item`
    __device__ __forceinline__ StreamOf(const WalkArgs& a, const int item, const int i, const int NBK, const int streams = WALK_STREAMS) {
        g  = (long long)item * streams + i;
        on = g < (long long)a.nseg * a.sps;
        const long long gg = on ? g : 0;
        sg = (int)(gg / a.sps);
        const int s = (int)(gg - (long long)sg * a.sps);
        p  = sg / a.D;
        stream_blocks(s, a.sps, NBK, b0, b1);
        nblk = on ? b1 - b0 : 0;
    }
};

// where the events of key blocks before b end, among all events of all segments
__device__ __forceinline__ long long events_end(const WalkArgs& a, const int sg, const int b) {
    return (long long)sg * estride(a.N, a.M) + min(b * KB, a.N) + (int)__ldg(a.mstart + (long long)sg * mstride(a.N) + b);
}

// The first passes' staging: LPS lanes per stream with CPL = 4 or 8 channels each (quads ln, and LPS + ln, of the row). Rows go straight to
// registers, those of the next block as soon as the block in use is done with (through shared memory, as above, the load/store pipe
// moves them twice: Laplace at 48 heads x 16384 keys 1.12 -> 0.79 ms, abs at
// 96 x 4096 0.43 -> 0.36; the gathers alone take 0.75 and 0.33). Indices and scalars are shared by the lanes of a stream and arrive in shared
// memory a block ahead. Small CTAs, one item each: they spread over the SMs however few streams there are.
constexpr int KEY_THREADS = 64, KEY_CTAS = 8, KEY_REC = KB * 8;

template <int LPS, int CPL, bool WITH_X, int DIR>
struct KeyFeeder {
    static constexpr int STREAMS = KEY_THREADS / LPS, SMEM = STREAMS * 3 * KEY_REC, Q = CPL / 4;
    uint32_t    rec, next, after;  // shared addresses: the indices and scalars of the block in use, the next one and the one after it
    int         ln, N, j0;         // j0: first key of the block in use
    bool        on[Q];             // quad q lies inside the row (idle ones read the first)
    uint32_t    row_bytes, second; // from the first quad to the second
    const char* rows;              // + p * N * row_bytes + my first quad
    const char* aux;               // lanes 0, 1: the indices of the next block to copy; lanes 2, 3: its scalars, + my 16 bytes
    int         nblk;

    __device__ __forceinline__ int channel(const int q) const { return on[q] ? (q * LPS + ln) * 4 : 0; }
    __device__ __forceinline__ void init(const uint32_t smem, const int N_, const int C4) {
        ln = threadIdx.x % LPS; N = N_;
        rec = smem + (threadIdx.x / LPS) * 3 * KEY_REC; next = rec + KEY_REC; after = next + KEY_REC;
        #pragma unroll
        for (int q = 0; q < Q; q++) on[q] = (q * LPS + ln) * 4 < C4;
        second = Q > 1 && on[Q - 1] ? LPS * 16 : 0;
        row_bytes = (uint32_t)C4 * 4u;
    }
    __device__ __forceinline__ void copy_records(const int t, const uint32_t dst) {
        if (t < nblk && ln < (WITH_X ? 4 : 2)) { cp_async16(dst + ln * 16, aux); aux += DIR * KB * 4; }
    }
    __device__ __forceinline__ void read_index(const uint32_t r, uint32_t (&n)[KB]) const {
        const uint4 a = lds128u(r), b = lds128u(r + 16);
        n[0] = a.x; n[1] = a.y; n[2] = a.z; n[3] = a.w; n[4] = b.x; n[5] = b.y; n[6] = b.z; n[7] = b.w;
    }
    __device__ __forceinline__ void scalars(float (&s)[KB]) const {
        const float4 a = lds128(rec + KB * 4), b = lds128(rec + KB * 4 + 16);
        s[0] = a.x; s[1] = a.y; s[2] = a.z; s[3] = a.w; s[4] = b.x; s[5] = b.y; s[6] = b.z; s[7] = b.w;
    }
    __device__ __forceinline__ Vec<CPL> row(const uint32_t i) const {
        const char* at = rows + (unsigned long long)(i & ~(KEY_FIRST | KEY_LATER)) * row_bytes;
        Vec<CPL> v;
        #pragma unroll
        for (int q = 0; q < Q; q++)
            asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v.x[4 * q]), "=f"(v.x[4 * q + 1]), "=f"(v.x[4 * q + 2]), "=f"(v.x[4 * q + 3]) : "l"(at + (q ? second : 0u)));
        return v;
    }
    // the stream's blocks in steps t = 0 .. nblk - 1; rows of the first under way, indices of the second as well
    __device__ __forceinline__ void start(const WalkArgs& a, const StreamOf& st, Vec<CPL> (&x)[KB]) {
        nblk = st.nblk;
        const int b = DIR > 0 ? st.b0 : max(st.b1 - 1, 0);
        j0   = (b - DIR) * KB;
        rows = reinterpret_cast<const char*>(a.rows + (long long)st.p * a.N * a.C4 + channel(0));
        aux  = ln < 2 ? reinterpret_cast<const char*>(a.xperm + (long long)st.sg * npad(a.N) + b * KB) + ln * 16
                      : reinterpret_cast<const char*>(a.xval + (long long)st.sg * xstride(a.N) + b * KB) + (ln - 2) * 16;
        copy_records(0, next);
        cp_async_commit();
        cp_async_wait<0>();
        __syncwarp();
        copy_records(1, after);
        cp_async_commit();
        if (nblk > 0) {
            uint32_t n[KB];
            read_index(next, n);
            #pragma unroll
            for (int i = 0; i < KB; i++) x[i] = row(n[i]);
        }
    }
    // the next block becomes the one in use; the indices after it are readable
    __device__ __forceinline__ void step(const int t, Vec<CPL> (&x)[KB]) {
        const uint32_t r = rec;
        rec = next; next = after; after = r;
        j0 += DIR * KB;
        cp_async_wait<0>();
        __syncwarp();                  // ... by every lane; and every lane has left block t - 1
        copy_records(t + 2, after);
        cp_async_commit();
        if (j0 + KB > N) {             // (positions past the last key point at row 0)
            #pragma unroll
            for (int i = 0; i < KB; i++) if (j0 + i >= N) x[i].zero();
        }
    }
};

}  // namespace qlka
