// Short sequences: the sums evaluated pair by pair, tile by tile, without sorting anything.
//
//   A_mn = sum_d f(q_dm - k_dn)          f(x) = exp(-|x|), |x| or max(0, 1 - |x|)
//   out[p, m, :] = sum_n A_mn v[p, n, :],   out_u[p, m] = sum_n A_mn
//
// The sorted walk costs a fixed amount per (feature, key): one gathered row, one row reduction in the L2 and a share of the
// sort, whatever the length. The pairwise evaluation costs N times a few instructions instead, all of them in registers, in one
// launch, with the layout change, the scaling, the key mask and the normalisation of the attention entry points folded in.
//
// dense_stage brings queries and keys into tiles of 64 rows, feature-major, as the main kernel wants them (scaled,
// exponentiated or negated), so that the main kernel copies tiles with coalesced 16-byte cp.async and does nothing else to
// them. dense_forward: one CTA owns 64 queries of one head and runs over its tiles of 64 keys. Per tile the 64 x 64 block of A
// is accumulated in registers over the features (4 x 8 pairs per thread, operands from shared memory in chunks of features,
// chunks in flight ahead of their use), goes to shared memory, and is multiplied with the tile's value rows (4 rows x C / 8
// channels per thread). When heads x query tiles do not fill the GPU, a cluster of CTAs shares one query tile: each takes a
// share of the keys and the partial results meet through distributed shared memory.
//
// exp(-|q - k|) = min(e^q e^-k, e^-q e^k) = min(e^q, e^k) min(e^-q, e^-k): the exponentials are taken once per value when a
// tile is staged; a pair costs three or four plain instructions instead of a special-function one (16 per SM and clock).
// The first form leans on the FMA pipe, the second on the ALU pipe (minimum: half rate); half of the pairs take each.
// That needs |q|, |k| <= LAP_RANGE (e^80 squared would overflow, and no product may be 0 * inf); tiles with larger values
// are staged as they are and their pairs take the plain form.
// Bound by instruction issue and the FMA / ALU pipes (Laplace, 96 heads x 777 keys: 73 % of the issue slots, 52 % of the ALU pipe);
// measured at B=4, H=12, D=C=64 as pairs x features per second: 5.2e12 (Laplace), 8.1e12 (riesz), 6.7e12 (bump) at 2048 keys.
// Times of attention calls, pairwise / sorted: 96 heads x 256 keys 114 / 335 us (Laplace), 77 / 363 (riesz), 88 / 518 (bump); 48 x 1024
// 710 / 443, 462 / 475, 552 / 892. On the way: 4 x 4 pairs per thread instead of 4 x 8 was bound by shared-memory reads (Laplace 4.1e12);
// tiles transposed and exponentiated by the main kernel itself cost a quarter of its time (4.5e12); only the product form
// or only the minimum form of the pair, two or four features unrolled: within 5 %.
#include "qlka_common.cuh"
#include "dense_tiles.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace qlka {

constexpr int TM = 64, TN = 64, DT_THREADS = 128;
constexpr int AT_LD = TM + 4;                 // row pitch of the transposed A tile: 16-byte stores of a warp hit all banks
static_assert(DT_THREADS == 2 * TN, "two threads clear a masked row");
constexpr int KSTAGES = 3;                    // chunks of the key tile in shared memory: one in use, two on their way

namespace {

__device__ __forceinline__ void cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

// two floats in one 64-bit register pair: one instruction issues two additions or multiply-adds
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack(const float a, const float b) { f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpack(const f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 add(const f2 a, const f2 b) { f2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f2 fma(const f2 a, const f2 b, const f2 c) { f2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ float rcp(const float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }

}  // namespace

// arrays per staged key: Laplace e^-k and e^k, the others -k; features per chunk of the main kernel
template <int KIND> __host__ __device__ constexpr int kind_arrays() { return KIND == DENSE_LAPLACE ? 2 : 1; }
template <int KIND> __host__ __device__ constexpr int kind_chunk()  { return KIND == DENSE_LAPLACE ? 16 : 32; }

// staged area, in floats: query tiles [P][mtiles][D][64] | key tiles [P][ntiles][arrays][D][64] | norms of the query rows and
// of the key rows (RIESZ) | one word per tile: a value beyond LAP_RANGE is in it (Laplace)
struct StagedView {
    long long q, k, qn, kn, qflag, kflag, floats;
    __host__ __device__ StagedView(int kind, int P, int D, int N, int M) {
        const long long mt = (M + TM - 1) / TM, nt = (N + TN - 1) / TN;
        const int na = kind == DENSE_LAPLACE ? 2 : 1;
        q = 0;
        k = q + P * mt * D * TM;
        qn = k + P * nt * na * D * TN;
        kn = qn + (kind == DENSE_RIESZ ? P * mt * TM : 0);
        qflag = kn + (kind == DENSE_RIESZ ? P * nt * TN : 0);
        kflag = qflag + (kind == DENSE_LAPLACE ? P * mt : 0);
        floats = kflag + (kind == DENSE_LAPLACE ? P * nt : 0);
    }
};

size_t dense_workspace_bytes(int kind, int P, int D, int N, int M) { return sizeof(float) * (size_t)StagedView(kind, P, D, N, M).floats; }

// One CTA stages one tile of 64 rows (queries first, then keys). Streaming: bound by memory.
template <int KIND>
__global__ void __launch_bounds__(256) dense_stage(const DenseArgs a)
{
    extern __shared__ float tr[];                        // rows layout: [64][D + 1]
    const int tid = threadIdx.x, D = a.D, lane64 = tid & 63, d4 = tid >> 6;
    const int mt = (a.M + TM - 1) / TM, nt = (a.N + TN - 1) / TN;
    const StagedView sv(KIND, a.P, D, a.N, a.M);
    const bool keys = blockIdx.x >= (unsigned)(a.P * mt);
    const int  tile = keys ? blockIdx.x - a.P * mt : blockIdx.x;
    const int  L = keys ? a.N : a.M, tiles = keys ? nt : mt;
    const int  p = tile / tiles, r0 = (tile % tiles) * 64, rows = min(64, L - r0);
    const float* src = (keys ? a.k : a.q) + (long long)p * L * D;
    float* dst = a.staged + (keys ? sv.k + (long long)tile * kind_arrays<KIND>() * D * TN : sv.q + (long long)tile * D * TM);

    if (a.rows_layout) {
        const float* s = src + (long long)r0 * D;
        if (a.vec) {
            for (int i = tid * 4; i < rows * D; i += 1024) {
                const float4 x = ldg4(s + i);
                float* t = tr + (i / D) * (D + 1) + i % D;
                t[0] = x.x; t[1] = x.y; t[2] = x.z; t[3] = x.w;
            }
        } else {
            for (int i = tid; i < rows * D; i += 256) tr[(i / D) * (D + 1) + i % D] = __ldg(s + i);
        }
        __syncthreads();
    }
    // (a masked key is staged as zeros: its values neither reach a result nor send its tile to the slow form)
    const float* keep = keys ? a.keep : a.row_keep;
    const bool   kept = lane64 < rows && (!keep || __ldg(keep + (long long)(p / a.H) * L + r0 + lane64) != 0.0f);
    auto value = [&](const int d) -> float {
        if (!kept) return 0.0f;
        return (a.rows_layout ? tr[lane64 * (D + 1) + d] : __ldg(src + (long long)d * L + r0 + lane64)) * a.scale;
    };
    if (KIND == DENSE_LAPLACE) {
        int bad = 0;
        for (int d = d4; d < D; d += 4) bad |= !(fabsf(value(d)) <= LAP_RANGE);
        bad = __syncthreads_or(bad);
        for (int d = d4; d < D; d += 4) {
            const float x = value(d);
            if (!keys) dst[d * TM + lane64] = bad ? x : expf(x);
            else {
                dst[d * TN + lane64]       = bad ? x : expf(-x);
                dst[(D + d) * TN + lane64] = bad ? x : expf(x);
            }
        }
        if (tid == 0) reinterpret_cast<int*>(a.staged)[(keys ? sv.kflag : sv.qflag) + tile] = bad;
    } else {
        float norm = 0.0f;
        for (int d = d4; d < D; d += 4) {
            const float x = value(d);
            norm += fabsf(x);
            dst[d * 64 + lane64] = keys ? -x : x;
        }
        if (KIND == DENSE_RIESZ) {
            __shared__ float part[4][64];
            part[d4][lane64] = norm;
            __syncthreads();
            if (tid < 64)
                a.staged[(keys ? sv.kn : sv.qn) + (long long)tile * 64 + tid] = (part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]) + (keys ? 0.0f : a.eps);
        }
    }
}

// shared memory of the main kernel, in floats: q tile | k chunks | A tile | v tile | key weights | key norms | row sums | tile list
template <int KIND, int CT>
static size_t dense_smem_bytes(int D, int list) {
    return sizeof(float) * (list + (size_t)D * TM + KSTAGES * kind_arrays<KIND>() * kind_chunk<KIND>() * TN + TN * AT_LD + TN * CT * 8 + 2 * TN + TM);
}

// CT: channels per thread (C <= 8 CT). Thread (mg, ng) of 16 x 8 owns the pairs of queries 4 mg .. 4 mg + 3 with the keys
// 4 ng + 0..3 and 32 + 4 ng + 0..3, and of the output the same queries and the channels 32 h + 4 ng + 0..3.
template <int KIND, int CT>
__global__ void __launch_bounds__(DT_THREADS, CT > 8 ? 2 : 3) dense_forward(const DenseArgs a)
{
    constexpr int NA = kind_arrays<KIND>(), CP = CT * 8, DK = kind_chunk<KIND>(), CHUNK = NA * DK * TN;
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                                      // [D][TM]
    float* ks = qs + (size_t)a.D * TM;                   // [KSTAGES][NA][DK][TN]
    float* at = ks + KSTAGES * CHUNK;                    // [TN][AT_LD]
    float* vs = at + TN * AT_LD;                         // [TN][CP]
    float* kw = vs + TN * CP;                            // [TN] weight of a key: keep mask, 0 beyond the last key
    float* kns = kw + TN;                                // [TN] |k|_1 (RIESZ)
    float* rsum = kns + TN;                              // [TM]
    int*   list = reinterpret_cast<int*>(rsum + TM);     // [ntiles + 1] with a keep mask: its active tiles and their number

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int mg = warp * 4 + (lane & 3), ng = lane >> 2;
    const int split = a.split;
    const int rank  = blockIdx.x % split;
    const int qt    = blockIdx.x / split;
    const int D = a.D, N = a.N, M = a.M, C = a.C;
    const int mtiles = (M + TM - 1) / TM, ntiles = (N + TN - 1) / TN;
    const int p = qt / mtiles, m0 = (qt % mtiles) * TM;
    const StagedView sv(KIND, a.P, D, N, M);
    const float* kst = a.staged + sv.k + (long long)p * ntiles * NA * D * TN;
    const float* v = a.v + (long long)p * N * C;
    const float* keep = a.keep ? a.keep + (long long)(p / a.H) * N : nullptr;
    const int active = keep ? active_tiles(keep, N, list, list + ntiles) : ntiles;
    int tile0 = (int)((long long)rank * active / split), tile1 = (int)((long long)(rank + 1) * active / split);
    if (a.row_keep) {                                    // rows that all are masked
        const bool on = tid < TM && m0 + tid < M && __ldg(a.row_keep + (long long)(p / a.H) * M + m0 + tid) != 0.0f;
        if (!__syncthreads_or(on)) tile1 = tile0;
    }
    auto tile_at = [&](const int t) -> int { return keep ? list[t] >> 1 : t; };
    const int nchunks = (D + DK - 1) / DK;

    // chunk c of this CTA's sequence (tile tile0 + c / nchunks, features DK (c mod nchunks) on) into its stage
    int it = tile0, ic = 0, istage = 0;                  // next chunk to start
    auto issue_chunk = [&]() {
        if (it < tile1) {
            const int d0 = ic * DK, n4 = min(DK, D - d0) * (TN / 4);         // float4s per array
            const float* src = kst + ((long long)tile_at(it) * NA * D + d0) * TN;
            float* dst = ks + istage * CHUNK;
            #pragma unroll
            for (int b = 0; b < NA; b++)
                #pragma unroll
                for (int i = 0; i < DK * TN / 4; i += DT_THREADS)
                    if (i + tid < n4) cp16(dst + b * DK * TN + (i + tid) * 4, src + (long long)b * D * TN + (i + tid) * 4);
            if (++ic == nchunks) { ic = 0; it++; }
            istage = istage + 1 == KSTAGES ? 0 : istage + 1;
        }
        cp_commit();
    };

    {   // the query tile rides with the first chunk
        const float* src = a.staged + sv.q + (long long)qt * D * TM;
        for (int i = tid; i < D * (TM / 4); i += DT_THREADS) cp16(qs + i * 4, src + i * 4);
    }
    #pragma unroll
    for (int i = 0; i < KSTAGES - 1; i++) issue_chunk();
    const bool qbad = KIND == DENSE_LAPLACE && __ldg(reinterpret_cast<const int*>(a.staged) + sv.qflag + qt) != 0;
    float qv[4] = {0.f, 0.f, 0.f, 0.f};                  // RIESZ: |q|_1 + eps of my queries
    if (KIND == DENSE_RIESZ) {
        const float4 s = ldg4(a.staged + sv.qn + (long long)qt * TM + mg * 4);
        qv[0] = s.x; qv[1] = s.y; qv[2] = s.z; qv[3] = s.w;
    }

    f2 o[4][CT / 2];
    float rs[4];
    #pragma unroll
    for (int i = 0; i < 4; i++) {
        rs[i] = 0.0f;
        #pragma unroll
        for (int c = 0; c < CT / 2; c++) o[i][c] = 0ull;
    }
    int stage = 0;
    for (int i = tile0; i < tile1; i++) {
        const int t = tile_at(i), n0 = t * TN;
        float acc[4][8];
        #pragma unroll
        for (int i = 0; i < 4; i++)
            #pragma unroll
            for (int j = 0; j < 8; j++) acc[i][j] = 0.0f;
        const bool kbad = KIND == DENSE_LAPLACE && __ldg(reinterpret_cast<const int*>(a.staged) + sv.kflag + (long long)p * ntiles + t) != 0;
        for (int ch = 0; ch < nchunks; ch++) {
            const int d0 = ch * DK, dc = min(DK, D - d0);
            const float* kc = ks + stage * CHUNK;
            if (ch == 0 && tid < TN) {
                kw[tid] = n0 + tid < N ? (keep ? __ldg(keep + n0 + tid) : 1.0f) : 0.0f;
                if (KIND == DENSE_RIESZ) kns[tid] = __ldg(a.staged + sv.kn + ((long long)p * ntiles + t) * TN + tid);
            }
            cp_wait<KSTAGES - 2>();
            __syncthreads();
            if (ch == 0) {                               // (everybody has left the previous tile's v and A)
                if ((C & 3) == 0) {
                    const int c4 = C >> 2;
                    for (int i = tid; i < TN * c4; i += DT_THREADS) {
                        const int r = i / c4, c = (i - r * c4) * 4;
                        if (n0 + r < N) cp16(vs + r * CP + c, v + (long long)(n0 + r) * C + c);
                        else *reinterpret_cast<float4*>(vs + r * CP + c) = make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                } else {
                    for (int i = tid; i < TN * C; i += DT_THREADS) {
                        const int r = i / C, c = i - r * C;
                        if (n0 + r < N) cp4(vs + r * CP + c, v + (long long)(n0 + r) * C + c);
                        else vs[r * CP + c] = 0.0f;
                    }
                }
            }
            issue_chunk();
            // ---- 4 x 8 pairs, feature by feature
            const float* qc = qs + d0 * TM + mg * 4;
            const float* kp = kc + ng * 4;
            if (KIND == DENSE_LAPLACE) {
                if (!(qbad | kbad)) {
                    #pragma unroll 4
                    for (int d = 0; d < dc; d++) {
                        const float4 qa = *reinterpret_cast<const float4*>(qc + d * TM);
                        const float4 i0 = *reinterpret_cast<const float4*>(kp + d * TN), i1 = *reinterpret_cast<const float4*>(kp + d * TN + 32);
                        const float4 e0 = *reinterpret_cast<const float4*>(kp + (DK + d) * TN), e1 = *reinterpret_cast<const float4*>(kp + (DK + d) * TN + 32);
                        const float qe[4] = {qa.x, qa.y, qa.z, qa.w}, qi[4] = {rcp(qa.x), rcp(qa.y), rcp(qa.z), rcp(qa.w)};
                        const float ki[8] = {i0.x, i0.y, i0.z, i0.w, i1.x, i1.y, i1.z, i1.w}, ke[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
                        #pragma unroll
                        for (int i = 0; i < 4; i++)
                            #pragma unroll
                            for (int j = 0; j < 8; j++) {
                                if (j & 1) acc[i][j] = fmaf(fminf(qe[i], ke[j]), fminf(qi[i], ki[j]), acc[i][j]);
                                else       acc[i][j] += fminf(qe[i] * ki[j], qi[i] * ke[j]);
                            }
                    }
                } else {                                 // (a tile within the range holds e^x: take its logarithm)
                    #pragma unroll 1
                    for (int d = 0; d < dc; d++) {
                        float y[8];
                        #pragma unroll
                        for (int j = 0; j < 8; j++) { const float s = kp[(DK + d) * TN + (j >> 2) * 32 + (j & 3)]; y[j] = kbad ? s : logf(s); }
                        #pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const float s = qc[d * TM + i], x = qbad ? s : logf(s);
                            #pragma unroll
                            for (int j = 0; j < 8; j++) acc[i][j] += __expf(-fabsf(x - y[j]));
                        }
                    }
                }
            } else {
                #pragma unroll 4
                for (int d = 0; d < dc; d++) {
                    const float4 qa = *reinterpret_cast<const float4*>(qc + d * TM);
                    const ulonglong2 k0 = *reinterpret_cast<const ulonglong2*>(kp + d * TN), k1 = *reinterpret_cast<const ulonglong2*>(kp + d * TN + 32);
                    const f2 kn[4] = {k0.x, k0.y, k1.x, k1.y};
                    const f2 qd[4] = {pack(qa.x, qa.x), pack(qa.y, qa.y), pack(qa.z, qa.z), pack(qa.w, qa.w)};
                    #pragma unroll
                    for (int i = 0; i < 4; i++)
                        #pragma unroll
                        for (int j = 0; j < 4; j++) {
                            float r0, r1;
                            unpack(add(qd[i], kn[j]), r0, r1);
                            if (KIND == DENSE_BUMP) { r0 = __saturatef(1.0f - fabsf(r0)); r1 = __saturatef(1.0f - fabsf(r1)); }
                            else                    { r0 = fabsf(r0); r1 = fabsf(r1); }
                            acc[i][2 * j]     += r0;
                            acc[i][2 * j + 1] += r1;
                        }
                }
            }
            stage = stage + 1 == KSTAGES ? 0 : stage + 1;
        }
        // ---- A, transposed, into shared memory; row sums
        #pragma unroll
        for (int h = 0; h < 2; h++) {
            const int nn = h * 32 + ng * 4;
            float kn[4] = {0.f, 0.f, 0.f, 0.f};
            if (KIND == DENSE_RIESZ) {
                const float4 s = *reinterpret_cast<const float4*>(kns + nn);
                kn[0] = s.x; kn[1] = s.y; kn[2] = s.z; kn[3] = s.w;
            }
            const float4 w4 = *reinterpret_cast<const float4*>(kw + nn);
            const float  w[4] = {w4.x, w4.y, w4.z, w4.w};
            #pragma unroll
            for (int j = 0; j < 4; j++) {
                float r[4];
                #pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float s = acc[i][h * 4 + j];
                    r[i] = w[j] != 0.0f ? (KIND == DENSE_RIESZ ? (qv[i] + kn[j]) - s : s) * w[j] : 0.0f;     // (0 for a masked or absent key)
                    rs[i] += r[i];
                }
                *reinterpret_cast<float4*>(at + (nn + j) * AT_LD + mg * 4) = make_float4(r[0], r[1], r[2], r[3]);
            }
        }
        cp_wait<0>();
        __syncthreads();
        if (keep && (list[i] & 1)) {
            // The rows of masked keys, whatever they hold, to zeros: their weight is 0, but 0 times NaN is not. (Here and not where the
            // rows are copied, which costs every call 0.4 %, masked or not; in tiles without masked keys too: 96 heads x 777 keys + 1.2 %.)
            const int r = tid >> 1;
            if (kw[r] == 0.0f)
                for (int c = (tid & 1) * 4; c < CP; c += 8) *reinterpret_cast<float4*>(vs + r * CP + c) = make_float4(0.f, 0.f, 0.f, 0.f);
            __syncthreads();
        }
        // ---- out += A v, 4 rows x CT channels per thread
        {
            const float* ap = at + mg * 4;
            const float* vp = vs + ng * 4;
            #pragma unroll 4
            for (int n = 0; n < TN; n++) {
                const float4 a4 = *reinterpret_cast<const float4*>(ap + n * AT_LD);
                const f2 ar[4] = {pack(a4.x, a4.x), pack(a4.y, a4.y), pack(a4.z, a4.z), pack(a4.w, a4.w)};
                #pragma unroll
                for (int h = 0; h < CT / 4; h++) {
                    const ulonglong2 vv = *reinterpret_cast<const ulonglong2*>(vp + n * CP + h * 32);
                    #pragma unroll
                    for (int i = 0; i < 4; i++) {
                        o[i][2 * h]     = fma(ar[i], vv.x, o[i][2 * h]);
                        o[i][2 * h + 1] = fma(ar[i], vv.y, o[i][2 * h + 1]);
                    }
                }
            }
        }
    }
    cp_wait<0>();
    // ---- row sums over the 8 key groups (all in one warp)
    #pragma unroll
    for (int i = 0; i < 4; i++) {
        #pragma unroll
        for (int off = 4; off < 32; off <<= 1) rs[i] += __shfl_xor_sync(FULL, rs[i], off);
    }
    auto row_weight = [&](const int m) -> float { return a.row_keep ? __ldg(a.row_keep + (long long)(p / a.H) * M + m) : 1.0f; };
    auto finish = [&](const float den) -> float { return a.normalise ? 1.0f / fmaxf(den, a.clamp) : 1.0f; };
    if (split == 1) {
        #pragma unroll
        for (int i = 0; i < 4; i++) {
            const int m = m0 + mg * 4 + i;
            if (m >= M) continue;
            const float f = finish(rs[i]) * row_weight(m);
            if (a.out_u && ng == 0) a.out_u[(long long)p * M + m] = rs[i];
            float* dst = a.out + ((long long)p * M + m) * C;
            #pragma unroll
            for (int h = 0; h < CT / 4; h++) {
                const int c = h * 32 + ng * 4;
                float r[4];
                unpack(o[i][2 * h], r[0], r[1]);
                unpack(o[i][2 * h + 1], r[2], r[3]);
                if ((C & 3) == 0) {
                    if (c < C) *reinterpret_cast<float4*>(dst + c) = make_float4(r[0] * f, r[1] * f, r[2] * f, r[3] * f);
                } else {
                    #pragma unroll
                    for (int e = 0; e < 4; e++) if (c + e < C) dst[c + e] = r[e] * f;
                }
            }
        }
    } else {
        // the CTAs of the cluster meet: partial tiles in shared memory (over the A and v tiles), every CTA finishes a share of the rows
        cg::cluster_group cl = cg::this_cluster();
        float* part = at;                                // [TM][CP]; TM * CP <= TN * AT_LD + TN * CP
        __syncthreads();
        #pragma unroll
        for (int i = 0; i < 4; i++) {
            if (ng == 0) rsum[mg * 4 + i] = rs[i];
            #pragma unroll
            for (int h = 0; h < CT / 4; h++)
                *reinterpret_cast<ulonglong2*>(part + (mg * 4 + i) * CP + h * 32 + ng * 4) = make_ulonglong2(o[i][2 * h], o[i][2 * h + 1]);
        }
        cl.sync();
        // (float4s, a few at a time: every remote load takes some hundred cycles)
        const int r0 = TM * rank / split, rn = TM / split, c4 = (C + 3) >> 2;
        #pragma unroll 4
        for (int i = tid; i < rn * c4; i += DT_THREADS) {
            const int r = r0 + i / c4, c = (i % c4) * 4;
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
            float  den = 0.0f;
            #pragma unroll
            for (int b = 0; b < 8; b++) {
                if (b >= split) break;
                const float4 x = *reinterpret_cast<const float4*>(cl.map_shared_rank(part, b) + r * CP + c);
                s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
                den += cl.map_shared_rank(rsum, b)[r];
            }
            if (m0 + r >= M) continue;
            const float f = finish(den) * row_weight(m0 + r);
            float* dst = a.out + ((long long)p * M + m0 + r) * C + c;
            if ((C & 3) == 0) {
                *reinterpret_cast<float4*>(dst) = make_float4(s.x * f, s.y * f, s.z * f, s.w * f);
            } else {
                const float y[4] = {s.x * f, s.y * f, s.z * f, s.w * f};
                #pragma unroll
                for (int e = 0; e < 4; e++) if (c + e < C) dst[e] = y[e];
            }
            if (a.out_u && c == 0) a.out_u[(long long)p * M + m0 + r] = den;
        }
        cl.sync();                                       // nobody leaves while its shared memory is still read
    }
}

template <int KIND, int CT>
static cudaError_t launch_dense_inst(const DenseArgs& a, cudaStream_t stream) {
    auto kern = dense_forward<KIND, CT>;
    const size_t smem = dense_smem_bytes<KIND, CT>(a.D, a.keep ? (a.N + TN - 1) / TN + 1 : 0);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim  = dim3((unsigned)((long long)a.P * ((a.M + TM - 1) / TM) * a.split));
    cfg.blockDim = dim3(DT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at{};                            // (a programmatic launch that overlaps dense_stage was measured slower: its CTAs take the room)
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = a.split; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, a);
}

template <int KIND>
static cudaError_t launch_dense_c(const DenseArgs& a, cudaStream_t stream) {
    const unsigned tiles = (unsigned)a.P * (unsigned)((a.M + TM - 1) / TM + (a.N + TN - 1) / TN);
    const size_t smem = a.rows_layout ? sizeof(float) * 64 * (a.D + 1) : 0;
    dense_stage<KIND><<<tiles, 256, smem, stream>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (a.C <= 32) return launch_dense_inst<KIND, 4>(a, stream);
    if (a.C <= 64) return launch_dense_inst<KIND, 8>(a, stream);
    return launch_dense_inst<KIND, 16>(a, stream);
}

cudaError_t launch_dense_forward(DenseArgs a, int kind, int sms, cudaStream_t stream) {
    a.split = dense_split((long long)a.P * ((a.M + TM - 1) / TM), (a.N + TN - 1) / TN, sms);
    a.vec = a.rows_layout && (a.D & 3) == 0 && ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k)) & 15) == 0;
    switch (kind) {
        case DENSE_LAPLACE: return launch_dense_c<DENSE_LAPLACE>(a, stream);
        case DENSE_ABS:     return launch_dense_c<DENSE_ABS>(a, stream);
        case DENSE_BUMP:    return launch_dense_c<DENSE_BUMP>(a, stream);
        case DENSE_RIESZ:   return launch_dense_c<DENSE_RIESZ>(a, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace qlka
