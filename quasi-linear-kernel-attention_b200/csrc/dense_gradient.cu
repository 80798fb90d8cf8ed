// Gradients of the pairwise sums of dense_tiles.cu, for the same short sequences. With the row matrices a (per query: the
// upstream gradient) and v (per key) and the scalars s (per query),
//
//   G_mn = <a_m, v_n> + s_m                         (0 where the key is masked)
//   grad_q[d, m] = sum_n f'(q_dm - k_dn) G_mn,   grad_k[d, n] = sum_m f'(k_dn - q_dm) G_mn    (f is even)
//   grad_v[n, :] = sum_m A_mn a_m                   dense_forward with the roles swapped
//
// Both of the first are the same kernel, x standing for the side that gets the gradient and y for the other: one CTA owns 64 x
// and runs over tiles of 64 y. Per tile G is formed like a GEMM tile (4 x 4 per thread), goes to shared memory, and is
// contracted over y with f' evaluated on the fly (4 x, 4 features per thread, the x values in registers).
//
// Where an x equals a y the derivative is the sorted walk's: u = y - x has its sign bit clear, which counts as y above x.
//   |x - y|          -1 there (both sides)          sum of -(G with the sign bit of u)
//   exp(-|x - y|)    +1 there (both sides)          sum of e^-|u| (G with the sign bit of u)
//   bump             -|q - k| + |q + 1 - k| / 2 + |q - 1 - k| / 2 term by term, the shifts added to q in fp32
//
// dense_stage_gradient stages rows (scaled, exponentiated) and transposed row matrices per tile; for the attention entry points
// it also forms a and s from the upstream gradient, the output and the row sums: a = g / den, s = -<g, out> / den.
// Bound by instruction issue like dense_forward (6 instructions per pair and feature for the Laplace kernel, 3 for the abs).
#include "qlka_common.cuh"
#include "dense_tiles.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace qlka {

namespace {

constexpr int GT = 64, G_THREADS = 256, G_LD = GT + 4;

typedef unsigned long long f2;
__device__ __forceinline__ f2 pack(const float a, const float b) { f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpack(const f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 fma(const f2 a, const f2 b, const f2 c) { f2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ void cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }
// b with the sign bit of u flipped in
__device__ __forceinline__ float signed_by(const float b, const float u) { return __uint_as_float(__float_as_uint(b) ^ (__float_as_uint(u) & 0x80000000u)); }

template <int KIND> __host__ __device__ constexpr int row_arrays() { return KIND == DENSE_LAPLACE ? 3 : 1; }      // x, e^x, e^-x

}  // namespace

__host__ __device__ inline int grad_pitch(int D) { return D <= 64 ? 64 : 128; }
__host__ __device__ inline int grad_c4(int C) { return (C + 3) & ~3; }

// staged area, in floats: rows of q [P][mt][arrays][64][pitch] | rows of k | a transposed [P][mt][C4][64] | v transposed |
// a rows [P][M][C] (attention) | s [P][mt * 64] | one word per tile, queries first: a value beyond LAP_RANGE is in it (Laplace)
struct GradView {
    long long qr, kr, at, vt, a, s, flag, floats;
    __host__ __device__ GradView(int kind, int P, int D, int N, int M, int C, bool attention) {
        const long long mt = (M + GT - 1) / GT, nt = (N + GT - 1) / GT, ra = kind == DENSE_LAPLACE ? 3 : 1, dp = grad_pitch(D), c4 = grad_c4(C);
        qr = 0;
        kr = qr + P * mt * ra * GT * dp;
        at = kr + P * nt * ra * GT * dp;
        vt = at + P * mt * c4 * GT;
        a  = vt + P * nt * c4 * GT;
        s  = a + (attention ? ((long long)P * M * C + 3) / 4 * 4 : 0);
        flag = s + P * mt * GT;
        floats = flag + P * (mt + nt);
    }
};

size_t dense_gradient_workspace_bytes(int kind, int P, int D, int N, int M, int C, bool attention) {
    const size_t own = sizeof(float) * (size_t)GradView(kind, P, D, N, M, C, attention).floats;
    return ((own + 255) & ~size_t(255)) + dense_workspace_bytes(kind, P, D, M, N);       // + the staged tiles of grad_v
}

template <int KIND>
__global__ void __launch_bounds__(256) dense_stage_gradient(const DenseGradArgs g)
{
    extern __shared__ float tr[];
    const int tid = threadIdx.x, D = g.D, C = g.C, DP = grad_pitch(D), C4 = grad_c4(C), row = tid & 63, sub = tid >> 6;
    const int mt = (g.M + GT - 1) / GT, nt = (g.N + GT - 1) / GT;
    const GradView gv(KIND, g.P, D, g.N, g.M, C, g.attention);
    const bool keys = blockIdx.x >= (unsigned)(g.P * mt);
    const int  tile = keys ? blockIdx.x - g.P * mt : blockIdx.x;
    const int  L = keys ? g.N : g.M, tiles = keys ? nt : mt;
    const int  p = tile / tiles, r0 = (tile % tiles) * GT, rows = min(GT, L - r0);
    constexpr int RA = row_arrays<KIND>();
    // masked keys are staged as zeros, their rows of v too: what stands there reaches no gradient
    const float* keep = keys && g.keep ? g.keep + (long long)(p / g.H) * L + r0 : nullptr;
    auto present = [&](const int r) -> bool { return r < rows && (!keep || __ldg(keep + r) != 0.0f); };

    // ---- rows of q or k
    const float* src = (keys ? g.k : g.q) + (long long)p * L * D;
    float*       dst = g.staged + (keys ? gv.kr : gv.qr) + (long long)tile * RA * GT * DP;
    if (!g.attention) {                                  // (P, D, L): through shared memory
        for (int d = sub; d < D; d += 4) tr[row * (D + 1) + d] = present(row) ? __ldg(src + (long long)d * L + r0 + row) : 0.0f;
        __syncthreads();
    }
    int bad = 0;
    for (int i = tid; i < GT * DP; i += 256) {
        const int r = i / DP, d = i % DP;
        float x = 0.0f;
        if (d < D && present(r)) x = g.attention ? __ldg(src + (long long)(r0 + r) * D + d) * g.scale : tr[r * (D + 1) + d];
        dst[i] = x;
        if (KIND == DENSE_LAPLACE) { dst[GT * DP + i] = expf(x); dst[2 * GT * DP + i] = expf(-x); bad |= !(fabsf(x) <= LAP_RANGE); }
    }
    if (KIND == DENSE_LAPLACE) {
        bad = __syncthreads_or(bad);
        if (tid == 0) reinterpret_cast<int*>(g.staged)[gv.flag + blockIdx.x] = bad;
    }
    // ---- the row matrix of the side, transposed; for the queries of an attention call a and s first
    const float* w = (keys ? g.v : g.a) + ((long long)p * L + r0) * C;
    float* wt = g.staged + (keys ? gv.vt : gv.at) + (long long)tile * C4 * GT;
    __syncthreads();
    if (!keys && g.attention) {
        const int warp = tid >> 5, lane = tid & 31;
        float* aw = g.staged + gv.a + ((long long)p * g.M + r0) * C;
        const float* o = g.out + ((long long)p * g.M + r0) * C;
        for (int r = warp; r < GT; r += 8) {
            float dot = 0.0f, inv = 0.0f, den = 1.0f;
            if (r < rows) { den = __ldg(g.den + (long long)p * g.M + r0 + r); inv = 1.0f / fmaxf(den, g.clamp); }
            for (int c = lane; c < C; c += 32) {
                const float x = r < rows ? __ldg(w + (long long)r * C + c) * inv : 0.0f;
                if (r < rows) { aw[(long long)r * C + c] = x; dot = fmaf(x, __ldg(o + (long long)r * C + c), dot); }
                tr[c * 65 + r] = x;
            }
            #pragma unroll
            for (int off = 16; off > 0; off >>= 1) dot += __shfl_xor_sync(FULL, dot, off);
            if (lane == 0) g.staged[gv.s + (long long)tile * GT + r] = r < rows && den >= g.clamp ? -dot : 0.0f;
        }
    } else {
        for (int i = tid; i < GT * C; i += 256) tr[(i % C) * 65 + i / C] = present(i / C) ? __ldg(w + i) : 0.0f;
        if (!keys && tid < GT) g.staged[gv.s + (long long)tile * GT + tid] = g.s && tid < rows ? __ldg(g.s + (long long)p * g.M + r0 + tid) : 0.0f;
    }
    __syncthreads();
    for (int i = tid; i < GT * C4; i += 256) wt[i] = i / GT < C ? tr[(i / GT) * 65 + i % GT] : 0.0f;
}

// x = queries (KEYS = false) or keys; ND: feature chunks of 64
template <int KIND, int ND>
__global__ void __launch_bounds__(G_THREADS, KIND == DENSE_LAPLACE && ND == 2 ? 1 : 2) dense_gradient(const DenseGradArgs g, const bool keys)
{
    constexpr int RA = row_arrays<KIND>(), DP = ND * 64;
    extern __shared__ __align__(16) float sm[];
    const int C4 = grad_c4(g.C);
    float* xt = sm;                                      // [C4][64] row matrix of x, transposed
    float* yt = xt + C4 * GT;                            // [C4][64] of the y tile
    float* yr = yt + C4 * GT;                            // [RA][64][DP] rows of the y tile
    float* Gs = yr + RA * GT * DP;                       // [64 y][G_LD]
    float* yw = Gs + GT * G_LD;                          // [64] weight of y: keep mask, 0 beyond the last
    float* ys = yw + GT;                                 // [64] scalar of y
    float* rg = ys + GT;                                 // [2][64] row sums of G (RIESZ)
    int*   list = reinterpret_cast<int*>(rg + 2 * GT);   // [ytiles + 1] with a keep mask over y: its active tiles and their number

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int mg = (warp & 3) * 4 + (lane & 3), ng = (warp >> 2) * 8 + (lane >> 2);
    const int split = g.split, rank = blockIdx.x % split, xtile = blockIdx.x / split;
    const int Lx = keys ? g.N : g.M, Ly = keys ? g.M : g.N, D = g.D;
    const int xtiles = (Lx + GT - 1) / GT, ytiles = (Ly + GT - 1) / GT;
    const int p = xtile / xtiles, x0 = (xtile % xtiles) * GT;
    const GradView gv(KIND, g.P, D, g.N, g.M, g.C, g.attention);
    const float* xr_g = g.staged + (keys ? gv.kr : gv.qr) + (long long)xtile * RA * GT * DP;
    const float* yr_g = g.staged + (keys ? gv.qr : gv.kr) + (long long)p * ytiles * RA * GT * DP;
    const float* xt_g = g.staged + (keys ? gv.vt : gv.at) + (long long)xtile * C4 * GT;
    const float* yt_g = g.staged + (keys ? gv.at : gv.vt) + (long long)p * ytiles * C4 * GT;
    const float* keep = g.keep ? g.keep + (long long)(p / g.H) * g.N : nullptr;
    const int active = keep && !keys ? active_tiles(keep, g.N, list, list + ytiles) : ytiles;
    int t0 = (int)((long long)rank * active / split), t1 = (int)((long long)(rank + 1) * active / split);
    if (keep && keys) {                                  // x that all are masked
        const bool on = tid < GT && x0 + tid < Lx && __ldg(keep + x0 + tid) != 0.0f;
        if (!__syncthreads_or(on)) t1 = t0;
    }
    auto tile_at = [&](const int t) -> int { return keep && !keys ? list[t] >> 1 : t; };

    auto copy = [&](float* dst, const float* src, const int n) { for (int i = tid * 4; i < n; i += G_THREADS * 4) cp16(dst + i, src + i); };
    auto issue_yt = [&](const int t) { if (t < t1) copy(yt, yt_g + (long long)tile_at(t) * C4 * GT, C4 * GT); cp_commit(); };
    auto issue_yr = [&](const int t) { if (t < t1) copy(yr, yr_g + (long long)tile_at(t) * RA * GT * DP, RA * GT * DP); cp_commit(); };
    copy(xt, xt_g, C4 * GT);
    issue_yt(t0);
    issue_yr(t0);

    // my x values: 4 rows x 4 features per chunk (bump: shifted; the shifts belong to the queries)
    const float dh = keys ? 0.0f : 1.0f, dl = keys ? 0.0f : -1.0f, ch = keys ? -1.0f : 0.0f, cl = keys ? 1.0f : 0.0f;
    float acc[ND][4][4];
    #pragma unroll
    for (int h = 0; h < ND; h++)
        #pragma unroll
        for (int i = 0; i < 4; i++)
            #pragma unroll
            for (int d = 0; d < 4; d++) acc[h][i][d] = 0.0f;
    float rs[4] = {0.f, 0.f, 0.f, 0.f};
    float sx[4] = {0.f, 0.f, 0.f, 0.f};
    if (!keys) {
        const float4 s = ldg4(g.staged + gv.s + (long long)xtile * GT + mg * 4);
        sx[0] = s.x; sx[1] = s.y; sx[2] = s.z; sx[3] = s.w;
    }
    const int* flag = reinterpret_cast<const int*>(g.staged) + gv.flag;
    const long long fx = keys ? g.P * (long long)ytiles : 0, fy = keys ? 0 : g.P * (long long)xtiles;       // flags of the x and of the y side
    for (int step = t0; step < t1; step++) {
        const int t = tile_at(step), y0 = t * GT;
        const bool plain = KIND == DENSE_LAPLACE && (__ldg(flag + fx + xtile) | __ldg(flag + fy + (long long)p * ytiles + t)) != 0;
        if (tid < GT) {
            yw[tid] = y0 + tid < Ly ? (keep && !keys ? __ldg(keep + y0 + tid) : 1.0f) : 0.0f;
            ys[tid] = keys ? __ldg(g.staged + gv.s + ((long long)p * ytiles + t) * GT + tid) : 0.0f;
        }
        cp_wait<1>();
        __syncthreads();
        // ---- G = x rows . y rows + s
        f2 ga[4][2];
        {
            const float4 s4 = *reinterpret_cast<const float4*>(ys + ng * 4);
            #pragma unroll
            for (int i = 0; i < 4; i++) { ga[i][0] = pack(sx[i] + s4.x, sx[i] + s4.y); ga[i][1] = pack(sx[i] + s4.z, sx[i] + s4.w); }
        }
        #pragma unroll 4
        for (int c = 0; c < C4; c++) {
            const float4 a4 = *reinterpret_cast<const float4*>(xt + c * GT + mg * 4);
            const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(yt + c * GT + ng * 4);
            const f2 ad[4] = {pack(a4.x, a4.x), pack(a4.y, a4.y), pack(a4.z, a4.z), pack(a4.w, a4.w)};
            #pragma unroll
            for (int i = 0; i < 4; i++) { ga[i][0] = fma(ad[i], b.x, ga[i][0]); ga[i][1] = fma(ad[i], b.y, ga[i][1]); }
        }
        {
            const float4 w4 = *reinterpret_cast<const float4*>(yw + ng * 4);
            const float  w[4] = {w4.x, w4.y, w4.z, w4.w};
            float G[4][4];
            #pragma unroll
            for (int i = 0; i < 4; i++) { unpack(ga[i][0], G[i][0], G[i][1]); unpack(ga[i][1], G[i][2], G[i][3]); }
            #pragma unroll
            for (int j = 0; j < 4; j++) {
                #pragma unroll
                for (int i = 0; i < 4; i++) {
                    G[i][j] = w[j] != 0.0f ? G[i][j] * w[j] : 0.0f;
                    if (KIND == DENSE_RIESZ) rs[i] += G[i][j];
                }
                *reinterpret_cast<float4*>(Gs + (ng * 4 + j) * G_LD + mg * 4) = make_float4(G[0][j], G[1][j], G[2][j], G[3][j]);
            }
        }
        cp_wait<0>();
        __syncthreads();
        issue_yt(step + 1);                                 // (everybody has left this tile's)
        // ---- contraction over y
        #pragma unroll
        for (int h = 0; h < ND; h++) {
            float xv[4][4], xa[4][4], xb[4][4];          // x; Laplace: e^x and e^-x; bump: the two shifted values
            #pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 v = ldg4(xr_g + (mg * 4 + i) * DP + h * 64 + ng * 4);
                xv[i][0] = v.x; xv[i][1] = v.y; xv[i][2] = v.z; xv[i][3] = v.w;
                if (KIND == DENSE_LAPLACE) {
                    const float4 e = ldg4(xr_g + GT * DP + (mg * 4 + i) * DP + h * 64 + ng * 4), n = ldg4(xr_g + 2 * GT * DP + (mg * 4 + i) * DP + h * 64 + ng * 4);
                    xa[i][0] = e.x; xa[i][1] = e.y; xa[i][2] = e.z; xa[i][3] = e.w;
                    xb[i][0] = n.x; xb[i][1] = n.y; xb[i][2] = n.z; xb[i][3] = n.w;
                } else if (KIND == DENSE_BUMP) {
                    #pragma unroll
                    for (int d = 0; d < 4; d++) { xa[i][d] = xv[i][d] + dh; xb[i][d] = xv[i][d] + dl; }
                }
            }
            const float* yp = yr + h * 64 + ng * 4;
            const float* gp = Gs + mg * 4;
            if (plain) {
                #pragma unroll 1
                for (int y = 0; y < GT; y++) {
                    #pragma unroll
                    for (int i = 0; i < 4; i++)
                        #pragma unroll
                        for (int d = 0; d < 4; d++) {
                            const float u = yp[y * DP + d] - xv[i][d];
                            acc[h][i][d] = fmaf(__expf(-fabsf(u)), signed_by(gp[y * G_LD + i], u), acc[h][i][d]);
                        }
                }
                continue;
            }
            #pragma unroll 2
            for (int y = 0; y < GT; y++) {
                const float4 g4 = *reinterpret_cast<const float4*>(gp + y * G_LD);
                const float4 y4 = *reinterpret_cast<const float4*>(yp + y * DP);
                const float  G[4] = {g4.x, g4.y, g4.z, g4.w}, yv[4] = {y4.x, y4.y, y4.z, y4.w};
                float ya[4], yb[4];
                if (KIND == DENSE_LAPLACE) {
                    const float4 e = *reinterpret_cast<const float4*>(yp + GT * DP + y * DP), n = *reinterpret_cast<const float4*>(yp + 2 * GT * DP + y * DP);
                    ya[0] = e.x; ya[1] = e.y; ya[2] = e.z; ya[3] = e.w;
                    yb[0] = n.x; yb[1] = n.y; yb[2] = n.z; yb[3] = n.w;
                } else if (KIND == DENSE_BUMP) {
                    #pragma unroll
                    for (int d = 0; d < 4; d++) { ya[d] = yv[d] + ch; yb[d] = yv[d] + cl; }
                }
                #pragma unroll
                for (int i = 0; i < 4; i++)
                    #pragma unroll
                    for (int d = 0; d < 4; d++) {
                        const float u = yv[d] - xv[i][d], t = signed_by(G[i], u);
                        if (KIND == DENSE_LAPLACE) {
                            acc[h][i][d] = fmaf(fminf(xa[i][d] * yb[d], xb[i][d] * ya[d]), t, acc[h][i][d]);
                        } else if (KIND == DENSE_BUMP) {
                            const uint32_t in = __float_as_uint(ya[d] - xa[i][d]) & ~__float_as_uint(yb[d] - xb[i][d]);       // sign bit: within the bump
                            acc[h][i][d] += __uint_as_float(__float_as_uint(t) & (uint32_t)((int)in >> 31));
                        } else {
                            acc[h][i][d] += t;
                        }
                    }
            }
        }
        __syncthreads();                                 // the y rows and G are free again
        issue_yr(step + 1);
    }
    cp_wait<0>();
    if (KIND == DENSE_RIESZ) {                           // |x|_1 in every A: sign(x) times the row sum of G
        #pragma unroll
        for (int i = 0; i < 4; i++)
            #pragma unroll
            for (int off = 4; off < 32; off <<= 1) rs[i] += __shfl_xor_sync(FULL, rs[i], off);
        if (lane < 4) {
            #pragma unroll
            for (int i = 0; i < 4; i++) rg[(warp >> 2) * GT + mg * 4 + i] = rs[i];
        }
    }
    __syncthreads();
    cg::cluster_group cl_g = cg::this_cluster();
    float* part = yt;                                    // [64][DP], over the y tile
    float* grad = (keys ? g.grad_k : g.grad_q) + (long long)p * Lx * D;
    const long long s_row = g.attention ? D : 1, s_d = g.attention ? 1 : Lx;
    const float sign = KIND == DENSE_ABS ? -1.0f : 1.0f;
    #pragma unroll
    for (int h = 0; h < ND; h++)
        #pragma unroll
        for (int i = 0; i < 4; i++)
            *reinterpret_cast<float4*>(part + (mg * 4 + i) * DP + h * 64 + ng * 4) = make_float4(acc[h][i][0], acc[h][i][1], acc[h][i][2], acc[h][i][3]);
    if (split > 1) cl_g.sync(); else __syncthreads();
    // this CTA's rows, as float4s of features, lanes along the contiguous direction of the gradient
    const int r0 = GT * rank / split, rn = GT / split, d4 = (D + 3) >> 2;
    #pragma unroll 4
    for (int i = tid; i < rn * d4; i += G_THREADS) {
        const int r = r0 + (g.attention ? i / d4 : i % rn), d = (g.attention ? i % d4 : i / rn) * 4;
        float y[4] = {0.f, 0.f, 0.f, 0.f}, G = 0.0f;
        #pragma unroll
        for (int b = 0; b < 8; b++) {
            if (b >= split) break;
            const float4 v = *reinterpret_cast<const float4*>((split > 1 ? cl_g.map_shared_rank(part, b) : part) + r * DP + d);
            y[0] += v.x; y[1] += v.y; y[2] += v.z; y[3] += v.w;
            if (KIND == DENSE_RIESZ) { const float* q = split > 1 ? cl_g.map_shared_rank(rg, b) : rg; G += q[r] + q[GT + r]; }
        }
        if (x0 + r >= Lx) continue;
        const float w = keys && keep ? __ldg(keep + x0 + r) : 1.0f;
        #pragma unroll
        for (int e = 0; e < 4; e++) {
            if (d + e >= D) continue;
            float s = y[e] * sign;
            if (KIND == DENSE_RIESZ) { const float x = __ldg(xr_g + r * DP + d + e); s += x > 0.0f ? G : x < 0.0f ? -G : 0.0f; }
            if (g.attention) s *= g.scale;
            grad[(x0 + r) * s_row + (d + e) * s_d] = w != 0.0f ? s * w : 0.0f;
        }
    }
    if (split > 1) cl_g.sync();                          // nobody leaves while its shared memory is still read
}

template <int KIND, int ND>
static cudaError_t launch_gradient_inst(DenseGradArgs g, int sms, cudaStream_t stream) {
    auto kern = dense_gradient<KIND, ND>;
    const int c4 = grad_c4(g.C);
    size_t smem = sizeof(float) * ((size_t)2 * c4 * GT + row_arrays<KIND>() * GT * ND * 64 + GT * G_LD + 2 * GT + 2 * GT);
    const size_t need = sizeof(float) * ((size_t)c4 * GT + GT * ND * 64 + 2 * GT);       // (the partial result overlies the y tile)
    if (smem < need) smem = need;
    if (g.keep) smem += sizeof(int) * ((g.N + GT - 1) / GT + 1);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    for (int keys = 0; keys < 2; keys++) {
        g.split = dense_split((long long)g.P * (((keys ? g.N : g.M) + GT - 1) / GT), ((keys ? g.M : g.N) + GT - 1) / GT, sms);
        cudaLaunchConfig_t cfg{};
        cfg.gridDim  = dim3((unsigned)((long long)g.P * (((keys ? g.N : g.M) + GT - 1) / GT) * g.split));
        cfg.blockDim = dim3(G_THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = g.split; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
        cfg.attrs = &at; cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, kern, g, keys != 0);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <int KIND>
static cudaError_t launch_gradient_kind(const DenseGradArgs& g, int sms, cudaStream_t stream) {
    const unsigned tiles = (unsigned)g.P * (unsigned)((g.M + GT - 1) / GT + (g.N + GT - 1) / GT);
    const size_t rows = g.attention ? 0 : sizeof(float) * GT * (g.D + 1), cols = sizeof(float) * g.C * 65;
    const size_t smem = rows > cols ? rows : cols;
    dense_stage_gradient<KIND><<<tiles, 256, smem, stream>>>(g);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return g.D <= 64 ? launch_gradient_inst<KIND, 1>(g, sms, stream) : launch_gradient_inst<KIND, 2>(g, sms, stream);
}

// grad_q, grad_k and grad_v of the pairwise sums; `g.staged` has dense_gradient_workspace_bytes()
cudaError_t launch_dense_gradient(const DenseGradArgs& g, int kind, int sms, cudaStream_t stream) {
    cudaError_t e = cudaErrorInvalidValue;
    switch (kind) {
        case DENSE_LAPLACE: e = launch_gradient_kind<DENSE_LAPLACE>(g, sms, stream); break;
        case DENSE_ABS:     e = launch_gradient_kind<DENSE_ABS>(g, sms, stream); break;
        case DENSE_BUMP:    e = launch_gradient_kind<DENSE_BUMP>(g, sms, stream); break;
        case DENSE_RIESZ:   e = launch_gradient_kind<DENSE_RIESZ>(g, sms, stream); break;
    }
    if (e != cudaSuccess) return e;
    const GradView gv(kind, g.P, g.D, g.N, g.M, g.C, g.attention);
    DenseArgs a{};                                       // grad_v: the queries are summed over, weighted rows a
    a.q = g.k; a.k = g.q; a.v = g.attention ? g.staged + gv.a : g.a; a.out = g.grad_v;
    a.P = g.P; a.H = g.H; a.D = g.D; a.N = g.M; a.M = g.N; a.C = g.C;
    a.scale = g.attention ? g.scale : 1.0f; a.eps = g.eps; a.rows_layout = g.attention; a.row_keep = g.keep;
    a.staged = g.staged + (((size_t)gv.floats * sizeof(float) + 255) & ~size_t(255)) / sizeof(float);
    return launch_dense_forward(a, kind, sms, stream);
}

}  // namespace qlka
