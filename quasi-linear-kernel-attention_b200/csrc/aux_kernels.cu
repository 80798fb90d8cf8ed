// Small streaming kernels around the walks: the pre-reductions and the rank-1 initial value
// of the abs sum (the reference uses ATen sum / bmm for the former,
// Weighted_Abs_Sum/csrc/binding.cpp:154-159,286-289,349-350, and abs_init for the latter,
// Weighted_Abs_Sum/csrc/abs_kernels.cu:23-70), and channel padding to a multiple of four
// (the reference pads odd C to even with constant_pad_nd, binding.cpp:87-89).
#include "qlka_common.cuh"

namespace qlka {

// out[p, l] = sum_d x[p, d, l]   (ABS: sum_d |x[p, d, l]|)
template <bool ABS>
__global__ void colsum_d_kernel(const float* __restrict__ x, float* __restrict__ out, const int D, const int L, const long long total) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const long long p = i / L, l = i % L;
    const float* src = x + p * D * L + l;
    float acc = 0.0f;
    for (int d = 0; d < D; d++) { const float t = src[(long long)d * L]; acc += ABS ? fabsf(t) : t; }
    out[i] = acc;
}

// Per p over rows r of w (P, R, C4) with optional row scalars s (P, R):
//   wsum[p, c] += sum_r w[r, c],  swsum[p, c] += sum_r s[r] w[r, c],  ssum[p] += sum_r s[r]
// (outputs must be zeroed; partial sums of a row tile are added atomically). grid (tiles, P).
// VEC: C4 is a multiple of four; 16 bytes per lane, eight rows of a thread in flight (one float per lane and row at a time: 0.064 -> 0.022 ms
// for 96 heads x 4096 rows x 64 channels, 101 MB). A CTA adds each of its sums once: with an atomic per row lane for ssum, and the partial sums added up one after
// the other, narrow rows took longer than one float per lane (48 heads x 9000 rows, 16 channels 39 us, then 59, now 12; 32 channels 40, 60, 15).
constexpr int RS_THREADS = 256, RS_ROWS = 256;
template <bool VEC>
__global__ void __launch_bounds__(RS_THREADS) rowstat_kernel(
    const float* __restrict__ w, const float* __restrict__ s,
    float* __restrict__ wsum, float* __restrict__ swsum, float* __restrict__ ssum,
    const int R, const int C4)
{
    constexpr int U = VEC ? 4 : 1;                                // channels of a lane
    __shared__ float red_w[U][RS_THREADS], red_k[U][RS_THREADS], red_s[RS_THREADS];
    const int chunks = (R + RS_ROWS - 1) / RS_ROWS;               // (p rides in blockIdx.x: a grid's y extent stops at 65535)
    const int p  = blockIdx.x / chunks;
    const int r0 = (blockIdx.x % chunks) * RS_ROWS, r1 = min(R, r0 + RS_ROWS);
    const int CW = (C4 <= 32 ? 32 : (C4 <= 64 ? 64 : 128)) / U;   // lanes of a row
    const int c  = threadIdx.x % CW * U, lane_r = threadIdx.x / CW, nr = RS_THREADS / CW;
    const float* rows = w + (long long)p * R * C4 + c;
    const float* sp   = s ? s + (long long)p * R : nullptr;
    float aw[U], ak[U], as = 0.0f;
    #pragma unroll
    for (int u = 0; u < U; u++) aw[u] = ak[u] = 0.0f;
    if (c < C4) {
        #pragma unroll 8
        for (int r = r0 + lane_r; r < r1; r += nr) {
            float x[U];
            if constexpr (VEC) { const float4 t = ldg4(rows + (long long)r * C4); x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w; }
            else               x[0] = rows[(long long)r * C4];
            const float sc = sp ? __ldg(sp + r) : 0.0f;
            #pragma unroll
            for (int u = 0; u < U; u++) { aw[u] += x[u]; ak[u] = fmaf(sc, x[u], ak[u]); }
            as += sc;
        }
    }
    for (int off = CW; off < 32; off <<= 1) {                     // the rows of a warp
        #pragma unroll
        for (int u = 0; u < U; u++) { aw[u] += __shfl_xor_sync(FULL, aw[u], off); ak[u] += __shfl_xor_sync(FULL, ak[u], off); }
        as += __shfl_xor_sync(FULL, as, off);
    }
    #pragma unroll
    for (int u = 0; u < U; u++) { red_w[u][threadIdx.x] = aw[u]; red_k[u][threadIdx.x] = ak[u]; }
    red_s[threadIdx.x] = as;
    __syncthreads();
    if (lane_r == 0 && c < C4) {
        const int apart = max(CW, 32);                            // threads from one partial sum to the next
        for (int j = apart + threadIdx.x; j < RS_THREADS; j += apart) {
            #pragma unroll
            for (int u = 0; u < U; u++) { aw[u] += red_w[u][j]; ak[u] += red_k[u][j]; }
            as += red_s[j];
        }
        #pragma unroll
        for (int u = 0; u < U; u++) {
            atomicAdd(wsum + (long long)p * C4 + c + u, aw[u]);
            if (swsum) atomicAdd(swsum + (long long)p * C4 + c + u, ak[u]);
        }
        if (ssum && c == 0) atomicAdd(ssum + p, as);
    }
}

// out[p] = sum_l x[p, l]; one CTA per p
__global__ void __launch_bounds__(256) vecsum_kernel(const float* __restrict__ x, float* __restrict__ out, const int L) {
    __shared__ float red[256];
    const int p = blockIdx.x;
    float acc = 0.0f;
    for (int l = threadIdx.x; l < L; l += 256) acc += x[(long long)p * L + l];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int off = 128; off > 0; off >>= 1) {
        if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[p] = red[0];
}

// out[p, m, c] = A * ktot[p, c] - (A * qsum[p, m] + Bq) * vsum[p, c];  out_u[p, m] = A * ksr[p] - Nk * (A * qsum[p, m] + Bq)
// (A = 1, Bq = 0 for the plain abs sum; a folded sum over shifted queries has A = sum of weights, Bq = D * sum w_s shift_s; without
// qsum the query terms are left out)
// The kernels over rows take ROW_TILE rows per CTA, so that what depends on the row is worked out once per CTA, not by a division per element.
constexpr int ROW_TILE = 64;
__global__ void __launch_bounds__(256) abs_init_kernel(
    const float* __restrict__ ktot, const float* __restrict__ vsum, const float* __restrict__ qsum,
    const float* __restrict__ ksr, float* __restrict__ out, float* __restrict__ out_u,
    const int M, const int C4, const float Nk, const long long rows, const float A, const float Bq)
{
    __shared__ float qs[ROW_TILE];
    __shared__ int   head[ROW_TILE];
    const long long r0 = (long long)blockIdx.x * ROW_TILE;
    const int n = (int)min((long long)ROW_TILE, rows - r0), q4 = C4 >> 2, tid = threadIdx.x;
    if (tid < n) {
        const int p = (int)((r0 + tid) / M);
        head[tid] = p;
        qs[tid]   = qsum ? fmaf(A, qsum[r0 + tid], Bq) : 0.0f;
        if (out_u) out_u[r0 + tid] = A * ksr[p] - Nk * qs[tid];
    }
    __syncthreads();
    #pragma unroll 4
    for (int i = tid; i < n * q4; i += 256) {
        const int r = i / q4, c = (i - r * q4) * 4;
        const float4 kt = ldg4(ktot + (long long)head[r] * C4 + c), vs = ldg4(vsum + (long long)head[r] * C4 + c);
        *reinterpret_cast<float4*>(out + r0 * C4 + 4 * i) =
            make_float4(fmaf(-qs[r], vs.x, A * kt.x), fmaf(-qs[r], vs.y, A * kt.y), fmaf(-qs[r], vs.z, A * kt.z), fmaf(-qs[r], vs.w, A * kt.w));
    }
}

// dst (rows, C4) <- src (rows, C), zero filled
__global__ void pad_rows_kernel(const float* __restrict__ src, float* __restrict__ dst, const int C, const int C4, const long long total) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const long long r = i / C4; const int c = (int)(i % C4);
    dst[i] = c < C ? src[r * C + c] : 0.0f;
}
// dst (rows, C) <- src (rows, C4)
__global__ void unpad_rows_kernel(const float* __restrict__ src, float* __restrict__ dst, const int C, const int C4, const long long total) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const long long r = i / C; const int c = (int)(i % C);
    dst[i] = src[r * C4 + c];
}

// ---- the caller's side of add_laplace attention (Experiments/kernel_attention/attention.py:67-72, 95-126) ----
// x under a key mask: what stands in a masked place counts nothing, NaN and infinities too
__device__ __forceinline__ float weighted(const float x, const float keep) { return keep != 0.0f ? x * keep : 0.0f; }

// dst[p, d, s] = src[p, s, d] * scale * (keep ? keep[p / H, s] : 1): the (B, H, S, D) -> (P, D, S) layout change of
// attention(), the division by tau and the zeroing of masked keys (whatever they hold) in one pass; 32 x 32 tiles through shared memory
__global__ void __launch_bounds__(256) transpose_scale_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                              const float* __restrict__ keep, const float scale,
                                                              const int S, const int D, const int H)
{
    __shared__ float tile[32][33];
    const int stiles = (S + 31) / 32;
    const int p  = blockIdx.x / stiles;
    const int s0 = (blockIdx.x % stiles) * 32, d0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;       // 32 x 8
    const float* sp = src + (long long)p * S * D;
    float*       dp = dst + (long long)p * D * S;
    #pragma unroll
    for (int r = ty; r < 32; r += 8) {
        const int s = s0 + r, d = d0 + tx;
        float x = 0.0f;
        if (s < S && d < D) {
            x = sp[(long long)s * D + d] * scale;
            if (keep) x = weighted(x, keep[(long long)(p / H) * S + s]);
        }
        tile[r][tx] = x;
    }
    __syncthreads();
    #pragma unroll
    for (int r = ty; r < 32; r += 8) {
        const int d = d0 + r, s = s0 + tx;
        if (d < D && s < S) dp[(long long)d * S + s] = tile[tx][r];
    }
}

// The way back for a gradient: dst[p, s, d] = (src[p, d, s] + c) * scale * (keep ? keep[p / H, s] : 1). With `qt` (the operator's
// queries) c takes out what the masked keys, which sit at the origin, added through the row sum's gradient dd[p, s]:
// c = n_pad[p / H] dd[p, s] sign(q) exp(-|q|), the sign at 0 as the walk has it: a key equal to the query counts as above it, derivative +1.
__global__ void __launch_bounds__(256) transpose_back_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                             const float* __restrict__ keep, const float scale,
                                                             const float* __restrict__ qt, const float* __restrict__ dd, const float* __restrict__ n_pad,
                                                             const int S, const int D, const int H)
{
    __shared__ float tile[32][33];
    const int stiles = (S + 31) / 32;
    const int p  = blockIdx.x / stiles;
    const int s0 = (blockIdx.x % stiles) * 32, d0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const float np = qt ? n_pad[p / H] : 0.0f;
    #pragma unroll
    for (int r = ty; r < 32; r += 8) {
        const int d = d0 + r, s = s0 + tx;
        float x = 0.0f;
        if (d < D && s < S) {
            const long long at = ((long long)p * D + d) * S + s;
            x = src[at];
            if (qt) { const float q = qt[at], w = np * __expf(-fabsf(q)); x += (q > 0.0f ? w : -w) * dd[(long long)p * S + s]; }
            x *= scale;
            if (keep) x = weighted(x, keep[(long long)(p / H) * S + s]);
        }
        tile[r][tx] = x;
    }
    __syncthreads();
    #pragma unroll
    for (int r = ty; r < 32; r += 8) {
        const int s = s0 + r, d = d0 + tx;
        if (s < S && d < D) dst[((long long)p * S + s) * D + d] = tile[tx][r];
    }
}

// dn[row, :] = g[row, :] / max(den[row], clamp),  dd[row] = den[row] >= clamp ? -<dn[row, :], out[row, :]> : 0; 8, 16 or 32 lanes per row with VEC (C a multiple of four), else a warp
template <bool VEC>
__global__ void __launch_bounds__(256) attention_gradient_rows_kernel(const float* __restrict__ g, const float* __restrict__ out, const float* __restrict__ den,
                                                                      float* __restrict__ dn, float* __restrict__ dd, const int C, const float clamp, const long long rows)
{
    constexpr int U = VEC ? 4 : 1;
    const int lanes = VEC ? (C <= 32 ? 8 : C <= 64 ? 16 : 32) : 32, step = 256 / lanes, ln = threadIdx.x % lanes;
    const long long r0 = (long long)blockIdx.x * ROW_TILE, r1 = min(rows, r0 + ROW_TILE);
    #pragma unroll 4
    for (long long r = r0 + threadIdx.x / lanes; r - threadIdx.x / lanes < r1; r += step) {      // (all lanes of a warp stay for the shuffles)
        const long long row = min(r, rows - 1);
        const float d = __ldg(den + row), inv = 1.0f / fmaxf(d, clamp);
        float dot = 0.0f;
        for (int c = ln * U; c < C; c += lanes * U) {
            if constexpr (VEC) {
                float4 x = ldg4(g + row * C + c);
                const float4 o = ldg4(out + row * C + c);
                x.x *= inv; x.y *= inv; x.z *= inv; x.w *= inv;
                if (r < r1) *reinterpret_cast<float4*>(dn + row * C + c) = x;
                dot = fmaf(x.x, o.x, fmaf(x.y, o.y, fmaf(x.z, o.z, fmaf(x.w, o.w, dot))));
            } else {
                const float x = g[row * C + c] * inv;
                if (r < r1) dn[row * C + c] = x;
                dot = fmaf(x, out[row * C + c], dot);
            }
        }
        for (int off = lanes / 2; off > 0; off >>= 1) dot += __shfl_xor_sync(FULL, dot, off);
        if (ln == 0 && r < r1) dd[row] = d >= clamp ? -dot : 0.0f;
    }
}

// dst[p, s, :] = src[p, s, :] * keep[p / H, s]   (src may be dst)
__global__ void mask_rows_kernel(const float* src, float* dst, const float* __restrict__ keep,
                                 const int S, const int C, const int H, const long long total)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const long long ps = i / C;
    const long long p = ps / S, s = ps % S;
    dst[i] = weighted(src[i], keep[(p / H) * S + s]);
}

// n_pad[b] = S - sum_s keep[b, s]; one CTA per b
__global__ void __launch_bounds__(256) npad_kernel(const float* __restrict__ keep, float* __restrict__ n_pad, const int S) {
    __shared__ float red[256];
    const int b = blockIdx.x;
    float acc = 0.0f;
    for (int s = threadIdx.x; s < S; s += 256) acc += keep[(long long)b * S + s];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int off = 128; off > 0; off >>= 1) {
        if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) n_pad[b] = (float)S - red[0];
}

// out[p, m, :] /= max(out_u[p, m] - n_pad[p / H] * sum_d f(qt[p, d, m]), clamp): the row normalisation of _add_laplace
// (BUMP = false, f(x) = exp(-|x|)) and of _add_bump (BUMP = true, f(x) = max(0, 1 - |x|)), with the row sum corrected for
// the masked keys (each sits at k = 0 with v = 0 and adds f(q_d) per dimension); the corrected sum goes to den_out if given.
// A warp per row took 53 us for 24 heads x 8192 rows x 64 channels (101 MB moved), this 15.
template <bool BUMP>
__global__ void __launch_bounds__(256) normalise_kernel(float* __restrict__ out, const float* __restrict__ out_u,
                                                        const float* __restrict__ qt, const float* __restrict__ n_pad,
                                                        const int M, const int D, const int C, const int H,
                                                        const float clamp, const long long rows, float* __restrict__ den_out)
{
    __shared__ float part[4][ROW_TILE], inv[ROW_TILE];
    const long long r0 = (long long)blockIdx.x * ROW_TILE;
    const int n = (int)min((long long)ROW_TILE, rows - r0), tid = threadIdx.x, t = tid % ROW_TILE;
    if (n_pad) {                                       // the weights of a masked key, whose coordinates are 0: neighbouring lanes on neighbouring rows
        if (t < n) {
            const int p = (int)((r0 + t) / M), m = (int)((r0 + t) - (long long)p * M);
            float acc = 0.0f;
            if (n_pad[p / H] != 0.0f) {
                #pragma unroll 8
                for (int d = tid / ROW_TILE; d < D; d += 4) {
                    const float x = fabsf(__ldg(qt + ((long long)p * D + d) * M + m));
                    acc += BUMP ? fmaxf(0.0f, 1.0f - x) : __expf(-x);
                }
            }
            part[tid / ROW_TILE][t] = acc;
        }
        __syncthreads();
    }
    if (tid < n) {
        float den = out_u[r0 + tid];
        if (n_pad) {
            const float np = n_pad[(int)((r0 + tid) / M) / H];
            if (np != 0.0f) den -= np * ((part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]));
        }
        if (den_out) den_out[r0 + tid] = den;
        inv[tid] = 1.0f / fmaxf(den, clamp);
    }
    __syncthreads();
    float* o = out + r0 * C;
    if (C % 4 == 0) {
        const int q = C >> 2;
        #pragma unroll 4
        for (int i = tid; i < n * q; i += 256) {
            float4 x = *reinterpret_cast<const float4*>(o + 4 * i);
            const float f = inv[i / q];
            x.x *= f; x.y *= f; x.z *= f; x.w *= f;
            *reinterpret_cast<float4*>(o + 4 * i) = x;
        }
    } else {
        for (int i = tid; i < n * C; i += 256) o[i] *= inv[i / C];
    }
}

// The add_riesz epilogue (Experiments/kernel_attention/attention.py:75-81), in place on out = the weighted abs sum:
//   a = aq[p, m] + eps;  num = a * vsum[p, :] + akv[p, :] - out;  den = a * S + aksum[p] - out_u[p, m] - eps * n_pad[p / H]
//   out = num / max(den, clamp).
__global__ void __launch_bounds__(256) riesz_epilogue_kernel(float* __restrict__ out, const float* __restrict__ out_u,
                                                             const float* __restrict__ aq, const float* __restrict__ vsum,
                                                             const float* __restrict__ akv, const float* __restrict__ aksum,
                                                             const float* __restrict__ n_pad,
                                                             const int M, const int C, const int H,
                                                             const float eps, const float clamp, const long long rows, float* __restrict__ den_out)
{
    __shared__ float as[ROW_TILE], inv[ROW_TILE];
    __shared__ int   head[ROW_TILE];
    const long long r0 = (long long)blockIdx.x * ROW_TILE;
    const int n = (int)min((long long)ROW_TILE, rows - r0), tid = threadIdx.x;
    if (tid < n) {
        const int   p   = (int)((r0 + tid) / M);
        const float a   = aq[r0 + tid] + eps;
        const float np  = n_pad ? n_pad[p / H] : 0.0f;
        const float den = a * (float)M + aksum[p] - out_u[r0 + tid] - eps * np;
        if (den_out) den_out[r0 + tid] = den;
        as[tid] = a; head[tid] = p; inv[tid] = 1.0f / fmaxf(den, clamp);
    }
    __syncthreads();
    float* o = out + r0 * C;
    if (C % 4 == 0) {
        const int q = C >> 2;
        #pragma unroll 4
        for (int i = tid; i < n * q; i += 256) {
            const int r = i / q, c = (i - r * q) * 4;
            const float4 vs = ldg4(vsum + (long long)head[r] * C + c), kv = ldg4(akv + (long long)head[r] * C + c);
            const float  a = as[r], f = inv[r];
            float4 x = *reinterpret_cast<const float4*>(o + 4 * i);
            x.x = (fmaf(a, vs.x, kv.x) - x.x) * f; x.y = (fmaf(a, vs.y, kv.y) - x.y) * f;
            x.z = (fmaf(a, vs.z, kv.z) - x.z) * f; x.w = (fmaf(a, vs.w, kv.w) - x.w) * f;
            *reinterpret_cast<float4*>(o + 4 * i) = x;
        }
    } else {
        for (int i = tid; i < n * C; i += 256) {
            const int r = i / C, c = i - r * C;
            o[i] = (fmaf(as[r], vsum[(long long)head[r] * C + c], akv[(long long)head[r] * C + c]) - o[i]) * inv[r];
        }
    }
}

static inline unsigned blocks_for(long long total, int threads) { return (unsigned)((total + threads - 1) / threads); }

cudaError_t launch_colsum_d(const float* x, float* out, int P, int D, int L, cudaStream_t st) {
    const long long total = (long long)P * L;
    colsum_d_kernel<false><<<blocks_for(total, 256), 256, 0, st>>>(x, out, D, L, total);
    return cudaGetLastError();
}
cudaError_t launch_abscolsum_d(const float* x, float* out, int P, int D, int L, cudaStream_t st) {
    const long long total = (long long)P * L;
    colsum_d_kernel<true><<<blocks_for(total, 256), 256, 0, st>>>(x, out, D, L, total);
    return cudaGetLastError();
}
cudaError_t launch_rowstat(const float* w, const float* s, float* wsum, float* swsum, float* ssum, int P, int R, int C4, cudaStream_t st) {
    const unsigned grid = (unsigned)((R + RS_ROWS - 1) / RS_ROWS) * (unsigned)P;
    if (C4 % 4 == 0) rowstat_kernel<true><<<grid, RS_THREADS, 0, st>>>(w, s, wsum, swsum, ssum, R, C4);
    else             rowstat_kernel<false><<<grid, RS_THREADS, 0, st>>>(w, s, wsum, swsum, ssum, R, C4);
    return cudaGetLastError();
}
cudaError_t launch_vecsum(const float* x, float* out, int P, int L, cudaStream_t st) {
    vecsum_kernel<<<P, 256, 0, st>>>(x, out, L);
    return cudaGetLastError();
}
cudaError_t launch_abs_init(const float* ktot, const float* vsum, const float* qsum, const float* ksr,
                            float* out, float* out_u, int P, int M, int C4, int Nk, float A, float Bq, cudaStream_t st) {
    const long long rows = (long long)P * M;
    abs_init_kernel<<<blocks_for(rows, ROW_TILE), 256, 0, st>>>(ktot, vsum, qsum, ksr, out, out_u, M, C4, (float)Nk, rows, A, Bq);
    return cudaGetLastError();
}
cudaError_t launch_pad_rows(const float* src, float* dst, long long rows, int C, int C4, cudaStream_t st) {
    const long long total = rows * C4;
    pad_rows_kernel<<<blocks_for(total, 256), 256, 0, st>>>(src, dst, C, C4, total);
    return cudaGetLastError();
}
cudaError_t launch_unpad_rows(const float* src, float* dst, long long rows, int C, int C4, cudaStream_t st) {
    const long long total = rows * C;
    unpad_rows_kernel<<<blocks_for(total, 256), 256, 0, st>>>(src, dst, C, C4, total);
    return cudaGetLastError();
}

cudaError_t launch_transpose_scale(const float* src, float* dst, const float* keep, float scale, int P, int S, int D, int H, cudaStream_t st) {
    dim3 grid((unsigned)((S + 31) / 32) * (unsigned)P, (D + 31) / 32);
    transpose_scale_kernel<<<grid, 256, 0, st>>>(src, dst, keep, scale, S, D, H);
    return cudaGetLastError();
}
cudaError_t launch_transpose_back(const float* src, float* dst, const float* keep, float scale, const float* qt, const float* dd, const float* n_pad,
                                  int P, int S, int D, int H, cudaStream_t st) {
    dim3 grid((unsigned)((S + 31) / 32) * (unsigned)P, (D + 31) / 32);
    transpose_back_kernel<<<grid, 256, 0, st>>>(src, dst, keep, scale, qt, dd, n_pad, S, D, H);
    return cudaGetLastError();
}
cudaError_t launch_attention_gradient_rows(const float* g, const float* out, const float* den, float* dn, float* dd, long long rows, int C, float clamp, cudaStream_t st) {
    if (C % 4 == 0) attention_gradient_rows_kernel<true><<<blocks_for(rows, ROW_TILE), 256, 0, st>>>(g, out, den, dn, dd, C, clamp, rows);
    else            attention_gradient_rows_kernel<false><<<blocks_for(rows, ROW_TILE), 256, 0, st>>>(g, out, den, dn, dd, C, clamp, rows);
    return cudaGetLastError();
}
cudaError_t launch_mask_rows(const float* src, float* dst, const float* keep, int P, int S, int C, int H, cudaStream_t st) {
    const long long total = (long long)P * S * C;
    mask_rows_kernel<<<blocks_for(total, 256), 256, 0, st>>>(src, dst, keep, S, C, H, total);
    return cudaGetLastError();
}
cudaError_t launch_npad(const float* keep, float* n_pad, int B, int S, cudaStream_t st) {
    npad_kernel<<<B, 256, 0, st>>>(keep, n_pad, S);
    return cudaGetLastError();
}
cudaError_t launch_normalise(float* out, const float* out_u, const float* qt, const float* n_pad,
                             int P, int M, int D, int C, int H, float clamp, bool bump, float* den_out, cudaStream_t st) {
    const long long rows = (long long)P * M;
    if (bump) normalise_kernel<true><<<blocks_for(rows, ROW_TILE), 256, 0, st>>>(out, out_u, qt, n_pad, M, D, C, H, clamp, rows, den_out);
    else      normalise_kernel<false><<<blocks_for(rows, ROW_TILE), 256, 0, st>>>(out, out_u, qt, n_pad, M, D, C, H, clamp, rows, den_out);
    return cudaGetLastError();
}
cudaError_t launch_riesz_epilogue(float* out, const float* out_u, const float* aq, const float* vsum, const float* akv,
                                  const float* aksum, const float* n_pad, int P, int M, int C, int H,
                                  float eps, float clamp, float* den_out, cudaStream_t st) {
    const long long rows = (long long)P * M;
    riesz_epilogue_kernel<<<blocks_for(rows, ROW_TILE), 256, 0, st>>>(out, out_u, aq, vsum, akv, aksum, n_pad, M, C, H, eps, clamp, rows, den_out);
    return cudaGetLastError();
}

}  // namespace qlka
