// Arguments of the pairwise (unsorted) kernels for short sequences, dense_tiles.cu.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace qlka {

enum DenseKind : int { DENSE_LAPLACE = 0, DENSE_ABS = 1, DENSE_BUMP = 2, DENSE_RIESZ = 3 };

struct DenseArgs {
    const float* q;          // (P, D, M), or (P, M, D) with rows_layout
    const float* k;          // (P, D, N), or (P, N, D)
    const float* v;          // (P, N, C), 16-byte aligned
    const float* keep;       // (P / H, N) key weights 0 / 1, or null
    const float* row_keep;   // (P / H, M) weights of the output rows 0 / 1, or null
    float*       staged;     // dense_workspace_bytes() of scratch
    float*       out;        // (P, M, C), 16-byte aligned
    float*       out_u;      // (P, M) row sums, or null
    int   P, H, D, N, M, C;
    float scale;             // applied to q and k: 1 / tau rounded, as torch divides by a scalar (ties between q and k depend on it)
    float eps;               // RIESZ: added to every A_mn
    float clamp;             // floor of the row sum when normalising
    bool  rows_layout, normalise;
    bool  vec;               // (set by the launcher) q and k can be read 16 bytes at a time
    int   split;             // (set by the launcher) CTAs per query tile
};

size_t      dense_workspace_bytes(int kind, int P, int D, int N, int M);
cudaError_t launch_dense_forward(DenseArgs a, int kind, int sms, cudaStream_t stream);

// Gradients of the same sums, dense_gradient.cu.
struct DenseGradArgs {
    const float *q, *k, *v;  // as in DenseArgs; attention: rows layout, scaled
    const float* a;          // (P, M, C) upstream gradient of the sums (attention: of the normalised output)
    const float* s;          // (P, M) upstream gradient of the row sums, or null (attention: unused)
    const float *out, *den;  // attention: (P, M, C) output and (P, M) row sums of the forward call
    const float* keep;       // (P / H, N) or null
    float *grad_q, *grad_k;  // in the layout of q and k
    float* grad_v;           // (P, N, C), 16-byte aligned
    float* staged;           // dense_gradient_workspace_bytes()
    int   P, H, D, N, M, C;
    float scale, eps, clamp;
    bool  attention;
    int   split;             // (set by the launcher)
};
size_t      dense_gradient_workspace_bytes(int kind, int P, int D, int N, int M, int C, bool attention);
cudaError_t launch_dense_gradient(const DenseGradArgs& g, int kind, int sms, cudaStream_t stream);

// CTAs that share one tile of 64 rows: the count that takes the busiest SM the least time, in tiles of the other side; a CTA's own
// start and end count as one and a half more, and an SM with one or two of these CTAs leaves a half or a fifth of itself idle.
inline double dense_sm_cost(long long ctas, int ntiles, int split, int sms) {
    const long long per_sm = (ctas * split + sms - 1) / sms;
    return per_sm * (per_sm < 2 ? 2.2 : per_sm < 3 ? 1.25 : 1.0) * ((ntiles + split - 1) / split + 1.5);
}
inline int dense_split(long long ctas, int ntiles, int sms) {
    int best = 1;
    for (int s = 2; s <= 8 && s <= ntiles; s *= 2)
        if (dense_sm_cost(ctas, ntiles, s, sms) < 0.97 * dense_sm_cost(ctas, ntiles, best, sms)) best = s;
    return best;
}

#ifdef __CUDACC__
// The tiles of 64 keys that hold an unmasked one, in order, into `list` (shared memory, one entry per tile: twice the tile, plus 1 if
// masked keys are in it too); returns their number.
// Padding at the end of a sequence costs nothing that way. All threads of the block call it; `keep` has N entries.
__device__ __forceinline__ int active_tiles(const float* __restrict__ keep, const int N, int* list, int* count) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5, tiles = (N + 63) / 64;
    for (int t = warp; t < tiles; t += warps) {
        const int  n = t * 64 + lane;
        const bool a = n < N && __ldg(keep + n) != 0.0f, b = n + 32 < N && __ldg(keep + n + 32) != 0.0f;
        const bool any = __any_sync(0xffffffffu, a || b), all = __all_sync(0xffffffffu, (a || n >= N) && (b || n + 32 >= N));
        if (lane == 0) list[t] = any ? (all ? 2 : 1) : 0;
    }
    __syncthreads();
    if (warp == 0) {
        int n = 0;
        for (int t0 = 0; t0 < tiles; t0 += 32) {
            const int      s = t0 + lane < tiles ? list[t0 + lane] : 0;
            const unsigned b = __ballot_sync(0xffffffffu, s != 0);
            __syncwarp();
            if (s) list[n + __popc(b & ((1u << lane) - 1u))] = 2 * (t0 + lane) + (s == 1);      // (never ahead of the entries still to be read)
            n += __popc(b);
            __syncwarp();
        }
        if (lane == 0) *count = n;
    }
    __syncthreads();
    return *count;
}
#endif

constexpr float LAP_RANGE = 80.0f;     // largest |value| whose exponentials the Laplace kernels multiply
constexpr int DENSE_MAX_D = 128;      // the query tile of all features stays in shared memory

}  // namespace qlka
