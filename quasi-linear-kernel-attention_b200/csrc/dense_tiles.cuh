// Arguments of the pairwise (unsorted) kernels for short sequences, dense_tiles.cu.
#pragma once
#include <cuda_runtime.h>

namespace qlka {

enum DenseKind : int { DENSE_LAPLACE = 0, DENSE_ABS = 1, DENSE_BUMP = 2, DENSE_RIESZ = 3 };

struct DenseArgs {
    const float* q;          // (P, D, M), or (P, M, D) with rows_layout
    const float* k;          // (P, D, N), or (P, N, D)
    const float* v;          // (P, N, C), 16-byte aligned
    const float* keep;       // (P / H, N) key weights 0 / 1, or null
    float*       staged;     // dense_workspace_bytes() of scratch
    float*       out;        // (P, M, C), 16-byte aligned
    float*       out_u;      // (P, M) row sums, or null
    int   P, H, D, N, M, C;
    float scale;             // applied to q and k
    float eps;               // RIESZ: added to every A_mn
    float clamp;             // floor of the row sum when normalising
    bool  rows_layout, normalise;
    bool  vec;               // (set by the launcher) q and k can be read 16 bytes at a time
    int   split;             // (set by the launcher) CTAs per query tile
};

size_t dense_workspace_bytes(int kind, int P, int D, int N, int M);

constexpr int DENSE_MAX_D = 128;      // the query tile of all features stays in shared memory

}  // namespace qlka
