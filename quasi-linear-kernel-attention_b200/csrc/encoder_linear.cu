// The linear layers of the encoder harness in fp32 accuracy on the bf16 tensor cores.
//
// Every fp32 operand is cut into three bf16 parts, x = x1 + x2 + x3 (each part the rounded rest of the ones before: 24 bits of
// mantissa, nothing of x is lost), and
//     x y = x1 y1  +  (x1 y2 + x2 y1 + x1 y3 + x2 y2 + x3 y1)  +  terms below 2^-24 |x y|, which an fp32 product rounds away too.
// The first term and the five small ones add up in accumulators of their own, so that the small ones lose nothing to the size of
// the first. The tensor cores' fp32 additions cut off rather than round, an error that grows with their number, so every 384
// of K the accumulators are added to fp32 sums in registers and start anew. Error against float64 (2-norm) at 16384 rows, K = 768
// / 3072: 3.2e-7 / 3.2e-7; torch's fp32 product 4.9e-7 / 9.7e-7; one accumulator over all of K 6.6e-7 / 3.1e-6.
//
// linear_kernel: persistent, one CTA per SM, 128 x 256 output tiles. One warp issues TMA copies (per stage 32 of K: the three parts
// of both operands, 72 KB, three stages), one thread issues tcgen05.mma (12 per stage: 2 steps of K = 16 times 6 products; the
// two accumulators take all 512 columns of TMEM), eight warps add the accumulators of every chunk into registers, hand TMEM back at
// once - the small one first: its next products cover the reading of the other - and finish (bias, rotary and head layout / GELU
// and the parts of the next layer's input / residual) while the next tile's products run. Loading all parts of a K step together
// is what keeps the L2 out of the way: 48 bytes per clock and SM for six products instead of 96 each.
// Bound by the tensor pipe (and, in long runs, by the power limit): 16384 x 3072 x 768 with GELU 414 us (1120 TFLOP/s of bf16
// products), torch's fp32 linear on the FP32 pipe 1492 us without the GELU.
//
// Every barrier wait has a limit. A CTA that reaches one sets the device's error word, writes NaN to the tiles it has left, waits for
// its copies and products in flight and ends. The word is in host memory: the next call sees it without waiting for the device.
#include "qlka_common.cuh"

#include <cuda.h>
#include <cuda_bf16.h>

#include <atomic>
#include <mutex>

namespace qlka {

namespace {

constexpr int BM = 128, BN = 256, BK = 32, STAGES = 3, PARTS = 3;
constexpr int KCHUNK_STEPS = 12;                                                // K steps per chunk: 384
constexpr int A_TILE = BM * BK * 2, B_TILE = BN * BK * 2;                       // bytes of one part
constexpr int STAGE_BYTES = PARTS * (A_TILE + B_TILE);
constexpr int EPI_WARPS = 8, LIN_THREADS = (EPI_WARPS + 2) * 32;
constexpr size_t LIN_SMEM = (size_t)STAGES * STAGE_BYTES + 1024 /* alignment */ + 256;
constexpr uint32_t WAIT_LIMIT = 1u << 21;        // tries of a barrier wait before a kernel gives up (a wait is some 100 us at most)

enum { EPI_QKV = 0, EPI_GELU = 1, EPI_RESIDUAL = 2 };

struct LinearArgs {
    int M, N, K;
    const float* bias;           // (N)
    float*       x;              // RESIDUAL: (M, N), added to
    __nv_bfloat16* out3;         // GELU: (3, M, N)
    float *q, *k, *v;            // QKV: (B, H, S, 64), M = B * S rows, N = 3 * H * 64 columns
    const float2* table;         // QKV: (S, 32) cos, sin
    int S, H;
    int* error;                  // set to 1 by a CTA that gave up on a barrier
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(const uint32_t b, const uint32_t n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(b), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_expect(const uint32_t b, const uint32_t bytes) { asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(b), "r"(bytes) : "memory"); }
__device__ __forceinline__ void bar_arrive(const uint32_t b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(b) : "memory"); }
// false: the limit was reached
__device__ __forceinline__ bool bar_wait(const uint32_t b, const uint32_t parity) {
    for (uint32_t i = 0; i < WAIT_LIMIT; i++) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(b), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ void tma_load3(const uint32_t dst, const CUtensorMap* map, const uint32_t bar, const int x, const int y, const int z) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 :: "r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
// K-major tile with rows of 64 bytes, 64-byte swizzle: groups of 8 rows 512 bytes apart
__device__ __forceinline__ uint64_t tile_desc(const uint32_t addr) {
    return (uint64_t)((addr & 0x3ffffu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}
// bf16 x bf16 -> f32, both K-major, 128 x 256
constexpr uint32_t MMA_DESC = 1u << 4 | 1u << 7 | 1u << 10 | (uint32_t)(BN >> 3) << 17 | (uint32_t)(BM >> 4) << 24;
__device__ __forceinline__ void mma(const uint32_t d, const uint64_t a, const uint64_t b, const bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 :: "r"(d), "l"(a), "l"(b), "r"(MMA_DESC), "r"((uint32_t)accumulate) : "memory");
}
__device__ __forceinline__ void mma_commit(const uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_load32(const uint32_t addr, float (&r)[32]) {
    uint32_t* u = reinterpret_cast<uint32_t*>(r);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]),
                   "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]), "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]),
                   "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
                 : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// the three parts of two neighbouring values, one word each (two conversions per instruction)
__device__ __forceinline__ void split3(const float x, const float y, uint32_t (&p)[3]) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(x, y);
    const float rx = x - __low2float(a), ry = y - __high2float(a);
    const __nv_bfloat162 b = __floats2bfloat162_rn(rx, ry);
    const __nv_bfloat162 c = __floats2bfloat162_rn(rx - __low2float(b), ry - __high2float(b));
    p[0] = *reinterpret_cast<const uint32_t*>(&a);
    p[1] = *reinterpret_cast<const uint32_t*>(&b);
    p[2] = *reinterpret_cast<const uint32_t*>(&c);
}

}  // namespace

template <int EPI>
__global__ void __launch_bounds__(LIN_THREADS, 1) linear_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const LinearArgs g)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)STAGES * STAGE_BYTES);       // full[STAGES] empty[STAGES] acc_full small_empty main_empty drained
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full = smem_addr(bars), empty = full + STAGES * 8, acc_full = empty + STAGES * 8, small_empty = acc_full + 8, main_empty = small_empty + 8, drained = main_empty + 8;
    const int mt = (g.M + BM - 1) / BM, nt = (g.N + BN - 1) / BN, tiles = mt * nt, ksteps = g.K / BK;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" :: "r"(smem_addr(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 32) {
        for (int s = 0; s < STAGES; s++) { bar_init(full + 8 * s, 1); bar_init(empty + 8 * s, 1); }
        bar_init(acc_full, 1);
        bar_init(small_empty, EPI_WARPS);
        bar_init(main_empty, EPI_WARPS);
        bar_init(drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    bool ok = true;

    if (warp == EPI_WARPS) {                             // ---- copies
        if (lane == 0) {
            int stage = 0;
            uint32_t parity = 1;                         // (a fresh barrier's previous phase counts as done)
            uint32_t uses[STAGES] = {};
            for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
                const int m0 = tile / nt * BM, n0 = tile % nt * BN;
                for (int ks = 0; ks < ksteps; ks++) {
                    if (!(ok = bar_wait(empty + 8 * stage, parity))) break;
                    const uint32_t a = smem_addr(smem) + stage * STAGE_BYTES, b = a + PARTS * A_TILE;
                    bar_expect(full + 8 * stage, STAGE_BYTES);
                    tma_load3(a, &map_a, full + 8 * stage, ks * BK, m0, 0);
                    tma_load3(b, &map_b, full + 8 * stage, ks * BK, n0, 0);
                    #pragma unroll
                    for (int i = 0; i < STAGES; i++) uses[i] += i == stage;
                    if (++stage == STAGES) { stage = 0; parity ^= 1; }
                }
            }
            #pragma unroll
            for (int i = 0; i < STAGES; i++)             // every copy has landed before the CTA may end
                if (uses[i]) ok &= bar_wait(full + 8 * i, (uses[i] - 1) & 1);
        }
    } else if (warp == EPI_WARPS + 1) {                  // ---- products
        if (lane == 0) {
            int stage = 0;
            uint32_t parity = 0, acc_parity = 1;
            for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
                for (int ks = 0; ks < ksteps; ks++) {
                    const bool first = ks % KCHUNK_STEPS == 0;
                    if (!(ok = bar_wait(full + 8 * stage, parity))) break;
                    if (first && !(ok = bar_wait(small_empty, acc_parity))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a = smem_addr(smem) + stage * STAGE_BYTES, b = a + PARTS * A_TILE;
                    #pragma unroll
                    for (int kk = 0; kk < BK / 16; kk++) {
                        uint64_t da[PARTS], db[PARTS];
                        #pragma unroll
                        for (int i = 0; i < PARTS; i++) { da[i] = tile_desc(a + i * A_TILE + kk * 32); db[i] = tile_desc(b + i * B_TILE + kk * 32); }
                        const bool more = !first || kk > 0;
                        mma(tmem + BN, da[2], db[0], more);              // the small ones, smallest first
                        mma(tmem + BN, da[1], db[1], true);
                        mma(tmem + BN, da[0], db[2], true);
                        mma(tmem + BN, da[1], db[0], true);
                        mma(tmem + BN, da[0], db[1], true);
                        if (first && kk == 0) {
                            if (!(ok = bar_wait(main_empty, acc_parity))) break;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        }
                        mma(tmem, da[0], db[0], more);
                    }
                    if (!ok) break;
                    mma_commit(empty + 8 * stage);
                    if (++stage == STAGES) { stage = 0; parity ^= 1; }
                    if (first) acc_parity ^= 1;
                    if ((ks + 1) % KCHUNK_STEPS == 0 || ks + 1 == ksteps) mma_commit(acc_full);
                }
            }
            mma_commit(drained);                         // no product is in flight any more when TMEM is handed back
            ok &= bar_wait(drained, 0);
        }
    } else {                                             // ---- results: warp w has rows 32 (w mod 4) .. + 31 and 128 of the 256 columns
        uint32_t parity = 0;
        const int row_in = (warp & 3) * 32 + lane, col_in = (warp >> 2) * 128;
        const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + col_in;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            float r[4][32];
            #pragma unroll
            for (int c = 0; c < 4; c++)
                #pragma unroll
                for (int j = 0; j < 32; j++) r[c][j] = 0.0f;
            #pragma unroll 1
            for (int ks = 0; ks < ksteps && ok; ks += KCHUNK_STEPS) {
                if (!(ok = __all_sync(FULL, bar_wait(acc_full, parity)))) break;
                parity ^= 1;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                #pragma unroll
                for (int which = 1; which >= 0; which--) {           // the small products, then the first ones
                    #pragma unroll
                    for (int c = 0; c < 4; c++) {
                        float s[32];
                        tmem_load32(taddr + which * BN + c * 32, s);
                        #pragma unroll
                        for (int j = 0; j < 32; j++) r[c][j] += s[j];
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) bar_arrive(which ? small_empty : main_empty);
                }
            }
            if (!ok) {                                   // (this tile and all that follow)
                #pragma unroll
                for (int c = 0; c < 4; c++)
                    #pragma unroll
                    for (int j = 0; j < 32; j++) r[c][j] = __int_as_float(0x7fffffff);
            }
            const int row = tile / nt * BM + row_in, n0 = tile % nt * BN + col_in;
            if (EPI == EPI_QKV) {
                // 64 columns are one head of q, k or v; pairs (i, i + 32) turn by the angle of the position
                const int b = row / g.S, s = row % g.S;
                #pragma unroll
                for (int h2 = 0; h2 < 2; h2++) {
                    const int n = n0 + h2 * 64;
                    if (n >= g.N || row >= g.M) continue;
                    const int which = n / (g.H * 64), head = n / 64 % g.H;
                    float* dst = (which == 0 ? g.q : which == 1 ? g.k : g.v) + (((long long)b * g.H + head) * g.S + s) * 64;
                    #pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        const float4 b1 = ldg4(g.bias + n + j), b2 = ldg4(g.bias + n + 32 + j);
                        const float  y1[4] = {r[2 * h2][j] + b1.x, r[2 * h2][j + 1] + b1.y, r[2 * h2][j + 2] + b1.z, r[2 * h2][j + 3] + b1.w};
                        const float  y2[4] = {r[2 * h2 + 1][j] + b2.x, r[2 * h2 + 1][j + 1] + b2.y, r[2 * h2 + 1][j + 2] + b2.z, r[2 * h2 + 1][j + 3] + b2.w};
                        float z1[4], z2[4];
                        if (which < 2) {
                            const float4 t0 = ldg4(reinterpret_cast<const float*>(g.table + (long long)s * 32 + j)), t1 = ldg4(reinterpret_cast<const float*>(g.table + (long long)s * 32 + j + 2));
                            const float  cs[4] = {t0.x, t0.z, t1.x, t1.z}, sn[4] = {t0.y, t0.w, t1.y, t1.w};
                            #pragma unroll
                            for (int e = 0; e < 4; e++) {
                                z1[e] = __fsub_rn(__fmul_rn(y1[e], cs[e]), __fmul_rn(y2[e], sn[e]));      // (each product rounded, as the separate operations do)
                                z2[e] = __fadd_rn(__fmul_rn(y1[e], sn[e]), __fmul_rn(y2[e], cs[e]));
                            }
                        } else {
                            #pragma unroll
                            for (int e = 0; e < 4; e++) { z1[e] = y1[e]; z2[e] = y2[e]; }
                        }
                        *reinterpret_cast<float4*>(dst + j)      = make_float4(z1[0], z1[1], z1[2], z1[3]);
                        *reinterpret_cast<float4*>(dst + 32 + j) = make_float4(z2[0], z2[1], z2[2], z2[3]);
                    }
                }
            } else {
                #pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int n = n0 + c * 32;
                    if (n >= g.N || row >= g.M) continue;
                    if (EPI == EPI_RESIDUAL) {
                        float* x = g.x + (long long)row * g.N + n;
                        #pragma unroll
                        for (int j = 0; j < 32; j += 4) {            // (reductions, one per element: nothing to wait for)
                            const float4 b4 = ldg4(g.bias + n + j);
                            red_add4(x + j, r[c][j] + b4.x, r[c][j + 1] + b4.y, r[c][j + 2] + b4.z, r[c][j + 3] + b4.w);
                        }
                    } else {
                        __nv_bfloat16* o = g.out3 + (long long)row * g.N + n;
                        const long long part = (long long)g.M * g.N;
                        #pragma unroll
                        for (int j = 0; j < 32; j += 8) {
                            uint32_t p[3][4];
                            const float4 b0 = ldg4(g.bias + n + j), b1 = ldg4(g.bias + n + j + 4);
                            const float  bias[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
                            #pragma unroll
                            for (int e = 0; e < 8; e += 2) {
                                float z[2];
                                #pragma unroll
                                for (int f = 0; f < 2; f++) {
                                    const float y = r[c][j + e + f] + bias[e + f];
                                    z[f] = 0.5f * y * (1.0f + erff(y * 0.70710678118654752440f));
                                }
                                uint32_t u[3];
                                split3(z[0], z[1], u);
                                #pragma unroll
                                for (int i = 0; i < 3; i++) p[i][e / 2] = u[i];
                            }
                            #pragma unroll
                            for (int i = 0; i < 3; i++) *reinterpret_cast<uint4*>(o + i * part + j) = make_uint4(p[i][0], p[i][1], p[i][2], p[i][3]);
                        }
                    }
                }
            }
        }
    }
    if (!ok) {
        *reinterpret_cast<volatile int*>(g.error) = 1;
        __threadfence_system();
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem));
}

// rows (R, K) -> parts (3, R, K), LN: layer norm with weight and bias first; one warp per row, K a multiple of 4
template <bool LN>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b,
                                                         __nv_bfloat16* __restrict__ out, const int K, const float eps, const long long rows)
{
    const long long row  = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int       lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float* src = x + row * K;
    float mean = 0.0f, inv = 1.0f;
    if (LN) {
        float s = 0.0f;
        for (int c = lane * 4; c < K; c += 128) { const float4 v = ldg4(src + c); s += (v.x + v.y) + (v.z + v.w); }
        #pragma unroll
        for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(FULL, s, off);
        mean = s / (float)K;
        float q = 0.0f;
        for (int c = lane * 4; c < K; c += 128) {
            const float4 v = ldg4(src + c);
            const float d0 = v.x - mean, d1 = v.y - mean, d2 = v.z - mean, d3 = v.w - mean;
            q += (d0 * d0 + d1 * d1) + (d2 * d2 + d3 * d3);
        }
        #pragma unroll
        for (int off = 16; off > 0; off >>= 1) q += __shfl_xor_sync(FULL, q, off);
        inv = rsqrtf(q / (float)K + eps);
    }
    for (int c = lane * 4; c < K; c += 128) {
        const float4 v = ldg4(src + c);
        float y[4] = {v.x, v.y, v.z, v.w};
        if (LN) {
            const float4 w4 = ldg4(w + c), b4 = ldg4(b + c);
            y[0] = fmaf((y[0] - mean) * inv, w4.x, b4.x); y[1] = fmaf((y[1] - mean) * inv, w4.y, b4.y);
            y[2] = fmaf((y[2] - mean) * inv, w4.z, b4.z); y[3] = fmaf((y[3] - mean) * inv, w4.w, b4.w);
        }
        uint32_t lo[3], hi[3];
        split3(y[0], y[1], lo);
        split3(y[2], y[3], hi);
        #pragma unroll
        for (int i = 0; i < 3; i++) *reinterpret_cast<uint2*>(out + (i * rows + row) * K + c) = make_uint2(lo[i], hi[i]);
    }
}

// o (B, H, S, D) -> parts of (B, S, H * D); a CTA per (b, h) and run of positions, so that no thread divides but by D / 4
constexpr int SPLIT_POS = 64;
__global__ void __launch_bounds__(256) split_heads_kernel(const float* __restrict__ o, __nv_bfloat16* __restrict__ out, const int H, const int S, const int D, const int runs, const long long total)
{
    const int bh = blockIdx.x / runs, s0 = (blockIdx.x % runs) * SPLIT_POS, n = min(SPLIT_POS, S - s0), d4 = D >> 2;
    const float* src = o + ((long long)bh * S + s0) * D;
    const long long dst = (((long long)(bh / H) * S + s0) * H + bh % H) * D;
    #pragma unroll 4
    for (int i = threadIdx.x; i < n * d4; i += 256) {
        const int s = i / d4, d = (i - s * d4) * 4;
        const float4 v = ldg4(src + 4 * i);
        uint32_t lo[3], hi[3];
        split3(v.x, v.y, lo);
        split3(v.z, v.w, hi);
        #pragma unroll
        for (int p = 0; p < 3; p++) *reinterpret_cast<uint2*>(out + p * total + dst + (long long)s * H * D + d) = make_uint2(lo[p], hi[p]);
    }
}

cudaError_t launch_split_rows(const float* x, const float* w, const float* b, void* out, long long rows, int K, float eps, cudaStream_t st) {
    const unsigned grid = (unsigned)((rows + 7) / 8);
    if (w) split_rows_kernel<true><<<grid, 256, 0, st>>>(x, w, b, static_cast<__nv_bfloat16*>(out), K, eps, rows);
    else   split_rows_kernel<false><<<grid, 256, 0, st>>>(x, nullptr, nullptr, static_cast<__nv_bfloat16*>(out), K, eps, rows);
    return cudaGetLastError();
}

cudaError_t launch_split_heads(const float* o, void* out, int B, int H, int S, int D, cudaStream_t st) {
    const int runs = (S + SPLIT_POS - 1) / SPLIT_POS;
    split_heads_kernel<<<(unsigned)B * H * runs, 256, 0, st>>>(o, static_cast<__nv_bfloat16*>(out), H, S, D, runs, (long long)B * H * S * D);
    return cudaGetLastError();
}

// The current device's error word, in pinned host memory that kernels can write to: allocated at the first use, one word per device,
// for as long as the process runs.
cudaError_t linear_error_word(int** host, int** device) {
    constexpr int MAX_DEV = 64;
    static std::mutex        lock;
    static std::atomic<int*> words;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= MAX_DEV) return cudaErrorInvalidDevice;
    int* base = words.load(std::memory_order_acquire);
    if (!base) {
        std::lock_guard<std::mutex> hold(lock);
        base = words.load(std::memory_order_relaxed);
        if (!base) {
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;        // (the first call may be under capture: this allocation is not part of it)
            e = cudaThreadExchangeStreamCaptureMode(&mode);
            if (e != cudaSuccess) return e;
            void* p = nullptr;
            e = cudaHostAlloc(&p, MAX_DEV * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped);
            cudaThreadExchangeStreamCaptureMode(&mode);
            if (e != cudaSuccess) return e;
            base = static_cast<int*>(p);
            for (int i = 0; i < MAX_DEV; i++) base[i] = 0;
            words.store(base, std::memory_order_release);
        }
    }
    *host = base + dev;
    void* d = nullptr;
    e = cudaHostGetDevicePointer(&d, base, 0);
    *device = static_cast<int*>(d) + dev;
    return e;
}

// (3, rows, K) bf16 parts, boxes of `box_rows` rows x 32 columns x 3 parts with the 64-byte swizzle
static cudaError_t make_map(CUtensorMap* map, const void* base, long long rows, int K, int box_rows) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                               CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static std::atomic<void*> entry;
    void* fn = entry.load(std::memory_order_acquire);
    if (!fn) {
        cudaDriverEntryPointQueryResult found;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found);
        if (e != cudaSuccess) return e;
        if (found != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
        entry.store(fn, std::memory_order_release);
    }
    const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, PARTS}, strides[2] = {(cuuint64_t)K * 2, (cuuint64_t)K * 2 * rows};
    const cuuint32_t box[3] = {BK, (cuuint32_t)box_rows, PARTS}, one[3] = {1, 1, 1};
    const CUresult r = reinterpret_cast<Encode>(fn)(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                                    CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int EPI>
static cudaError_t launch_linear(LinearArgs g, const void* a3, const void* w3, int sms, cudaStream_t st) {
    CUtensorMap ma, mb;
    int* word;
    cudaError_t e = linear_error_word(&word, &g.error);
    if (e == cudaSuccess) e = make_map(&ma, a3, g.M, g.K, BM);
    if (e == cudaSuccess) e = make_map(&mb, w3, g.N, g.K, BN);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(linear_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LIN_SMEM);
    if (e != cudaSuccess) return e;
    const int tiles = ((g.M + BM - 1) / BM) * ((g.N + BN - 1) / BN);
    linear_kernel<EPI><<<tiles < sms ? tiles : sms, LIN_THREADS, LIN_SMEM, st>>>(ma, mb, g);
    return cudaGetLastError();
}

cudaError_t launch_linear_qkv(const void* a3, const void* w3, const float* bias, const float* table, float* q, float* k, float* v,
                              int B, int S, int H, int K, int sms, cudaStream_t st) {
    LinearArgs g{};
    g.M = B * S; g.N = 3 * H * 64; g.K = K; g.bias = bias; g.q = q; g.k = k; g.v = v;
    g.table = reinterpret_cast<const float2*>(table); g.S = S; g.H = H;
    return launch_linear<EPI_QKV>(g, a3, w3, sms, st);
}
cudaError_t launch_linear_gelu(const void* a3, const void* w3, const float* bias, void* out3, int M, int N, int K, int sms, cudaStream_t st) {
    LinearArgs g{};
    g.M = M; g.N = N; g.K = K; g.bias = bias; g.out3 = static_cast<__nv_bfloat16*>(out3);
    return launch_linear<EPI_GELU>(g, a3, w3, sms, st);
}
cudaError_t launch_linear_residual(const void* a3, const void* w3, const float* bias, float* x, int M, int N, int K, int sms, cudaStream_t st) {
    LinearArgs g{};
    g.M = M; g.N = N; g.K = K; g.bias = bias; g.x = x;
    return launch_linear<EPI_RESIDUAL>(g, a3, w3, sms, st);
}

}  // namespace qlka
