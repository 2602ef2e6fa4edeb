// Weight gradients of the dense layers, C [m][n] = A^T B over k rows, in float32 on the FMA units (sm_100a).
//
// A weight gradient contracts over the rows of a mini-batch's layer -- 10^3 to 10^5 -- into an output of a few tiles.  cuBLAS's
// float32 kernels put one 64 x 64 tile on a CTA and do not cut the contraction, or cut it a little: 1 to 20 TFLOP/s.  Here it is
// cut over as many CTAs as fill the chip, every slice leaves its partial product in scratch and a second launch adds the slices
// in a fixed order (the same bits every run; partial sums over shorter runs round less: 2 to 4e-7 of the largest entry where
// cuBLAS has 4e-7 to 1.7e-6).  Before and after, m x n over k rows: 602 x 256 over 10073 114 -> 79 us (39 TFLOP/s), 100 x 64
// over 177148 268 -> 84 us, 64 x 64 over 42209 118 -> 19 us, 256 x 41 over 1024 10 -> 5 us.  (The layers' other products, whose
// rows are many and whose contraction is short, stay with cuBLAS, which runs them as fast as this kernel does: 30 to 40.)
//
// A thread owns an 8 x TN block of its CTA's BM x BN tile (as two halves 4 rows and 4 columns wide, so that a warp's
// shared-memory reads are broadcasts and whole 128-byte rows) and multiplies two columns per instruction.  The k-slab that the
// next iteration reads travels through registers while the current one is multiplied.  Operands may have any width and any
// leading dimension; 16-byte loads are used where the width and the base allow it.
#include <algorithm>
#include <cstdint>

#include "common.cuh"

namespace fgl {

constexpr int kBK = 16;

struct GemmParams {
    const float* a;
    const float* b;
    float* c;        // [m][n], or the slices' partial products [slices][m][n]
    int64_t lda, ldb, ldc;
    int m, n, k;
    int k_slice;     // contraction range of a slice, a multiple of kBK
    int64_t slice_stride;
};

// Two float32 multiply-adds in one instruction (each rounded as fmaf rounds): half the issue slots of the inner loop.
__device__ __forceinline__ unsigned long long pair(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void unpair(unsigned long long v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ void fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

// A kBK x W slab (W = BM or BN) of an operand on its way through registers; both operands are contiguous along W.
template <int W, int THREADS, bool VEC>
struct Slab {
    static constexpr int kVecs = (kBK * W / 4 + THREADS - 1) / THREADS;
    static_assert((kBK * W / 4) % THREADS == 0, "whole vectors per thread");
    float4 v[kVecs];

    __device__ __forceinline__ void load(const float* __restrict__ p, int64_t ld, int w0, int w_end, int k0, int k_end) {
#pragma unroll
        for (int i = 0; i < kVecs; ++i) {
            const int u = (int)threadIdx.x + i * THREADS;
            const int k = k0 + u / (W / 4), w = w0 + (u % (W / 4)) * 4;
            v[i] = fetch(p + (int64_t)k * ld + w, k < k_end ? w_end - w : 0);
        }
    }
    static __device__ __forceinline__ float4 fetch(const float* p, int left) {  // `left` elements are inside
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (VEC) {
            if (left > 0) r = __ldg(reinterpret_cast<const float4*>(p));
        } else {
            if (left > 0) r.x = __ldg(p);
            if (left > 1) r.y = __ldg(p + 1);
            if (left > 2) r.z = __ldg(p + 2);
            if (left > 3) r.w = __ldg(p + 3);
        }
        return r;
    }
    __device__ __forceinline__ void store(float (*s)[W + 4]) const {
#pragma unroll
        for (int i = 0; i < kVecs; ++i) {
            const int u = (int)threadIdx.x + i * THREADS;
            *reinterpret_cast<float4*>(&s[u / (W / 4)][(u % (W / 4)) * 4]) = v[i];
        }
    }
};

template <int BM, int BN, int TN, bool VA, bool VB>
__global__ void __launch_bounds__(BM / 8 * (BN / TN)) gemm_kernel(const GemmParams p) {
    if (!after_the_kernels_before()) return;
    constexpr int kThreads = BM / 8 * (BN / TN);
    constexpr int kCols = BN / TN;  // threads side by side
    __shared__ __align__(16) float sa[2][kBK][BM + 4];
    __shared__ __align__(16) float sb[2][kBK][BN + 4];
    const int tx = threadIdx.x % kCols, ty = threadIdx.x / kCols;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int k_lo = blockIdx.z * p.k_slice, k_hi = min(p.k, k_lo + p.k_slice);
    Slab<BM, kThreads, VA> ra;
    Slab<BN, kThreads, VB> rb;
    unsigned long long acc[8][TN / 2];  // pairs of neighbouring columns
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
    ra.load(p.a, p.lda, m0, p.m, k_lo, k_hi);
    rb.load(p.b, p.ldb, n0, p.n, k_lo, k_hi);
    int buf = 0;
    for (int k0 = k_lo; k0 < k_hi; k0 += kBK) {
        ra.store(sa[buf]);
        rb.store(sb[buf]);
        __syncthreads();
        if (k0 + kBK < k_hi) {
            ra.load(p.a, p.lda, m0, p.m, k0 + kBK, k_hi);
            rb.load(p.b, p.ldb, n0, p.n, k0 + kBK, k_hi);
        }
#pragma unroll
        for (int kk = 0; kk < kBK; ++kk) {
            float fa[8];
            unsigned long long fb[TN / 2];
            *reinterpret_cast<float4*>(fa) = *reinterpret_cast<const float4*>(&sa[buf][kk][ty * 4]);
            *reinterpret_cast<float4*>(fa + 4) = *reinterpret_cast<const float4*>(&sa[buf][kk][BM / 2 + ty * 4]);
#pragma unroll
            for (int j = 0; j < TN; j += 4)
                *reinterpret_cast<ulonglong2*>(fb + j / 2) = *reinterpret_cast<const ulonglong2*>(&sb[buf][kk][j / 4 * (kCols * 4) + tx * 4]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const unsigned long long aa = pair(fa[i], fa[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], aa, fb[j]);
            }
        }
        buf ^= 1;
    }
    float* c = p.c + (int64_t)blockIdx.z * p.slice_stride;
    const bool vec = p.ldc % 4 == 0 && ((uintptr_t)c & 15) == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = m0 + (i < 4 ? ty * 4 + i : BM / 2 + ty * 4 + i - 4);
        if (row >= p.m) continue;
#pragma unroll
        for (int j = 0; j < TN; j += 4) {
            const int col = n0 + j / 4 * (kCols * 4) + tx * 4;
            float* to = c + (int64_t)row * p.ldc + col;
            float4 v;
            unpair(acc[i][j / 2], v.x, v.y);
            unpair(acc[i][j / 2 + 1], v.z, v.w);
            if (vec && col + 3 < p.n) {
                *reinterpret_cast<float4*>(to) = v;
            } else {
                const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (col + q < p.n) to[q] = e[q];
            }
        }
    }
}

// C = sum of the slices in a fixed order: lane l of every warp has the l-th group of VEC elements of the CTA, warp w adds the
// slices w, w + 8, ..., and the eight partial sums meet in shared memory.
constexpr int kFoldThreads = 256;

template <int VEC>
__global__ void __launch_bounds__(kFoldThreads) gemm_fold_kernel(const float* __restrict__ part, int slices, int64_t slice_stride, int m, int n,
                                                                 float* __restrict__ c, int64_t ldc) {
    if (!after_the_kernels_before()) return;
    __shared__ float s[kFoldThreads / 32][32 * VEC];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t at = ((int64_t)blockIdx.x * 32 + lane) * VEC, total = (int64_t)m * n;
    float t[VEC] = {};
    if (at < total) {
        for (int s0 = warp; s0 < slices; s0 += 4 * (kFoldThreads / 32)) {
            float v[4][VEC];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int sl = s0 + u * (kFoldThreads / 32);
#pragma unroll
                for (int q = 0; q < VEC; ++q) v[u][q] = 0.f;
                if (sl < slices) {
                    const float* from = part + (int64_t)sl * slice_stride + at;
                    if (VEC == 4)
                        *reinterpret_cast<float4*>(v[u]) = __ldg(reinterpret_cast<const float4*>(from));
                    else
                        v[u][0] = __ldg(from);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int q = 0; q < VEC; ++q) t[q] += v[u][q];
        }
    }
#pragma unroll
    for (int q = 0; q < VEC; ++q) s[warp][lane * VEC + q] = t[q];
    __syncthreads();
    for (int i = threadIdx.x; i < 32 * VEC; i += kFoldThreads) {
        const int64_t e = (int64_t)blockIdx.x * 32 * VEC + i;
        if (e >= total) continue;
        float r = 0.f;
#pragma unroll
        for (int w = 0; w < kFoldThreads / 32; ++w) r += s[w][i];
        c[e / n * ldc + e % n] = r;
    }
}

struct GemmPlan {
    int bm, bn, slices, k_slice;
};

// The tile and the split of a shape.  Outputs of a few thousand elements and products below 10^8 operations are bound by the
// length of a CTA's chain of slabs: tiles of 64 x 32, cut until there are two CTAs per SM, down to two slabs a slice.  The others
// are bound by the FMA units: tiles of 128 x 64 and up to four CTAs per SM, slices of at least 64 terms (below that, storing and
// folding a slice's tile costs more than computing it).
static GemmPlan plan_gemm(int sms, int m, int n, int k) {
    GemmPlan g{};
    const bool small = (int64_t)m * n <= 64 * 64 || 2.0 * m * n * k < 1e8;
    g.bm = small ? 64 : 128;
    g.bn = small ? 32 : 64;
    const int64_t tiles = (int64_t)((m + g.bm - 1) / g.bm) * ((n + g.bn - 1) / g.bn);
    const int64_t want = (int64_t)sms * (small ? 2 : 4);
    const int64_t slices = std::max<int64_t>(1, std::min<int64_t>(want / tiles, k / (small ? 32 : 64)));
    g.k_slice = (int)((((int64_t)k + slices - 1) / slices + kBK - 1) / kBK * kBK);
    g.slices = (k + g.k_slice - 1) / g.k_slice;
    return g;
}

template <int BM, int BN, int TN>
static void launch_gemm(const GemmParams& p, dim3 grid, bool va, bool vb, cudaStream_t st) {
    constexpr int threads = BM / 8 * (BN / TN);
    if (va && vb) launch(gemm_kernel<BM, BN, TN, true, true>, grid, threads, 0, st, p);
    else if (va) launch(gemm_kernel<BM, BN, TN, true, false>, grid, threads, 0, st, p);
    else if (vb) launch(gemm_kernel<BM, BN, TN, false, true>, grid, threads, 0, st, p);
    else launch(gemm_kernel<BM, BN, TN, false, false>, grid, threads, 0, st, p);
}

static void launch_gemm_tile(const GemmPlan& g, const GemmParams& p, dim3 grid, bool va, bool vb, cudaStream_t st) {
    if (g.bm == 128) launch_gemm<128, 64, 8>(p, grid, va, vb, st);
    else launch_gemm<64, 32, 4>(p, grid, va, vb, st);
}

static void gemm_with(const GemmPlan& g, const float* a, int64_t lda, const float* b, int64_t ldb, float* c,
                      int64_t ldc, int m, int n, int k, float* scratch, cudaStream_t st) {
    const bool split = g.slices > 1;
    GemmParams p{};
    p.a = a;
    p.b = b;
    p.c = split ? scratch : c;
    p.lda = lda;
    p.ldb = ldb;
    p.ldc = split ? n : ldc;
    p.m = m;
    p.n = n;
    p.k = k;
    p.k_slice = g.k_slice;
    p.slice_stride = (int64_t)m * n;
    const dim3 grid((m + g.bm - 1) / g.bm, (n + g.bn - 1) / g.bn, g.slices);
    auto vec = [](const float* x, int64_t ld, int contiguous) { return ld % 4 == 0 && contiguous % 4 == 0 && ((uintptr_t)x & 15) == 0; };
    launch_gemm_tile(g, p, grid, vec(a, lda, m), vec(b, ldb, n), st);
    if (split) {
        const int64_t mn = (int64_t)m * n;
        if (mn % 4 == 0 && ((uintptr_t)scratch & 15) == 0)
            launch(gemm_fold_kernel<4>, (unsigned)((mn / 4 + 31) / 32), kFoldThreads, 0, st, scratch, g.slices, p.slice_stride, m, n, c, ldc);
        else
            launch(gemm_fold_kernel<1>, (unsigned)((mn + 31) / 32), kFoldThreads, 0, st, scratch, g.slices, p.slice_stride, m, n, c, ldc);
    }
}

}  // namespace fgl

using namespace fgl;

extern "C" {

int64_t fgl_weight_grad_scratch(fgl_ws* ws, int32_t m, int32_t n, int32_t k) {
    if (!ws || m < 1 || n < 1 || k < 1) return 0;
    const GemmPlan g = plan_gemm(ws->sm_count, m, n, k);
    return g.slices > 1 ? (int64_t)g.slices * m * n : 0;
}

int fgl_weight_grad(fgl_ws* ws, int32_t m, int32_t n, int32_t k, const float* x, int64_t ldx, const float* dy, int64_t ldy, float* dw,
                    int64_t ldw, float* scratch, void* stream) {
    if (!ws || m < 0 || n < 0 || k < 0 || ldx < m || ldy < n || ldw < n) return FGL_ERR_INVALID;
    if (m == 0 || n == 0) return FGL_OK;
    if (!dw || (k > 0 && (!x || !dy))) return FGL_ERR_INVALID;
    DeviceGuard guard(ws->device);
    cudaStream_t st = (cudaStream_t)stream;
    if (k == 0) {
        FGL_CUDA_OK(ws, cudaMemset2DAsync(dw, sizeof(float) * (size_t)ldw, 0, sizeof(float) * (size_t)n, (size_t)m, st));
        return FGL_OK;
    }
    const GemmPlan g = plan_gemm(ws->sm_count, m, n, k);
    if (g.slices > 1 && !scratch) return FGL_ERR_INVALID;
    if ((n + g.bn - 1) / g.bn > 65535 || (int64_t)m * n > (1LL << 36)) return FGL_ERR_INVALID;
    gemm_with(g, x, ldx, dy, ldy, dw, ldw, m, n, k, scratch, st);
    FGL_CUDA_OK(ws, cudaGetLastError());
    return FGL_OK;
}

}  // extern "C"
