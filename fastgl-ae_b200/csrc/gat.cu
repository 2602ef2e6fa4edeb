// The attention part of a GAT layer in three launches forward and two backward (sm_100a).
//
// Replaces, for the whole of GATConv.forward behind the linear map (GraphConv.py:262-283), the score sums, the edge
// softmax that the reference takes from DGL and K12 (aggregate_acc_kernel.cu:789-885), and their backward with the
// gradient of the attention coefficients that the reference drops (GraphConv.py:227).  Op by op that is some sixty
// launches of 2 us per layer and direction (gathers, scatters, sorts of an index_put, reductions) around a few megabytes;
// a sampled block's rows have a handful of edges, so a warp keeps everything of its row to itself: scores, softmax,
// weighted sum, and on the way back the coefficient gradients, the softmax and leaky-ReLU derivatives and one vector
// reduction per edge into the source's gradient row, which carries the aggregation's and the scores' part together.
#include <algorithm>
#include <cstdint>

#include "common.cuh"

namespace fgl {

constexpr int kGatThreads = 256;
constexpr int kGatWarps = kGatThreads / 32;

struct GatParams {
    const int32_t* indptr;
    const int32_t* src;
    const float* feat;    // [n_src][dim], dim = heads * width
    const float* attn_l;  // [dim]
    const float* attn_r;
    float* el;            // [n_src][heads]
    float* er;            // [n_dst][heads]
    float* alpha;         // [n_edges][heads]
    float* out;           // forward: [n_dst][dim]
    const float* dy;      // backward: [n_dst][dim]
    float* de;            // backward: [n_edges][heads] scratch
    float* der;           // backward: [n_dst][heads] scratch
    float* dfeat;         // backward: [n_src][dim], zero on entry
    float* partial;       // backward: [CTAs][2 * dim] column sums for the two attention vectors
    int64_t ldf, ldo, ldy;
    int32_t heads, width, dim, n_dst, n_src;
    float slope;
    int32_t* status;
};

__device__ __forceinline__ float leaky(float v, float slope) { return v > 0.f ? v : v * slope; }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// el[n, h] = <feat[n, h], attn_l[h]> for every source, er likewise for the destinations (the first n_dst sources): a warp
// per node and head.
__global__ void __launch_bounds__(kGatThreads) gat_scores_kernel(const GatParams p) {
    if (!after_the_kernels_before()) return;
    const int lane = threadIdx.x & 31;
    const int64_t n_warps = (int64_t)gridDim.x * kGatWarps;
    for (int64_t u = (int64_t)blockIdx.x * kGatWarps + (threadIdx.x >> 5); u < (int64_t)p.n_src * p.heads; u += n_warps) {
        const int64_t n = u / p.heads;
        const int h = (int)(u - n * p.heads);
        const float* x = p.feat + n * p.ldf + (int64_t)h * p.width;
        const bool dst = n < p.n_dst;
        float l = 0.f, r = 0.f;
        for (int f = lane; f < p.width; f += 32) {
            const float v = __ldg(x + f);
            l = fmaf(v, __ldg(p.attn_l + h * p.width + f), l);
            if (dst) r = fmaf(v, __ldg(p.attn_r + h * p.width + f), r);
        }
        l = warp_sum(l);
        if (dst) r = warp_sum(r);
        if (lane == 0) {
            p.el[u] = l;
            if (dst) p.er[u] = r;
        }
    }
}

// Lanes of a warp over the (edge, head) pairs of a row: `span` heads (a power of two, at most 32) side by side, 32 / span
// edges at once; sums and maxima over the edges are taken across the lanes of equal head.
struct PairLanes {
    int span, head, edge, stride;
    __device__ __forceinline__ PairLanes(int heads, int lane) {
        span = 1;
        while (span < heads && span < 32) span <<= 1;
        head = lane & (span - 1);
        edge = lane / span;
        stride = 32 / span;
    }
    __device__ __forceinline__ float sum(float v) const {
        for (int o = span; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    }
    __device__ __forceinline__ float max(float v) const {
        for (int o = span; o < 32; o <<= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    }
};

template <int VEC>
struct GVec;
template <>
struct GVec<4> {
    using T = float4;
};
template <>
struct GVec<1> {
    using T = float;
};

template <int VEC>
__device__ __forceinline__ void vfma(typename GVec<VEC>::T& a, float w, const typename GVec<VEC>::T& x) {
    float* pa = reinterpret_cast<float*>(&a);
    const float* px = reinterpret_cast<const float*>(&x);
#pragma unroll
    for (int q = 0; q < VEC; ++q) pa[q] = fmaf(w, px[q], pa[q]);
}

// A warp per destination row.  An edge whose source is out of range gets the coefficient zero and is reported.
template <int VEC>
__global__ void __launch_bounds__(kGatThreads) gat_fwd_kernel(const GatParams p) {
    if (!after_the_kernels_before()) return;
    using T = typename GVec<VEC>::T;
    const int lane = threadIdx.x & 31;
    const int n_warps = gridDim.x * kGatWarps;
    const PairLanes pl(p.heads, lane);
    const int chunks = p.dim / VEC;
    for (int d = blockIdx.x * kGatWarps + (threadIdx.x >> 5); d < p.n_dst; d += n_warps) {
        const int a = __ldg(p.indptr + d), b = __ldg(p.indptr + d + 1);
        T* out = reinterpret_cast<T*>(p.out + (int64_t)d * p.ldo);
        if (a >= b) {  // no in-edges: the row's own input row, as the reference's kernel has it
            const T* x = reinterpret_cast<const T*>(p.feat + (int64_t)d * p.ldf);
            for (int c = lane; c < chunks; c += 32) out[c] = __ldg(x + c);
            continue;
        }
        for (int h0 = 0; h0 < p.heads; h0 += 32) {
            const int h = h0 + pl.head;
            const bool on = h < p.heads;
            const float er = on ? p.er[(int64_t)d * p.heads + h] : 0.f;
            float top = -INFINITY;
            for (int e = a + pl.edge; e < b; e += pl.stride) {
                const int s = __ldg(p.src + e);
                const bool ok = s >= 0 && s < p.n_src;
                if (!ok && p.status) set_status(p.status, FGL_ERR_BOUNDS);
                if (on && ok) top = fmaxf(top, leaky(p.el[(int64_t)s * p.heads + h] + er, p.slope));
            }
            top = pl.max(top);
            float sum = 0.f;
            for (int e = a + pl.edge; e < b; e += pl.stride) {
                const int s = __ldg(p.src + e);
                if (on) {
                    const float ex = (s >= 0 && s < p.n_src) ? expf(leaky(p.el[(int64_t)s * p.heads + h] + er, p.slope) - top) : 0.f;
                    p.alpha[(int64_t)e * p.heads + h] = ex;
                    sum += ex;
                }
            }
            sum = pl.sum(sum);
            for (int e = a + pl.edge; e < b; e += pl.stride)
                if (on) p.alpha[(int64_t)e * p.heads + h] = sum > 0.f ? p.alpha[(int64_t)e * p.heads + h] / sum : 0.f;
        }
        __syncwarp();  // the coefficients are read by other lanes than wrote them
        for (int c = lane; c < chunks; c += 32) {
            const int h = (c * VEC) / p.width;
            T acc{};
            constexpr int U = 4;
            for (int e = a; e < b; e += U) {
                T v[U];
                float w[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int k = min(e + u, b - 1);
                    const int s = __ldg(p.src + k);
                    w[u] = p.alpha[(int64_t)k * p.heads + h];
                    v[u] = __ldg(reinterpret_cast<const T*>(p.feat + (int64_t)((s >= 0 && s < p.n_src) ? s : 0) * p.ldf) + c);
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (e + u < b) vfma<VEC>(acc, w[u], v[u]);
            }
            out[c] = acc;
        }
    }
}

// A warp per destination row: coefficient gradients, softmax and leaky-ReLU backward, then per edge one vector reduction
// into the source's row.  The gradients of the attention vectors are column sums over all rows: every CTA adds its rows'
// up in shared memory and leaves one row of `partial`.
template <int VEC>
__global__ void __launch_bounds__(kGatThreads) gat_bwd_kernel(const GatParams p) {
    if (!after_the_kernels_before()) return;
    using T = typename GVec<VEC>::T;
    extern __shared__ float cols[];  // [2 * dim]: attn_l's columns, then attn_r's
    const int lane = threadIdx.x & 31;
    const int n_warps = gridDim.x * kGatWarps;
    const PairLanes pl(p.heads, lane);
    const int chunks = p.dim / VEC;
    for (int i = threadIdx.x; i < 2 * p.dim; i += kGatThreads) cols[i] = 0.f;
    __syncthreads();
    for (int d = blockIdx.x * kGatWarps + (threadIdx.x >> 5); d < p.n_dst; d += n_warps) {
        const int a = __ldg(p.indptr + d), b = __ldg(p.indptr + d + 1);
        if (a >= b) continue;  // as the reference's backward: no gradient through a row without in-edges
        const float* dy = p.dy + (int64_t)d * p.ldy;
        // <dy[d, h], feat[src, h]> for every edge and head: the whole row at a time where a head is 1, 2, 4 .. 32 lanes' vectors
        // (eight heads of 32 columns: an eighth of the rounds), else head by head
        const int seg = p.width / VEC;
        const bool whole = seg * VEC == p.width && seg <= 32 && (seg & (seg - 1)) == 0;
        for (int c0 = 0; whole && c0 < chunks; c0 += 32) {
            const int c = c0 + lane;
            const bool in = c < chunks;
            T g{};
            if (in) g = __ldg(reinterpret_cast<const T*>(dy) + c);
            constexpr int U = 4;
            for (int e = a; e < b; e += U) {
                T x[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int s = __ldg(p.src + min(e + u, b - 1));
                    const bool ok = s >= 0 && s < p.n_src;
                    if (!ok && p.status && e + u < b) set_status(p.status, FGL_ERR_BOUNDS);
                    x[u] = __ldg(reinterpret_cast<const T*>(p.feat + (int64_t)(ok ? s : 0) * p.ldf) + (in ? c : 0));
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    float v = 0.f;
#pragma unroll
                    for (int q = 0; q < VEC; ++q) v = fmaf(reinterpret_cast<const float*>(&g)[q], reinterpret_cast<const float*>(&x[u])[q], v);
                    for (int o = 1; o < seg; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    if (in && (lane & (seg - 1)) == 0 && e + u < b) p.de[(int64_t)(e + u) * p.heads + c / seg] = v;
                }
            }
        }
        for (int h = 0; !whole && h < p.heads; ++h) {
            constexpr int U = 4;
            for (int e = a; e < b; e += U) {
                float v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int s = __ldg(p.src + min(e + u, b - 1));
                    const bool ok = s >= 0 && s < p.n_src;
                    if (!ok && p.status && e + u < b) set_status(p.status, FGL_ERR_BOUNDS);
                    const float* x = p.feat + (int64_t)(ok ? s : 0) * p.ldf + (int64_t)h * p.width;
                    v[u] = 0.f;
                    for (int f = lane; f < p.width; f += 32) v[u] = fmaf(__ldg(dy + (int64_t)h * p.width + f), __ldg(x + f), v[u]);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = warp_sum(v[u]);
                if (lane < U && e + lane < b) p.de[(int64_t)(e + lane) * p.heads + h] = lane == 0 ? v[0] : lane == 1 ? v[1] : lane == 2 ? v[2] : v[3];
            }
        }
        __syncwarp();
        for (int h0 = 0; h0 < p.heads; h0 += 32) {
            const int h = h0 + pl.head;
            const bool on = h < p.heads;
            float dot = 0.f;
            for (int e = a + pl.edge; e < b; e += pl.stride)
                if (on) dot = fmaf(p.alpha[(int64_t)e * p.heads + h], p.de[(int64_t)e * p.heads + h], dot);
            dot = pl.sum(dot);
            const float er = on ? p.er[(int64_t)d * p.heads + h] : 0.f;
            float sum = 0.f;
            for (int e = a + pl.edge; e < b; e += pl.stride) {
                const int s = __ldg(p.src + e);
                if (on && s >= 0 && s < p.n_src) {
                    float g = p.alpha[(int64_t)e * p.heads + h] * (p.de[(int64_t)e * p.heads + h] - dot);
                    if (!(p.el[(int64_t)s * p.heads + h] + er > 0.f)) g *= p.slope;
                    p.de[(int64_t)e * p.heads + h] = g;
                    sum += g;
                }
            }
            sum = pl.sum(sum);
            if (on && pl.edge == 0) p.der[(int64_t)d * p.heads + h] = sum;
        }
        __syncwarp();
        for (int c = lane; c < chunks; c += 32) {
            const int h = (c * VEC) / p.width;
            const T g = __ldg(reinterpret_cast<const T*>(dy) + c);
            const T al = __ldg(reinterpret_cast<const T*>(p.attn_l) + c);
            T sum_l{};
            constexpr int U = 4;
            for (int e = a; e < b; e += U) {
                int s[U];
                float w[U], q[U];
                T x[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int k = min(e + u, b - 1);
                    s[u] = __ldg(p.src + k);
                    if (s[u] < 0 || s[u] >= p.n_src || e + u >= b) s[u] = -1;
                    w[u] = p.alpha[(int64_t)k * p.heads + h];
                    q[u] = p.de[(int64_t)k * p.heads + h];
                    x[u] = __ldg(reinterpret_cast<const T*>(p.feat + (int64_t)max(s[u], 0) * p.ldf) + c);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (s[u] < 0) continue;
                    T v{};
                    vfma<VEC>(v, w[u], g);
                    vfma<VEC>(v, q[u], al);
                    atomicAdd(reinterpret_cast<T*>(p.dfeat + (int64_t)s[u] * p.dim) + c, v);
                    vfma<VEC>(sum_l, q[u], x[u]);
                }
            }
            const float r = p.der[(int64_t)d * p.heads + h];
            T v{}, sum_r{};
            vfma<VEC>(v, r, __ldg(reinterpret_cast<const T*>(p.attn_r) + c));
            atomicAdd(reinterpret_cast<T*>(p.dfeat + (int64_t)d * p.dim) + c, v);
            vfma<VEC>(sum_r, r, __ldg(reinterpret_cast<const T*>(p.feat + (int64_t)d * p.ldf) + c));
            const float* pl_ = reinterpret_cast<const float*>(&sum_l);
            const float* pr_ = reinterpret_cast<const float*>(&sum_r);
#pragma unroll
            for (int q = 0; q < VEC; ++q) {
                atomicAdd(cols + c * VEC + q, pl_[q]);
                atomicAdd(cols + p.dim + c * VEC + q, pr_[q]);
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * p.dim; i += kGatThreads) p.partial[(int64_t)blockIdx.x * 2 * p.dim + i] = cols[i];
}

// Column sums of [n_rows][n_cols]: a CTA per 32 columns, its warps take every eighth row each.
__global__ void __launch_bounds__(kGatThreads) column_sums_kernel(const float* __restrict__ x, int n_rows, int n_cols, float* __restrict__ out) {
    if (!after_the_kernels_before()) return;
    __shared__ float part[kGatWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + lane;
    float t = 0.f;
    if (c < n_cols)
        for (int r = warp; r < n_rows; r += kGatWarps) t += x[(int64_t)r * n_cols + c];
    part[warp][lane] = t;
    __syncthreads();
    if (warp == 0 && c < n_cols) {
        t = 0.f;
#pragma unroll
        for (int w = 0; w < kGatWarps; ++w) t += part[w][lane];
        out[c] = t;
    }
}

static bool vec4_rows(int dim, int width, const void* a, int64_t lda, const void* b, int64_t ldb, const void* c, const void* d) {
    return width % 4 == 0 && dim % 4 == 0 && lda % 4 == 0 && ldb % 4 == 0 &&
           (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d) & 15) == 0;
}

constexpr int kGatMaxDim = 24 * 1024;  // two rows of column sums in shared memory

}  // namespace fgl

using namespace fgl;

extern "C" {

int fgl_gat_fwd(fgl_ws* ws, const int32_t* indptr, const int32_t* src, const float* feat, int64_t ldf, const float* attn_l,
                const float* attn_r, int32_t heads, int32_t width, int32_t n_dst, int32_t n_src, float slope, float* el, float* er,
                float* alpha, float* out, int64_t ldo, void* stream) {
    if (!ws || heads < 1 || width < 1 || (int64_t)heads * width > 0x7fffffffLL || n_dst < 0 || n_src < n_dst || ldf < (int64_t)heads * width ||
        ldo < (int64_t)heads * width)
        return FGL_ERR_INVALID;
    if (n_dst == 0) return FGL_OK;
    if (!indptr || !feat || !attn_l || !attn_r || !el || !er || !out) return FGL_ERR_INVALID;
    GatParams p{};
    p.indptr = indptr;
    p.src = src;
    p.feat = feat;
    p.attn_l = attn_l;
    p.attn_r = attn_r;
    p.el = el;
    p.er = er;
    p.alpha = alpha;
    p.out = out;
    p.ldf = ldf;
    p.ldo = ldo;
    p.heads = heads;
    p.width = width;
    p.dim = heads * width;
    p.n_dst = n_dst;
    p.n_src = n_src;
    p.slope = slope;
    p.status = ws->status;
    DeviceGuard guard(ws->device);
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t cap = (int64_t)ws->sm_count * 8;
    const int score_grid = (int)std::min<int64_t>(((int64_t)n_src * heads + kGatWarps - 1) / kGatWarps, cap);
    launch(gat_scores_kernel, score_grid, kGatThreads, 0, st, p);
    const int grid = (int)std::min<int64_t>(((int64_t)n_dst + kGatWarps - 1) / kGatWarps, cap);
    if (vec4_rows(p.dim, width, feat, ldf, out, ldo, nullptr, nullptr))
        launch(gat_fwd_kernel<4>, grid, kGatThreads, 0, st, p);
    else
        launch(gat_fwd_kernel<1>, grid, kGatThreads, 0, st, p);
    return cudaGetLastError() == cudaSuccess ? FGL_OK : FGL_ERR_CUDA;
}

int fgl_gat_bwd_partials(fgl_ws* ws, int32_t heads, int32_t width, int32_t n_dst) {
    if (!ws || heads < 1 || width < 1 || (int64_t)heads * width > kGatMaxDim) return 0;
    return (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)n_dst + kGatWarps - 1) / kGatWarps, (int64_t)ws->sm_count * 2));
}

int fgl_gat_bwd(fgl_ws* ws, const int32_t* indptr, const int32_t* src, const float* feat, int64_t ldf, const float* attn_l,
                const float* attn_r, const float* el, const float* er, const float* alpha, const float* dy, int64_t ldy, int32_t heads,
                int32_t width, int32_t n_dst, int32_t n_src, int64_t n_edges, float slope, float* scratch, float* dfeat, float* dattn,
                void* stream) {
    const int grid = fgl_gat_bwd_partials(ws, heads, width, n_dst);
    if (grid == 0 || n_dst < 0 || n_src < n_dst || n_edges < 0 || ldf < (int64_t)heads * width || ldy < (int64_t)heads * width)
        return FGL_ERR_INVALID;
    if (!scratch || !dattn || (n_src > 0 && !dfeat) || (n_dst > 0 && (!indptr || !feat || !dy || !attn_l || !attn_r || !el || !er)))
        return FGL_ERR_INVALID;
    GatParams p{};
    p.indptr = indptr;
    p.src = src;
    p.feat = feat;
    p.attn_l = attn_l;
    p.attn_r = attn_r;
    p.el = const_cast<float*>(el);
    p.er = const_cast<float*>(er);
    p.alpha = const_cast<float*>(alpha);
    p.dy = dy;
    p.dim = heads * width;
    p.partial = scratch;  // first: its rows are not vectors, but every part that follows is read by element as well
    p.de = p.partial + (int64_t)grid * 2 * p.dim;
    p.der = p.de + n_edges * heads;
    p.dfeat = dfeat;
    p.ldf = ldf;
    p.ldy = ldy;
    p.heads = heads;
    p.width = width;
    p.n_dst = n_dst;
    p.n_src = n_src;
    p.slope = slope;
    p.status = ws->status;
    DeviceGuard guard(ws->device);
    cudaStream_t st = (cudaStream_t)stream;
    if (n_src > 0) FGL_CUDA_OK(ws, cudaMemsetAsync(dfeat, 0, sizeof(float) * (size_t)n_src * p.dim, st));
    const size_t dyn = sizeof(float) * 2 * (size_t)p.dim;
    const bool vec = vec4_rows(p.dim, width, feat, ldf, dy, ldy, attn_l, attn_r) && ((uintptr_t)dfeat & 15) == 0;
    void (*kernel)(const GatParams) = vec ? gat_bwd_kernel<4> : gat_bwd_kernel<1>;
    if (dyn > 48 * 1024) FGL_CUDA_OK(ws, cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
    launch(kernel, grid, kGatThreads, dyn, st, p);
    launch(column_sums_kernel, (2 * p.dim + 31) / 32, kGatThreads, 0, st, p.partial, grid, 2 * p.dim, dattn);
    return cudaGetLastError() == cudaSuccess ? FGL_OK : FGL_ERR_CUDA;
}

}  // extern "C"
