// Sum / mean / sym-norm aggregation over a block CSR, forward (gather) and backward (scatter), sm_100a.
//
// The work is HBM-bound (one FMA per 4 bytes read), so no tensor cores: a warp owns one destination row,
// its lanes sweep the feature dimension with 128-bit loads (64- or 32-bit when the row stride is not a
// multiple of 16 bytes, e.g. 602 floats), the neighbour ids of the row are read once, coalesced, and handed
// round by shuffle, the loads of several neighbours are issued before the first FMA, the ids of the warp's
// next row are fetched while the current row is summed, and the row's sum stays in registers until one
// coalesced store.  The number of accumulators is a template parameter chosen from
// the row width, so narrow rows (100 / 128 floats) run with few registers and full occupancy.
//
// The forward kernel also runs over a whole window of mini-batches (per-batch strides, rows in batch-major
// order), so the first layer of the window -- which reads only the feature table and does not depend on the
// weights -- is one launch that is long enough to reach a steady state.
//
// Replaces K8 / K10 (aggregate_acc_kernel.cu:271-331, :376-427: 8 rows x 4 floats per warp, shared-memory
// read-modify-write per neighbour) and K9 / K11 (:468-517, :555-596: scalar atomics, the GCN one built from
// two atomicExch in a retry loop).
#include <algorithm>
#include <atomic>

#include <cooperative_groups.h>

#include "common.cuh"

namespace fgl {

#ifndef FGL_AGG_THREADS
#define FGL_AGG_THREADS 256
#endif
constexpr int kAggThreads = FGL_AGG_THREADS;
constexpr int kAggWarps = kAggThreads / 32;
#ifndef FGL_AGG_UNR1
#define FGL_AGG_UNR1 8  // neighbour rows in flight per lane for rows of up to 32 vectors
#endif
#ifndef FGL_AGG_MIN_CTAS
#define FGL_AGG_MIN_CTAS 2
#endif

template <int VEC>
struct Vec;
template <>
struct Vec<4> {
    using T = float4;
    static __device__ __forceinline__ T zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
    static __device__ __forceinline__ void fma(T& a, float w, const T& x) {
        a.x = fmaf(w, x.x, a.x);
        a.y = fmaf(w, x.y, a.y);
        a.z = fmaf(w, x.z, a.z);
        a.w = fmaf(w, x.w, a.w);
    }
    static __device__ __forceinline__ T scale(const T& a, float w) { return make_float4(a.x * w, a.y * w, a.z * w, a.w * w); }
};
template <>
struct Vec<2> {
    using T = float2;
    static __device__ __forceinline__ T zero() { return make_float2(0.f, 0.f); }
    static __device__ __forceinline__ void fma(T& a, float w, const T& x) {
        a.x = fmaf(w, x.x, a.x);
        a.y = fmaf(w, x.y, a.y);
    }
    static __device__ __forceinline__ T scale(const T& a, float w) { return make_float2(a.x * w, a.y * w); }
};
template <>
struct Vec<1> {
    using T = float;
    static __device__ __forceinline__ T zero() { return 0.f; }
    static __device__ __forceinline__ void fma(T& a, float w, const T& x) { a = fmaf(w, x, a); }
    static __device__ __forceinline__ T scale(const T& a, float w) { return a * w; }
};

struct AggParams {
    const int32_t* indptr;
    const int32_t* src;
    const int32_t* src_deg;
    const int32_t* dst_deg;
    const int32_t* row_map;
    const float* x;  // forward: input rows; backward: dy
    float* out;      // forward: out; backward: dx
    float* self_out; // forward, optional: copy of the row's own input row x[row(d)]
    int64_t ldx, ldo, ld_self;
    int32_t dim, n_dst, n_src;
    int32_t passthrough;
    // window forward: all zero / NULL for a single block
    int64_t indptr_stride, src_stride, row_map_stride;
    int32_t n_batches;
    const int64_t* out_row_off;  // [n_batches + 1]: first output row of batch b, then the total
    const int32_t* counts;       // or: rows of batch b at counts[b * counts_stride]
    int64_t counts_stride;
    // optional: the real number of destination rows, read on the device (n_dst is then the padded row count
    // the launch is sized for; forward rows beyond the real count are zero-filled)
    const int32_t* n_dst_dev;
    // optional: x is row-sharded over several tables (one per GPU, peer-mapped); global row r lives in
    // shards[r / rows_per_shard] at local row r % rows_per_shard
    const float* const* shards;
    int64_t rows_per_shard;
    // FGL_AGG_EDGE: one weight per (edge, head), edge_w[e * n_heads + h]; head h covers dim / n_heads columns
    const float* edge_w;
    int32_t n_heads;
    // bounds of the ids the kernels dereference: x (or the sharded table) has n_rows rows; with a row map the local
    // ids index a map of n_map entries.  An id outside its range is never dereferenced: the edge (or the gathered
    // row) contributes zeros and FGL_ERR_BOUNDS goes to *status (may be NULL).
    int64_t n_rows;
    int64_t n_map;
    int32_t* status;
    // forward, optional: the result (also) as TF32 parts, [hi | lo] or [hi | lo | hi] split_stride columns apart
    float* split;
    int64_t ld_split, split_stride;
    int32_t split_blocks;
    // backward, optional: a self gradient that is added to dx[d] as one more edge of row d
    const float* dy_self;
    int64_t ld_dy_self;
};

__device__ __forceinline__ void agg_bad_id(const AggParams& p) {
    if (p.status) set_status(p.status, FGL_ERR_BOUNDS);
}

// Row of x that local id s stands for, or -1 (recorded) when s or the mapped row is out of range.
template <bool HAS_MAP>
__device__ __forceinline__ int64_t checked_row(const AggParams& p, const int32_t* row_map, int s) {
    int64_t r = (int64_t)s;
    if (HAS_MAP) {
        if (s < 0 || (int64_t)s >= p.n_map) {
            agg_bad_id(p);
            return -1;
        }
        r = (int64_t)__ldg(row_map + s);
    }
    if (r < 0 || r >= p.n_rows) {
        agg_bad_id(p);
        return -1;
    }
    return r;
}

// Start of input row r: in the single table, or in the shard (possibly another GPU's HBM, read with plain
// peer loads over NVLink) that owns it.
__device__ __forceinline__ const float* x_row(const AggParams& p, int64_t r) {
    if (p.shards == nullptr) return p.x + r * p.ldx;
    const int64_t s = r / p.rows_per_shard;
    return p.shards[s] + (r - s * p.rows_per_shard) * p.ldx;
}

constexpr int kAggMaxWindow = 512;  // mini-batches per window launch (their row offsets are staged in shared memory)

// First output row of every mini-batch of the window, into shared memory.
__device__ __forceinline__ void window_offsets(const AggParams& p, long long* s_off) {
    if (p.counts == nullptr) {
        for (int i = threadIdx.x; i <= p.n_batches; i += blockDim.x) s_off[i] = __ldg(p.out_row_off + i);
    } else if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        long long before = 0;
        for (int b0 = 0; b0 < p.n_batches; b0 += 32) {
            const int n = b0 + lane < p.n_batches ? max(__ldg(p.counts + (int64_t)(b0 + lane) * p.counts_stride), 0) : 0;
            const int incl = warp_incl_scan(n, lane);
            if (b0 + lane < p.n_batches) s_off[b0 + lane] = before + incl - n;
            before += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) s_off[p.n_batches] = before;
    }
    __syncthreads();
}

// Forward: out[d,:] = scale_d * sum_e w_e * x[row(src[e]),:]
// NACC vector accumulators per lane cover 32 * NACC * VEC floats per pass; UNR neighbours' loads are in
// flight before their FMAs.  In window mode (out_row_off != NULL) the rows of all mini-batches form one
// sequence in batch-major order and the grid sweeps it front to back, so that at any moment the CTAs work
// on one or two mini-batches and the rows those batches re-read stay in L2.
//
// A warp issues its instructions in order, so a value that was just requested from memory stalls the warp at its
// first use.  The ids of a row form a dependent chain -- indptr[d] -> src[a + lane] -> row_map[s] -> the feature
// rows -- and walked one row at a time that chain is four round trips per destination row, more than the row data
// itself costs.  The chain is therefore software-pipelined over the warp's rows: while row i is summed, the map
// entries of row i+1, the source ids of row i+2 and the offsets of row i+3 are in flight, and every loaded value is
// first touched one iteration after it was requested.  The row's own input row (the "self" copy) is requested
// together with the first batch of neighbour rows, not before it.
//
// SPLIT: the result leaves as the TF32 parts that an error-compensated product reads ([hi | lo | hi], see split_tf32_kernel),
// beside or instead of the plain rows, so that no pass of its own reads the rows again to split them.
template <int VEC, bool SPLIT>
__device__ __forceinline__ void put_out(const AggParams& p, int64_t row, int c, const typename Vec<VEC>::T& v) {
    using T = typename Vec<VEC>::T;
    if (!SPLIT || p.out) reinterpret_cast<T*>(p.out + row * p.ldo)[c] = v;
    if (SPLIT) {
        T h, l;
#pragma unroll
        for (int q = 0; q < VEC; ++q) {
            const float x = reinterpret_cast<const float*>(&v)[q], xh = to_tf32(x);
            reinterpret_cast<float*>(&h)[q] = xh;
            reinterpret_cast<float*>(&l)[q] = to_tf32(x - xh);
        }
        float* s = p.split + row * p.ld_split;
        reinterpret_cast<T*>(s)[c] = h;
        reinterpret_cast<T*>(s + p.split_stride)[c] = l;
        if (p.split_blocks > 2) reinterpret_cast<T*>(s + 2 * p.split_stride)[c] = h;
    }
}

template <int VEC, int MODE, bool HAS_MAP, int NACC, int UNR, bool SPLIT = false>
__global__ void __launch_bounds__(kAggThreads, FGL_AGG_MIN_CTAS) agg_fwd_kernel(const AggParams p) {
    if (!after_the_kernels_before()) return;
    using V = Vec<VEC>;
    using T = typename V::T;
    __shared__ long long s_off[kAggMaxWindow + 1];
    const int lane = threadIdx.x & 31;
    const int warp_global = blockIdx.x * kAggWarps + (threadIdx.x >> 5);
    const int n_warps = gridDim.x * kAggWarps;
    const int chunks = p.dim / VEC;  // dim % VEC == 0 by dispatch
    const bool window = p.n_batches > 0;
    if (window) window_offsets(p, s_off);
    const int64_t padded = window ? s_off[p.n_batches] : (int64_t)p.n_dst;
    const int64_t total = p.n_dst_dev ? min((int64_t)max(__ldg(p.n_dst_dev), 0), padded) : padded;
    // padding rows of a launch sized for more rows than the block has: zero them
    for (int64_t g = total + warp_global; g < padded; g += n_warps) {
        for (int c = lane; c < chunks; c += 32) put_out<VEC, SPLIT>(p, g, c, V::zero());
    }
    const bool want_self = p.self_out != nullptr || p.passthrough != 0;

    // ---- pipeline state: stage A (offsets), B (source ids), C (map entries / degrees) ------------------------------
    int bA = 0, dA = 0, aA = 0, eA = 0;              // row i+3 after its stage A: batch, local row, edge range
    int bB = 0, dB = 0, aB = 0, eB = 0, sB = -1;      // row i+2 after stage B: + this lane's source id
    int selfB = -1;                                   //                         + the row's own input row (raw)
    int ddegB = 1;
    int bC = 0, dC = 0, aC = 0, eC = 0, sC = -1;      // row i+1 after stage C: + raw map entry / degree of the lane's source
    int rowC = 0, selfC = -1;
    int sdegC = 1, ddegC = 1;
    int batch_ptr = 0;                                // window mode: batch of the row stage A looks at (monotonic)

    auto stage_a = [&](int64_t g) {  // offsets of row g
        aA = 0;
        eA = 0;
        if (g >= total) return;
        if (window) {
            while (g >= s_off[batch_ptr + 1]) ++batch_ptr;
            bA = batch_ptr;
            dA = (int)(g - s_off[batch_ptr]);
        } else {
            bA = 0;
            dA = (int)g;
        }
        const int32_t* indptr = p.indptr + (int64_t)bA * p.indptr_stride;
        aA = __ldg(indptr + dA);
        eA = __ldg(indptr + dA + 1);
    };
    auto stage_b = [&]() {  // source ids of the row stage A saw one iteration ago (its offsets have arrived)
        bB = bA;
        dB = dA;
        aB = aA;
        eB = eA;
        sB = -1;
        selfB = -1;
        if (lane < eB - aB) sB = __ldg(p.src + (int64_t)bB * p.src_stride + aB + lane);
        if (want_self) {
            if (HAS_MAP)
                selfB = (int64_t)dB < p.n_map ? __ldg(p.row_map + (int64_t)bB * p.row_map_stride + dB) : -1;
            else
                selfB = dB;
        }
        if (MODE == FGL_AGG_SYMNORM && eB > aB) ddegB = __ldg(p.dst_deg + dB);
    };
    auto stage_c = [&]() {  // map entry and degree of this lane's source (the id has arrived)
        bC = bB;
        dC = dB;
        aC = aB;
        eC = eB;
        sC = sB;
        selfC = selfB;
        ddegC = ddegB;
        rowC = sB;
        sdegC = 1;
        const bool id_ok = sB >= 0 && (HAS_MAP ? (int64_t)sB < p.n_map : (int64_t)sB < p.n_rows);
        if (id_ok) {
            if (HAS_MAP) rowC = __ldg(p.row_map + (int64_t)bC * p.row_map_stride + sB);
            if (MODE == FGL_AGG_SYMNORM) sdegC = __ldg(p.src_deg + sB);
        } else {
            rowC = -1;  // no such edge in this lane, or an id out of range (told apart when the row is summed)
        }
    };

    // prologue: fill the pipeline (each stage waits for the one before it, once)
    stage_a(warp_global);
    stage_b();
    stage_c();
    stage_a(warp_global + (int64_t)n_warps);
    stage_b();
    stage_a(warp_global + 2 * (int64_t)n_warps);

    for (int64_t g = warp_global; g < total; g += n_warps) {
        // ---- the current row: everything below was requested at least one iteration ago ----------------------------
        const int b = bC, a = aC, e_end = eC;
        const int cnt_first = min(32, e_end - a);
        const bool has_edge = lane < cnt_first;
        bool bad = has_edge && (rowC < 0 || (int64_t)rowC >= p.n_rows);
        if (bad) agg_bad_id(p);
        const int first_row = (has_edge && !bad) ? rowC : 0;
        const unsigned first_bad = __ballot_sync(0xffffffffu, bad);
        float first_w = 1.0f;
        if (MODE == FGL_AGG_SYMNORM && has_edge && !bad) first_w = 1.0f / sqrtf((float)sdegC);
        int self_row = selfC;
        const int ddeg = ddegC;
        const bool need_self = p.self_out != nullptr || (a >= e_end && p.passthrough);
        if (need_self && (self_row < 0 || (int64_t)self_row >= p.n_rows)) {
            agg_bad_id(p);
            self_row = -1;
        }
        const int32_t* src = p.src + (int64_t)b * p.src_stride;
        const int32_t* row_map = HAS_MAP ? p.row_map + (int64_t)b * p.row_map_stride : nullptr;

        // ---- requests of this iteration, all issued before anything is consumed ------------------------------------
        // (1) the row's own input row (narrow rows: one vector per lane, kept in a register until it is stored)
        T self_v = V::zero();
        const bool self_in_reg = NACC == 1 && need_self && self_row >= 0;
        if (self_in_reg && lane < chunks) self_v = __ldg(reinterpret_cast<const T*>(x_row(p, self_row)) + lane);
        // (2) the first batch of neighbour rows, first pass over the columns
        T v0[UNR][NACC];
        if (a < e_end) {
#pragma unroll
            for (int u = 0; u < UNR; ++u) {
                const int j = min(u, cnt_first - 1);  // past the end: reload the last row, skip its FMA
                const int r = __shfl_sync(0xffffffffu, first_row, j);
                const T* xr = reinterpret_cast<const T*>(x_row(p, r));
#pragma unroll
                for (int k = 0; k < NACC; ++k) {
                    const int c = k * 32 + lane;
                    v0[u][k] = (c < chunks) ? __ldg(xr + c) : V::zero();
                }
            }
        }
        // (3) the pipeline stages of the warp's next rows
        stage_c();
        stage_b();
        stage_a(g + 3 * (int64_t)n_warps);

        // ---- consume ------------------------------------------------------------------------------------------------
        if (p.self_out) {
            T* srow = reinterpret_cast<T*>(p.self_out + g * p.ld_self);
            if (NACC == 1) {
                if (lane < chunks) srow[lane] = self_v;
            } else {
                const T* xr = reinterpret_cast<const T*>(x_row(p, self_row < 0 ? 0 : self_row));
                for (int c = lane; c < chunks; c += 32) srow[c] = self_row < 0 ? V::zero() : __ldg(xr + c);
            }
        }
        if (a >= e_end) {  // aggregate_acc_kernel.cu:307-308, :405-406
            if (NACC == 1) {
                if (lane < chunks) put_out<VEC, SPLIT>(p, g, lane, p.passthrough ? self_v : V::zero());
            } else {
                const T* xr = reinterpret_cast<const T*>(x_row(p, self_row < 0 ? 0 : self_row));
                for (int c = lane; c < chunks; c += 32)
                    put_out<VEC, SPLIT>(p, g, c, (p.passthrough && self_row >= 0) ? __ldg(xr + c) : V::zero());
            }
            continue;
        }
        float scale = 1.0f;
        if (MODE == FGL_AGG_MEAN) scale = 1.0f / (float)(e_end - a);
        if (MODE == FGL_AGG_SYMNORM) scale = 1.0f / sqrtf((float)ddeg);

        for (int c0 = 0; c0 < chunks; c0 += 32 * NACC) {
            T acc[NACC];
            int head[NACC];
#pragma unroll
            for (int k = 0; k < NACC; ++k) {
                acc[k] = V::zero();
                head[k] = (MODE == FGL_AGG_EDGE) ? min(((c0 + k * 32 + lane) * VEC) / (p.dim / p.n_heads), p.n_heads - 1) : 0;
            }
            for (int e0 = a; e0 < e_end; e0 += 32) {
                const int cnt = min(32, e_end - e0);
                int my_row = first_row;
                float my_w = first_w;
                unsigned bad_mask = first_bad;
                if (e0 != a) {  // rows with more than 32 in-edges: their further ids are fetched in line
                    my_row = 0;
                    my_w = 1.0f;
                    bool bad2 = false;
                    if (lane < cnt) {
                        const int s = __ldg(src + e0 + lane);
                        my_row = (int)checked_row<HAS_MAP>(p, row_map, s);
                        bad2 = my_row < 0;
                        if (bad2) my_row = 0;
                        if (MODE == FGL_AGG_SYMNORM && !bad2) my_w = 1.0f / sqrtf((float)__ldg(p.src_deg + s));
                    }
                    bad_mask = __ballot_sync(0xffffffffu, bad2);
                }
                int j0 = 0;
                if (c0 == 0 && e0 == a) {  // warp-uniform: the batch requested before the pipeline stages
#pragma unroll
                    for (int u = 0; u < UNR; ++u) {
                        const float wu = (MODE == FGL_AGG_SYMNORM) ? __shfl_sync(0xffffffffu, my_w, min(u, cnt - 1)) : 1.0f;
                        if (u < cnt && !((bad_mask >> u) & 1u)) {
#pragma unroll
                            for (int k = 0; k < NACC; ++k) {
                                const float wk = (MODE == FGL_AGG_EDGE) ? __ldg(p.edge_w + (int64_t)(e0 + u) * p.n_heads + head[k]) : wu;
                                V::fma(acc[k], wk, v0[u][k]);
                            }
                        }
                    }
                    j0 = UNR;
                }
                for (; j0 < cnt; j0 += UNR) {
                    T v[UNR][NACC];
                    float w[UNR];
#pragma unroll
                    for (int u = 0; u < UNR; ++u) {
                        const int j = min(j0 + u, cnt - 1);  // past the end: reload the last row, skip its FMA
                        const int r = __shfl_sync(0xffffffffu, my_row, j);
                        w[u] = (MODE == FGL_AGG_SYMNORM) ? __shfl_sync(0xffffffffu, my_w, j) : 1.0f;
                        const T* xr = reinterpret_cast<const T*>(x_row(p, r));
#pragma unroll
                        for (int k = 0; k < NACC; ++k) {
                            const int c = c0 + k * 32 + lane;
                            v[u][k] = (c < chunks) ? __ldg(xr + c) : V::zero();
                        }
                    }
#pragma unroll
                    for (int u = 0; u < UNR; ++u) {
                        if (j0 + u < cnt && !((bad_mask >> (j0 + u)) & 1u)) {  // warp-uniform
#pragma unroll
                            for (int k = 0; k < NACC; ++k) {
                                const float wk = (MODE == FGL_AGG_EDGE)
                                                     ? __ldg(p.edge_w + (int64_t)(e0 + j0 + u) * p.n_heads + head[k])
                                                     : w[u];
                                V::fma(acc[k], wk, v[u][k]);
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < NACC; ++k) {
                const int c = c0 + k * 32 + lane;
                if (c < chunks)
                    put_out<VEC, SPLIT>(p, g, c, (MODE == FGL_AGG_SUM || MODE == FGL_AGG_EDGE) ? acc[k] : V::scale(acc[k], scale));
            }
        }
    }
}

// The same forward aggregation for the shapes a sampled mini-batch has on its widest hop -- rows of at most 32
// 128-bit vectors (D <= 128 floats), a single dense table, sum / mean / sym-norm -- with the rows staged through
// shared memory by asynchronous copies (cp.async, 16 bytes per lane, L2 only) instead of through registers.
//
// Why: a warp of agg_fwd_kernel holds every byte it has in flight in registers; at 120 registers a thread an SM keeps
// 16 warps x 8 rows = 50 KB in flight, and on 400-byte rows fetched at random from HBM that -- not bandwidth -- bounds
// the kernel (measured: 2.6 TB/s of DRAM traffic, 40 % of the copy peak).  Here every warp owns kAggSlots row slots of
// shared memory and needs few registers, so an SM runs 24 warps with 16 rows each in flight (150 KB; measured best).  Per
// destination row a warp requests its own input row (slot 0, the self copy) and up to 15 neighbour rows (a row sampled
// with fanout 15 is exactly one pass), moves the id pipeline (indptr -> src -> row_map, three rows ahead, as in
// agg_fwd_kernel) while the copies fly, waits for its copies, and adds the rows out of shared memory.  Per neighbour
// row that is one shuffle, one multiply-add and one cp.async, later one 128-bit shared-memory load and four adds.  Rows
// with more than 15 in-edges take further passes whose ids are fetched in line.
constexpr int kAggSlots = 16;
#ifndef FGL_AGG_STAGED_WARPS
#define FGL_AGG_STAGED_WARPS 24
#endif
constexpr int kAggStagedMaxWarps = FGL_AGG_STAGED_WARPS;  // per CTA (one CTA per SM); fewer when the rows are wider

__device__ __forceinline__ void cp_async16(unsigned smem_dst, const void* gmem_src) {  // smem_dst: shared-space address
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_dst), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ float4 lds128(unsigned smem_src) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(smem_src));
    return v;
}

template <int MODE, bool HAS_MAP>
__global__ void __launch_bounds__(kAggStagedMaxWarps * 32, 1) agg_fwd_staged_kernel(const AggParams p) {
    if (!after_the_kernels_before()) return;
    using V = Vec<4>;
    using T = float4;
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    __shared__ long long s_off[kAggMaxWindow + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cta_warps = blockDim.x >> 5;
    const int warp_global = blockIdx.x * cta_warps + warp;
    const int n_warps = gridDim.x * cta_warps;
    const int chunks = p.dim / 4;  // <= 32
    const unsigned slot_bytes = (unsigned)chunks * 16u;
    const bool window = p.n_batches > 0;
    if (window) window_offsets(p, s_off);
    const int64_t padded = window ? s_off[p.n_batches] : (int64_t)p.n_dst;
    const int64_t total = p.n_dst_dev ? min((int64_t)max(__ldg(p.n_dst_dev), 0), padded) : padded;
    const bool lane_on = lane < chunks;
    for (int64_t g = total + warp_global; g < padded; g += n_warps)
        if (lane_on) reinterpret_cast<T*>(p.out + g * p.ldo)[lane] = V::zero();
    const bool want_self = p.self_out != nullptr || p.passthrough != 0;
    // Lanes beyond the row's last vector repeat that vector (same source, same destination: a duplicate request inside
    // one instruction), so that no copy, load or add in the loops below needs a per-lane predicate.
    const int lane_c = min(lane, chunks - 1);
    const char* lane_base = reinterpret_cast<const char*>(p.x) + lane_c * 16;
    const unsigned ld_bytes = (unsigned)(p.ldx * 4);
    auto row_ptr = [&](int r) { return lane_base + (uint64_t)(unsigned)r * ld_bytes; };  // one 32 x 32 + 64 multiply-add
    const unsigned slots = (unsigned)__cvta_generic_to_shared(dyn_smem) + (unsigned)warp * kAggSlots * slot_bytes + lane_c * 16;

    // ---- id pipeline, three destination rows ahead (see agg_fwd_kernel) ------------------------------------------------
    int bA = 0, dA = 0, aA = 0, eA = 0;
    int bB = 0, dB = 0, aB = 0, eB = 0, sB = -1, selfB = -1, ddegB = 1;
    int bC = 0, aC = 0, eC = 0, rowC = 0, selfC = -1, sdegC = 1, ddegC = 1;
    int batch_ptr = 0;
    auto stage_a = [&](int64_t g) {
        aA = 0;
        eA = 0;
        if (g >= total) return;
        if (window) {
            while (g >= s_off[batch_ptr + 1]) ++batch_ptr;
            bA = batch_ptr;
            dA = (int)(g - s_off[batch_ptr]);
        } else {
            bA = 0;
            dA = (int)g;
        }
        const int32_t* indptr = p.indptr + (int64_t)bA * p.indptr_stride;
        aA = __ldg(indptr + dA);
        eA = __ldg(indptr + dA + 1);
    };
    auto stage_b = [&]() {
        bB = bA;
        dB = dA;
        aB = aA;
        eB = eA;
        sB = -1;
        selfB = -1;
        if (lane < min(eB - aB, kAggSlots - 1)) sB = __ldg(p.src + (int64_t)bB * p.src_stride + aB + lane);
        if (want_self) {
            if (HAS_MAP)
                selfB = (int64_t)dB < p.n_map ? __ldg(p.row_map + (int64_t)bB * p.row_map_stride + dB) : -1;
            else
                selfB = dB;
        }
        if (MODE == FGL_AGG_SYMNORM && eB > aB) ddegB = __ldg(p.dst_deg + dB);
    };
    auto stage_c = [&]() {
        bC = bB;
        aC = aB;
        eC = eB;
        selfC = selfB;
        ddegC = ddegB;
        rowC = sB;
        sdegC = 1;
        const bool id_ok = sB >= 0 && (HAS_MAP ? (int64_t)sB < p.n_map : (int64_t)sB < p.n_rows);
        if (id_ok) {
            if (HAS_MAP) rowC = __ldg(p.row_map + (int64_t)bC * p.row_map_stride + sB);
            if (MODE == FGL_AGG_SYMNORM) sdegC = __ldg(p.src_deg + sB);
        } else {
            rowC = -1;
        }
    };
    stage_a(warp_global);
    stage_b();
    stage_c();
    stage_a(warp_global + (int64_t)n_warps);
    stage_b();
    stage_a(warp_global + 2 * (int64_t)n_warps);

    // Copy `cnt` rows (lane u holds row u) into slots 1 .. cnt; add them out of shared memory.
    auto request = [&](int my_row, int cnt) {
        unsigned dst = slots;
        if (cnt == kAggSlots - 1) {  // the common case: a row sampled with the full fanout
#pragma unroll
            for (int u = 0; u < kAggSlots - 1; ++u) {
                dst += slot_bytes;
                cp_async16(dst, row_ptr(__shfl_sync(0xffffffffu, my_row, u)));
            }
        } else {
            for (int u = 0; u < cnt; ++u) {
                dst += slot_bytes;
                cp_async16(dst, row_ptr(__shfl_sync(0xffffffffu, my_row, u)));
            }
        }
    };
    auto add_up = [&](T& acc, int cnt, unsigned bad_mask, float my_w) {
        unsigned from = slots;
        if (cnt == kAggSlots - 1 && bad_mask == 0u) {
#pragma unroll
            for (int u = 0; u < kAggSlots - 1; ++u) {
                from += slot_bytes;
                V::fma(acc, (MODE == FGL_AGG_SYMNORM) ? __shfl_sync(0xffffffffu, my_w, u) : 1.0f, lds128(from));
            }
        } else {
            for (int u = 0; u < cnt; ++u) {
                from += slot_bytes;
                const float wu = (MODE == FGL_AGG_SYMNORM) ? __shfl_sync(0xffffffffu, my_w, u) : 1.0f;
                if (!((bad_mask >> u) & 1u)) V::fma(acc, wu, lds128(from));
            }
        }
    };

    for (int64_t g = warp_global; g < total; g += n_warps) {
        // the current row: its ids were requested at least one iteration ago
        const int b = bC, a = aC, e_end = eC, ddeg = ddegC;
        const int cnt = min(kAggSlots - 1, e_end - a);
        const bool has_edge = lane < cnt;
        const bool bad = has_edge && (rowC < 0 || (int64_t)rowC >= p.n_rows);
        if (bad) agg_bad_id(p);
        const int my_row = (has_edge && !bad) ? rowC : 0;
        const unsigned bad_mask = __ballot_sync(0xffffffffu, bad);
        float my_w = 1.0f;
        if (MODE == FGL_AGG_SYMNORM && has_edge && !bad) my_w = 1.0f / sqrtf((float)sdegC);
        int self_row = selfC;
        const bool need_self = p.self_out != nullptr || (a >= e_end && p.passthrough);
        if (need_self && (self_row < 0 || (int64_t)self_row >= p.n_rows)) {
            agg_bad_id(p);
            self_row = -1;
        }
        // requests: the row's own input row, its first 15 neighbours, the next rows' ids
        if (need_self && self_row >= 0) cp_async16(slots, row_ptr(self_row));
        request(my_row, cnt);
        stage_c();
        stage_b();
        stage_a(g + 3 * (int64_t)n_warps);
        cp_async_wait_all();
        __syncwarp();
        // consume
        T self_v = V::zero();
        if (need_self && self_row >= 0) self_v = lds128(slots);
        if (p.self_out && lane_on) reinterpret_cast<T*>(p.self_out + g * p.ld_self)[lane] = self_v;
        T* orow = reinterpret_cast<T*>(p.out + g * p.ldo);
        if (a >= e_end) {  // aggregate_acc_kernel.cu:307-308, :405-406
            if (lane_on) orow[lane] = p.passthrough ? self_v : V::zero();
            __syncwarp();
            continue;
        }
        T acc = V::zero();
        add_up(acc, cnt, bad_mask, my_w);
        __syncwarp();  // every lane is done with the slots before the next copies overwrite them
        if (e_end - a > kAggSlots - 1) {  // further passes of a long row: ids in line, same slots
            const int32_t* src = p.src + (int64_t)b * p.src_stride;
            const int32_t* row_map = HAS_MAP ? p.row_map + (int64_t)b * p.row_map_stride : nullptr;
            for (int e0 = a + kAggSlots - 1; e0 < e_end; e0 += kAggSlots - 1) {
                const int n = min(kAggSlots - 1, e_end - e0);
                int row2 = 0;
                float w2 = 1.0f;
                bool bad2 = false;
                if (lane < n) {
                    const int s = __ldg(src + e0 + lane);
                    row2 = (int)checked_row<HAS_MAP>(p, row_map, s);
                    bad2 = row2 < 0;
                    if (bad2) row2 = 0;
                    if (MODE == FGL_AGG_SYMNORM && !bad2) w2 = 1.0f / sqrtf((float)__ldg(p.src_deg + s));
                }
                const unsigned bad2_mask = __ballot_sync(0xffffffffu, bad2);
                request(row2, n);
                cp_async_wait_all();
                __syncwarp();
                add_up(acc, n, bad2_mask, w2);
                __syncwarp();
            }
        }
        float scale = 1.0f;
        if (MODE == FGL_AGG_MEAN) scale = 1.0f / (float)(e_end - a);
        if (MODE == FGL_AGG_SYMNORM) scale = 1.0f / sqrtf((float)ddeg);
        if (lane_on) orow[lane] = (MODE == FGL_AGG_SUM) ? acc : V::scale(acc, scale);
    }
}

// Row gather: out[i,:] = x[ids[i],:] (single or sharded table).  A warp per row, UNR rows in flight per warp.
// Replaces the CPU index_select + host-to-device copy of load_subtensors (train_fastgl.py:161-184).
template <int VEC>
__global__ void __launch_bounds__(kAggThreads) gather_rows_kernel(const AggParams p, const int32_t* __restrict__ ids, int64_t n_ids) {
    if (!after_the_kernels_before()) return;
    using T = typename Vec<VEC>::T;
    const int lane = threadIdx.x & 31;
    const int64_t warp_global = (int64_t)blockIdx.x * kAggWarps + (threadIdx.x >> 5);
    const int64_t n_warps = (int64_t)gridDim.x * kAggWarps;
    const int chunks = p.dim / VEC;
    constexpr int UNR = 4;
    for (int64_t i0 = warp_global * UNR; i0 < n_ids; i0 += n_warps * UNR) {
        const T* src[UNR];
        bool ok[UNR];
#pragma unroll
        for (int u = 0; u < UNR; ++u) {
            const int64_t i = i0 + u < n_ids ? i0 + u : n_ids - 1;
            const int64_t r = (int64_t)__ldg(ids + i);
            ok[u] = r >= 0 && r < p.n_rows;
            if (!ok[u]) agg_bad_id(p);
            src[u] = reinterpret_cast<const T*>(x_row(p, ok[u] ? r : 0));
        }
        for (int c = lane; c < chunks; c += 32) {
            T v[UNR];
#pragma unroll
            for (int u = 0; u < UNR; ++u) v[u] = __ldg(src[u] + c);
#pragma unroll
            for (int u = 0; u < UNR; ++u)
                if (i0 + u < n_ids) reinterpret_cast<T*>(p.out + (i0 + u) * p.ldo)[c] = ok[u] ? v[u] : Vec<VEC>::zero();
        }
    }
}

__device__ __forceinline__ void red_add(float4* addr, const float4& v) { atomicAdd(addr, v); }
__device__ __forceinline__ void red_add(float2* addr, const float2& v) { atomicAdd(addr, v); }
__device__ __forceinline__ void red_add(float* addr, const float& v) { atomicAdd(addr, v); }

// Backward: dx[src[e],:] += w_e * scale_d * dy[d,:]; vector reductions (red.global.add.v4.f32 on sm_100a)
template <int VEC, int MODE, int NACC>
__global__ void __launch_bounds__(kAggThreads) agg_bwd_kernel(const AggParams p) {
    if (!after_the_kernels_before()) return;
    using V = Vec<VEC>;
    using T = typename V::T;
    const int lane = threadIdx.x & 31;
    const int warp_global = blockIdx.x * kAggWarps + (threadIdx.x >> 5);
    const int n_warps = gridDim.x * kAggWarps;
    const int chunks = p.dim / VEC;

    const int n_dst = p.n_dst_dev ? min(max(__ldg(p.n_dst_dev), 0), p.n_dst) : p.n_dst;
    for (int d = warp_global; d < n_dst; d += n_warps) {
        const int a = __ldg(p.indptr + d), b = __ldg(p.indptr + d + 1);
        if (p.dy_self) {
            const T* srow = reinterpret_cast<const T*>(p.dy_self + (int64_t)d * p.ld_dy_self);
            T* xr = reinterpret_cast<T*>(p.out + (int64_t)d * p.ldo);
            for (int c = lane; c < chunks; c += 32) red_add(xr + c, __ldg(srow + c));
        }
        if (a >= b) continue;  // aggregate_acc_kernel.cu:498-500, :580-582
        float scale = 1.0f;
        if (MODE == FGL_AGG_MEAN) scale = 1.0f / (float)(b - a);
        if (MODE == FGL_AGG_SYMNORM) scale = 1.0f / sqrtf((float)__ldg(p.dst_deg + d));
        const T* grow = reinterpret_cast<const T*>(p.x + (int64_t)d * p.ldx);

        for (int c0 = 0; c0 < chunks; c0 += 32 * NACC) {
            T g[NACC];
            int head[NACC];
#pragma unroll
            for (int k = 0; k < NACC; ++k) {
                const int c = c0 + k * 32 + lane;
                g[k] = (c < chunks) ? V::scale(__ldg(grow + c), scale) : V::zero();
                head[k] = (MODE == FGL_AGG_EDGE) ? min((c * VEC) / (p.dim / p.n_heads), p.n_heads - 1) : 0;
            }
            for (int e0 = a; e0 < b; e0 += 32) {
                const int cnt = min(32, b - e0);
                int my_s = 0;
                float my_w = 1.0f;
                if (lane < cnt) {
                    my_s = __ldg(p.src + e0 + lane);
                    if (MODE == FGL_AGG_SYMNORM && my_s >= 0 && my_s < p.n_src) my_w = 1.0f / sqrtf((float)__ldg(p.src_deg + my_s));
                }
                for (int j = 0; j < cnt; ++j) {
                    const int s = __shfl_sync(0xffffffffu, my_s, j);
                    const float w = (MODE == FGL_AGG_SYMNORM) ? __shfl_sync(0xffffffffu, my_w, j) : 1.0f;
                    if (s < 0 || s >= p.n_src) {  // warp-uniform
                        agg_bad_id(p);
                        continue;
                    }
                    T* xr = reinterpret_cast<T*>(p.out + (int64_t)s * p.ldo);
#pragma unroll
                    for (int k = 0; k < NACC; ++k) {
                        const int c = c0 + k * 32 + lane;
                        if (c < chunks) {
                            if (MODE == FGL_AGG_EDGE)
                                red_add(xr + c, V::scale(g[k], __ldg(p.edge_w + (int64_t)(e0 + j) * p.n_heads + head[k])));
                            else
                                red_add(xr + c, (MODE == FGL_AGG_SYMNORM) ? V::scale(g[k], w) : g[k]);
                        }
                    }
                }
            }
        }
    }
}

// Gradient of the edge weights: dw[e, h] = sum over head h's columns f of dy[d, f] * x[src[e], f] for every edge e of
// row d (the term the reference drops, GraphConv.py:227).  A warp per destination row; per neighbour the lanes
// multiply their vectors, reduce within runs of lanes that share a head, and the first lane of each run adds.
template <int VEC>
__global__ void __launch_bounds__(kAggThreads) agg_edge_wgrad_kernel(const AggParams p, float* __restrict__ dw) {
    if (!after_the_kernels_before()) return;
    using T = typename Vec<VEC>::T;
    const int lane = threadIdx.x & 31;
    const int warp_global = blockIdx.x * kAggWarps + (threadIdx.x >> 5);
    const int n_warps = gridDim.x * kAggWarps;
    const int chunks = p.dim / VEC;
    const int unit = p.dim / p.n_heads;
    for (int d = warp_global; d < p.n_dst; d += n_warps) {
        const int a = __ldg(p.indptr + d), b = __ldg(p.indptr + d + 1);
        const T* grow = reinterpret_cast<const T*>(p.out + (int64_t)d * p.ldo);  // dy
        for (int c0 = 0; c0 < chunks; c0 += 32) {
            const int c = c0 + lane;
            const bool live = c < chunks;
            const int head = live ? (c * VEC) / unit : -1;
            T g = Vec<VEC>::zero();
            if (live) g = __ldg(grow + c);
            const int prev_head = __shfl_up_sync(0xffffffffu, head, 1);
            const bool leader = live && (lane == 0 || prev_head != head);
            for (int e = a; e < b; ++e) {
                const int s = __ldg(p.src + e);
                if (s < 0 || s >= p.n_src) {  // warp-uniform: dw[e, :] stays zero
                    agg_bad_id(p);
                    continue;
                }
                float v = 0.0f;
                if (live) {
                    const T xv = __ldg(reinterpret_cast<const T*>(p.x + (int64_t)s * p.ldx) + c);
                    const float* gp = reinterpret_cast<const float*>(&g);
                    const float* xp = reinterpret_cast<const float*>(&xv);
#pragma unroll
                    for (int q = 0; q < VEC; ++q) v = fmaf(gp[q], xp[q], v);
                }
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {  // segmented suffix sum over lanes of the same head
                    const float ov = __shfl_down_sync(0xffffffffu, v, off);
                    const int oh = __shfl_down_sync(0xffffffffu, head, off);
                    if (lane + off < 32 && oh == head) v += ov;
                }
                if (leader) atomicAdd(dw + (int64_t)e * p.n_heads + head, v);
            }
        }
    }
}

static bool aligned_for(int v, const void* a, int64_t lda) { return lda % v == 0 && ((uintptr_t)a % (4 * v)) == 0; }

static int pick_vec(int dim, const void* a, int64_t lda, const void* b, int64_t ldb, const void* c = nullptr, int64_t ldc = 4) {
    auto ok = [&](int v) {
        return dim % v == 0 && aligned_for(v, a, lda) && aligned_for(v, b, ldb) && (!c || aligned_for(v, c, ldc));
    };
    if (ok(4)) return 4;
    if (ok(2)) return 2;
    return 1;
}

// Asked once: every call costs as much as a launch's arguments (the GPUs of a box are alike).
static int sm_count() {
    static std::atomic<int> cached{0};
    int sms = cached.load(std::memory_order_relaxed);
    if (sms == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
            return 148;
        cached.store(sms, std::memory_order_relaxed);
    }
    return sms;
}

// dx[0 .. n_src) = 0
static cudaError_t zero_rows(float* dx, int64_t ldx, int32_t dim, int32_t n_src, cudaStream_t st) {
    if (ldx == dim) return cudaMemsetAsync(dx, 0, sizeof(float) * (size_t)dim * (size_t)n_src, st);
    return cudaMemset2DAsync(dx, sizeof(float) * (size_t)ldx, 0, sizeof(float) * (size_t)dim, (size_t)n_src, st);
}

static int agg_grid_x(int n_rows, int n_batches) {
    const int sms = sm_count();
    const int64_t want = ((int64_t)n_rows + kAggWarps - 1) / kAggWarps;
    const int64_t cap = std::max<int64_t>(1, ((int64_t)sms * 8 + n_batches - 1) / n_batches);
    return (int)std::max<int64_t>(1, std::min<int64_t>(want, cap));
}

template <int VEC, int MODE, int NACC, int UNR>
static void launch_fwd(const AggParams& p, dim3 grid, cudaStream_t st) {
    if (p.row_map)
        launch(agg_fwd_kernel<VEC, MODE, true, NACC, UNR>, grid, kAggThreads, 0, st, p);
    else
        launch(agg_fwd_kernel<VEC, MODE, false, NACC, UNR>, grid, kAggThreads, 0, st, p);
}

// Whether agg_fwd_staged_kernel applies: 128-bit rows of at most 32 vectors in a single dense table.
static bool staged_applies(const AggParams& p, int vec) {
    return vec == 4 && p.shards == nullptr && p.dim / 4 <= 32 && p.ldx * 4 <= 0xffffffffLL;
}

// The shared memory a kernel may ask for, set once per kernel and device instead of before every launch.
template <auto kernel>
static void allow_shared(int bytes) {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return;
    const uint64_t bit = 1ULL << (dev & 63);
    if (done.load(std::memory_order_relaxed) & bit) return;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess)
        done.fetch_or(bit, std::memory_order_relaxed);
}

template <int MODE>
static void launch_fwd_staged(const AggParams& p, cudaStream_t st) {
    const int sms = sm_count();
    constexpr int64_t kRoom = (227 - 8) * 1024;  // beside the kernel's static shared memory
    const int64_t per_warp = (int64_t)kAggSlots * (p.dim / 4) * 16;
    // As many warps per SM as their row slots fit; a block of few rows is spread over the SMs instead of filling a few.
    const int64_t rows = p.n_batches > 0 ? 0x7fffffff : p.n_dst;  // window launches fill the GPU
    const int64_t fit = std::min<int64_t>(kAggStagedMaxWarps, kRoom / per_warp);
    const int warps = (int)std::max<int64_t>(1, std::min<int64_t>(fit, std::max<int64_t>(4, (rows + sms - 1) / sms)));
    const size_t dyn = (size_t)warps * per_warp;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(sms, (rows + warps - 1) / warps));
    if (p.row_map) {
        allow_shared<agg_fwd_staged_kernel<MODE, true>>((int)kRoom);
        launch(agg_fwd_staged_kernel<MODE, true>, grid, warps * 32, dyn, st, p);
    } else {
        allow_shared<agg_fwd_staged_kernel<MODE, false>>((int)kRoom);
        launch(agg_fwd_staged_kernel<MODE, false>, grid, warps * 32, dyn, st, p);
    }
}

template <int VEC, int MODE>
static void launch_fwd_nacc(const AggParams& p, dim3 grid, cudaStream_t st) {
    const int chunks = p.dim / VEC;
    if (MODE != FGL_AGG_EDGE && staged_applies(p, VEC)) {
        launch_fwd_staged<MODE == FGL_AGG_EDGE ? FGL_AGG_SUM : MODE>(p, st);
    } else if (chunks <= 32)
        launch_fwd<VEC, MODE, 1, FGL_AGG_UNR1>(p, grid, st);
    else if (VEC == 4) {
        if (chunks <= 64) launch_fwd<VEC, MODE, 2, 4>(p, grid, st);
        else launch_fwd<VEC, MODE, 4, 2>(p, grid, st);
    // Rows that are only 8- or 4-byte aligned: a load brings half or a quarter of the bytes, so twice or four times as many
    // are kept in flight (602 floats: 16 -> 40 KB per SM), and a row of up to 320 vectors is one pass.
    } else if (chunks <= 64)
        launch_fwd<VEC, MODE, 2, 8>(p, grid, st);
    else if (chunks <= 128)
        launch_fwd<VEC, MODE, 4, VEC == 2 ? 4 : 8>(p, grid, st);
    else if (chunks <= 160)
        launch_fwd<VEC, MODE, 5, VEC == 2 ? 3 : 6>(p, grid, st);
    else if (chunks <= 320)
        launch_fwd<VEC, MODE, 10, VEC == 2 ? 2 : 3>(p, grid, st);
    else
        launch_fwd<VEC, MODE, 8, VEC == 2 ? 2 : 4>(p, grid, st);
}

template <int VEC>
static void launch_fwd_mode(int mode, const AggParams& p, dim3 grid, cudaStream_t st) {
    if (mode == FGL_AGG_SUM) launch_fwd_nacc<VEC, FGL_AGG_SUM>(p, grid, st);
    if (mode == FGL_AGG_MEAN) launch_fwd_nacc<VEC, FGL_AGG_MEAN>(p, grid, st);
    if (mode == FGL_AGG_SYMNORM) launch_fwd_nacc<VEC, FGL_AGG_SYMNORM>(p, grid, st);
    if (mode == FGL_AGG_EDGE) launch_fwd_nacc<VEC, FGL_AGG_EDGE>(p, grid, st);
}

static int launch_fwd_any(int mode, const AggParams& p, dim3 grid, int vec, cudaStream_t st) {
    switch (vec) {
        case 4: launch_fwd_mode<4>(mode, p, grid, st); break;
        case 2: launch_fwd_mode<2>(mode, p, grid, st); break;
        default: launch_fwd_mode<1>(mode, p, grid, st); break;
    }
    return cudaGetLastError() == cudaSuccess ? FGL_OK : FGL_ERR_CUDA;
}


template <int VEC, int MODE>
static void launch_bwd_nacc(const AggParams& p, int grid, cudaStream_t st) {
    const int chunks = p.dim / VEC;
    if (chunks <= 32)
        launch(agg_bwd_kernel<VEC, MODE, 1>, grid, kAggThreads, 0, st, p);
    else if (chunks <= 64)
        launch(agg_bwd_kernel<VEC, MODE, 2>, grid, kAggThreads, 0, st, p);
    else
        launch(agg_bwd_kernel<VEC, MODE, 4>, grid, kAggThreads, 0, st, p);
}

template <int VEC>
static void launch_bwd_mode(int mode, const AggParams& p, int grid, cudaStream_t st) {
    if (mode == FGL_AGG_SUM) launch_bwd_nacc<VEC, FGL_AGG_SUM>(p, grid, st);
    if (mode == FGL_AGG_MEAN) launch_bwd_nacc<VEC, FGL_AGG_MEAN>(p, grid, st);
    if (mode == FGL_AGG_SYMNORM) launch_bwd_nacc<VEC, FGL_AGG_SYMNORM>(p, grid, st);
    if (mode == FGL_AGG_EDGE) launch_bwd_nacc<VEC, FGL_AGG_EDGE>(p, grid, st);
}

// dx[r, :] = dy_self[r, :] for r < n_dst (the real count when n_dst_dev is given), 0 for n_dst <= r < n_src: the
// start value of the scatter of a layer with a self term.  Scalar columns: the two matrices may have different
// alignment.
__global__ void __launch_bounds__(256)
init_self_rows_kernel(float* __restrict__ dx, int64_t ldx, const float* __restrict__ dy_self, int64_t ld_self, int dim,
                      int n_dst, int n_src, const int32_t* __restrict__ n_dst_dev) {
    if (!after_the_kernels_before()) return;
    if (n_dst_dev) n_dst = min(max(__ldg(n_dst_dev), 0), n_dst);  // padded launch: rows at or beyond the real count are zero
    const int groups = (dim + 3) / 4;
    const int64_t total = (int64_t)n_src * groups;
    const bool vec = dim % 4 == 0 && ldx % 4 == 0 && ld_self % 4 == 0 && (((uintptr_t)dx | (uintptr_t)dy_self) & 15) == 0;
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = g / groups;
        const int c = (int)(g - r * groups) * 4;
        if (vec) {
            const float4 v = r < n_dst ? *reinterpret_cast<const float4*>(dy_self + r * ld_self + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<float4*>(dx + r * ldx + c) = v;
        } else {
            for (int j = c; j < c + 4 && j < dim; ++j) dx[r * ldx + j] = r < n_dst ? dy_self[r * ld_self + j] : 0.f;
        }
    }
}

}  // namespace fgl

using namespace fgl;

static int32_t* status_of(fgl_ws* ws) { return ws ? ws->status : nullptr; }

extern "C" {

int fgl_agg_fwd(fgl_ws* ws, int32_t mode, const int32_t* indptr, const int32_t* src, const int32_t* src_deg,
                const int32_t* dst_deg, const int32_t* row_map, int64_t n_map, const float* x, int64_t n_rows, int64_t ldx,
                int32_t dim, int32_t n_dst, int32_t flags, float* out, int64_t ldo, const int32_t* n_dst_dev, void* stream) {
    return fgl_agg_fwd_sharded(ws, mode, indptr, src, src_deg, dst_deg, row_map, n_map, x, nullptr, 0, n_rows, ldx, dim, n_dst,
                               flags, out, ldo, n_dst_dev, stream);
}

int fgl_agg_fwd_sharded(fgl_ws* ws, int32_t mode, const int32_t* indptr, const int32_t* src, const int32_t* src_deg,
                        const int32_t* dst_deg, const int32_t* row_map, int64_t n_map, const float* x,
                        const float* const* shards, int64_t rows_per_shard, int64_t n_rows, int64_t ldx, int32_t dim,
                        int32_t n_dst, int32_t flags, float* out, int64_t ldo, const int32_t* n_dst_dev, void* stream) {
    if (mode < FGL_AGG_SUM || mode > FGL_AGG_SYMNORM || n_dst < 0 || dim < 1 || ldx < dim || ldo < dim || n_rows < 0 ||
        (row_map && n_map < 0))
        return FGL_ERR_INVALID;
    if (n_dst == 0) return FGL_OK;
    if (!indptr || (!x && !shards) || (shards && rows_per_shard < 1) || !out || n_rows < 1) return FGL_ERR_INVALID;
    if (mode == FGL_AGG_SYMNORM && (!src_deg || !dst_deg)) return FGL_ERR_INVALID;
    AggParams p{};
    p.indptr = indptr;
    p.src = src;
    p.src_deg = src_deg;
    p.dst_deg = dst_deg;
    p.row_map = row_map;
    p.x = x;
    p.out = out;
    p.ldx = ldx;
    p.ldo = ldo;
    p.dim = dim;
    p.n_dst = n_dst;
    p.n_dst_dev = n_dst_dev;
    p.shards = shards;
    p.rows_per_shard = rows_per_shard;
    p.n_rows = n_rows;
    p.n_map = n_map;
    p.status = status_of(ws);
    p.passthrough = (flags & FGL_AGG_ZERO_DEG_PASSTHROUGH) ? 1 : 0;
    return launch_fwd_any(mode, p, dim3(agg_grid_x(n_dst, 1), 1), pick_vec(dim, shards ? nullptr : x, ldx, out, ldo),
                          (cudaStream_t)stream);
}

static int agg_fwd_window(fgl_ws* ws, int32_t mode, int32_t n_batches, const int32_t* indptr, int64_t indptr_stride,
                       const int32_t* src, int64_t src_stride, const int32_t* row_map, int64_t row_map_stride,
                       const int64_t* out_row_off, const int32_t* counts, int64_t counts_stride, int64_t total_rows, const float* x, const float* const* shards,
                       int64_t rows_per_shard, int64_t n_rows, int64_t ldx, int32_t dim, int32_t flags, float* out,
                       int64_t ldo, float* self_out, int64_t ld_self, void* stream) {
    if ((mode != FGL_AGG_SUM && mode != FGL_AGG_MEAN) || n_batches < 0 || n_batches > kAggMaxWindow || total_rows < 0 ||
        total_rows > 0x7fffffffLL ||
        dim < 1 || ldx < dim || ldo < dim || (self_out && ld_self < dim) || n_rows < 0)
        return FGL_ERR_INVALID;
    if (n_batches == 0 || total_rows == 0) return FGL_OK;
    if (!indptr || !src || (!out_row_off && !counts) || (!x && !shards) || (shards && rows_per_shard < 1) || !out || n_rows < 1)
        return FGL_ERR_INVALID;
    AggParams p{};
    p.indptr = indptr;
    p.src = src;
    p.row_map = row_map;
    p.x = x;
    p.shards = shards;
    p.rows_per_shard = rows_per_shard;
    p.n_rows = n_rows;
    p.n_map = row_map_stride;  // a batch's local ids index its own row of the map
    p.status = status_of(ws);
    p.out = out;
    p.self_out = self_out;
    p.ldx = ldx;
    p.ldo = ldo;
    p.ld_self = ld_self;
    p.dim = dim;
    p.passthrough = (flags & FGL_AGG_ZERO_DEG_PASSTHROUGH) ? 1 : 0;
    p.indptr_stride = indptr_stride;
    p.src_stride = src_stride;
    p.row_map_stride = row_map_stride;
    p.n_batches = n_batches;
    p.out_row_off = out_row_off;
    p.counts = counts;
    p.counts_stride = counts_stride;
    const int vec = pick_vec(dim, shards ? nullptr : x, ldx, out, ldo, self_out, self_out ? ld_self : 4);
    timing_begin(ws, (cudaStream_t)stream);
    const int rc = launch_fwd_any(mode, p, dim3(agg_grid_x((int)total_rows, 1), 1), vec, (cudaStream_t)stream);
    timing_end(ws, (cudaStream_t)stream);
    return rc;
}

int fgl_agg_fwd_window(fgl_ws* ws, int32_t mode, int32_t n_batches, const int32_t* indptr, int64_t indptr_stride,
                       const int32_t* src, int64_t src_stride, const int32_t* row_map, int64_t row_map_stride,
                       const int64_t* out_row_off, int64_t total_rows, const float* x, const float* const* shards,
                       int64_t rows_per_shard, int64_t n_rows, int64_t ldx, int32_t dim, int32_t flags, float* out,
                       int64_t ldo, float* self_out, int64_t ld_self, void* stream) {
    return agg_fwd_window(ws, mode, n_batches, indptr, indptr_stride, src, src_stride, row_map, row_map_stride, out_row_off, nullptr, 0, total_rows, x, shards, rows_per_shard, n_rows, ldx, dim, flags, out, ldo, self_out, ld_self, stream);
}

int fgl_agg_fwd_window_counts(fgl_ws* ws, int32_t mode, int32_t n_batches, const int32_t* indptr, int64_t indptr_stride,
                       const int32_t* src, int64_t src_stride, const int32_t* row_map, int64_t row_map_stride,
                       const int32_t* counts, int64_t counts_stride, int64_t total_rows, const float* x, const float* const* shards,
                       int64_t rows_per_shard, int64_t n_rows, int64_t ldx, int32_t dim, int32_t flags, float* out,
                       int64_t ldo, float* self_out, int64_t ld_self, void* stream) {
    return agg_fwd_window(ws, mode, n_batches, indptr, indptr_stride, src, src_stride, row_map, row_map_stride, nullptr, counts, counts_stride, total_rows, x, shards, rows_per_shard, n_rows, ldx, dim, flags, out, ldo, self_out, ld_self, stream);
}

int fgl_agg_edge_fwd(fgl_ws* ws, const int32_t* indptr, const int32_t* src, const float* edge_w, int32_t n_heads,
                     const float* x, int32_t n_src, int64_t ldx, int32_t dim, int32_t n_dst, int32_t flags, float* out,
                     int64_t ldo, void* stream) {
    if (n_dst < 0 || n_src < 0 || dim < 1 || n_heads < 1 || dim % n_heads != 0 || ldx < dim || ldo < dim) return FGL_ERR_INVALID;
    if (n_dst == 0) return FGL_OK;
    if (!indptr || !x || !out || !edge_w || n_src < 1) return FGL_ERR_INVALID;
    AggParams p{};
    p.indptr = indptr;
    p.src = src;
    p.x = x;
    p.out = out;
    p.ldx = ldx;
    p.ldo = ldo;
    p.dim = dim;
    p.n_dst = n_dst;
    p.n_rows = n_src;
    p.status = status_of(ws);
    p.edge_w = edge_w;
    p.n_heads = n_heads;
    p.passthrough = (flags & FGL_AGG_ZERO_DEG_PASSTHROUGH) ? 1 : 0;
    int vec = pick_vec(dim, x, ldx, out, ldo);
    while (vec > 1 && (dim / n_heads) % vec != 0) vec /= 2;  // a vector never straddles two heads
    return launch_fwd_any(FGL_AGG_EDGE, p, dim3(agg_grid_x(n_dst, 1), 1), vec, (cudaStream_t)stream);
}

int fgl_agg_edge_bwd(fgl_ws* ws, const int32_t* indptr, const int32_t* src, const float* edge_w, int32_t n_heads,
                     const float* dy, int64_t ldy, int32_t dim, int32_t n_dst, int32_t n_src, float* dx, int64_t ldx,
                     void* stream) {
    if (n_dst < 0 || n_src < 0 || dim < 1 || n_heads < 1 || dim % n_heads != 0 || ldy < dim || ldx < dim) return FGL_ERR_INVALID;
    if (n_src == 0) return FGL_OK;
    if (!dx) return FGL_ERR_INVALID;
    cudaStream_t st = (cudaStream_t)stream;
    if (zero_rows(dx, ldx, dim, n_src, st) != cudaSuccess) return FGL_ERR_CUDA;
    if (n_dst == 0) return FGL_OK;
    if (!indptr || !dy || !edge_w) return FGL_ERR_INVALID;
    AggParams p{};
    p.indptr = indptr;
    p.src = src;
    p.x = dy;
    p.out = dx;
    p.ldx = ldy;
    p.ldo = ldx;
    p.dim = dim;
    p.n_dst = n_dst;
    p.n_src = n_src;
    p.status = status_of(ws);
    p.edge_w = edge_w;
    p.n_heads = n_heads;
    int vec = pick_vec(dim, dy, ldy, dx, ldx);
    while (vec > 1 && (dim / n_heads) % vec != 0) vec /= 2;
    const int grid = agg_grid_x(n_dst, 1);
    switch (vec) {
        case 4: launch_bwd_mode<4>(FGL_AGG_EDGE, p, grid, st); break;
        case 2: launch_bwd_mode<2>(FGL_AGG_EDGE, p, grid, st); break;
        default: launch_bwd_mode<1>(FGL_AGG_EDGE, p, grid, st); break;
    }
    return cudaGetLastError() == cudaSuccess ? FGL_OK : FGL_ERR_CUDA;
}

int fgl_agg_edge_wgrad(fgl_ws* ws, const int32_t* indptr, const int32_t* src, int32_t n_heads, const float* x, int32_t n_src,
                       int64_t ldx, const float* dy, int64_t ldy, int32_t dim, int32_t n_dst, int64_t n_edges, float* dw,
                       void* stream) {
    if (n_dst < 0 || n_src < 0 || n_edges < 0 || dim < 1 || n_heads < 1 || dim % n_heads != 0 || ldx < dim || ldy < dim)
        return FGL_ERR_INVALID;
    if (n_edges == 0) return FGL_OK;
    if (!dw) return FGL_ERR_INVALID;
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemsetAsync(dw, 0, sizeof(float) * (size_t)n_edges * (size_t)n_heads, st) != cudaSuccess) return FGL_ERR_CUDA;
    if (n_dst == 0) return FGL_OK;
    if (!indptr || !src || !x || !dy) return FGL_ERR_INVALID;
    AggParams p{};
    p.indptr = indptr;
    p.src = src;
    p.x = x;
    p.out = const_cast<float*>(dy);
    p.ldx = ldx;
    p.ldo = ldy;
    p.dim = dim;
    p.n_dst = n_dst;
    p.n_src = n_src;
    p.status = status_of(ws);
    p.n_heads = n_heads;
    int vec = pick_vec(dim, x, ldx, dy, ldy);
    while (vec > 1 && (dim / n_heads) % vec != 0) vec /= 2;
    const int grid = agg_grid_x(n_dst, 1);
    switch (vec) {
        case 4: launch(agg_edge_wgrad_kernel<4>, grid, kAggThreads, 0, st, p, dw); break;
        case 2: launch(agg_edge_wgrad_kernel<2>, grid, kAggThreads, 0, st, p, dw); break;
        default: launch(agg_edge_wgrad_kernel<1>, grid, kAggThreads, 0, st, p, dw); break;
    }
    return cudaGetLastError() == cudaSuccess ? FGL_OK : FGL_ERR_CUDA;
}

int fgl_gather_rows(fgl_ws* ws, const float* table, const float* const* shards, int64_t rows_per_shard, int64_t n_rows,
                    int64_t ld, int32_t dim, const int32_t* ids, int64_t n_ids, float* out, int64_t ldo, void* stream) {
    if ((!table && !shards) || (shards && rows_per_shard < 1) || dim < 1 || ld < dim || ldo < dim || n_ids < 0 || n_rows < 0)
        return FGL_ERR_INVALID;
    if (n_ids == 0) return FGL_OK;
    if (!ids || !out || n_rows < 1) return FGL_ERR_INVALID;
    AggParams p{};
    p.x = table;
    p.shards = shards;
    p.rows_per_shard = rows_per_shard;
    p.n_rows = n_rows;
    p.status = status_of(ws);
    p.out = out;
    p.ldx = ld;
    p.ldo = ldo;
    p.dim = dim;
    // the shard bases cannot be inspected on the host: rely on the leading dimension and cudaMalloc alignment
    const int vec = pick_vec(dim, shards ? (const void*)nullptr : (const void*)table, ld, out, ldo);
    const int grid = agg_grid_x((int)std::min<int64_t>((n_ids + 3) / 4, 0x7fffffff), 1);
    cudaStream_t st = (cudaStream_t)stream;
    switch (vec) {
        case 4: launch(gather_rows_kernel<4>, grid, kAggThreads, 0, st, p, ids, n_ids); break;
        case 2: launch(gather_rows_kernel<2>, grid, kAggThreads, 0, st, p, ids, n_ids); break;
        default: launch(gather_rows_kernel<1>, grid, kAggThreads, 0, st, p, ids, n_ids); break;
    }
    return cudaGetLastError() == cudaSuccess ? FGL_OK : FGL_ERR_CUDA;
}

static int agg_bwd_impl(fgl_ws* ws, int32_t mode, const int32_t* indptr, const int32_t* src, const int32_t* src_deg,
                        const int32_t* dst_deg, const float* dy, int64_t ldy, const float* dy_self, int64_t ld_self,
                        int32_t dim, int32_t n_dst, int32_t n_src, float* dx, int64_t ldx, const int32_t* n_dst_dev,
                        bool accumulate, void* stream) {
    if (mode < FGL_AGG_SUM || mode > FGL_AGG_SYMNORM || n_dst < 0 || n_src < 0 || dim < 1 || ldy < dim || ldx < dim)
        return FGL_ERR_INVALID;
    if (dy_self && (ld_self < dim || n_dst > n_src)) return FGL_ERR_INVALID;
    if (n_src == 0) return FGL_OK;
    if (!dx) return FGL_ERR_INVALID;
    cudaStream_t st = (cudaStream_t)stream;
    if (accumulate) {
        // dx holds what the scatter adds to
    } else if (dy_self && n_dst > 0) {
        const int64_t items = (int64_t)n_src * ((dim + 3) / 4);
        const int grid = (int)std::min<int64_t>((items + 255) / 256, 148 * 16);
        launch(init_self_rows_kernel, grid, 256, 0, st, dx, ldx, dy_self, ld_self, dim, n_dst, n_src, n_dst_dev);
    } else if (zero_rows(dx, ldx, dim, n_src, st) != cudaSuccess) {
        return FGL_ERR_CUDA;
    }
    if (n_dst == 0) return FGL_OK;
    if (!indptr || !dy) return FGL_ERR_INVALID;
    if (mode == FGL_AGG_SYMNORM && (!src_deg || !dst_deg)) return FGL_ERR_INVALID;
    AggParams p{};
    p.indptr = indptr;
    p.src = src;
    p.src_deg = src_deg;
    p.dst_deg = dst_deg;
    p.x = dy;
    p.out = dx;
    p.ldx = ldy;
    p.ldo = ldx;
    p.dim = dim;
    p.n_dst = n_dst;
    p.n_src = n_src;
    p.n_dst_dev = n_dst_dev;
    p.status = status_of(ws);
    const int grid = agg_grid_x(n_dst, 1);
    int vec = pick_vec(dim, dy, ldy, dx, ldx);
    if (accumulate && dy_self) {
        p.dy_self = dy_self;
        p.ld_dy_self = ld_self;
        vec = std::min(vec, pick_vec(dim, dy_self, ld_self, dx, ldx));
    }
    switch (vec) {
        case 4: launch_bwd_mode<4>(mode, p, grid, st); break;
        case 2: launch_bwd_mode<2>(mode, p, grid, st); break;
        default: launch_bwd_mode<1>(mode, p, grid, st); break;
    }
    return cudaGetLastError() == cudaSuccess ? FGL_OK : FGL_ERR_CUDA;
}

int fgl_agg_bwd(fgl_ws* ws, int32_t mode, const int32_t* indptr, const int32_t* src, const int32_t* src_deg,
                const int32_t* dst_deg, const float* dy, int64_t ldy, int32_t dim, int32_t n_dst, int32_t n_src, float* dx,
                int64_t ldx, const int32_t* n_dst_dev, void* stream) {
    return agg_bwd_impl(ws, mode, indptr, src, src_deg, dst_deg, dy, ldy, nullptr, 0, dim, n_dst, n_src, dx, ldx, n_dst_dev,
                        false, stream);
}

int fgl_agg_bwd_add(fgl_ws* ws, int32_t mode, const int32_t* indptr, const int32_t* src, const int32_t* src_deg,
                    const int32_t* dst_deg, const float* dy, int64_t ldy, const float* dy_self, int64_t ld_self,
                    int32_t dim, int32_t n_dst, int32_t n_src, float* dx, int64_t ldx, const int32_t* n_dst_dev,
                    void* stream) {
    return agg_bwd_impl(ws, mode, indptr, src, src_deg, dst_deg, dy, ldy, dy_self, ld_self, dim, n_dst, n_src, dx, ldx, n_dst_dev,
                        true, stream);
}

int fgl_agg_fwd_split(fgl_ws* ws, const int32_t* indptr, const int32_t* src, const float* x, int64_t n_rows, int64_t ldx,
                      int32_t dim, int32_t n_dst, float* out, int64_t ldo, float* split, int64_t ld_split,
                      int64_t split_stride, int32_t blocks, const int32_t* n_dst_dev, void* stream) {
    if (n_dst < 0 || dim < 1 || ldx < dim || (out && ldo < dim) || n_rows < 0 || blocks < 2 || blocks > 3 || split_stride < dim ||
        ld_split < (blocks - 1) * split_stride + dim)
        return FGL_ERR_INVALID;
    if (n_dst == 0) return FGL_OK;
    if (!indptr || !x || !split || n_rows < 1) return FGL_ERR_INVALID;
    // 128-bit rows alone: a caller with other rows splits them in a pass of its own
    if (dim % 4 != 0 || split_stride % 4 != 0 || pick_vec(dim, x, ldx, split, ld_split) != 4 ||
        (out && pick_vec(dim, x, ldx, out, ldo) != 4))
        return FGL_ERR_INVALID;
    AggParams p{};
    p.indptr = indptr;
    p.src = src;
    p.x = x;
    p.out = out;
    p.ldx = ldx;
    p.ldo = ldo;
    p.dim = dim;
    p.n_dst = n_dst;
    p.n_dst_dev = n_dst_dev;
    p.n_rows = n_rows;
    p.status = status_of(ws);
    p.split = split;
    p.ld_split = ld_split;
    p.split_stride = split_stride;
    p.split_blocks = blocks;
    const int grid = agg_grid_x(n_dst, 1);
    cudaStream_t st = (cudaStream_t)stream;
    if (dim <= 128) launch(agg_fwd_kernel<4, FGL_AGG_MEAN, false, 1, FGL_AGG_UNR1, true>, grid, kAggThreads, 0, st, p);
    else if (dim <= 256) launch(agg_fwd_kernel<4, FGL_AGG_MEAN, false, 2, 4, true>, grid, kAggThreads, 0, st, p);
    else launch(agg_fwd_kernel<4, FGL_AGG_MEAN, false, 4, 2, true>, grid, kAggThreads, 0, st, p);
    return cudaGetLastError() == cudaSuccess ? FGL_OK : FGL_ERR_CUDA;
}

int fgl_agg_bwd_self(fgl_ws* ws, int32_t mode, const int32_t* indptr, const int32_t* src, const int32_t* src_deg,
                     const int32_t* dst_deg, const float* dy, int64_t ldy, const float* dy_self, int64_t ld_self,
                     int32_t dim, int32_t n_dst, int32_t n_src, float* dx, int64_t ldx, const int32_t* n_dst_dev,
                     void* stream) {
    if (!dy_self && n_dst > 0) return FGL_ERR_INVALID;
    return agg_bwd_impl(ws, mode, indptr, src, src_deg, dst_deg, dy, ldy, dy_self, ld_self, dim, n_dst, n_src, dx, ldx,
                        n_dst_dev, false, stream);
}

}  // extern "C"

// ================================================================================================================
// Backward as a gather over the transposed block CSR (deterministic, no atomics on the gradient, no zero-fill pass)
// ================================================================================================================
// The scatter above adds every edge's contribution with a vector reduction: its speed is the L2's reduction rate
// and the order of the additions -- hence the last bits of the result -- changes from run to run.  Here the block is
// transposed once (per-source lists of destination rows: histogram, scan, fill) and every gradient row dx[s] is
// then produced by exactly one warp (sources with at most kHubThreshold in-block out-edges) or one CTA per tile (hubs), which adds the
// rows dy[d] of its list in ascending order of d.  The order is a property of the block, not of the schedule, so two
// runs give the same bits; dx[s] is written once, with the self term folded in, so it needs no initialisation.
// Replaces K9 / K11 (aggregate_acc_kernel.cu:468-517, :555-596) like agg_bwd_kernel does.
namespace fgl {

struct GatherParams {
    const int32_t* indptr;    // block CSR over destinations (mean weights)
    const int32_t* t_indptr;  // transposed: per source, [n_src + 1]
    const int32_t* t_dst;     // destination rows, grouped by source (order within a group: arbitrary)
    const int32_t* hubs;      // [0] number of sources with more than kHubThreshold entries, then their ids
    const int32_t* src_deg;
    const int32_t* dst_deg;
    const float* dy;
    const float* dy_self;
    float* dx;
    int64_t ldy, ld_self, ldx;
    int32_t dim, n_dst, n_src;
    const int32_t* n_dst_dev;
    int32_t hub_ctas;  // agg_bwd_gather_kernel: so many CTAs take the hubs
};

constexpr int kHubThreshold = 128;  // sources with more entries than a warp sorts in its registers

template <int MODE>
__device__ __forceinline__ float gather_weight(const GatherParams& p, int d) {
    if (MODE == FGL_AGG_MEAN) return 1.0f / (float)(__ldg(p.indptr + d + 1) - __ldg(p.indptr + d));
    if (MODE == FGL_AGG_SYMNORM) return 1.0f / sqrtf((float)__ldg(p.dst_deg + d));
    return 1.0f;
}

// The whole transposition in one cooperative launch: sixteen lanes per destination row count their edges' sources and keep
// (source, rank, destination) in registers over the scan of the counts (two levels, over the CTAs' runs of sources) until they
// place them.  Edges beyond what the registers hold (rows past the first kKeep of a group of lanes, or entries past the
// sixteenth of a row) are counted apart and placed behind the others of their source with a second round of atomics.
// As seven launches -- zeroing, histogram, scan, placement, hubs -- it was 36 us on the device and 20 us on the host for a
// block of 374 k edges.
constexpr int kTransposeThreads = 512;
constexpr int kTransposeMaxCtas = kWsTeamMax;
constexpr int kKeep = 4;

struct TransposeParams {
    const int32_t* indptr;
    const int32_t* src;
    int32_t n_dst, n_src;
    const int32_t* n_dst_dev;
    int32_t* t_indptr;
    int32_t* t_dst;
    int64_t t_cap;
    int32_t* hubs;
    int32_t* counts;            // 2 * n_src words: kept edges, then the others
    unsigned long long* bar;    // barrier counter; the next word: what it was at when the last launch ended, read by all
                                // before the first barrier and raised behind the last
    int32_t* partial;           // one word per CTA
    int32_t* status;
};

__global__ void __launch_bounds__(kTransposeThreads) transpose_block_kernel(const TransposeParams p) {
    __shared__ int s_scan[40];
    Team t;
    t.rank = blockIdx.x;
    t.size = gridDim.x;
    t.epoch = 0;
    t.bar = p.bar;
    t.base = *(volatile unsigned long long*)(p.bar + 1);
    t.status = p.status;
    const int n_dst = p.n_dst_dev ? min(max(__ldg(p.n_dst_dev), 0), p.n_dst) : p.n_dst;
    const int tid = blockIdx.x * kTransposeThreads + (int)threadIdx.x, n_threads = gridDim.x * kTransposeThreads;
    int32_t* const more = p.counts + p.n_src;
    for (int64_t i = tid; i < 2 * (int64_t)p.n_src; i += n_threads) __stcg(p.counts + i, 0);
    if (tid == 0) p.hubs[0] = 0;
    const int lane = threadIdx.x & 15, group = tid >> 4, groups = n_threads >> 4;
    int a[kKeep], b[kKeep], src[kKeep], rank[kKeep];
#pragma unroll
    for (int q = 0; q < kKeep; ++q) {
        const int64_t d = group + (int64_t)q * groups;
        a[q] = d < n_dst ? __ldg(p.indptr + d) : 0;
        b[q] = d < n_dst ? __ldg(p.indptr + d + 1) : 0;
    }
#pragma unroll
    for (int q = 0; q < kKeep; ++q) src[q] = a[q] + lane < b[q] ? __ldg(p.src + a[q] + lane) : -2;
    if (!team_barrier(t)) return;

    auto count_more = [&](int from, int to) {
        for (int e = from + lane; e < to; e += 16) {
            const int s = __ldg(p.src + e);
            if (s >= 0 && s < p.n_src) atomicAdd(more + s, 1);
            else if (p.status) set_status(p.status, FGL_ERR_BOUNDS);
        }
    };
#pragma unroll
    for (int q = 0; q < kKeep; ++q) {
        rank[q] = 0;
        if (src[q] >= 0 && src[q] < p.n_src) {
            rank[q] = atomicAdd(p.counts + src[q], 1);
        } else {
            if (src[q] != -2 && p.status) set_status(p.status, FGL_ERR_BOUNDS);
            src[q] = -2;
        }
    }
#pragma unroll
    for (int q = 0; q < kKeep; ++q) count_more(a[q] + 16, b[q]);
    for (int64_t d = group + (int64_t)kKeep * groups; d < n_dst; d += groups) count_more(__ldg(p.indptr + d), __ldg(p.indptr + d + 1));
    if (!team_barrier(t)) return;

    // every CTA scans a run of sources
    constexpr int kPer = 4;
    const int per = ((p.n_src + t.size - 1) / t.size + kPer - 1) / kPer * kPer;
    const int lo = min((int64_t)p.n_src, (int64_t)t.rank * per), hi = min(p.n_src, lo + per);
    int acc = 0;
    for (int i = lo + (int)threadIdx.x; i < hi; i += kTransposeThreads) acc += __ldcg(p.counts + i) + __ldcg(more + i);
    const int mine = block_sum(acc, s_scan);
    if (threadIdx.x == 0) __stcg(p.partial + t.rank, mine);
    if (!team_barrier(t)) return;

    int before = 0, total = 0;
    for (int q = threadIdx.x; q < t.size; q += kTransposeThreads) {
        const int x = __ldcg(p.partial + q);
        total += x;
        if (q < t.rank) before += x;
    }
    int running = block_sum(before, s_scan);
    total = block_sum(total, s_scan);
    if (tid == 0) p.t_indptr[p.n_src] = total;
    for (int tile = lo; tile < hi; tile += kPer * kTransposeThreads) {
        const int base = tile + (int)threadIdx.x * kPer;
        int v[kPer], sum = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            v[k] = base + k < hi ? __ldcg(p.counts + base + k) + __ldcg(more + base + k) : 0;
            sum += v[k];
        }
        int tile_total;
        int excl = running + block_excl_scan(sum, s_scan, tile_total);
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            if (base + k < hi) __stcg(p.t_indptr + base + k, excl);
            if (v[k] > kHubThreshold) p.hubs[1 + atomicAdd(p.hubs, 1)] = base + k;
            excl += v[k];
        }
        running += tile_total;
    }
    if (!team_barrier(t)) return;

    auto place = [&](int64_t at, int d) {
        if (at < p.t_cap) p.t_dst[at] = d;
        else if (p.status) set_status(p.status, FGL_ERR_CAPACITY);
    };
    auto place_more = [&](int from, int to, int d) {
        for (int e = from + lane; e < to; e += 16) {
            const int s = __ldg(p.src + e);
            if (s >= 0 && s < p.n_src)
                place((int64_t)__ldcg(p.t_indptr + s) + __ldcg(p.counts + s) + atomicSub(more + s, 1) - 1, d);
        }
    };
#pragma unroll
    for (int q = 0; q < kKeep; ++q)
        if (src[q] != -2) place((int64_t)__ldcg(p.t_indptr + src[q]) + rank[q], group + q * groups);
#pragma unroll
    for (int q = 0; q < kKeep; ++q) place_more(a[q] + 16, b[q], group + q * groups);
    for (int64_t d = group + (int64_t)kKeep * groups; d < n_dst; d += groups) place_more(__ldg(p.indptr + d), __ldg(p.indptr + d + 1), (int)d);
    if (tid == 0) p.bar[1] = t.base + (t.size > 1 ? (unsigned long long)t.epoch * t.size : 0ULL);
}

// acc += sum over j < deg of w_j * dy[d_j, columns c0 ..], lane j holding (d_j, w_j); U rows' loads in flight.
template <int VEC, int NACC, int U>
__device__ __forceinline__ void gather_add_rows(const GatherParams& p, int d, float w, int deg, int c0, int chunks, int lane,
                                                typename Vec<VEC>::T (&acc)[NACC]) {
    using V = Vec<VEC>;
    using T = typename V::T;
    for (int j0 = 0; j0 < deg; j0 += U) {
        T v[U][NACC];
        float wj[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = min(j0 + u, deg - 1);
            const int dj = __shfl_sync(0xffffffffu, d, j);
            wj[u] = __shfl_sync(0xffffffffu, w, j);
            const T* row = reinterpret_cast<const T*>(p.dy + (int64_t)dj * p.ldy);
#pragma unroll
            for (int k = 0; k < NACC; ++k) {
                const int c = c0 + k * 32 + lane;
                v[u][k] = c < chunks ? __ldg(row + c) : V::zero();
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (j0 + u < deg) {
#pragma unroll
                for (int k = 0; k < NACC; ++k) V::fma(acc[k], wj[u], v[u][k]);
            }
    }
}

__device__ __forceinline__ int warp_sort_ascending(int v, int lane) {
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const int other = __shfl_xor_sync(0xffffffffu, v, j);
            const bool up = (lane & k) == 0, lower = (lane & j) == 0;
            v = (lower == up) ? min(v, other) : max(v, other);
        }
    }
    return v;
}

// Up to 32 * R keys of a warp (lane l holds the keys r * 32 + l), sorted ascending.
template <int R>
__device__ __forceinline__ void warp_sort_regs(int (&v)[R], int lane) {
#pragma unroll
    for (int k = 2; k <= 32 * R; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int o = r ^ (j / 32);
                    if (o > r) {
                        const bool up = ((r * 32) & k) == 0;
                        const int x = v[r], y = v[o];
                        v[r] = up ? min(x, y) : max(x, y);
                        v[o] = up ? max(x, y) : min(x, y);
                    }
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int other = __shfl_xor_sync(0xffffffffu, v[r], j);
                    const bool up = ((r * 32 + lane) & k) == 0, lower = (lane & j) == 0;
                    v[r] = (lower == up) ? min(v[r], other) : max(v[r], other);
                }
            }
        }
    }
}

// One source row: the sorted list of `deg` <= 32 * R destination rows, lane l holding entries r * 32 + l.
template <int VEC, int MODE, int NACC, int R>
__device__ __forceinline__ void gather_one_source(const GatherParams& p, int s, int a, int deg, int chunks, int n_dst, int lane) {
    using V = Vec<VEC>;
    using T = typename V::T;
    constexpr int UNR = NACC == 1 ? 8 : (NACC == 2 ? 4 : 2);
    int d[R];
    float w[R];
#pragma unroll
    for (int r = 0; r < R; ++r) d[r] = r * 32 + lane < deg ? __ldg(p.t_dst + a + r * 32 + lane) : 0x7fffffff;
    warp_sort_regs<R>(d, lane);
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = r * 32 + lane < deg ? gather_weight<MODE>(p, d[r]) : 0.0f;
    const float ws = MODE == FGL_AGG_SYMNORM ? 1.0f / sqrtf((float)__ldg(p.src_deg + s)) : 1.0f;
    const bool self = p.dy_self != nullptr && s < n_dst;
    const T* self_row = reinterpret_cast<const T*>(p.dy_self + (self ? (int64_t)s * p.ld_self : 0));
    T* out = reinterpret_cast<T*>(p.dx + (int64_t)s * p.ldx);
    for (int c0 = 0; c0 < chunks; c0 += 32 * NACC) {
        T acc[NACC];
#pragma unroll
        for (int k = 0; k < NACC; ++k) acc[k] = V::zero();
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (deg > r * 32) gather_add_rows<VEC, NACC, UNR>(p, d[r], w[r], min(32, deg - r * 32), c0, chunks, lane, acc);
#pragma unroll
        for (int k = 0; k < NACC; ++k) {
            const int c = c0 + k * 32 + lane;
            if (c < chunks) {
                T v = (MODE == FGL_AGG_SYMNORM) ? V::scale(acc[k], ws) : acc[k];
                if (self) V::fma(v, 1.0f, __ldg(self_row + c));
                out[c] = v;
            }
        }
    }
}

// Sources with at most kHubThreshold entries: a warp takes eight at a time, a quarter of the ids' range apart from one
// another (popular sources have neighbouring numbers).  Most sources of a sampled block have one to four entries: their offsets,
// lists and weights are read by the eight quads at once, sorted in the quads, and then G sources' rows at a time are in flight
// -- one at a time, the chain offset -> list -> weight -> row of every source stood in the way of the next one's.
// Sources with more entries follow one by one, their lists sorted in the warp's registers.
template <int VEC, int MODE, int NACC>
__device__ __forceinline__ void gather_small_sources(const GatherParams& p, int block, int n_blocks) {
    using V = Vec<VEC>;
    using T = typename V::T;
    constexpr int G = NACC == 1 ? 4 : (NACC == 2 ? 2 : 1);
    const int lane = threadIdx.x & 31, quad = lane >> 2, j = lane & 3;
    const int warp_global = block * 8 + (threadIdx.x >> 5), n_warps = n_blocks * 8;
    const int chunks = p.dim / VEC;
    const int n_dst = p.n_dst_dev ? min(max(__ldg(p.n_dst_dev), 0), p.n_dst) : p.n_dst;
    const int eighth = (p.n_src + 7) / 8;
    for (int u = warp_global; u < eighth; u += n_warps) {
        const int s = quad * eighth + u;
        int a = 0, deg = 0;
        if (s < p.n_src) {
            a = __ldg(p.t_indptr + s);
            deg = __ldg(p.t_indptr + s + 1) - a;
        }
        int d = j < deg ? __ldg(p.t_dst + a + j) : 0x7fffffff;
        if (deg > 4) d = 0x7fffffff;
        {  // sorted within the quad
            int o = __shfl_xor_sync(0xffffffffu, d, 1);
            d = ((j & 1) == ((j >> 1) & 1)) ? min(d, o) : max(d, o);
            o = __shfl_xor_sync(0xffffffffu, d, 2);
            d = (j & 2) ? max(d, o) : min(d, o);
            o = __shfl_xor_sync(0xffffffffu, d, 1);
            d = (j & 1) ? max(d, o) : min(d, o);
        }
        const bool on = j < deg && deg <= 4;
        const float w = on ? gather_weight<MODE>(p, d) : 0.0f;
        const float ws = (MODE == FGL_AGG_SYMNORM && deg > 0 && deg <= 4) ? 1.0f / sqrtf((float)__ldg(p.src_deg + s)) : 1.0f;
        const unsigned few = __ballot_sync(0xffffffffu, s < p.n_src && deg <= 4);   // bit 4 * i: source i is settled here
        const unsigned many = __ballot_sync(0xffffffffu, deg > 4 && deg <= kHubThreshold);
        const unsigned entry = __ballot_sync(0xffffffffu, on);
#pragma unroll 1
        for (int i0 = 0; i0 < 8; i0 += G) {
            if (((few >> (4 * i0)) & (G == 4 ? 0xffffu : (G == 2 ? 0xffu : 0xfu))) == 0) continue;
            for (int c0 = 0; c0 < chunks; c0 += 32 * NACC) {
                T acc[G][NACC];
#pragma unroll
                for (int g = 0; g < G; ++g)
#pragma unroll
                    for (int k = 0; k < NACC; ++k) {
                        acc[g][k] = V::zero();
                    }
#pragma unroll 1
                for (int e = 0; e < 4; ++e) {
                    unsigned any = 0;
#pragma unroll
                    for (int g = 0; g < G; ++g) any |= (entry >> (4 * (i0 + g) + e)) & 1u;
                    if (!any) break;  // warp-uniform; the entries of a source fill its quad from the front
                    T v[G][NACC];
                    float we[G];
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        const int from = 4 * (i0 + g) + e;
                        const bool has = (entry >> from) & 1u;
                        const int de = __shfl_sync(0xffffffffu, d, from);
                        we[g] = __shfl_sync(0xffffffffu, w, from);
                        const T* row = reinterpret_cast<const T*>(p.dy + (int64_t)(has ? de : 0) * p.ldy);
#pragma unroll
                        for (int k = 0; k < NACC; ++k) {
                            const int c = c0 + k * 32 + lane;
                            v[g][k] = has && c < chunks ? __ldg(row + c) : V::zero();
                        }
                    }
#pragma unroll
                    for (int g = 0; g < G; ++g)
#pragma unroll
                        for (int k = 0; k < NACC; ++k) V::fma(acc[g][k], we[g], v[g][k]);
                }
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    if (!((few >> (4 * (i0 + g))) & 1u)) continue;
                    const int sg = (i0 + g) * eighth + u;
                    const float wg = MODE == FGL_AGG_SYMNORM ? __shfl_sync(0xffffffffu, ws, 4 * (i0 + g)) : 1.0f;
                    const bool self = p.dy_self != nullptr && sg < n_dst;
                    const T* self_row = reinterpret_cast<const T*>(p.dy_self + (self ? (int64_t)sg * p.ld_self : 0));
                    T* out = reinterpret_cast<T*>(p.dx + (int64_t)sg * p.ldx);
#pragma unroll
                    for (int k = 0; k < NACC; ++k) {
                        const int c = c0 + k * 32 + lane;
                        if (c < chunks) {
                            T r = (MODE == FGL_AGG_SYMNORM) ? V::scale(acc[g][k], wg) : acc[g][k];
                            if (self) V::fma(r, 1.0f, __ldg(self_row + c));
                            out[c] = r;
                        }
                    }
                }
            }
        }
        for (unsigned m = many & 0x11111111u; m; m &= m - 1) {  // warp-uniform
            const int from = __ffs(m) - 1;
            const int sm = (from >> 2) * eighth + u, am = __shfl_sync(0xffffffffu, a, from), dm = __shfl_sync(0xffffffffu, deg, from);
            if (dm <= 32) gather_one_source<VEC, MODE, NACC, 1>(p, sm, am, dm, chunks, n_dst, lane);
            else if (dm <= 64) gather_one_source<VEC, MODE, NACC, 2>(p, sm, am, dm, chunks, n_dst, lane);
            else gather_one_source<VEC, MODE, NACC, 4>(p, sm, am, dm, chunks, n_dst, lane);
        }
    }
}

// Hubs, a tile of 32 vectors of the row at a time.  The list is sorted (bitonic network in shared memory, over the list padded to
// a power of two), warp k of the CTA adds the k-th eighth of it and the eight partial sums are folded in warp order, so the result
// does not depend on the order in which the transposition's atomics filled the list.
//   CLUSTER = false: a CTA per hub of up to kHubSplitMin entries and tile.
//   CLUSTER = true:  a cluster of eight CTAs per longer hub and tile, for the longest list of a block is what a launch waits for
//                    (4800 entries: 200 us in one CTA).  CTA r keeps the entries whose destination lies in the r-th eighth of the
//                    destination range -- a fixed partition, whatever the order of the list -- and rank 0 folds the CTAs' sums in
//                    rank order through distributed shared memory.  An eighth with more than kHubSort entries is not sorted but
//                    counted, over windows of kHubWindow destination rows (16-bit counts), which orders it as well.
constexpr int kHubSplitMin = 512;
constexpr int kHubSort = 2048;
constexpr int kHubWindow = 4096;
constexpr int kHubCluster = 8;
constexpr int kHubEvery = 4;  // one of so many clusters of the launch takes hubs

template <typename T>
struct HubSmem {
    uint32_t words[kHubSort];  // the list, or the counts of a window
    T part[8][32];
    T sum[32];
    int sel[256];
    int wcnt[8];
    int count;
};

// This thread's column of sum over the sorted list[lo .. hi) of w * dy[d].
template <int VEC, int MODE>
__device__ __forceinline__ void hub_add_rows(const GatherParams& p, const int* list, int lo, int hi, const typename Vec<VEC>::T* dy,
                                             typename Vec<VEC>::T& acc) {
    using T = typename Vec<VEC>::T;
    constexpr int UNR = 8;
    for (int j0 = lo; j0 < hi; j0 += UNR) {
        T v[UNR];
        float w[UNR];
#pragma unroll
        for (int u = 0; u < UNR; ++u) {
            const int dj = list[min(j0 + u, hi - 1)];
            w[u] = gather_weight<MODE>(p, dj);
            v[u] = __ldg(dy + (int64_t)dj * (p.ldy / VEC));
        }
#pragma unroll
        for (int u = 0; u < UNR; ++u)
            if (j0 + u < hi) Vec<VEC>::fma(acc, w[u], v[u]);
    }
}

template <int VEC, int MODE, bool CLUSTER>
__device__ __forceinline__ void gather_hubs(const GatherParams& p, int block, int n_blocks, HubSmem<typename Vec<VEC>::T>& sm) {
    namespace cg = cooperative_groups;
    using V = Vec<VEC>;
    using T = typename V::T;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int chunks = p.dim / VEC, tiles = (chunks + 31) / 32;
    const int n_dst = p.n_dst_dev ? min(max(__ldg(p.n_dst_dev), 0), p.n_dst) : p.n_dst;
    const int rank = CLUSTER ? (int)cg::this_cluster().block_rank() : 0;
    const int unit = CLUSTER ? block / kHubCluster : block;
    const int n_units = CLUSTER ? n_blocks / kHubCluster : n_blocks;
    const int64_t n_work = (int64_t)min(__ldg(p.hubs), p.n_src) * tiles;  // (hub, tile) pairs; this unit has unit, unit + n_units, ...
    int* list = reinterpret_cast<int*>(sm.words);
    // Which of them are of this size class is found 256 at a time, a thread per pair, and compacted in order -- every CTA of a
    // cluster arrives at the same selection -- instead of one dependent pair of loads per hub in turn.
    for (int64_t base = 0; base * n_units + unit < n_work; base += 256) {
        const int64_t mine = (base + threadIdx.x) * n_units + unit;
        bool ok = false;
        if (mine < n_work) {
            const int s = __ldg(p.hubs + 1 + mine / tiles);
            const int deg = __ldg(p.t_indptr + s + 1) - __ldg(p.t_indptr + s);
            ok = CLUSTER ? deg > kHubSplitMin : deg <= kHubSplitMin;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, ok);
        if (lane == 0) sm.wcnt[warp] = __popc(bal);
        __syncthreads();
        int before = 0, n_sel = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (q < warp) before += sm.wcnt[q];
            n_sel += sm.wcnt[q];
        }
        if (ok) sm.sel[before + __popc(bal & ((1u << lane) - 1u))] = (int)threadIdx.x;
        __syncthreads();
        for (int i_sel = 0; i_sel < n_sel; ++i_sel) {
            const int64_t work = (base + sm.sel[i_sel]) * n_units + unit;
            const int s = __ldg(p.hubs + 1 + work / tiles), c = (int)(work % tiles) * 32 + lane;
            const bool in = c < chunks;
            const int a = __ldg(p.t_indptr + s), deg = __ldg(p.t_indptr + s + 1) - a;
            const T* dy = reinterpret_cast<const T*>(p.dy) + (in ? c : 0);
            const int seg = CLUSTER ? (n_dst + kHubCluster - 1) / kHubCluster : n_dst;
            const int d_lo = rank * seg, d_hi = min(n_dst, d_lo + seg);
            T acc = V::zero();
            int m = deg;
            if (CLUSTER) {
                if (threadIdx.x == 0) sm.count = 0;
                __syncthreads();
                for (int i = threadIdx.x; i < deg; i += 256) {
                    const int d = __ldg(p.t_dst + a + i);
                    if (d >= d_lo && d < d_hi) {
                        const int at = atomicAdd(&sm.count, 1);
                        if (at < kHubSort) list[at] = d;
                    }
                }
                __syncthreads();
                m = sm.count;
            } else {
                for (int i = threadIdx.x; i < deg; i += 256) list[i] = __ldg(p.t_dst + a + i);
            }
            if (m <= kHubSort) {
                int n2 = 64;
                while (n2 < m) n2 <<= 1;
                for (int i = m + (int)threadIdx.x; i < n2; i += 256) list[i] = 0x7fffffff;
                __syncthreads();
                for (int k = 2; k <= n2; k <<= 1) {
                    for (int q = k >> 1; q > 0; q >>= 1) {
                        for (int i = threadIdx.x; i < n2 / 2; i += 256) {
                            const int x0 = 2 * i - (i & (q - 1)), x1 = x0 + q;  // the i-th pair of this step
                            const int x = list[x0], y = list[x1];
                            if ((x > y) == ((x0 & k) == 0)) {
                                list[x0] = y;
                                list[x1] = x;
                            }
                        }
                        __syncthreads();
                    }
                }
                const int per = (m + 7) / 8;
                hub_add_rows<VEC, MODE>(p, list, warp * per, min(warp * per + per, m), dy, acc);
            } else {
                for (int w0 = d_lo; w0 < d_hi; w0 += kHubWindow) {
                    __syncthreads();  // the previous window's counts have been read
                    for (int i = threadIdx.x; i < kHubWindow / 2; i += 256) sm.words[i] = 0u;
                    __syncthreads();
                    for (int e = a + (int)threadIdx.x; e < a + deg; e += 256) {
                        const int d = __ldg(p.t_dst + e), off = d - w0;
                        if (d < d_hi && off >= 0 && off < kHubWindow) atomicAdd(sm.words + (off >> 1), 1u << (16 * (off & 1)));
                    }
                    __syncthreads();
                    const int hi = min(kHubWindow, d_hi - w0);
                    for (int off = warp * (kHubWindow / 8); off < min((warp + 1) * (kHubWindow / 8), hi); ++off) {
                        const int n = (int)((sm.words[off >> 1] >> (16 * (off & 1))) & 0xffffu);
                        if (n) V::fma(acc, (float)n * gather_weight<MODE>(p, w0 + off), __ldg(dy + (int64_t)(w0 + off) * (p.ldy / VEC)));
                    }
                }
            }
            sm.part[warp][lane] = acc;
            __syncthreads();
            T total = V::zero();
            if (warp == 0) {
#pragma unroll
                for (int q = 0; q < 8; ++q) V::fma(total, 1.0f, sm.part[q][lane]);
                if (CLUSTER) sm.sum[lane] = total;
            }
            if (CLUSTER) {
                cg::this_cluster().sync();
                if (rank == 0 && warp == 0)
                    for (int q = 1; q < kHubCluster; ++q) V::fma(total, 1.0f, cg::this_cluster().map_shared_rank(sm.sum, q)[lane]);
            }
            if (rank == 0 && warp == 0 && in) {
                if (MODE == FGL_AGG_SYMNORM) total = V::scale(total, 1.0f / sqrtf((float)__ldg(p.src_deg + s)));
                if (p.dy_self != nullptr && s < n_dst)
                    V::fma(total, 1.0f, __ldg(reinterpret_cast<const T*>(p.dy_self + (int64_t)s * p.ld_self) + c));
                reinterpret_cast<T*>(p.dx + (int64_t)s * p.ldx)[c] = total;
            }
            if (CLUSTER) cg::this_cluster().sync();  // rank 0 has read the sums
            __syncthreads();                         // list and partial sums are consumed
        }
        __syncthreads();
    }
}

// One launch of clusters: of every kHubEvery one takes hubs (while there are hub clusters), the others' CTAs the remaining sources.
// What the launch needs is row data in flight: held to 64 registers (four CTAs per SM; six where a lane's load is 8 or 4 bytes)
// it is faster than with the 110 the compiler would take, a few spills included (inner block of 26 k x 173 k rows, 374 k edges:
// 256 floats 166 -> 108 us; reads of the rows, 410 MB, and writes, 177 MB, then go through the L2 at 5.4 TB/s).
template <int VEC, int MODE, int NACC>
__global__ void __cluster_dims__(kHubCluster, 1, 1) __launch_bounds__(256, VEC == 4 ? 4 : 6) agg_bwd_gather_kernel(const GatherParams p) {
    __shared__ HubSmem<typename Vec<VEC>::T> sm;
    const int cluster = (int)blockIdx.x / kHubCluster, r = (int)blockIdx.x % kHubCluster;
    const int hub_clusters = p.hub_ctas / kHubCluster;
    if (cluster < hub_clusters * kHubEvery && cluster % kHubEvery == 0) {
        const int block = cluster / kHubEvery * kHubCluster + r;
        gather_hubs<VEC, MODE, true>(p, block, p.hub_ctas, sm);
        gather_hubs<VEC, MODE, false>(p, block, p.hub_ctas, sm);
    } else {
        const int others = cluster - min(cluster / kHubEvery + 1, hub_clusters);
        gather_small_sources<VEC, MODE, NACC>(p, others * kHubCluster + r, (int)gridDim.x - p.hub_ctas);
    }
}

template <int VEC, int MODE>
static void launch_gather_nacc(const GatherParams& p, int sms, cudaStream_t st) {
    const int chunks = p.dim / VEC;
    GatherParams q = p;
    const int64_t want = ((int64_t)p.n_src + 64 * kHubCluster - 1) / (64 * kHubCluster);  // clusters, eight sources per warp
    const int small = (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)sms * 8 / kHubCluster));
    const int hub_clusters = std::max(1, std::min(2 * sms / kHubCluster, small / (kHubEvery - 1)));
    q.hub_ctas = hub_clusters * kHubCluster;
    const int grid = std::max(small + hub_clusters, hub_clusters * kHubEvery - (kHubEvery - 2)) * kHubCluster;
    if (chunks <= 32) agg_bwd_gather_kernel<VEC, MODE, 1><<<grid, 256, 0, st>>>(q);
    else if (chunks <= 64) agg_bwd_gather_kernel<VEC, MODE, 2><<<grid, 256, 0, st>>>(q);
    else agg_bwd_gather_kernel<VEC, MODE, 4><<<grid, 256, 0, st>>>(q);
}

template <int VEC>
static void launch_gather_mode(int mode, const GatherParams& p, int sms, cudaStream_t st) {
    if (mode == FGL_AGG_SUM) launch_gather_nacc<VEC, FGL_AGG_SUM>(p, sms, st);
    if (mode == FGL_AGG_MEAN) launch_gather_nacc<VEC, FGL_AGG_MEAN>(p, sms, st);
    if (mode == FGL_AGG_SYMNORM) launch_gather_nacc<VEC, FGL_AGG_SYMNORM>(p, sms, st);
}

}  // namespace fgl

extern "C" {

int fgl_block_transpose(fgl_ws* ws, const int32_t* indptr, const int32_t* src, int32_t n_dst, int32_t n_src, int32_t* t_indptr,
                        int32_t* t_dst, int64_t t_cap, int32_t* hubs, int32_t* work, const int32_t* n_dst_dev, void* stream) {
    if (!ws || n_dst < 0 || n_src < 0 || t_cap < 0) return FGL_ERR_INVALID;
    if (!t_indptr || !hubs || (n_src > 0 && !work) || (t_cap > 0 && !t_dst) || (n_dst > 0 && (!indptr || !src))) return FGL_ERR_INVALID;
    cudaStream_t st = (cudaStream_t)stream;
    std::lock_guard<std::mutex> lock(ws->mu);
    DeviceGuard guard(ws->device);
    static std::atomic<int> cached{0};  // the same on every device of this architecture
    int per_sm = cached.load(std::memory_order_relaxed);
    if (per_sm == 0) {
        FGL_CUDA_OK(ws, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, transpose_block_kernel, kTransposeThreads, 0));
        cached.store(per_sm, std::memory_order_relaxed);
    }
    // two rows per group of lanes and four sources per thread: fewer CTAs make the phases longer, more the barriers
    const int64_t items = std::max<int64_t>((int64_t)n_dst * 8, n_src / 4);
    const int64_t most = std::min<int64_t>(kTransposeMaxCtas, (int64_t)std::min(per_sm, 2) * ws->sm_count);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(most, (items + kTransposeThreads - 1) / kTransposeThreads));
    TransposeParams p{indptr, src, n_dst, n_src, n_dst_dev, t_indptr, t_dst, t_cap, hubs, work,
                      (unsigned long long*)(ws->status + kWsTeamWord), ws->status + kWsTeamWord + 32, ws->status};
    void* args[] = {(void*)&p};
    FGL_CUDA_OK(ws, cudaLaunchCooperativeKernel((const void*)transpose_block_kernel, dim3(grid), dim3(kTransposeThreads), args, 0, st));
    return FGL_OK;
}

int fgl_agg_bwd_gather(fgl_ws* ws, int32_t mode, const int32_t* indptr, const int32_t* t_indptr, const int32_t* t_dst,
                       const int32_t* hubs, const int32_t* src_deg, const int32_t* dst_deg, const float* dy, int64_t ldy,
                       const float* dy_self, int64_t ld_self, int32_t dim, int32_t n_dst, int32_t n_src, float* dx, int64_t ldx,
                       const int32_t* n_dst_dev, void* stream) {
    if (!ws || mode < FGL_AGG_SUM || mode > FGL_AGG_SYMNORM || n_dst < 0 || n_src < 0 || dim < 1 || ldy < dim || ldx < dim)
        return FGL_ERR_INVALID;
    if (dy_self && (ld_self < dim || n_dst > n_src)) return FGL_ERR_INVALID;
    if (n_src == 0) return FGL_OK;
    if (!dx || !t_indptr || !hubs || (n_dst > 0 && (!dy || !t_dst || !indptr))) return FGL_ERR_INVALID;
    if (mode == FGL_AGG_SYMNORM && (!src_deg || !dst_deg)) return FGL_ERR_INVALID;
    GatherParams p{};
    p.indptr = indptr;
    p.t_indptr = t_indptr;
    p.t_dst = t_dst;
    p.hubs = hubs;
    p.src_deg = src_deg;
    p.dst_deg = dst_deg;
    p.dy = dy;
    p.dy_self = dy_self;
    p.dx = dx;
    p.ldy = ldy;
    p.ld_self = ld_self;
    p.ldx = ldx;
    p.dim = dim;
    p.n_dst = n_dst;
    p.n_src = n_src;
    p.n_dst_dev = n_dst_dev;
    DeviceGuard guard(ws->device);
    cudaStream_t st = (cudaStream_t)stream;
    const int sms = ws->sm_count > 0 ? ws->sm_count : 148;
    switch (pick_vec(dim, dy, ldy, dx, ldx, dy_self, dy_self ? ld_self : 4)) {
        case 4: launch_gather_mode<4>(mode, p, sms, st); break;
        case 2: launch_gather_mode<2>(mode, p, sms, st); break;
        default: launch_gather_mode<1>(mode, p, sms, st); break;
    }
    return cudaGetLastError() == cudaSuccess ? FGL_OK : FGL_ERR_CUDA;
}

}  // extern "C"
