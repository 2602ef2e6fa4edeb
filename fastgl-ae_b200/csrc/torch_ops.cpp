// The host path of the ``fastgl`` operators: argument checks, output allocation and the call into the C ABI, in one
// native call per operator.  Spelled in Python (ctypes), a call spent 10 to 20 us on the host for kernels of 2 to 5 us,
// and a layer is a dozen of them; here it is 2 to 4 us, most of it the launch.
//
// The kernels stay behind the C ABI: this module resolves the entry points from the library it is given (init) and holds
// no device code.  Every failed check and every status is a RuntimeError.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <array>
#include <atomic>
#include <chrono>
#include <mutex>
#include <string>
#include <vector>

#include "fastgl_b200.h"

namespace py = pybind11;

namespace {

// ---------------------------------------------------------------------------------------------------------------------
// the library
// ---------------------------------------------------------------------------------------------------------------------
void* g_lib = nullptr;

#define FGL_ENTRIES(X)                                                                                                  \
    X(fgl_status_str) X(fgl_last_error) X(fgl_ws_create) X(fgl_ws_check) X(fgl_sample) X(fgl_map) X(fgl_fused_capacity) \
    X(fgl_sample_map_fused_extra) X(fgl_cal_deg) X(fgl_exclusive_sum) X(fgl_stage_segments) X(fgl_agg_fwd)              \
    X(fgl_agg_fwd_window_counts) X(fgl_agg_edge_fwd) X(fgl_agg_edge_bwd) X(fgl_agg_edge_wgrad) X(fgl_agg_bwd)            \
    X(fgl_agg_bwd_self) X(fgl_agg_bwd_add) X(fgl_block_transpose) X(fgl_agg_bwd_gather) X(fgl_gather_rows) X(fgl_ws_time_next_launch)           \
    X(fgl_gat_fwd) X(fgl_gat_bwd) X(fgl_gat_bwd_partials) X(fgl_softmax_xent) X(fgl_adam_step) \
    X(fgl_block_degrees) X(fgl_mask_rows) X(fgl_weight_grad) X(fgl_weight_grad_scratch)

struct Api {
#define FGL_FIELD(name) decltype(&::name) name = nullptr;
    FGL_ENTRIES(FGL_FIELD)
#undef FGL_FIELD
} api;

void init(const std::string& path) {
    g_lib = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
    TORCH_CHECK(g_lib, "cannot load ", path, ": ", dlerror());
#define FGL_LOAD(name)                                                       \
    api.name = reinterpret_cast<decltype(&::name)>(dlsym(g_lib, #name));     \
    TORCH_CHECK(api.name, path, " lacks the symbol " #name);
    FGL_ENTRIES(FGL_LOAD)
#undef FGL_LOAD
}

std::mutex g_ws_lock;
std::array<fgl_ws*, 64> g_ws{};

fgl_ws* workspace(int device) {
    TORCH_CHECK(device >= 0 && device < (int)g_ws.size(), "device index ", device, " out of range");
    std::lock_guard<std::mutex> lock(g_ws_lock);
    if (!g_ws[device]) {
        const int rc = api.fgl_ws_create(device, &g_ws[device]);
        TORCH_CHECK(rc == FGL_OK, "fgl_ws_create(device=", device, ") failed: ", api.fgl_status_str(rc));
    }
    return g_ws[device];
}

void check(int rc, const char* what, fgl_ws* ws = nullptr) {
    if (rc == FGL_OK) return;
    const char* msg = ws ? api.fgl_last_error(ws) : "";
    TORCH_CHECK(false, what, " failed: ", api.fgl_status_str(rc), msg && *msg ? std::string(" (") + msg + ")" : std::string());
}

// ---------------------------------------------------------------------------------------------------------------------
// arguments
// ---------------------------------------------------------------------------------------------------------------------
// CHECK_INPUT of the reference: CUDA and contiguous (aggregate_acc.cpp:4-6)
const at::Tensor& tensor(const py::handle& o, const char* name) {
    TORCH_CHECK(THPVariable_Check(o.ptr()), name, " must be a torch.Tensor");
    return THPVariable_Unpack(o.ptr());
}

const at::Tensor& input(const py::handle& o, const char* name) {
    const at::Tensor& t = tensor(o, name);
    TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
    TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
    return t;
}

const at::Tensor& i32(const py::handle& o, const char* name) {
    const at::Tensor& t = input(o, name);
    TORCH_CHECK(t.scalar_type() == at::kInt, name, " must be int32 (got ", t.scalar_type(), ")");
    return t;
}

const at::Tensor& f32(const py::handle& o, const char* name) {
    const at::Tensor& t = input(o, name);
    TORCH_CHECK(t.scalar_type() == at::kFloat, name, " must be float32 (got ", t.scalar_type(), ")");
    return t;
}

const at::Tensor& matrix(const py::handle& o, const char* name) {
    const at::Tensor& t = f32(o, name);
    TORCH_CHECK(t.dim() == 2, name, " must be 2-D");
    return t;
}

// A float32 CUDA matrix whose rows are contiguous (a column slice of a wider buffer is fine).
const at::Tensor& rows_f32(const py::handle& o, const char* name) {
    const at::Tensor& t = tensor(o, name);
    TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kFloat && t.dim() == 2 && t.stride(1) == 1, name,
                " must be a float32 CUDA matrix with unit column stride");
    return t;
}

template <typename T>
T* ptr(const at::Tensor& t) {
    return t.defined() && t.numel() > 0 ? static_cast<T*>(t.data_ptr()) : nullptr;
}

at::Tensor optional_i32(const py::handle& o, const char* name) { return o.is_none() ? at::Tensor() : i32(o, name); }

struct Call {  // the device of a call, made current, with its stream and workspace
    c10::cuda::CUDAGuard guard;
    int device;
    fgl_ws* ws;
    c10::cuda::CUDAStream stream;
    explicit Call(const at::Tensor& t)
        : guard(t.device()), device(t.device().index()), ws(workspace(device)), stream(c10::cuda::getCurrentCUDAStream(device)) {}
    void* st() const { return stream.stream(); }
};

// ---------------------------------------------------------------------------------------------------------------------
// sampling and mapping
// ---------------------------------------------------------------------------------------------------------------------
bool is_64(const at::Tensor& edge_ptr) {
    TORCH_CHECK(edge_ptr.scalar_type() == at::kInt || edge_ptr.scalar_type() == at::kLong, "edge_ptr must be int32 or int64");
    return edge_ptr.scalar_type() == at::kLong;
}

py::tuple sample_node_csr(py::handle src_o, py::handle ptr_o, py::handle seeds_o, int64_t fanout, int flags, uint64_t rng_seed,
                          uint64_t rng_ctr, bool want_dst) {
    const at::Tensor &src = i32(src_o, "src_edges"), &edge_ptr = input(ptr_o, "edge_ptr"), &seeds = i32(seeds_o, "seed_nodes");
    const bool wide = is_64(edge_ptr);
    const int64_t S = seeds.numel();
    TORCH_CHECK(fanout >= 1 && fanout <= FGL_MAX_FANOUT && S * fanout <= 0x7fffffffLL, "sample_node failed: ",
                api.fgl_status_str(FGL_ERR_INVALID));
    Call c(seeds);
    auto opt = seeds.options();
    at::Tensor out_src = at::empty({std::max<int64_t>(1, S * fanout)}, opt);
    at::Tensor out_dst = want_dst ? at::empty({std::max<int64_t>(1, S * fanout)}, opt) : at::Tensor();
    at::Tensor out_ptr = at::empty({S + 1}, opt);
    int64_t n_edges = 0;
    int rc;
    {
        py::gil_scoped_release nogil;
        rc = api.fgl_sample(c.ws, ptr<void>(edge_ptr), wide, ptr<int32_t>(src), edge_ptr.numel() - 1, ptr<int32_t>(seeds), (int32_t)S,
                            (int32_t)fanout, flags, rng_seed, rng_ctr, ptr<int32_t>(out_ptr), ptr<int32_t>(out_src),
                            ptr<int32_t>(out_dst), &n_edges, c.st());
    }
    check(rc, "sample_node", c.ws);
    return py::make_tuple(out_src.slice(0, 0, n_edges), want_dst ? py::cast(out_dst.slice(0, 0, n_edges)) : py::none(), out_ptr, n_edges);
}

at::Tensor transfer_edge_id(py::handle src_o, py::handle dst_o, py::handle seeds_o, int64_t dst_nodes, int64_t unique_num,
                            int64_t n_edges, int flags) {
    const at::Tensor &src = i32(src_o, "src_edges"), &dst = i32(dst_o, "dst_edges"), &seeds = i32(seeds_o, "dst_edges_unique");
    const int64_t S = std::min<int64_t>(dst_nodes, seeds.numel());
    TORCH_CHECK(n_edges <= src.numel() && n_edges <= dst.numel(), "edge_nums exceeds the edge arrays");
    const int64_t cap = S + std::max<int64_t>(0, std::min<int64_t>(unique_num, n_edges));
    Call c(src);
    at::Tensor unique = at::empty({std::max<int64_t>(1, cap)}, src.options());
    int64_t n_unique = 0;
    int rc;
    {
        py::gil_scoped_release nogil;
        rc = api.fgl_map(c.ws, ptr<int32_t>(src), ptr<int32_t>(dst), ptr<int32_t>(seeds), (int32_t)S, n_edges, ptr<int32_t>(unique), cap,
                         flags, &n_unique, c.st());
    }
    check(rc, "transfer_edge_id", c.ws);
    return unique.slice(0, 0, n_unique);
}

struct FusedShape {
    int hops;
    int32_t fanout[FGL_MAX_HOPS];
    int64_t cap[FGL_MAX_HOPS + 1];
};

bool fused_shape(FusedShape& f, int64_t n_nodes, int64_t max_seeds, const std::vector<int64_t>& fanouts) {
    f.hops = (int)fanouts.size();
    if (f.hops < 1 || f.hops > FGL_MAX_HOPS || max_seeds > 0x7fffffffLL) return false;
    for (int h = 0; h < f.hops; ++h) {
        if (fanouts[h] < 1 || fanouts[h] > FGL_MAX_FANOUT) return false;
        f.fanout[h] = (int32_t)fanouts[h];
    }
    return api.fgl_fused_capacity(n_nodes, (int32_t)max_seeds, f.hops, f.fanout, f.cap) == FGL_OK;
}

void fused_graph(fgl_fused_args& a, const at::Tensor& edge_ptr, const at::Tensor& src, const FusedShape& f) {
    a.indptr = ptr<void>(edge_ptr);
    a.indices = ptr<int32_t>(src);
    a.n_nodes = edge_ptr.numel() - 1;
    a.indptr_is_64 = is_64(edge_ptr);
    a.n_hops = f.hops;
    for (int h = 0; h < f.hops; ++h) a.fanout[h] = f.fanout[h];
}

std::atomic<uint32_t> g_seq{0};

int32_t next_seq() {
    return (g_seq.fetch_add(1, std::memory_order_relaxed) & 0x3fffffff) + 1;  // never zero
}

// Waits until the rows of a launch's counts are closed with `seq`; false if the launch gave up, or if it takes so long that the
// caller had better sleep on an event.
bool poll_counts(const volatile int32_t* rows, const volatile int32_t* status, int64_t n, int32_t seq) {
    const auto until = std::chrono::steady_clock::now() + std::chrono::milliseconds(5);
    for (int64_t b = 0; b < n; ++b) {
        for (unsigned spins = 0; rows[b * FGL_COUNTS_STRIDE + FGL_COUNTS_STRIDE - 1] != seq; ++spins) {
            if (*status != FGL_OK) return false;
            if ((spins & 1023) == 1023 && std::chrono::steady_clock::now() > until) return false;
        }
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    return true;
}

bool wait_counts(const at::Tensor& counts_host, const at::Tensor& status_host, int32_t seq) {
    const auto* rows = static_cast<const int32_t*>(counts_host.data_ptr());
    const auto* status = static_cast<const int32_t*>(status_host.data_ptr());
    const int64_t n = counts_host.size(0);
    py::gil_scoped_release nogil;
    return poll_counts(rows, status, n, seq);
}

// One launch for a window of mini-batches, into the buffers of a FusedBatch; counts_host / status_host: its pinned copies, whose
// rows the launch closes with the number returned.
int32_t sample_map_fused(py::handle ptr_o, py::handle src_o, py::handle seeds_o, py::handle seed_counts_o, const std::vector<int64_t>& fanouts,
                      int flags, uint64_t rng_seed, uint64_t rng_ctr, int n_teams, int64_t table_slots, const at::Tensor& nodes,
                      const at::Tensor& counts, const std::vector<at::Tensor>& indptr, const std::vector<at::Tensor>& block_src,
                      py::handle counts_host, py::handle status_host) {
    const at::Tensor &src = i32(src_o, "src_edges"), &edge_ptr = input(ptr_o, "edge_ptr"), &seeds = i32(seeds_o, "seeds"),
                     &seed_counts = i32(seed_counts_o, "seed_counts");
    FusedShape f;
    TORCH_CHECK(fused_shape(f, edge_ptr.numel() - 1, seeds.size(1), fanouts), "sample_map_fused failed: ", api.fgl_status_str(FGL_ERR_INVALID));
    Call c(seeds);
    fgl_fused_args a{};
    fused_graph(a, edge_ptr, src, f);
    a.n_batches = (int32_t)seeds.size(0);
    for (int h = 0; h < f.hops; ++h) {
        a.block_indptr[h] = ptr<int32_t>(indptr[h]);
        a.block_indptr_stride[h] = indptr[h].stride(0);
        a.block_src[h] = ptr<int32_t>(block_src[h]);
        a.block_src_stride[h] = block_src[h].stride(0);
    }
    a.flags = flags;
    a.n_teams = n_teams;
    a.table_slots_hint = table_slots;
    a.rng_seed = rng_seed;
    a.rng_ctr = rng_ctr;
    a.seeds = ptr<int32_t>(seeds);
    a.seed_stride = seeds.stride(0);
    a.seed_counts = ptr<int32_t>(seed_counts);
    a.nodes = ptr<int32_t>(nodes);
    a.nodes_stride = nodes.stride(0);
    a.counts = ptr<int32_t>(counts);
    fgl_fused_extra x{};
    if (!counts_host.is_none()) {
        x.counts_host = static_cast<int32_t*>(tensor(counts_host, "counts_host").data_ptr());
        x.status_host = static_cast<int32_t*>(tensor(status_host, "status_host").data_ptr());
        *x.status_host = 0;
        x.seq = next_seq();
    }
    check(api.fgl_sample_map_fused_extra(c.ws, &a, &x, c.st()), "sample_map_fused", c.ws);
    return x.seq;
}

// Pinned words the blocking calls of a thread are answered in (one per thread: two threads may wait at once).
int32_t* answer_words() {
    static thread_local at::Tensor words;
    if (!words.defined()) words = at::empty({2 * FGL_COUNTS_STRIDE}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    return static_cast<int32_t*>(words.data_ptr());
}

// Above this size of the worst case, results are copied out of it into tensors of their own size: what a caller keeps then
// holds the memory it needs.  Below, the copy costs more than the memory.
constexpr int64_t kKeepArena = 1 << 18;       // int32 words
constexpr int64_t kMaxArena = 1LL << 29;      // beyond 2 GB of worst case the caller walks the hops one by one

// All hops of one mini-batch in one launch: (input nodes, [(indptr, src, dst, n_src, n_dst)] input layer first), or None when
// the worst case is too large for that.  ``fanouts`` in sampling order.
py::object sample_blocks(py::handle src_o, py::handle ptr_o, py::handle seeds_o, const std::vector<int64_t>& fanouts, int flags,
                         uint64_t rng_seed, uint64_t rng_ctr) {
    const at::Tensor &src = i32(src_o, "src_edges"), &edge_ptr = input(ptr_o, "edge_ptr"), &seeds = i32(seeds_o, "seed_nodes");
    FusedShape f;
    const int64_t S = seeds.numel();
    if (S == 0 || !fused_shape(f, edge_ptr.numel() - 1, S, fanouts)) return py::none();
    auto up = [](int64_t n) { return (n + 31) / 32 * 32; };
    const int64_t head = 2 * 32;  // the seed count, then the counts row
    int64_t total = head + up(f.cap[f.hops]);
    for (int h = 0; h < f.hops; ++h) total += up(f.cap[h] + 1) + 2 * up(f.cap[h] * f.fanout[h]);
    if (total > kMaxArena) return py::none();
    Call c(seeds);
    at::Tensor arena = at::empty({total}, seeds.options());
    int32_t* base = static_cast<int32_t*>(arena.data_ptr());
    fgl_fused_args a{};
    fused_graph(a, edge_ptr, src, f);
    fgl_fused_extra x{};
    int32_t* words = answer_words();
    x.counts_host = words;
    x.status_host = words + FGL_COUNTS_STRIDE;
    *x.status_host = 0;
    x.seq = next_seq();
    int64_t at_word = head, ptr_at[FGL_MAX_HOPS], src_at[FGL_MAX_HOPS], dst_at[FGL_MAX_HOPS];
    const int64_t nodes_at = at_word;
    at_word += up(f.cap[f.hops]);
    for (int h = 0; h < f.hops; ++h) {
        ptr_at[h] = at_word;
        src_at[h] = ptr_at[h] + up(f.cap[h] + 1);
        dst_at[h] = src_at[h] + up(f.cap[h] * f.fanout[h]);
        at_word = dst_at[h] + up(f.cap[h] * f.fanout[h]);
        a.block_indptr[h] = base + ptr_at[h];
        a.block_indptr_stride[h] = up(f.cap[h] + 1);
        a.block_src[h] = base + src_at[h];
        a.block_src_stride[h] = up(f.cap[h] * f.fanout[h]);
        x.block_dst[h] = base + dst_at[h];
    }
    a.n_batches = 1;
    a.flags = flags;
    a.rng_seed = rng_seed;
    a.rng_ctr = rng_ctr;
    a.seeds = ptr<int32_t>(seeds);
    a.seed_stride = S;
    a.seed_counts = nullptr;  // every seed
    a.nodes = base + nodes_at;
    a.nodes_stride = up(f.cap[f.hops]);
    a.counts = base + 32;
    int rc;
    {
        py::gil_scoped_release nogil;
        rc = api.fgl_sample_map_fused_extra(c.ws, &a, &x, c.st());
        if (rc == FGL_OK) {
            if (!poll_counts(words, x.status_host, 1, x.seq)) c.stream.synchronize();
            if (*(volatile int32_t*)x.status_host != FGL_OK) rc = api.fgl_ws_check(c.ws, c.st());
        }
    }
    check(rc, "sample_blocks", c.ws);
    const int32_t* n = words;
    if (total > kKeepArena) {
        int64_t exact = up(n[f.hops]);
        for (int h = 0; h < f.hops; ++h) exact += up(n[h] + 1) + 2 * up(n[8 + h]);
        at::Tensor own = at::empty({exact}, seeds.options());
        int32_t* to = static_cast<int32_t*>(own.data_ptr());
        std::vector<fgl_segment> seg;
        at_word = 0;
        auto move = [&](int64_t from, int64_t words_n) {
            seg.push_back({to + at_word, base + from, words_n * 4});
            const int64_t where = at_word;
            at_word += up(words_n);
            return where;
        };
        const int64_t new_nodes = move(nodes_at, n[f.hops]);
        TORCH_INTERNAL_ASSERT(new_nodes == 0);
        for (int h = 0; h < f.hops; ++h) {
            ptr_at[h] = move(ptr_at[h], n[h] + 1);
            src_at[h] = move(src_at[h], n[8 + h]);
            dst_at[h] = move(dst_at[h], n[8 + h]);
        }
        for (size_t i = 0; i < seg.size(); i += FGL_MAX_SEGMENTS)
            check(api.fgl_stage_segments(seg.data() + i, (int32_t)std::min<size_t>(FGL_MAX_SEGMENTS, seg.size() - i), nullptr, nullptr, 0,
                                         c.st()), "sample_blocks");
        arena = own;
    }
    py::list blocks;
    for (int h = f.hops - 1; h >= 0; --h)
        blocks.append(py::make_tuple(arena.slice(0, ptr_at[h], ptr_at[h] + n[h] + 1), arena.slice(0, src_at[h], src_at[h] + n[8 + h]),
                                     arena.slice(0, dst_at[h], dst_at[h] + n[8 + h]), n[h + 1], n[h]));
    const int64_t first = total > kKeepArena ? 0 : nodes_at;
    return py::make_tuple(arena.slice(0, first, first + n[f.hops]), blocks);
}

// ---------------------------------------------------------------------------------------------------------------------
// block CSR
// ---------------------------------------------------------------------------------------------------------------------
at::Tensor cal_deg(py::handle edges_o, int64_t n) {
    const at::Tensor& edges = i32(edges_o, "edges");
    Call c(edges);
    at::Tensor deg = at::empty({n}, edges.options());
    check(api.fgl_cal_deg(ptr<int32_t>(edges), edges.numel(), ptr<int32_t>(deg), (int32_t)n, c.st()), "cal_deg");
    return deg;
}

at::Tensor exclusive_sum(py::handle degs_o) {
    const at::Tensor& degs = i32(degs_o, "in_degs");
    Call c(degs);
    at::Tensor out = at::empty({degs.numel() + 1}, degs.options());
    check(api.fgl_exclusive_sum(c.ws, ptr<int32_t>(degs), degs.numel(), ptr<int32_t>(out), c.st()), "exclusive_sum", c.ws);
    return out;
}

void stage_segments(const std::vector<std::pair<py::object, py::object>>& copies, py::handle words_dst, const std::vector<int64_t>& words) {
    TORCH_CHECK(copies.size() <= FGL_MAX_SEGMENTS && words.size() <= FGL_MAX_SEGMENTS, "at most 8 copies and 8 words per call");
    fgl_segment seg[FGL_MAX_SEGMENTS];
    int32_t values[FGL_MAX_SEGMENTS];
    const at::Tensor* on = nullptr;
    for (size_t i = 0; i < copies.size(); ++i) {
        const at::Tensor &dst = tensor(copies[i].first, "dst"), &src = tensor(copies[i].second, "src");
        TORCH_CHECK(dst.element_size() == 4 && src.element_size() == 4 && dst.is_cuda() && src.is_cuda(),
                    "stage_segments copies 4-byte CUDA tensors");
        TORCH_CHECK(dst.numel() >= src.numel() && src.is_contiguous() && dst.is_contiguous(),
                    "stage_segments needs contiguous tensors and a destination at least as large as the source");
        seg[i] = {dst.data_ptr(), src.data_ptr(), src.numel() * 4};
        on = &dst;
    }
    int32_t* to = nullptr;
    if (!words_dst.is_none()) {
        const at::Tensor& w = i32(words_dst, "words_dst");
        to = ptr<int32_t>(w);
        on = &w;
    }
    for (size_t i = 0; i < words.size(); ++i) values[i] = (int32_t)words[i];
    TORCH_CHECK(on, "stage_segments needs a destination");
    Call c(*on);
    check(api.fgl_stage_segments(seg, (int32_t)copies.size(), to, values, (int32_t)words.size(), c.st()), "stage_segments");
}

// ---------------------------------------------------------------------------------------------------------------------
// aggregation
// ---------------------------------------------------------------------------------------------------------------------
at::Tensor agg_fwd(int mode, const at::Tensor& edge_ptr, const at::Tensor& src, const at::Tensor& x, int64_t n_dst, const at::Tensor& src_deg,
                   const at::Tensor& dst_deg, bool passthrough, const at::Tensor& row_map, const at::Tensor& out_given,
                   const at::Tensor& n_dst_dev) {
    TORCH_CHECK(edge_ptr.numel() >= n_dst + 1, "edge_ptr is shorter than dst_nodes + 1");
    if (mode == FGL_AGG_SYMNORM) {
        const int64_t n_src = row_map.defined() ? row_map.numel() : x.size(0);
        TORCH_CHECK(src_deg.defined() && dst_deg.defined() && dst_deg.numel() >= n_dst && src_deg.numel() >= n_src,
                    "sym-norm needs src_norm_degs[n_src] and dst_norm_degs[n_dst]");
    }
    Call c(x);
    at::Tensor out = out_given.defined() ? out_given : at::empty({n_dst, x.size(1)}, x.options());
    check(api.fgl_agg_fwd(c.ws, mode, ptr<int32_t>(edge_ptr), ptr<int32_t>(src), ptr<int32_t>(src_deg), ptr<int32_t>(dst_deg),
                          ptr<int32_t>(row_map), row_map.defined() ? row_map.numel() : 0, ptr<float>(x), x.size(0), x.stride(0),
                          (int32_t)x.size(1), (int32_t)n_dst, passthrough ? FGL_AGG_ZERO_DEG_PASSTHROUGH : 0, ptr<float>(out),
                          out.stride(0), ptr<int32_t>(n_dst_dev), c.st()), "aggregate");
    return out;
}

at::Tensor aggregate(int mode, py::handle ptr_o, py::handle src_o, py::handle x_o, int64_t n_dst, py::handle src_deg, py::handle dst_deg,
                     bool passthrough, py::handle row_map, py::handle out, py::handle n_dst_dev) {
    return agg_fwd(mode, i32(ptr_o, "edge_ptr"), i32(src_o, "src_edges"), matrix(x_o, "input_feat"), n_dst,
                   optional_i32(src_deg, "src_norm_degs"), optional_i32(dst_deg, "dst_norm_degs"), passthrough,
                   optional_i32(row_map, "row_map"), out.is_none() ? at::Tensor() : rows_f32(out, "out"),
                   n_dst_dev.is_none() ? at::Tensor() : tensor(n_dst_dev, "n_dst_dev"));
}

// dw = x^T dy, into `out` if given.  A caller who lets torch multiply in TF32 gets torch's product; so does a contraction that is
// shorter than the output is wide (nothing to split).
at::Tensor weight_grad(const Call& c, const at::Tensor& x, const at::Tensor& dy, const at::Tensor& out_given = at::Tensor(),
                       const at::Tensor& scratch_given = at::Tensor()) {
    const int64_t k = x.size(0), m = x.size(1), n = dy.size(1);
    TORCH_CHECK(dy.size(0) == k, "x and dy must have the same number of rows");
    at::Tensor out = out_given.defined() ? out_given : at::empty({m, n}, x.options());
    auto rows = [](const at::Tensor& t) { return t.stride(1) == 1 && t.stride(0) >= t.size(1); };
    if (!rows(x) || !rows(dy) || !rows(out) || k < std::max(m, n) || k > 0x7fffffffLL || at::globalContext().allowTF32CuBLAS())
        return at::mm_out(out, x.t(), dy);
    at::Tensor scratch = scratch_given;
    const int64_t floats = api.fgl_weight_grad_scratch(c.ws, (int32_t)m, (int32_t)n, (int32_t)k);
    TORCH_CHECK(!scratch.defined() || scratch.numel() >= floats, "scratch must hold weight_grad_scratch(...) floats");
    if (!scratch.defined() && floats > 0) scratch = at::empty({floats}, x.options());
    check(api.fgl_weight_grad(c.ws, (int32_t)m, (int32_t)n, (int32_t)k, ptr<float>(x), x.stride(0), ptr<float>(dy), dy.stride(0),
                              ptr<float>(out), out.stride(0), ptr<float>(scratch), c.st()), "weight_grad", c.ws);
    return out;
}

at::Tensor weight_grad_op(py::handle x_o, py::handle dy_o, py::handle out_o, py::handle scratch_o) {
    const at::Tensor &x = rows_f32(x_o, "x"), &dy = rows_f32(dy_o, "dy");
    Call c(x);
    return weight_grad(c, x, dy, out_o.is_none() ? at::Tensor() : rows_f32(out_o, "out"),
                       scratch_o.is_none() ? at::Tensor() : f32(scratch_o, "scratch"));
}

int64_t weight_grad_scratch(int device, int64_t m, int64_t n, int64_t k) {
    return api.fgl_weight_grad_scratch(workspace(device), (int32_t)m, (int32_t)n, (int32_t)k);
}

struct Transposed {
    at::Tensor t_indptr, t_dst, hubs;
};

at::Tensor agg_bwd(int mode, const at::Tensor& edge_ptr, const at::Tensor& src, const at::Tensor& dy, int64_t n_src, const at::Tensor& src_deg,
                   const at::Tensor& dst_deg, const at::Tensor& n_dst_dev, const at::Tensor& d_self, const at::Tensor& out_given,
                   const Transposed* tb, bool accumulate = false) {
    const int64_t n_dst = dy.size(0), dim = dy.size(1);
    TORCH_CHECK(mode != FGL_AGG_SYMNORM || (src_deg.defined() && dst_deg.defined() && src_deg.numel() >= n_src && dst_deg.numel() >= n_dst),
                "sym-norm needs src_norm_degs[src_nodes] and dst_norm_degs[n_dst]");
    TORCH_CHECK(edge_ptr.numel() >= n_dst + 1, "edge_ptr is shorter than n_dst + 1");
    TORCH_CHECK(!out_given.defined() || (out_given.size(0) >= n_src && out_given.size(1) == dim), "out must be float32[src_nodes, dim]");
    TORCH_CHECK(!d_self.defined() || (d_self.size(0) == n_dst && d_self.size(1) == dim), "d_self must be float32[n_dst, dim]");
    Call c(dy);
    at::Tensor dx = out_given.defined() ? out_given : at::empty({n_src, dim}, dy.options());
    int rc;
    if (tb)
        rc = api.fgl_agg_bwd_gather(c.ws, mode, ptr<int32_t>(edge_ptr), ptr<int32_t>(tb->t_indptr), ptr<int32_t>(tb->t_dst),
                                    ptr<int32_t>(tb->hubs), ptr<int32_t>(src_deg), ptr<int32_t>(dst_deg), ptr<float>(dy), dy.stride(0),
                                    ptr<float>(d_self), d_self.defined() ? d_self.stride(0) : dim, (int32_t)dim, (int32_t)n_dst,
                                    (int32_t)n_src, ptr<float>(dx), dx.stride(0), ptr<int32_t>(n_dst_dev), c.st());
    else if (accumulate)
        rc = api.fgl_agg_bwd_add(c.ws, mode, ptr<int32_t>(edge_ptr), ptr<int32_t>(src), ptr<int32_t>(src_deg), ptr<int32_t>(dst_deg),
                                 ptr<float>(dy), dy.stride(0), ptr<float>(d_self), d_self.defined() ? d_self.stride(0) : dim,
                                 (int32_t)dim, (int32_t)n_dst, (int32_t)n_src, ptr<float>(dx), dx.stride(0), ptr<int32_t>(n_dst_dev),
                                 c.st());
    else if (d_self.defined())
        rc = api.fgl_agg_bwd_self(c.ws, mode, ptr<int32_t>(edge_ptr), ptr<int32_t>(src), ptr<int32_t>(src_deg), ptr<int32_t>(dst_deg),
                                  ptr<float>(dy), dy.stride(0), ptr<float>(d_self), d_self.stride(0), (int32_t)dim, (int32_t)n_dst,
                                  (int32_t)n_src, ptr<float>(dx), dx.stride(0), ptr<int32_t>(n_dst_dev), c.st());
    else
        rc = api.fgl_agg_bwd(c.ws, mode, ptr<int32_t>(edge_ptr), ptr<int32_t>(src), ptr<int32_t>(src_deg), ptr<int32_t>(dst_deg),
                             ptr<float>(dy), dy.stride(0), (int32_t)dim, (int32_t)n_dst, (int32_t)n_src, ptr<float>(dx), dx.stride(0),
                             ptr<int32_t>(n_dst_dev), c.st());
    check(rc, tb ? "aggregate_backward (gather)" : "aggregate_backward", tb ? c.ws : nullptr);
    return dx;
}

at::Tensor aggregate_backward(int mode, py::handle ptr_o, py::handle src_o, py::handle dy_o, int64_t n_src, py::handle src_deg,
                              py::handle dst_deg, py::handle n_dst_dev, py::handle d_self, py::handle out, py::handle t_indptr,
                              py::handle t_dst, py::handle hubs, bool accumulate) {
    Transposed tb;
    const bool gather = !t_indptr.is_none();
    if (gather) tb = {tensor(t_indptr, "t_indptr"), tensor(t_dst, "t_dst"), tensor(hubs, "hubs")};
    return agg_bwd(mode, i32(ptr_o, "edge_ptr"), i32(src_o, "src_edges"), rows_f32(dy_o, "d_input"), n_src,
                   optional_i32(src_deg, "src_norm_degs"), optional_i32(dst_deg, "dst_norm_degs"),
                   n_dst_dev.is_none() ? at::Tensor() : tensor(n_dst_dev, "n_dst_dev"),
                   d_self.is_none() ? at::Tensor() : rows_f32(d_self, "d_self"), out.is_none() ? at::Tensor() : rows_f32(out, "out"),
                   gather ? &tb : nullptr, accumulate);
}

void transpose_block(py::handle ptr_o, py::handle src_o, int64_t n_dst, int64_t n_src, py::handle n_dst_dev, const at::Tensor& t_indptr,
                     const at::Tensor& t_dst, int64_t edge_cap, const at::Tensor& hubs, const at::Tensor& work) {
    const at::Tensor &edge_ptr = i32(ptr_o, "edge_ptr"), &src = i32(src_o, "src_edges");
    Call c(edge_ptr);
    check(api.fgl_block_transpose(c.ws, ptr<int32_t>(edge_ptr), ptr<int32_t>(src), (int32_t)n_dst, (int32_t)n_src, ptr<int32_t>(t_indptr),
                                  ptr<int32_t>(t_dst), edge_cap, ptr<int32_t>(hubs), ptr<int32_t>(work),
                                  n_dst_dev.is_none() ? nullptr : ptr<int32_t>(tensor(n_dst_dev, "n_dst_dev")), c.st()),
          "transpose_block", c.ws);
}

// One layer of a window from the counts on the device; n_dst: the batches' destination counts as the host read them.
// start / end: addresses of CUDA events to record around the launch, or 0.
void aggregate_window(int mode, const at::Tensor& counts, int64_t hop, int64_t total, const at::Tensor& indptr, const at::Tensor& src,
                      py::handle nodes_o, py::handle x_o, py::handle out_o, py::handle self_o, uint64_t start, uint64_t end) {
    const at::Tensor &x = rows_f32(x_o, "input_feat"), &out = rows_f32(out_o, "out");
    const at::Tensor self = self_o.is_none() ? at::Tensor() : rows_f32(self_o, "self_out");
    const at::Tensor nodes = nodes_o.is_none() ? at::Tensor() : tensor(nodes_o, "nodes");
    TORCH_CHECK(out.size(0) >= total && (!self.defined() || self.size(0) >= total), "out is too small for the window's destination rows");
    Call c(x);
    if (start) check(api.fgl_ws_time_next_launch(c.ws, (void*)start, (void*)end), "time_next_launch");
    check(api.fgl_agg_fwd_window_counts(c.ws, mode, (int32_t)counts.size(0), ptr<int32_t>(indptr), indptr.stride(0), ptr<int32_t>(src),
                                        src.stride(0), ptr<int32_t>(nodes), nodes.defined() ? nodes.stride(0) : 0,
                                        ptr<int32_t>(counts) + hop, counts.stride(0), total, ptr<float>(x), nullptr, 0, x.size(0),
                                        x.stride(0), (int32_t)x.size(1), 0, ptr<float>(out), out.stride(0), ptr<float>(self),
                                        self.defined() ? self.stride(0) : x.size(1), c.st()),
          "aggregate_window");
}

at::Tensor gather_rows(py::handle table_o, py::handle ids_o, py::handle out_o) {
    const at::Tensor &x = rows_f32(table_o, "input_feat"), &ids = i32(ids_o, "ids");
    Call c(x);
    at::Tensor out = out_o.is_none() ? at::empty({ids.numel(), x.size(1)}, x.options()) : rows_f32(out_o, "out");
    check(api.fgl_gather_rows(c.ws, ptr<float>(x), nullptr, 0, x.size(0), x.stride(0), (int32_t)x.size(1), ptr<int32_t>(ids), ids.numel(),
                              ptr<float>(out), out.stride(0), c.st()), "gather_rows");
    return out;
}

// ---------------------------------------------------------------------------------------------------------------------
// the reference's layer operators
// ---------------------------------------------------------------------------------------------------------------------
std::vector<at::Tensor> forward_gcn(py::handle ptr_o, py::handle src_o, py::handle src_deg, py::handle dst_deg, py::handle x_o, py::handle w_o,
                                    int64_t n_dst) {
    const at::Tensor &w = f32(w_o, "weight"), &x = f32(x_o, "input_feat");
    return {agg_fwd(FGL_AGG_SYMNORM, i32(ptr_o, "edge_ptr"), i32(src_o, "src_edges"), at::mm(x, w), n_dst, i32(src_deg, "src_norm_degs"),
                    i32(dst_deg, "dst_norm_degs"), true, at::Tensor(), at::Tensor(), at::Tensor())};
}

std::vector<at::Tensor> backward_gcn(py::handle ptr_o, py::handle src_o, py::handle src_deg, py::handle dst_deg, py::handle dy_o,
                                     py::handle w_o, py::handle x_o) {
    const at::Tensor &w = f32(w_o, "weight"), &x = f32(x_o, "input_feat");
    const at::Tensor d = agg_bwd(FGL_AGG_SYMNORM, i32(ptr_o, "edge_ptr"), i32(src_o, "src_edges"), rows_f32(dy_o, "d_input"), x.size(0),
                                 i32(dst_deg, "src_norm_degs"), i32(src_deg, "dst_norm_degs"), at::Tensor(), at::Tensor(), at::Tensor(), nullptr);
    Call c(x);
    return {at::mm(d, w.t()), weight_grad(c, x, d)};
}

std::vector<at::Tensor> forward_gin(py::handle ptr_o, py::handle src_o, py::handle x_o, py::handle w_o, int64_t n_dst) {
    const at::Tensor& w = f32(w_o, "weight");
    at::Tensor tmp = agg_fwd(FGL_AGG_SUM, i32(ptr_o, "edge_ptr"), i32(src_o, "src_edges"), matrix(x_o, "input_feat"), n_dst, at::Tensor(),
                             at::Tensor(), true, at::Tensor(), at::Tensor(), at::Tensor());
    return {at::mm(tmp, w), tmp};
}

std::vector<at::Tensor> backward_gin(py::handle ptr_o, py::handle src_o, py::handle dy_o, py::handle w_o, py::handle x_o, int64_t n_src) {
    const at::Tensor &w = f32(w_o, "weight"), &x = f32(x_o, "input_feat"), &dy = f32(dy_o, "d_input");
    const at::Tensor d_tmp = at::mm(dy, w.t());
    Call c(x);
    at::Tensor d_w = weight_grad(c, x, dy);
    return {agg_bwd(FGL_AGG_SUM, i32(ptr_o, "edge_ptr"), i32(src_o, "src_edges"), d_tmp, n_src, at::Tensor(), at::Tensor(), at::Tensor(),
                    at::Tensor(), at::Tensor(), nullptr), d_w};
}

std::vector<at::Tensor> forward_gat(py::handle ptr_o, py::handle w_o, py::handle src_o, py::handle x_o, int64_t n_dst, int64_t heads) {
    const at::Tensor &edge_ptr = i32(ptr_o, "edge_ptr"), &src = i32(src_o, "src_edges"), &w = f32(w_o, "edge_data"),
                     &x = f32(x_o, "input_feat");
    TORCH_CHECK(x.dim() == 2 && w.dim() == 2 && w.size(1) == heads && x.size(1) % heads == 0 && w.size(0) >= src.numel(),
                "edge_data must be [n_edges, num_heads] and num_heads must divide the feature width");
    const int64_t dim = x.size(1);
    Call c(x);
    at::Tensor out = at::empty({n_dst, dim}, x.options());
    check(api.fgl_agg_edge_fwd(c.ws, ptr<int32_t>(edge_ptr), ptr<int32_t>(src), ptr<float>(w), (int32_t)heads, ptr<float>(x),
                               (int32_t)x.size(0), x.stride(0), (int32_t)dim, (int32_t)n_dst, FGL_AGG_ZERO_DEG_PASSTHROUGH, ptr<float>(out),
                               dim, c.st()), "forward_gat");
    return {out};
}

std::vector<at::Tensor> backward_gat(py::handle ptr_o, py::handle w_o, py::handle src_o, py::handle dy_o, int64_t n_src, int64_t heads) {
    const at::Tensor &edge_ptr = i32(ptr_o, "edge_ptr"), &src = i32(src_o, "src_edges"), &w = f32(w_o, "edge_data"), &dy = f32(dy_o, "d_input");
    TORCH_CHECK(dy.dim() == 2 && w.dim() == 2 && w.size(1) == heads && dy.size(1) % heads == 0,
                "edge_data must be [n_edges, num_heads] and num_heads must divide the feature width");
    const int64_t dim = dy.size(1);
    Call c(dy);
    at::Tensor dx = at::empty({n_src, dim}, dy.options());
    check(api.fgl_agg_edge_bwd(c.ws, ptr<int32_t>(edge_ptr), ptr<int32_t>(src), ptr<float>(w), (int32_t)heads, ptr<float>(dy), dy.stride(0),
                               (int32_t)dim, (int32_t)dy.size(0), (int32_t)n_src, ptr<float>(dx), dim, c.st()), "backward_gat");
    return {dx};
}

at::Tensor edge_weight_grad(py::handle ptr_o, py::handle src_o, py::handle x_o, py::handle dy_o, int64_t heads) {
    const at::Tensor &edge_ptr = i32(ptr_o, "edge_ptr"), &src = i32(src_o, "src_edges"), &x = matrix(x_o, "input_feat"),
                     &dy = matrix(dy_o, "d_out");
    Call c(dy);
    at::Tensor dw = at::empty({src.numel(), heads}, dy.options());
    check(api.fgl_agg_edge_wgrad(c.ws, ptr<int32_t>(edge_ptr), ptr<int32_t>(src), (int32_t)heads, ptr<float>(x), (int32_t)x.size(0),
                                 x.stride(0), ptr<float>(dy), dy.stride(0), (int32_t)dy.size(1), (int32_t)dy.size(0), src.numel(),
                                 ptr<float>(dw), c.st()), "edge_weight_grad");
    return dw;
}

// Attention of a GAT layer behind its linear map: (out, alpha, el, er).
py::tuple gat_attention(py::handle ptr_o, py::handle src_o, py::handle feat_o, py::handle l_o, py::handle r_o, int64_t n_dst, int64_t heads,
                        double slope) {
    const at::Tensor &edge_ptr = i32(ptr_o, "edge_ptr"), &src = i32(src_o, "src_edges"), &feat = rows_f32(feat_o, "feat"),
                     &l = f32(l_o, "attn_l"), &r = f32(r_o, "attn_r");
    const int64_t dim = feat.size(1);
    TORCH_CHECK(heads >= 1 && dim % heads == 0 && l.numel() == dim && r.numel() == dim && n_dst <= feat.size(0) && edge_ptr.numel() >= n_dst + 1,
                "gat_attention: the attention vectors must have the feature width, and the destinations be the first sources");
    Call c(feat);
    auto opt = feat.options();
    at::Tensor out = at::empty({n_dst, dim}, opt), alpha = at::empty({src.numel(), heads}, opt), el = at::empty({feat.size(0), heads}, opt),
               er = at::empty({n_dst, heads}, opt);
    check(api.fgl_gat_fwd(c.ws, ptr<int32_t>(edge_ptr), ptr<int32_t>(src), ptr<float>(feat), feat.stride(0), ptr<float>(l), ptr<float>(r),
                          (int32_t)heads, (int32_t)(dim / heads), (int32_t)n_dst, (int32_t)feat.size(0), (float)slope, ptr<float>(el),
                          ptr<float>(er), ptr<float>(alpha), ptr<float>(out), dim, c.st()), "gat_attention");
    return py::make_tuple(out, alpha, el, er);
}

// (d_feat, d_attn_l, d_attn_r)
py::tuple gat_attention_backward(py::handle ptr_o, py::handle src_o, py::handle feat_o, py::handle l_o, py::handle r_o, py::handle el,
                                 py::handle er, py::handle alpha, py::handle dy_o, int64_t heads, double slope) {
    const at::Tensor &edge_ptr = i32(ptr_o, "edge_ptr"), &src = i32(src_o, "src_edges"), &feat = rows_f32(feat_o, "feat"),
                     &dy = rows_f32(dy_o, "d_out"), &l = f32(l_o, "attn_l"), &r = f32(r_o, "attn_r");
    const int64_t dim = feat.size(1), n_dst = dy.size(0), E = src.numel();
    Call c(feat);
    auto opt = feat.options();
    const int rows = api.fgl_gat_bwd_partials(c.ws, (int32_t)heads, (int32_t)(dim / heads), (int32_t)n_dst);
    at::Tensor scratch = at::empty({(int64_t)rows * 2 * dim + (E + n_dst) * heads}, opt);
    at::Tensor dfeat = at::empty({feat.size(0), dim}, opt), dattn = at::empty({2, dim}, opt);
    check(api.fgl_gat_bwd(c.ws, ptr<int32_t>(edge_ptr), ptr<int32_t>(src), ptr<float>(feat), feat.stride(0), ptr<float>(l), ptr<float>(r),
                          ptr<float>(f32(el, "el")), ptr<float>(f32(er, "er")), ptr<float>(f32(alpha, "alpha")), ptr<float>(dy),
                          dy.stride(0), (int32_t)heads, (int32_t)(dim / heads), (int32_t)n_dst, (int32_t)feat.size(0), E, (float)slope,
                          ptr<float>(scratch), ptr<float>(dfeat), ptr<float>(dattn), c.st()), "gat_attention_backward");
    return py::make_tuple(dfeat, dattn.select(0, 0).view(l.sizes()), dattn.select(0, 1).view(r.sizes()));
}

// ---------------------------------------------------------------------------------------------------------------------
// loss and optimizer
// ---------------------------------------------------------------------------------------------------------------------
py::tuple softmax_xent(py::handle logits_o, py::handle labels_o, py::handle ids_o, py::handle n_valid_o, py::handle loss_o, py::handle d_o,
                       py::handle rows_o) {
    const at::Tensor &logits = rows_f32(logits_o, "logits"), &labels = input(labels_o, "labels");
    TORCH_CHECK(labels.scalar_type() == at::kLong, "labels must be int64");
    const at::Tensor ids = optional_i32(ids_o, "label_ids");
    const int64_t n = logits.size(0), classes = logits.size(1);
    Call c(logits);
    auto opt = logits.options();
    at::Tensor loss = loss_o.is_none() ? at::empty({1}, opt) : tensor(loss_o, "loss");
    at::Tensor d = d_o.is_none() ? at::empty({n, classes}, opt) : rows_f32(d_o, "dlogits");
    at::Tensor rows = rows_o.is_none() ? at::empty({std::max<int64_t>(n, 1)}, opt) : f32(rows_o, "row_loss");
    TORCH_CHECK(rows.numel() >= n, "row_loss must hold one float per row");
    const bool on_device = THPVariable_Check(n_valid_o.ptr());
    const at::Tensor n_dev = on_device ? i32(n_valid_o, "n_valid") : at::Tensor();
    const int64_t n_host = on_device || n_valid_o.is_none() ? n : n_valid_o.cast<int64_t>();
    check(api.fgl_softmax_xent(c.ws, ptr<float>(logits), logits.stride(0), ptr<int64_t>(labels), ptr<int32_t>(ids), labels.numel(), (int32_t)n,
                               (int32_t)classes, ptr<int32_t>(n_dev), (int32_t)n_host, ptr<float>(loss), ptr<float>(d), d.stride(0),
                               ptr<float>(rows), c.st()), "softmax_xent", c.ws);
    return py::make_tuple(loss, d);
}

void adam_step(py::handle p_o, py::handle g_o, py::handle m_o, py::handle v_o, py::handle step_o, double lr, double b1, double b2, double eps,
               double wd) {
    const at::Tensor &p = f32(p_o, "param"), &g = f32(g_o, "grad"), &m = f32(m_o, "exp_avg"), &v = f32(v_o, "exp_avg_sq"),
                     &step = i32(step_o, "step_dev");
    TORCH_CHECK(g.numel() == p.numel() && m.numel() == p.numel() && v.numel() == p.numel(),
                "param, grad and the two moment buffers must have the same length");
    TORCH_CHECK(step.numel() >= 2, "step_dev must hold two int32 words");
    Call c(p);
    check(api.fgl_adam_step(ptr<float>(p), ptr<float>(g), ptr<float>(m), ptr<float>(v), p.numel(), (float)lr, (float)b1, (float)b2, (float)eps,
                            (float)wd, ptr<int32_t>(step), c.st()), "adam_step_");
}

// ---------------------------------------------------------------------------------------------------------------------
// one training step of the reference's models, without autograd
// ---------------------------------------------------------------------------------------------------------------------
// Forward, loss and backward of GCN / GIN / GAT (layers.py) on one mini-batch of a window, as the launches they are.  Under
// autograd a two-layer step is some forty operators and graph nodes and 0.6 ms of host time; spelled out it is about
// twenty launches.  The arithmetic is that of the layers' autograd functions, call by call.
struct BlockRef {
    const int32_t *indptr, *src;
    int32_t n_src, n_dst;
    int64_t n_edges;
};

struct StepBatch {
    std::vector<BlockRef> blocks;  // input layer first
    const int32_t* nodes;          // global ids of the input layer's sources, seeds first
};

StepBatch step_batch(const at::Tensor& nodes, const std::vector<at::Tensor>& indptr, const std::vector<at::Tensor>& src, int64_t b,
                     const std::vector<int64_t>& counts) {
    StepBatch s;
    s.nodes = ptr<int32_t>(nodes) + b * nodes.stride(0);
    for (int h = (int)indptr.size() - 1; h >= 0; --h)
        s.blocks.push_back({ptr<int32_t>(indptr[h]) + b * indptr[h].stride(0), ptr<int32_t>(src[h]) + b * src[h].stride(0),
                            (int32_t)counts[h + 1], (int32_t)counts[h], counts[8 + h]});
    return s;
}

// out [n_dst][x's width] = aggregation of x over the block; rows of x through `map` (n_map entries) if that is given.
at::Tensor step_agg(const Call& c, int mode, const BlockRef& b, const at::Tensor& x, const int32_t* map, const int32_t* sdeg, const int32_t* ddeg) {
    at::Tensor out = at::empty({b.n_dst, x.size(1)}, x.options());
    check(api.fgl_agg_fwd(c.ws, mode, b.indptr, b.src, sdeg, ddeg, map, map ? b.n_src : 0, ptr<float>(x), x.size(0), x.stride(0),
                          (int32_t)x.size(1), b.n_dst, FGL_AGG_ZERO_DEG_PASSTHROUGH, ptr<float>(out), out.stride(0), nullptr, c.st()),
          "aggregate");
    return out;
}

at::Tensor step_agg_bwd(const Call& c, int mode, const BlockRef& b, const at::Tensor& dy, const int32_t* sdeg, const int32_t* ddeg) {
    at::Tensor dx = at::empty({b.n_src, dy.size(1)}, dy.options());
    check(api.fgl_agg_bwd(c.ws, mode, b.indptr, b.src, sdeg, ddeg, ptr<float>(dy), dy.stride(0), (int32_t)dy.size(1), b.n_dst, b.n_src,
                          ptr<float>(dx), dx.stride(0), nullptr, c.st()), "aggregate_backward");
    return dx;
}

// Inverted dropout between two layers, drawing as torch's does.
struct Drop {
    double p;
    std::vector<at::Tensor> masks;
    at::Tensor forward(const at::Tensor& h) {
        if (p == 0.0 || h.numel() == 0) {
            masks.emplace_back();
            return h;
        }
        auto [out, mask] = at::native_dropout(h, p, true);
        masks.push_back(mask);
        return out;
    }
    at::Tensor backward(const at::Tensor& d) {
        at::Tensor mask = masks.back();
        masks.pop_back();
        return mask.defined() ? at::native_dropout_backward(d, mask, 1.0 / (1.0 - p)) : d;
    }
};

std::pair<at::Tensor, at::Tensor> step_loss(const Call& c, const at::Tensor& logits, const at::Tensor& labels, const StepBatch& s) {
    const int32_t n = s.blocks.back().n_dst;
    at::Tensor loss = at::empty({1}, logits.options()), d = at::empty_like(logits), rows = at::empty({std::max(n, 1)}, logits.options());
    check(api.fgl_softmax_xent(c.ws, ptr<float>(logits), logits.stride(0), ptr<int64_t>(labels), s.nodes, labels.numel(), n,
                               (int32_t)logits.size(1), nullptr, n, ptr<float>(loss), ptr<float>(d), d.stride(0), ptr<float>(rows), c.st()),
          "softmax_xent", c.ws);
    return {loss, d};
}

// GCN with the input layer's rows read in the feature table through the mini-batch's node ids.  aggregate_first: per layer,
// whether (A x) W is evaluated instead of A (x W).
at::Tensor gcn_step(const at::Tensor& table, const at::Tensor& nodes, const std::vector<at::Tensor>& indptr, const std::vector<at::Tensor>& src,
                    int64_t batch, const std::vector<int64_t>& counts, const std::vector<at::Tensor>& weights,
                    const std::vector<at::Tensor>& grads, const std::vector<bool>& aggregate_first, double p_drop, const at::Tensor& labels) {
    at::AutoDispatchBelowADInplaceOrView no_autograd;
    Call c(table);
    const StepBatch s = step_batch(nodes, indptr, src, batch, counts);
    const int L = (int)s.blocks.size();
    const auto words = nodes.options();
    Drop drop{p_drop, {}};
    std::vector<at::Tensor> kept(L), deg(L);  // per layer: the left operand of the weight gradient; both sides' degrees
    std::vector<const int32_t*> sdeg(L), ddeg(L);
    at::Tensor h = table;
    for (int i = 0; i < L; ++i) {
        const BlockRef& b = s.blocks[i];
        if (i > 0) h = drop.forward(h);
        const int64_t pad = (b.n_dst + 31) / 32 * 32;
        deg[i] = at::empty({pad + b.n_src}, words);
        int32_t* d = ptr<int32_t>(deg[i]);
        ddeg[i] = d;
        sdeg[i] = d + pad;
        check(api.fgl_block_degrees(b.indptr, b.src, b.n_dst, b.n_src, b.n_edges, d, d + pad, c.st()), "block_degrees");
        if (i == 0 || aggregate_first[i]) {
            kept[i] = step_agg(c, FGL_AGG_SYMNORM, b, h, i == 0 ? s.nodes : nullptr, sdeg[i], ddeg[i]);
            h = at::mm(kept[i], weights[i]);
        } else {
            kept[i] = h;
            h = step_agg(c, FGL_AGG_SYMNORM, b, at::mm(h, weights[i]), nullptr, sdeg[i], ddeg[i]);
        }
    }
    auto [loss, d] = step_loss(c, h, labels, s);
    for (int i = L - 1; i >= 0; --i) {
        const BlockRef& b = s.blocks[i];
        at::Tensor g = grads[i];
        if (i == 0 || aggregate_first[i]) {
            at::Tensor masked = at::empty_like(d);
            check(api.fgl_mask_rows(b.indptr, b.n_dst, (int32_t)d.size(1), ptr<float>(d), d.stride(0), ptr<float>(masked), masked.stride(0),
                                    c.st()), "mask_rows");
            weight_grad(c, kept[i], masked, g);
            if (i > 0) d = step_agg_bwd(c, FGL_AGG_SYMNORM, b, at::mm(masked, weights[i].t()), sdeg[i], ddeg[i]);
        } else {
            const at::Tensor dx = step_agg_bwd(c, FGL_AGG_SYMNORM, b, d, sdeg[i], ddeg[i]);
            weight_grad(c, kept[i], dx, g);
            d = at::mm(dx, weights[i].t());
        }
        if (i > 0) d = drop.backward(d);
    }
    return loss;
}

// GIN; the input layer sums the rows of the feature table in place, and its input takes no gradient.
at::Tensor gin_step(const at::Tensor& table, const at::Tensor& nodes, const std::vector<at::Tensor>& indptr, const std::vector<at::Tensor>& src,
                    int64_t batch, const std::vector<int64_t>& counts, const std::vector<at::Tensor>& weights,
                    const std::vector<at::Tensor>& grads, double p_drop, const at::Tensor& labels) {
    at::AutoDispatchBelowADInplaceOrView no_autograd;
    Call c(table);
    const StepBatch s = step_batch(nodes, indptr, src, batch, counts);
    const int L = (int)s.blocks.size();
    Drop drop{p_drop, {}};
    std::vector<at::Tensor> kept(L);
    at::Tensor h = table;
    for (int i = 0; i < L; ++i) {
        if (i > 0) h = drop.forward(h);
        kept[i] = step_agg(c, FGL_AGG_SUM, s.blocks[i], h, i == 0 ? s.nodes : nullptr, nullptr, nullptr);
        h = at::mm(kept[i], weights[i]);
    }
    auto [loss, d] = step_loss(c, h, labels, s);
    for (int i = L - 1; i >= 0; --i) {
        at::Tensor g = grads[i];
        weight_grad(c, kept[i], d, g);
        if (i > 0) d = drop.backward(step_agg_bwd(c, FGL_AGG_SUM, s.blocks[i], at::mm(d, weights[i].t()), nullptr, nullptr));
    }
    return loss;
}

// GAT.  params / grads: per layer the linear map's weight [heads * width][in] and the two attention vectors; without
// attention_grad the latter take no gradient (theirs stays zero).
at::Tensor gat_step(const at::Tensor& table, const at::Tensor& nodes, const std::vector<at::Tensor>& indptr, const std::vector<at::Tensor>& src,
                    int64_t batch, const std::vector<int64_t>& counts, const std::vector<at::Tensor>& params,
                    const std::vector<at::Tensor>& grads, const std::vector<int64_t>& heads, const std::vector<double>& slope,
                    const std::vector<bool>& attention_grad, const at::Tensor& labels) {
    at::AutoDispatchBelowADInplaceOrView no_autograd;
    Call c(table);
    const StepBatch s = step_batch(nodes, indptr, src, batch, counts);
    const int L = (int)s.blocks.size();
    const auto opt = table.options();
    std::vector<at::Tensor> x(L), feat(L), scores(L);   // scores: alpha [edges][heads], el [n_src][heads], er [n_dst][heads]
    at::Tensor h = at::empty({s.blocks[0].n_src, table.size(1)}, opt);
    check(api.fgl_gather_rows(c.ws, ptr<float>(table), nullptr, 0, table.size(0), table.stride(0), (int32_t)table.size(1), s.nodes,
                              s.blocks[0].n_src, ptr<float>(h), h.stride(0), c.st()), "gather_rows");
    for (int i = 0; i < L; ++i) {
        const BlockRef& b = s.blocks[i];
        const at::Tensor &w = params[3 * i], &l = params[3 * i + 1], &r = params[3 * i + 2];
        const int64_t dim = w.size(0);
        x[i] = h;
        feat[i] = at::mm(h, w.t());
        h = at::empty({b.n_dst, dim}, opt);
        scores[i] = at::empty({(b.n_edges + b.n_src + b.n_dst) * heads[i]}, opt);
        float* alpha = ptr<float>(scores[i]);
        check(api.fgl_gat_fwd(c.ws, b.indptr, b.src, ptr<float>(feat[i]), dim, ptr<float>(l), ptr<float>(r), (int32_t)heads[i],
                              (int32_t)(dim / heads[i]), b.n_dst, b.n_src, (float)slope[i], alpha + b.n_edges * heads[i],
                              alpha + (b.n_edges + b.n_src) * heads[i], alpha, ptr<float>(h), dim, c.st()), "gat_attention");
    }
    auto [loss, d] = step_loss(c, h, labels, s);
    for (int i = L - 1; i >= 0; --i) {
        const BlockRef& b = s.blocks[i];
        const at::Tensor &w = params[3 * i], &l = params[3 * i + 1], &r = params[3 * i + 2];
        const int64_t dim = w.size(0);
        at::Tensor dfeat = at::empty({b.n_src, dim}, opt);
        float* alpha = ptr<float>(scores[i]);
        if (attention_grad[i]) {
            const int rows = api.fgl_gat_bwd_partials(c.ws, (int32_t)heads[i], (int32_t)(dim / heads[i]), b.n_dst);
            at::Tensor scratch = at::empty({(int64_t)rows * 2 * dim + (b.n_edges + b.n_dst) * heads[i]}, opt);
            // both vectors' gradients in one piece, if the flat gradient holds them so
            const bool in_place = ptr<float>(grads[3 * i + 2]) == ptr<float>(grads[3 * i + 1]) + dim;
            at::Tensor dattn = in_place ? grads[3 * i + 1] : at::empty({2, dim}, opt);
            check(api.fgl_gat_bwd(c.ws, b.indptr, b.src, ptr<float>(feat[i]), dim, ptr<float>(l), ptr<float>(r),
                                  alpha + b.n_edges * heads[i], alpha + (b.n_edges + b.n_src) * heads[i], alpha, ptr<float>(d),
                                  d.stride(0), (int32_t)heads[i],
                                  (int32_t)(dim / heads[i]), b.n_dst, b.n_src, b.n_edges, (float)slope[i], ptr<float>(scratch),
                                  ptr<float>(dfeat), ptr<float>(dattn), c.st()), "gat_attention_backward");
            if (!in_place) {
                fgl_segment seg[2] = {{ptr<float>(grads[3 * i + 1]), ptr<float>(dattn), dim * 4},
                                      {ptr<float>(grads[3 * i + 2]), ptr<float>(dattn) + dim, dim * 4}};
                check(api.fgl_stage_segments(seg, 2, nullptr, nullptr, 0, c.st()), "gat_attention_backward");
            }
        } else {
            check(api.fgl_agg_edge_bwd(c.ws, b.indptr, b.src, alpha, (int32_t)heads[i], ptr<float>(d), d.stride(0),
                                       (int32_t)dim, b.n_dst, b.n_src, ptr<float>(dfeat), dim, c.st()), "backward_gat");
        }
        at::Tensor g = grads[3 * i];
        weight_grad(c, dfeat, x[i], g);
        if (i > 0) d = at::mm(dfeat, w);
    }
    return loss;
}

}  // namespace

PYBIND11_MODULE(_ops, m) {
    m.def("init", &init);
    m.def("workspace", [](int device) { return (uintptr_t)workspace(device); });
    m.def("sample_node_csr", &sample_node_csr);
    m.def("transfer_edge_id", &transfer_edge_id);
    m.def("sample_map_fused", &sample_map_fused);
    m.def("wait_counts", &wait_counts);
    m.def("sample_blocks", &sample_blocks);
    m.def("cal_deg", &cal_deg);
    m.def("exclusive_sum", &exclusive_sum);
    m.def("stage_segments", &stage_segments);
    m.def("aggregate", &aggregate);
    m.def("aggregate_backward", &aggregate_backward);
    m.def("transpose_block", &transpose_block);
    m.def("aggregate_window", &aggregate_window);
    m.def("gather_rows", &gather_rows);
    m.def("forward_gcn", &forward_gcn);
    m.def("backward_gcn", &backward_gcn);
    m.def("forward_gin", &forward_gin);
    m.def("backward_gin", &backward_gin);
    m.def("forward_gat", &forward_gat);
    m.def("backward_gat", &backward_gat);
    m.def("edge_weight_grad", &edge_weight_grad);
    m.def("softmax_xent", &softmax_xent);
    m.def("weight_grad", &weight_grad_op);
    m.def("weight_grad_scratch", &weight_grad_scratch);
    m.def("gcn_step", &gcn_step);
    m.def("gin_step", &gin_step);
    m.def("gat_step", &gat_step);
    m.def("adam_step", &adam_step);
    m.def("gat_attention", &gat_attention);
    m.def("gat_attention_backward", &gat_attention_backward);
}
