// Host path of the differentiable operators: checks, allocations, launches and autograd nodes in C++.
//
// The Python operators of this package cost about 0.8 ms of interpreter time per camera and training step (ctypes calls,
// torch.autograd.Function, tensor views of scratch buffers), several times what the kernels of a small step take on the
// device.  These nodes call the same C ABI (include/cgx_raster.h) through the addresses that Python resolved, so one
// library serves both; the raw entry points of diff_gaussian_rasterization._C and its per-stage profiling stay in Python.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <array>
#include <atomic>
#include <chrono>
#include <map>
#include <mutex>

#include "../../include/cgx_raster.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

// ---------------------------------------------------------------------------------------------- the library
#define CGX_FUNCTIONS(X)                                                                                             \
    X(cgx_anchor_stats) X(cgx_anchor_stats_workspace_bytes) X(cgx_filter_preprocess) X(cgx_preprocess_fwd) X(cgx_preprocess_bwd) X(cgx_preprocess_fwd_batched_planes) X(cgx_preprocess_bwd_batched_planes) \
    X(cgx_all_map_fwd) X(cgx_all_map_bwd) X(cgx_strip_loss_fwd) X(cgx_strip_loss_bwd) X(cgx_depth_normal_fwd)        \
    X(cgx_depth_normal_bwd) X(cgx_bin_workspace_bytes) X(cgx_bin_count_scan) X(cgx_emit_keys)                        \
    X(cgx_tile_bins_workspace_bytes) X(cgx_tile_bins_longest) X(cgx_tile_bins_count) X(cgx_tile_bins_sort)          \
    X(cgx_sort_workspace_bytes) X(cgx_sort_passes) X(cgx_sort_pairs_pingpong) X(cgx_tile_ranges) X(cgx_higher_msb)   \
    X(cgx_render_records_bytes) X(cgx_render_pack) X(cgx_render_fwd_packed) X(cgx_render_bwd_workspace_bytes) X(cgx_render_bwd_table)
struct Library {
#define X(f) decltype(&::f) f = nullptr;
    CGX_FUNCTIONS(X)
#undef X
} L;
PyObject* error_class = nullptr;      // _lib.CgxError

void bind(const py::dict& addresses, py::object error)
{
#define X(f) L.f = reinterpret_cast<decltype(L.f)>(addresses[#f].cast<uintptr_t>());
    CGX_FUNCTIONS(X)
#undef X
    error_class = error.release().ptr();
}

void check(int status, const char* where)
{
    if (status == CGX_OK) return;
    py::gil_scoped_acquire gil;
    py::object e = py::reinterpret_borrow<py::object>(error_class)(status, where);
    PyErr_SetObject(error_class, e.ptr());
    throw py::error_already_set();
}

// ---------------------------------------------------------------------------------------------- small helpers
Tensor cuda_f32(const Tensor& t, const char* name)
{
    if (!t.is_cuda()) throw std::runtime_error(std::string(name) + " must be a CUDA tensor (this rasterizer has no CPU path)");
    if (t.scalar_type() != at::kFloat) throw std::runtime_error(std::string(name) + " must be float32");
    return t.contiguous();
}
Tensor cuda_any(const Tensor& t, const char* name)
{
    if (!t.defined() || !t.is_cuda())
        throw std::runtime_error(std::string(name) + " must be a CUDA tensor (this rasterizer has no CPU path)");
    return t.contiguous();
}
float* f32(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }
int32_t* i32(const Tensor& t) { return static_cast<int32_t*>(t.data_ptr()); }
void* stream() { return at::cuda::getCurrentCUDAStream().stream(); }

Tensor empty_f32(at::IntArrayRef shape, const Tensor& like) { return at::empty(shape, like.options().dtype(at::kFloat).requires_grad(false)); }
Tensor empty_i32(at::IntArrayRef shape, const Tensor& like) { return at::empty(shape, like.options().dtype(at::kInt).requires_grad(false)); }

// The fields of GaussianRasterizationSettings, by position.
struct Settings {
    int H, W;
    float tanfovx, tanfovy, scale_modifier;
    Tensor bg, view, proj, campos;
    bool geo;
};
Tensor tensor_item(PyObject* tuple, int i) { return py::handle(PyTuple_GET_ITEM(tuple, i)).cast<Tensor>(); }
Settings read_settings(const py::handle& h, bool projection_only = false)
{
    PyObject* t = h.ptr();
    if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != 13) throw std::runtime_error("raster_settings must be a GaussianRasterizationSettings");
    auto item = [&](int i) { return py::reinterpret_borrow<py::object>(PyTuple_GET_ITEM(t, i)); };
    auto whole = [&](int i) { return (int)py::int_(item(i)); };              // whatever int() and float() take
    auto real = [&](int i) { return (float)(double)py::float_(item(i)); };
    Settings s;
    s.H = whole(0);
    s.W = whole(1);
    s.tanfovx = real(2);
    s.tanfovy = real(3);
    s.scale_modifier = real(5);
    s.view = tensor_item(t, 6);
    s.proj = tensor_item(t, 7);
    if (projection_only) return s;
    s.bg = tensor_item(t, 4);
    s.campos = tensor_item(t, 9);
    s.geo = PyObject_IsTrue(PyTuple_GET_ITEM(t, 11));
    return s;
}

// What a node keeps that is no tensor of the graph.
template <class T>
struct Holder : torch::CustomClassHolder {
    T v;
    explicit Holder(T x) : v(std::move(x)) {}
};
template <class T>
void keep(AutogradContext* ctx, T v)
{
    ctx->saved_data["s"] = c10::IValue::make_capsule(c10::make_intrusive<Holder<T>>(std::move(v)));
}
template <class T>
T& kept(AutogradContext* ctx)
{
    return static_cast<Holder<T>*>(ctx->saved_data["s"].toCapsule().get())->v;
}

// Sub-arrays of one buffer on 128-byte boundaries, in the order in which they are asked for.
struct Carver {
    size_t size = 0;
    size_t add(size_t bytes)
    {
        const size_t at = (size + 127) / 128 * 128;
        size = at + bytes;
        return at;
    }
};
struct GeometryLayout {
    size_t tiles_touched, bins, bins_bytes, records, total;
    GeometryLayout(int64_t P, int W, int H)
    {
        Carver c;
        tiles_touched = c.add(4 * P);
        bins_bytes = L.cgx_tile_bins_workspace_bytes(W, H);      // its first words are the tile ranges
        bins = c.add(bins_bytes);
        records = c.add(L.cgx_render_records_bytes((int)P));
        total = c.size + 128;
    }
};
struct ImageLayout {
    size_t accum_alpha, n_contrib, n_contrib2loss, total;
    explicit ImageLayout(int64_t N)
    {
        Carver c;
        accum_alpha = c.add(4 * N);
        n_contrib = c.add(4 * N);
        n_contrib2loss = c.add(4 * N);
        total = c.size + 128;
    }
};
Tensor bytes_like(size_t n, const Tensor& like) { return at::empty({(int64_t)n}, like.options().dtype(at::kByte).requires_grad(false)); }
template <class T>
T* at_offset(const Tensor& buf, size_t off)
{
    return reinterpret_cast<T*>(static_cast<char*>(buf.data_ptr()) + off);
}

// ---------------------------------------------------------------------------------------------- elapsed milliseconds
// Resolved on first numeric use, so that the operators never block the host.
constexpr int MOST_DEVICES = 64;
struct EventMs {
    cudaEvent_t a = nullptr, b = nullptr;
    double ms = 0;
    bool have = false;
    int device = 0;
    // Pairs that a collector dropped are taken up again, as many as EVENTS_KEPT: creating and destroying one took 4 us.
    struct Pool {
        std::mutex lock;
        std::vector<std::array<cudaEvent_t, 2>> pairs[MOST_DEVICES];
    };
    static constexpr size_t EVENTS_KEPT = 64;
    static Pool& pool()
    {
        static Pool* p = new Pool;      // outlives every collector
        return *p;
    }
    EventMs()
    {
        cudaGetDevice(&device);
        if (device < MOST_DEVICES) {
            Pool& p = pool();
            std::lock_guard<std::mutex> g(p.lock);
            if (!p.pairs[device].empty()) {
                a = p.pairs[device].back()[0], b = p.pairs[device].back()[1];
                p.pairs[device].pop_back();
                return;
            }
        }
        cudaEventCreate(&a);
        cudaEventCreate(&b);
    }
    EventMs(const EventMs&) = delete;
    ~EventMs()
    {
        if (device < MOST_DEVICES && a && b) {
            Pool& p = pool();
            std::lock_guard<std::mutex> g(p.lock);
            if (p.pairs[device].size() < EVENTS_KEPT) {
                p.pairs[device].push_back({a, b});
                return;
            }
        }
        if (a) cudaEventDestroy(a);
        if (b) cudaEventDestroy(b);
    }
    double get()
    {
        if (!have) {
            float f = 0.f;
            cudaEventSynchronize(b);
            cudaEventElapsedTime(&f, a, b);
            ms = f;
            have = true;
        }
        return ms;
    }
};

// The caller's stats_collector dict (or nothing), usable without the interpreter lock.
using Stats = std::shared_ptr<PyObject>;
Stats hold(const py::object& o)
{
    if (o.is_none()) return nullptr;
    return Stats(o.inc_ref().ptr(), [](PyObject* p) {
        if (!Py_IsInitialized()) return;
        py::gil_scoped_acquire gil;
        Py_DECREF(p);
    });
}
void report(const Stats& stats, const char* key, std::shared_ptr<EventMs> ms)
{
    py::gil_scoped_acquire gil;
    py::object v = py::cast(std::move(ms));
    if (PyObject_SetItem(stats.get(), py::str(key).ptr(), v.ptr()) != 0) throw py::error_already_set();
}

// ---------------------------------------------------------------------------------------------- pair counts
// The counting stage leaves the number of pairs and what the tiles' lists look like in page-locked memory, each with a
// flag that the host watches: neither a copy nor an event stands between the kernel and the launches that need them.
constexpr int SLOTS = 256;
struct Slot {
    volatile uint64_t word[6];          // see cgx_tile_bins_count
    uint64_t pad[2];
    bool arrived() const
    {
        uint64_t all = ~0ull;
        for (int k = 0; k < 6; k++) all &= word[k];
        return all >> 32;
    }
};
Slot* slots()
{
    static Slot* mem = [] {
        void* p = nullptr;
        if (cudaHostAlloc(&p, SLOTS * sizeof(Slot), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess)
            throw std::runtime_error("no page-locked memory for the pair counts");
        return static_cast<Slot*>(p);
    }();
    return mem;
}
struct Count {
    Tensor geom;
    int slot = -1;
    cudaStream_t stream = nullptr;
    uint32_t word[6];
    Tensor keep[3];            // a prefetched count's inputs: their addresses stay taken
};
std::mutex slot_lock;
std::vector<int> free_slots = [] {
    std::vector<int> v;
    for (int i = SLOTS - 1; i >= 0; i--) v.push_back(i);
    return v;
}();
int take_slot()
{
    std::lock_guard<std::mutex> g(slot_lock);
    if (free_slots.empty()) throw std::runtime_error("too many pair counts in flight");
    const int s = free_slots.back();
    free_slots.pop_back();
    return s;
}
void give_slot(int s)
{
    std::lock_guard<std::mutex> g(slot_lock);
    free_slots.push_back(s);
}

Count start_count(int64_t P, int W, int H, const Tensor& means2D, const Tensor& radii, const Tensor& local)
{
    const GeometryLayout gl(P, W, H);
    Count c;
    c.geom = bytes_like(gl.total, means2D);
    c.slot = take_slot();
    c.stream = at::cuda::getCurrentCUDAStream().stream();
    Slot& s = slots()[c.slot];
    for (int k = 0; k < 6; k++) s.word[k] = 0;
    check(L.cgx_tile_bins_count((int)P, W, H, i32(radii), f32(means2D), static_cast<uint8_t*>(local.data_ptr()),
                                at_offset<uint32_t>(c.geom, gl.tiles_touched), at_offset<void>(c.geom, gl.bins),
                                gl.bins_bytes, const_cast<uint64_t*>(s.word), c.stream), "cgx_tile_bins_count");
    return c;
}
// Waits for the count; gives the slot back.
void finish_count(Count& c)
{
    Slot& s = slots()[c.slot];
    const auto t0 = std::chrono::steady_clock::now();
    int spins = 0;
    while (!s.arrived()) {
        if (++spins % 1024 == 0 && std::chrono::steady_clock::now() - t0 > std::chrono::milliseconds(2)) {
            // a long queue in front of it, or an error: let the driver wait, and say so if there was one
            const cudaError_t e = cudaStreamSynchronize(c.stream);
            if (e != cudaSuccess) throw std::runtime_error(std::string("cgx_tile_bins_count: ") + cudaGetErrorString(e));
            if (!s.arrived()) throw std::runtime_error("cgx_tile_bins_count: the pair count did not arrive");
        }
    }
    for (int k = 0; k < 6; k++) c.word[k] = (uint32_t)s.word[k];
    give_slot(c.slot);
    c.slot = -1;
}

// Counts started ahead of their render call, found by the identity (and version) of its inputs.
using PrefetchKey = std::array<int64_t, 10>;
PrefetchKey prefetch_key(const Tensor& m, const Tensor& r, const Tensor& l, int H, int W)
{
    return {(int64_t)m.data_ptr(), (int64_t)r.data_ptr(), (int64_t)l.data_ptr(), m.size(0), H, W, m.device().index(),
            (int64_t)m._version(), (int64_t)r._version(), (int64_t)l._version()};
}
std::mutex prefetch_lock;
std::map<PrefetchKey, Count> prefetched;
constexpr size_t PREFETCH_MOST = SLOTS / 2;

bool find_prefetched(Count& c, const Tensor& means2D, const Tensor& radii, const Tensor& local, int H, int W)
{
    std::lock_guard<std::mutex> g(prefetch_lock);
    if (prefetched.empty()) return false;
    const auto it = prefetched.find(prefetch_key(means2D, radii, local, H, W));
    if (it == prefetched.end()) return false;
    c = std::move(it->second);
    prefetched.erase(it);
    return true;
}

void prefetch(int H, int W, const Tensor& means2D_, const Tensor& radii_, const Tensor& local_)
{
    const Tensor means2D = cuda_f32(means2D_, "means2D"), radii = cuda_any(radii_, "radii"),
                 local = cuda_any(local_, "compute_locally");
    const int64_t P = means2D.size(0);
    if (P == 0 || radii.scalar_type() != at::kInt) return;
    const c10::cuda::CUDAGuard guard(means2D.device());
    std::lock_guard<std::mutex> g(prefetch_lock);
    if (prefetched.size() >= PREFETCH_MOST) {              // counts nobody picked up
        for (auto& e : prefetched) finish_count(e.second);
        prefetched.clear();
    }
    const PrefetchKey key = prefetch_key(means2D, radii, local, H, W);
    const auto old = prefetched.find(key);
    if (old != prefetched.end()) {
        finish_count(old->second);
        prefetched.erase(old);
    }
    Count c = start_count(P, W, H, means2D, radii, local);
    c.keep[0] = means2D;
    c.keep[1] = radii;
    c.keep[2] = local;
    prefetched.emplace(key, std::move(c));
}

// The pairs of a count started ahead, or None.
py::object take_prefetched(int H, int W, const Tensor& means2D, const Tensor& radii, const Tensor& local)
{
    Count c;
    {
        py::gil_scoped_release nogil;
        if (find_prefetched(c, means2D, radii, local, H, W)) finish_count(c);
    }
    if (!c.geom.defined()) return py::none();
    return py::int_(c.word[0]);
}
size_t prefetched_counts()
{
    std::lock_guard<std::mutex> g(prefetch_lock);
    return prefetched.size();
}

// ---------------------------------------------------------------------------------------------- render
struct RenderState {
    int64_t P;
    int H, W;
    float tanfovx, tanfovy;
    bool geo;
    Stats stats;
};

// Lists with a tile longer than the per-tile sort takes: emission, global sort, ranges.
void sort_globally(int64_t P, int64_t R, int W, int H, int64_t T, const Tensor& radii, const Tensor& means2D,
                   const Tensor& depths, uint8_t* local, uint32_t* tiles, uint32_t* list, uint32_t* ranges, cudaStream_t st)
{
    Carver c;
    const size_t scan_bytes = L.cgx_bin_workspace_bytes((int)P), sort_bytes = L.cgx_sort_workspace_bytes(R);
    const size_t scan = c.add(scan_bytes), words = c.add(128), offsets = c.add(4 * P), list_b = c.add(4 * R),
                 keys_a = c.add(8 * R), keys_b = c.add(8 * R), sort = c.add(sort_bytes);
    const Tensor buf = bytes_like(c.size + 128, means2D);
    const int bit = (int)L.cgx_higher_msb((uint32_t)T);
    // the sort ping-pongs: the pairs are emitted where the last pass lands in `list`
    const bool even = L.cgx_sort_passes(32 + bit) % 2 == 0;
    uint32_t* v[2] = {list, at_offset<uint32_t>(buf, list_b)};
    uint64_t* k[2] = {at_offset<uint64_t>(buf, keys_a), at_offset<uint64_t>(buf, keys_b)};
    const int first = even ? 0 : 1;
    check(L.cgx_bin_count_scan((int)P, W, H, i32(radii), f32(means2D), local, tiles, at_offset<uint32_t>(buf, words),
                               at_offset<void>(buf, scan), scan_bytes, st), "cgx_bin_count_scan");
    check(L.cgx_emit_keys((int)P, W, H, i32(radii), f32(means2D), f32(depths), tiles, local,
                          at_offset<uint32_t>(buf, offsets), k[first], v[first], R, at_offset<void>(buf, scan), st),
          "cgx_emit_keys");
    check(L.cgx_sort_pairs_pingpong(R, 32 + bit, 32, k[first], v[first], k[1 - first], v[1 - first],
                                    at_offset<void>(buf, sort), sort_bytes, 0, st), "cgx_sort_pairs");
    check(L.cgx_tile_ranges(R, (int)T, k[0], ranges, st), "cgx_tile_ranges");
}

struct Render : torch::autograd::Function<Render> {
    static variable_list forward(AutogradContext* ctx, const Tensor& means2D_, const c10::optional<Tensor>& means2D_abs,
                                 const Tensor& conic_, const Tensor& rgb_, const Tensor& all_map_, const Tensor& depths_,
                                 const Tensor& radii_, const Tensor& local_, const Tensor& local_bwd, const Settings& s,
                                 const Stats& stats)
    {
        const Tensor means2D = cuda_f32(means2D_, "means2D");
        const int64_t P = means2D.size(0);
        const int H = s.H, W = s.W;
        const int64_t T = (int64_t)((W + 15) / 16) * ((H + 15) / 16), HW = (int64_t)H * W;
        const Tensor depths = cuda_f32(depths_, "depths"), conic = cuda_f32(conic_, "conic_opacity"),
                     rgb = cuda_f32(rgb_, "rgb"), all_map = cuda_f32(all_map_, "all_map"),
                     radii = cuda_any(radii_, "radii").to(at::kInt), local = cuda_any(local_, "compute_locally"),
                     bg = cuda_f32(s.bg, "background");
        if (local.scalar_type() != at::kBool || local.numel() != T)
            throw std::runtime_error("compute_locally must be a bool tensor with one entry per tile");
        if (means2D.size(1) != 2 || conic.numel() != 4 * P || rgb.numel() != 3 * P || all_map.numel() != 5 * P ||
            conic.size(0) != P || rgb.size(0) != P || all_map.size(0) != P || depths.numel() != P || radii.numel() != P)
            throw std::runtime_error("render_gaussians: per-Gaussian tensors must be (P,2) (P,4) (P,3) (P,5) (P) (P)");
        const c10::cuda::CUDAGuard guard(means2D.device());
        const cudaStream_t st = at::cuda::getCurrentCUDAStream().stream();

        Count count;
        if (!find_prefetched(count, means2D, radii, local, H, W))
            count = start_count(P, W, H, means2D, radii, local);
        // allocated, and the records packed, while the count is on its way: it reaches the host about 8 us after the
        // device has it, and the device would wait as long for the launches that need it
        const GeometryLayout gl(P, W, H);
        const ImageLayout il(HW);
        const Tensor n_render = empty_i32({T}, means2D), n_consider = empty_i32({T}, means2D),
                     n_contrib = empty_i32({T}, means2D), observe = empty_i32({P}, means2D),
                     color = empty_f32({3, H, W}, means2D), out_map = empty_f32({5, H, W}, means2D),
                     depth = empty_f32({1, H, W}, means2D), img = bytes_like(il.total, means2D);
        std::shared_ptr<EventMs> ms = stats ? std::make_shared<EventMs>() : nullptr;
        if (ms) cudaEventRecord(ms->a, st);
        check(L.cgx_render_pack((int)P, i32(radii), f32(means2D), f32(rgb), f32(all_map), f32(conic), s.geo,
                                at_offset<void>(count.geom, gl.records), i32(observe), st), "cgx_render_pack");
        finish_count(count);

        const int64_t R = count.word[0];
        const Tensor list = at::empty({R}, means2D.options().dtype(at::kInt).requires_grad(false));
        uint32_t* tiles = at_offset<uint32_t>(count.geom, gl.tiles_touched);
        uint32_t* ranges = at_offset<uint32_t>(count.geom, gl.bins);
        uint8_t* loc = static_cast<uint8_t*>(local.data_ptr());
        uint32_t* ids = static_cast<uint32_t*>(list.data_ptr());
        if (count.word[1] <= (uint32_t)L.cgx_tile_bins_longest()) {
            const Tensor pairs = bytes_like(8 * R, means2D);
            check(L.cgx_tile_bins_sort((int)P, W, H, i32(radii), f32(means2D), f32(depths), loc, count.word,
                                       at_offset<void>(count.geom, gl.bins), gl.bins_bytes,
                                       static_cast<uint64_t*>(pairs.data_ptr()), ids, st), "cgx_tile_bins_sort");
        } else {
            sort_globally(P, R, W, H, T, radii, means2D, depths, loc, tiles, ids, ranges, st);
        }
        check(L.cgx_render_fwd_packed((int)P, W, H, s.tanfovx, s.tanfovy, ranges, ids, i32(radii), f32(means2D), f32(rgb),
                               f32(all_map), f32(conic), loc, f32(bg), s.geo, at_offset<void>(count.geom, gl.records),
                               at_offset<float>(img, il.accum_alpha), at_offset<uint32_t>(img, il.n_contrib),
                               at_offset<uint32_t>(img, il.n_contrib2loss), f32(color), i32(observe), f32(out_map),
                               f32(depth), i32(n_render), i32(n_consider), i32(n_contrib), st), "cgx_render_fwd");
        if (ms) {
            cudaEventRecord(ms->b, st);
            report(stats, "forward_render_time", std::move(ms));
        }
        ctx->set_materialize_grads(false);
        ctx->mark_non_differentiable({n_render, n_consider, n_contrib, observe});
        ctx->save_for_backward({out_map, count.geom, list, img, cuda_any(local_bwd, "compute_locally"), bg});
        keep(ctx, RenderState{P, H, W, s.tanfovx, s.tanfovy, s.geo, stats});
        return {color, n_render, n_consider, n_contrib, observe, out_map, depth};
    }

    static variable_list backward(AutogradContext* ctx, variable_list g)
    {
        const RenderState& s = kept<RenderState>(ctx);
        const variable_list saved = ctx->get_saved_variables();
        const Tensor &out_map = saved[0], &geom = saved[1], &list = saved[2], &img = saved[3], &local = saved[4], &bg = saved[5];
        const c10::cuda::CUDAGuard guard(out_map.device());
        const cudaStream_t st = at::cuda::getCurrentCUDAStream().stream();
        auto cotangent = [&](const Tensor& t, int n, const char* name, bool needed) {
            if (t.defined()) return cuda_f32(t, name);
            return needed ? at::zeros({n, s.H, s.W}, out_map.options()) : Tensor();
        };
        const Tensor d_color = cotangent(g[0], 3, "dL_dout_color", true), d_map = cotangent(g[5], 5, "dL_dout_all_map", s.geo),
                     d_depth = cotangent(g[6], 1, "dL_dout_plane_depth", s.geo);
        const int64_t P = s.P, HW = (int64_t)s.H * s.W;
        const GeometryLayout gl(P, s.W, s.H);
        const ImageLayout il(HW);
        const Tensor m2 = empty_f32({P, 2}, out_map), abs2 = empty_f32({P, 3}, out_map), co = empty_f32({P, 4}, out_map),
                     rgb = empty_f32({P, 3}, out_map), am = empty_f32({P, 5}, out_map);
        const size_t ws_bytes = L.cgx_render_bwd_workspace_bytes((int)P);
        const Tensor ws = bytes_like(ws_bytes, out_map);
        std::shared_ptr<EventMs> ms = s.stats ? std::make_shared<EventMs>() : nullptr;
        if (ms) cudaEventRecord(ms->a, st);
        check(L.cgx_render_bwd_table((int)P, s.W, s.H, s.tanfovx, s.tanfovy, at_offset<uint32_t>(geom, gl.bins),
                                     static_cast<uint32_t*>(list.data_ptr()), f32(bg), at_offset<void>(geom, gl.records),
                                     f32(out_map), at_offset<float>(img, il.accum_alpha),
                                     at_offset<uint32_t>(img, il.n_contrib), static_cast<uint8_t*>(local.data_ptr()),
                                     f32(d_color), f32(d_map), f32(d_depth), s.geo, f32(m2), f32(abs2), f32(co), f32(rgb),
                                     f32(am), 0, at_offset<uint32_t>(geom, gl.tiles_touched), ws.data_ptr(), ws_bytes, st),
              "cgx_render_bwd");
        if (ms) {
            cudaEventRecord(ms->b, st);
            report(s.stats, "backward_render_time", std::move(ms));
        }
        return {m2, abs2, co, rgb, am, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

std::vector<Tensor> render(const Tensor& means2D, const c10::optional<Tensor>& means2D_abs, const Tensor& conic,
                           const Tensor& rgb, const Tensor& all_map, const Tensor& depths, const Tensor& radii,
                           const Tensor& local, const Tensor& local_bwd, const py::object& settings, const py::object& stats)
{
    const Settings s = read_settings(settings);
    const Stats held = hold(stats);
    py::gil_scoped_release nogil;
    return Render::apply(means2D, means2D_abs, conic, rgb, all_map, depths, radii, local, local_bwd, s, held);
}

// ---------------------------------------------------------------------------------------------- preprocess
struct Preprocess : torch::autograd::Function<Preprocess> {
    static variable_list forward(AutogradContext* ctx, const Tensor& means3D_, const Tensor& scales_,
                                 const Tensor& rotations_, const Tensor& sh, const Tensor& opacities_, const Settings& s)
    {
        if (means3D_.dim() != 2 || means3D_.size(1) != 3)
            throw std::runtime_error("means3D must have dimensions (num_points, 3)");
        const Tensor means3D = cuda_f32(means3D_, "means3D");
        const int64_t P = means3D.size(0);
        const c10::cuda::CUDAGuard guard(means3D.device());
        const Tensor m2 = empty_f32({P, 2}, means3D), depths = empty_f32({P}, means3D), radii = empty_i32({P}, means3D),
                     co = empty_f32({P, 4}, means3D);
        // SH evaluation is compiled out upstream: rgb stays zero
        const Tensor rgb = at::zeros({P, 3}, means3D.options().requires_grad(false));
        const Tensor scales = cuda_f32(scales_, "scales"), rotations = cuda_f32(rotations_, "rotations"),
                     opacities = cuda_f32(opacities_, "opacity"), view = cuda_f32(s.view, "viewmatrix"),
                     proj = cuda_f32(s.proj, "projmatrix");
        if (P)
            check(L.cgx_preprocess_fwd((int)P, f32(means3D), f32(scales), s.scale_modifier, f32(rotations), f32(opacities),
                                       f32(view), f32(proj), s.W, s.H, s.tanfovx, s.tanfovy, f32(m2), f32(depths),
                                       i32(radii), nullptr, f32(co), stream()), "cgx_preprocess_fwd");
        ctx->set_materialize_grads(false);
        ctx->mark_non_differentiable({radii, depths});
        ctx->save_for_backward({means3D_, scales_, rotations_, radii, view, proj});
        Settings lean = s;
        lean.bg = lean.view = lean.proj = lean.campos = Tensor();
        keep(ctx, std::make_pair(lean, sh.requires_grad()));
        return {m2, rgb, co, radii, depths};
    }
    static variable_list backward(AutogradContext* ctx, variable_list g)
    {
        const auto& k = kept<std::pair<Settings, bool>>(ctx);
        const Settings& s = k.first;
        const variable_list v = ctx->get_saved_variables();
        const Tensor means3D = v[0].contiguous(), scales = v[1].contiguous(), rotations = v[2].contiguous();
        const int64_t P = means3D.size(0);
        const c10::cuda::CUDAGuard guard(means3D.device());
        const auto opt = means3D.options().requires_grad(false);
        const Tensor g_m2 = g[0].defined() ? cuda_f32(g[0], "dL_dmeans2D") : at::zeros({P, 2}, opt);
        const Tensor g_co = g[2].defined() ? cuda_f32(g[2], "dL_dconic_opacity") : at::zeros({P, 4}, opt);
        const Tensor dm = empty_f32({P, 3}, means3D), ds = empty_f32({P, 3}, means3D), dr = empty_f32({P, 4}, means3D),
                     dop = empty_f32({P, 1}, means3D);
        if (P)
            check(L.cgx_preprocess_bwd((int)P, f32(means3D), f32(scales), s.scale_modifier, f32(rotations), i32(v[3]),
                                       f32(v[4]), f32(v[5]), s.W, s.H, s.tanfovx, s.tanfovy, f32(g_m2), f32(g_co), f32(dm),
                                       f32(ds), f32(dr), f32(dop), stream()), "cgx_preprocess_bwd");
        return {dm, ds, dr, k.second ? at::zeros({P, 3}, opt) : Tensor(), dop, Tensor()};
    }
};

std::vector<Tensor> preprocess(const Tensor& means3D, const Tensor& scales, const Tensor& rotations, const Tensor& sh,
                               const Tensor& opacities, const py::object& settings)
{
    const Settings s = read_settings(settings);
    py::gil_scoped_release nogil;
    return Preprocess::apply(means3D, scales, rotations, sh, opacities, s);
}

// Radii of the Gaussians whose projection touches the image.  A trainer asks this for every camera of a batch in turn:
// through Python a call took 12 us of host time, as long as the kernel with 200 K Gaussians.
Tensor visible_filter(const Tensor& means3D_, const Tensor& scales_, const Tensor& rotations_, const py::object& settings)
{
    const Settings s = read_settings(settings, true);
    py::gil_scoped_release nogil;
    if (means3D_.dim() != 2 || means3D_.size(1) != 3)
        throw std::runtime_error("means3D must have dimensions (num_points, 3)");
    const Tensor means3D = cuda_f32(means3D_, "means3D");
    const int64_t P = means3D.size(0);
    const c10::cuda::CUDAGuard guard(means3D.device());
    const Tensor radii = empty_i32({P}, means3D);
    if (P == 0) return radii;
    if (scales_.numel() == 0 || rotations_.numel() == 0)
        throw std::runtime_error("visible_filter needs scales and rotations, or precomputed covariances");
    const Tensor scales = cuda_f32(scales_, "scales"), rotations = cuda_f32(rotations_, "rotations"),
                 view = cuda_f32(s.view, "viewmatrix"), proj = cuda_f32(s.proj, "projmatrix");
    check(L.cgx_filter_preprocess((int)P, f32(means3D), f32(scales), s.scale_modifier, f32(rotations), f32(view), f32(proj),
                                  s.W, s.H, s.tanfovx, s.tanfovy, i32(radii), stream()), "cgx_filter_preprocess");
    return radii;
}

// All cameras of a batch in one launch; per camera means2D, conic_opacity, radii, depths[, all_map].
struct Cameras {
    std::vector<cgx_camera> cam;
    std::vector<Tensor> matrices, campos;
    float scale_modifier = 1.f;
    bool planes = false;
};
constexpr size_t MAX_CAMS = 16;

struct PreprocessBatch : torch::autograd::Function<PreprocessBatch> {
    static variable_list forward(AutogradContext* ctx, const Tensor& means3D_, const Tensor& scales_,
                                 const Tensor& rotations_, const Tensor& opacities_, std::shared_ptr<Cameras> c)
    {
        if (means3D_.dim() != 2 || means3D_.size(1) != 3)
            throw std::runtime_error("means3D must have dimensions (num_points, 3)");
        const Tensor means3D = cuda_f32(means3D_, "means3D"), scales = cuda_f32(scales_, "scales"),
                     rotations = cuda_f32(rotations_, "rotations"), opacities = cuda_f32(opacities_, "opacities");
        const int64_t P = means3D.size(0);
        const size_t B = c->cam.size();
        const c10::cuda::CUDAGuard guard(means3D.device());
        variable_list out, fixed, saved = {means3D_, scales_, rotations_};
        float *m2[MAX_CAMS], *dep[MAX_CAMS], *co[MAX_CAMS], *am[MAX_CAMS];
        int32_t* rad[MAX_CAMS];
        const float* campos[MAX_CAMS];
        for (size_t b = 0; b < B; b++) {
            const Tensor t_m2 = empty_f32({P, 2}, means3D), t_co = empty_f32({P, 4}, means3D),
                         t_rad = empty_i32({P}, means3D), t_dep = empty_f32({P}, means3D);
            m2[b] = f32(t_m2), co[b] = f32(t_co), rad[b] = i32(t_rad), dep[b] = f32(t_dep);
            out.insert(out.end(), {t_m2, t_co, t_rad, t_dep});
            if (c->planes) {
                const Tensor t_am = empty_f32({P, 5}, means3D);
                am[b] = f32(t_am);
                campos[b] = f32(c->campos[b]);
                out.push_back(t_am);
            }
            fixed.insert(fixed.end(), {t_rad, t_dep});
            saved.push_back(t_rad);
        }
        if (P)
            check(L.cgx_preprocess_fwd_batched_planes((int)P, (int)B, f32(means3D), f32(scales), c->scale_modifier,
                                                      f32(rotations), f32(opacities), c->cam.data(),
                                                      c->planes ? campos : nullptr, m2, dep, rad, co,
                                                      c->planes ? am : nullptr, stream()), "cgx_preprocess_fwd_batched");
        ctx->set_materialize_grads(false);
        ctx->mark_non_differentiable(fixed);
        ctx->save_for_backward(std::move(saved));
        keep(ctx, std::move(c));
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g)
    {
        const Cameras& c = *kept<std::shared_ptr<Cameras>>(ctx);
        const variable_list v = ctx->get_saved_variables();
        const Tensor means3D = v[0].contiguous(), scales = v[1].contiguous(), rotations = v[2].contiguous();
        const int64_t P = means3D.size(0);
        const size_t B = c.cam.size(), n_out = c.planes ? 5 : 4;
        const c10::cuda::CUDAGuard guard(means3D.device());
        const auto opt = means3D.options().requires_grad(false);
        const Tensor dm = empty_f32({P, 3}, means3D), ds = empty_f32({P, 3}, means3D), dr = empty_f32({P, 4}, means3D),
                     dop = empty_f32({P, 1}, means3D);
        std::vector<cgx_camera> cam;
        std::vector<Tensor> hold;
        const float *gm[MAX_CAMS], *gc[MAX_CAMS], *ga[MAX_CAMS], *campos[MAX_CAMS];
        const int32_t* rad[MAX_CAMS];
        bool planes = false;
        auto ready = [&](const Tensor& t, int64_t n) {
            hold.push_back(t.defined() ? cuda_f32(t, "cotangent") : at::zeros({P, n}, opt));
            return (const float*)f32(hold.back());
        };
        for (size_t b = 0; b < B; b++) {
            const Tensor &m = g[n_out * b], &o = g[n_out * b + 1];
            const Tensor a = c.planes ? g[n_out * b + 4] : Tensor();
            if (!m.defined() && !o.defined() && !a.defined()) continue;      // no cotangent: contributes nothing
            const size_t i = cam.size();
            cam.push_back(c.cam[b]);
            gm[i] = ready(m, 2);
            gc[i] = ready(o, 4);
            ga[i] = a.defined() ? ready(a, 5) : nullptr;
            planes |= a.defined();
            campos[i] = c.planes ? f32(c.campos[b]) : nullptr;
            rad[i] = i32(v[3 + b]);
        }
        if (P && !cam.empty()) {
            check(L.cgx_preprocess_bwd_batched_planes((int)P, (int)cam.size(), f32(means3D), f32(scales), c.scale_modifier,
                                                      f32(rotations), cam.data(), planes ? campos : nullptr, rad, gm, gc,
                                                      planes ? ga : nullptr, f32(dm), f32(ds), f32(dr), f32(dop), stream()),
                  "cgx_preprocess_bwd_batched");
        } else {
            for (const Tensor& t : {dm, ds, dr, dop}) t.zero_();
        }
        return {dm, ds, dr, dop, Tensor()};
    }
};

std::vector<Tensor> preprocess_batched(const Tensor& means3D, const Tensor& scales, const Tensor& rotations,
                                       const Tensor& opacities, const py::list& settings, bool planes)
{
    const size_t B = settings.size();
    if (!means3D.is_cuda()) throw std::runtime_error("means3D must be a CUDA tensor (this rasterizer has no CPU path)");
    if (B < 1 || B > MAX_CAMS) throw std::runtime_error("between 1 and 16 cameras per batched call");
    auto c = std::make_shared<Cameras>();
    c->planes = planes;
    for (size_t b = 0; b < B; b++) {
        const Settings s = read_settings(settings[b]);
        if (b == 0) c->scale_modifier = s.scale_modifier;
        if (!s.view.is_cuda() || !s.proj.is_cuda()) throw std::runtime_error("camera matrices must be CUDA tensors");
        const Tensor view = s.view.contiguous(), proj = s.proj.contiguous();
        c->matrices.insert(c->matrices.end(), {view, proj});
        if (planes) c->campos.push_back(s.campos.contiguous());
        cgx_camera k;
        k.viewmatrix = f32(view);
        k.projmatrix = f32(proj);
        k.tanfovx = s.tanfovx;
        k.tanfovy = s.tanfovy;
        k.W = s.W;
        k.H = s.H;
        c->cam.push_back(k);
    }
    py::gil_scoped_release nogil;
    return PreprocessBatch::apply(means3D, scales, rotations, opacities, c);
}

// ---------------------------------------------------------------------------------------------- plane descriptors
struct PlaneMap : torch::autograd::Function<PlaneMap> {
    static Tensor forward(AutogradContext* ctx, const Tensor& means3D_, const Tensor& scales_, const Tensor& rotations_,
                          const c10::optional<Tensor>& radii_, const Tensor& view_, const Tensor& campos_)
    {
        auto ready = [](const Tensor& t, const char* name) {
            if (!t.is_cuda() || t.scalar_type() != at::kFloat)
                throw std::runtime_error(std::string("plane_map: ") + name + " must be a float32 CUDA tensor (no CPU path)");
            return t.contiguous();
        };
        const Tensor means3D = ready(means3D_, "means3D"), scales = ready(scales_, "scales"),
                     rotations = ready(rotations_, "rotations"), view = ready(view_, "viewmatrix"),
                     campos = ready(campos_, "campos");
        const Tensor radii = radii_ && radii_->defined() ? radii_->contiguous() : Tensor();
        const int64_t P = means3D.size(0);
        const c10::cuda::CUDAGuard guard(means3D.device());
        const Tensor out = empty_f32({P, 5}, means3D);
        if (P)
            check(L.cgx_all_map_fwd((int)P, f32(means3D), f32(scales), f32(rotations), radii.defined() ? i32(radii) : nullptr,
                                    f32(view), f32(campos), f32(out), stream()), "cgx_all_map_fwd");
        ctx->save_for_backward({means3D, scales, rotations, radii, view, campos});
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g)
    {
        const variable_list v = ctx->get_saved_variables();
        const Tensor &means3D = v[0], &radii = v[3], g5 = g[0].contiguous();
        const int64_t P = means3D.size(0);
        const c10::cuda::CUDAGuard guard(means3D.device());
        const Tensor dm = empty_f32({P, 3}, means3D), dr = empty_f32({P, 4}, means3D);
        if (P)
            check(L.cgx_all_map_bwd((int)P, f32(means3D), f32(v[1]), f32(v[2]), radii.defined() ? i32(radii) : nullptr,
                                    f32(v[4]), f32(v[5]), f32(g5), f32(dm), f32(dr), stream()), "cgx_all_map_bwd");
        return {dm, Tensor(), dr, Tensor(), Tensor(), Tensor()};
    }
};
Tensor plane_map(const Tensor& means3D, const Tensor& scales, const Tensor& rotations, const c10::optional<Tensor>& radii,
                 const Tensor& view, const Tensor& campos)
{
    return PlaneMap::apply(means3D, scales, rotations, radii, view, campos);
}

// ---------------------------------------------------------------------------------------------- loss
struct StripLoss : torch::autograd::Function<StripLoss> {
    static variable_list forward(AutogradContext* ctx, const Tensor& image_, const Tensor& gt_,
                                 const c10::optional<Tensor>& mask_)
    {
        if (!image_.is_cuda() || image_.scalar_type() != at::kFloat || !gt_.is_cuda() || gt_.scalar_type() != at::kFloat)
            throw std::runtime_error("strip_loss: image and gt must be float32 CUDA tensors (no CPU path)");
        if (image_.dim() != 3 || gt_.sizes() != image_.sizes())
            throw std::runtime_error("strip_loss: image and gt must both be (C, H, W)");
        const Tensor image = image_.contiguous(), gt = gt_.contiguous();
        const int64_t C = image.size(0), H = image.size(1), W = image.size(2);
        Tensor mask;
        if (mask_ && mask_->defined()) {
            if (mask_->dim() != 2 || mask_->size(0) != H || mask_->size(1) != W || !mask_->is_cuda())
                throw std::runtime_error("strip_loss: mask must be a (H, W) CUDA tensor");
            mask = mask_->to(at::kBool).contiguous();
        }
        const c10::cuda::CUDAGuard guard(image.device());
        const Tensor sums = at::empty({2}, image.options().dtype(at::kDouble).requires_grad(false));
        // the three derivative maps are for the backward pass
        const Tensor maps = image_.requires_grad() ? empty_f32({3, C, H, W}, image) : Tensor();
        const int64_t n = C * H * W;
        float* m = f32(maps);
        if (n)
            check(L.cgx_strip_loss_fwd((int)C, (int)H, (int)W, f32(image), f32(gt),
                                       mask.defined() ? static_cast<uint8_t*>(mask.data_ptr()) : nullptr,
                                       static_cast<double*>(sums.data_ptr()), m, m ? m + n : nullptr,
                                       m ? m + 2 * n : nullptr, stream()), "cgx_strip_loss_fwd");
        else
            sums.zero_();
        ctx->set_materialize_grads(false);
        ctx->save_for_backward({image, gt, mask, maps});
        const Tensor f = sums.to(at::kFloat);
        return {f.select(0, 0), f.select(0, 1)};
    }
    static variable_list backward(AutogradContext* ctx, variable_list g)
    {
        const variable_list v = ctx->get_saved_variables();
        const Tensor &image = v[0], &mask = v[2];
        const int64_t C = image.size(0), H = image.size(1), W = image.size(2), n = C * H * W;
        const c10::cuda::CUDAGuard guard(image.device());
        const auto opt = image.options().requires_grad(false);
        Tensor w[2];
        for (int k = 0; k < 2; k++) w[k] = g[k].defined() ? g[k].to(at::kFloat) : at::zeros({}, opt);
        const Tensor weights = at::stack({w[0], w[1]}), grad = at::empty_like(image);
        const float* m = f32(v[3]);
        if (n)
            check(L.cgx_strip_loss_bwd((int)C, (int)H, (int)W, f32(image), f32(v[1]),
                                       mask.defined() ? static_cast<uint8_t*>(mask.data_ptr()) : nullptr, f32(weights), m,
                                       m + n, m + 2 * n, f32(grad), stream()), "cgx_strip_loss_bwd");
        return {grad, Tensor(), Tensor()};
    }
};
std::vector<Tensor> strip_loss(const Tensor& image, const Tensor& gt, const c10::optional<Tensor>& mask)
{
    return StripLoss::apply(image, gt, mask);
}

struct DepthNormal : torch::autograd::Function<DepthNormal> {
    static Tensor forward(AutogradContext* ctx, const Tensor& depth_, double fx, double fy, double cx, double cy)
    {
        if (!depth_.is_cuda() || depth_.scalar_type() != at::kFloat || depth_.dim() != 2)
            throw std::runtime_error("depth_normal: depth must be a (H, W) float32 CUDA tensor (no CPU path)");
        const Tensor depth = depth_.contiguous();
        const int64_t H = depth.size(0), W = depth.size(1);
        const c10::cuda::CUDAGuard guard(depth.device());
        const Tensor normal = empty_f32({3, H, W}, depth);
        if (H * W)
            check(L.cgx_depth_normal_fwd((int)H, (int)W, (float)fx, (float)fy, (float)cx, (float)cy, f32(depth),
                                         f32(normal), stream()), "cgx_depth_normal_fwd");
        ctx->save_for_backward({depth});
        keep(ctx, std::array<float, 4>{(float)fx, (float)fy, (float)cx, (float)cy});
        return normal;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g)
    {
        const Tensor depth = ctx->get_saved_variables()[0];
        const auto& k = kept<std::array<float, 4>>(ctx);
        const c10::cuda::CUDAGuard guard(depth.device());
        const Tensor out = at::empty_like(depth), gn = g[0].contiguous();
        if (depth.numel())
            check(L.cgx_depth_normal_bwd((int)depth.size(0), (int)depth.size(1), k[0], k[1], k[2], k[3], f32(depth), f32(gn),
                                         f32(out), stream()), "cgx_depth_normal_bwd");
        return {out, Tensor(), Tensor(), Tensor(), Tensor()};
    }
};
Tensor depth_normal_op(const Tensor& depth, double fx, double fy, double cx, double cy)
{
    return DepthNormal::apply(depth, fx, fy, cx, cy);
}

// ---------------------------------------------------------------------------------------------- statistics
// The anchors' statistics in one call; false where a tensor's type, layout or size asks for the tensor expressions.
bool anchor_stats(int n_offsets, const Tensor& opacity_accum, const Tensor& anchor_demon, const Tensor& gradient_accum,
                  const Tensor& denom, const Tensor& on_screen, const Tensor& selected, const Tensor& seen,
                  const Tensor& grad, const Tensor& opacity)
{
    const auto device = opacity.device();
    auto plain = [&](const Tensor& t, at::ScalarType type) {
        return t.is_cuda() && t.scalar_type() == type && t.is_contiguous() && t.device() == device;
    };
    for (const Tensor* t : {&opacity_accum, &anchor_demon, &gradient_accum, &denom, &opacity})
        if (!plain(*t, at::kFloat)) return false;
    for (const Tensor* t : {&on_screen, &selected, &seen})
        if (!plain(*t, at::kBool)) return false;
    if (!grad.is_cuda() || grad.device() != device || grad.scalar_type() != at::kFloat || grad.dim() != 2 ||
        grad.size(1) < 2 || grad.stride(1) != 1 || opacity.numel() != selected.numel() || seen.numel() == 0 ||
        on_screen.numel() != grad.size(0))
        return false;
    const c10::cuda::CUDAGuard guard(device);
    const int64_t n = seen.numel(), slots = selected.numel();
    const size_t bytes = L.cgx_anchor_stats_workspace_bytes((int)n, slots);
    const Tensor ws = bytes_like(bytes, opacity);
    auto bits = [](const Tensor& t) { return static_cast<const uint8_t*>(t.data_ptr()); };
    check(L.cgx_anchor_stats((int)n, n_offsets, slots, on_screen.numel(), f32(grad),
                             (int)std::max<int64_t>(2, grad.stride(0)), f32(opacity), bits(on_screen), bits(selected),
                             bits(seen), f32(opacity_accum), f32(anchor_demon), f32(gradient_accum), f32(denom),
                             ws.data_ptr(), bytes, stream()), "cgx_anchor_stats");
    return true;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m)
{
    const auto nogil = py::call_guard<py::gil_scoped_release>();
    m.def("bind", &bind);
    m.def("prefetch", &prefetch, nogil);
    m.def("take_prefetched", &take_prefetched);
    m.def("prefetched", &prefetched_counts, nogil);
    m.def("render", &render);
    m.def("preprocess", &preprocess);
    m.def("anchor_stats", &anchor_stats, nogil);
    m.def("visible_filter", &visible_filter);
    m.def("preprocess_batched", &preprocess_batched);
    m.def("plane_map", &plane_map, nogil);
    m.def("strip_loss", &strip_loss, nogil);
    m.def("depth_normal", &depth_normal_op, nogil);
    auto num = [](const py::object& o) { return py::float_(o).cast<double>(); };
    py::class_<EventMs, std::shared_ptr<EventMs>>(m, "EventMs")
        .def("__float__", &EventMs::get)
        .def("__add__", [num](EventMs& a, const py::object& o) { return a.get() + num(o); })
        .def("__radd__", [num](EventMs& a, const py::object& o) { return a.get() + num(o); })
        .def("__mul__", [num](EventMs& a, const py::object& o) { return a.get() * num(o); })
        .def("__rmul__", [num](EventMs& a, const py::object& o) { return a.get() * num(o); })
        .def("__sub__", [num](EventMs& a, const py::object& o) { return a.get() - num(o); })
        .def("__rsub__", [num](EventMs& a, const py::object& o) { return num(o) - a.get(); })
        .def("__truediv__", [num](EventMs& a, const py::object& o) { return a.get() / num(o); })
        .def("__repr__", [](EventMs& a) { return std::to_string(a.get()); });
}
