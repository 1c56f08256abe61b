// The operators' host path as native autograd nodes (Python module `triton_helpers_b200._native`).
//
// A small call of these operators is bound by the host: a few microseconds of kernel behind 40 us of Python
// (argument checks, the autograd Function, ctypes) in forward and 170 us with a backward pass.  The functions
// here take the usual call - plain CUDA tensors, no autocast, no event timing - from the public Python function
// straight to the C ABI of include/th_b200.h and record a C++ autograd node when a gradient is wanted, so that
// the backward pass runs on the autograd thread without the interpreter lock.  Measured on a B200, host time of
// one pass, calls back to back: encoding query (777 points) 40 -> 6.3 us, MLP query (1000 rows) 38 -> 8.8 us, encoding forward +
// backward (65536 points) 178 -> 77 us and reversible stack (5003 rows) 233 -> 89 us, both now bound by their kernels.
//
// Every function returns NotImplemented when the call is not the usual one or when any argument is not exactly
// what the kernels take; the Python implementation then runs (copies where strides ask for them, autocast,
// timing) or raises its own error, so the set of accepted calls and the error texts live in one place.  Nothing
// is launched before a function has made up its mind.
#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <atomic>
#include <cstring>
#include <memory>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "../../include/th_b200.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// ---- what the usual call looks like ---------------------------------------------------------------

std::atomic<bool> g_deferred{false};  // event timing of every launch is on: leave the calls to Python

// A CUDA tensor nothing else has a say in: no Python or functorch dispatch, no lazy conjugation or negation.
bool plain(const Tensor &t) {
    using c10::DispatchKey;
    static const c10::DispatchKeySet others({DispatchKey::Python, DispatchKey::PythonTLSSnapshot, DispatchKey::FuncTorchBatched,
                                             DispatchKey::FuncTorchGradWrapper, DispatchKey::Batched, DispatchKey::Functionalize,
                                             DispatchKey::Conjugate, DispatchKey::Negative, DispatchKey::ZeroTensor, DispatchKey::NestedTensor});
    return t.defined() && t.is_cuda() && !t.key_set().has_any(others) && t.layout() == at::kStrided;
}

bool usual_mode() {
    // a dispatch or function mode, or a functorch level, shows up in the thread's included keys
    using c10::DispatchKey;
    static const c10::DispatchKeySet modes({DispatchKey::Python, DispatchKey::PythonTLSSnapshot, DispatchKey::FuncTorchDynamicLayerFrontMode,
                                            DispatchKey::FuncTorchDynamicLayerBackMode, DispatchKey::Functionalize});
    return !g_deferred.load(std::memory_order_relaxed) && !at::autocast::is_autocast_enabled(at::kCUDA) &&
           !c10::impl::tls_local_dispatch_key_set().included_.has_any(modes);
}

// One optional tensor argument; false when it is neither None nor a tensor.
bool take(PyObject *o, Tensor &t) {
    if (o == Py_None) return true;
    if (!THPVariable_Check(o)) return false;
    t = THPVariable_Unpack(o);
    return true;
}

bool take(PyObject *o, int64_t &v) {
    if (!PyLong_CheckExact(o)) return false;
    v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}

bool take(PyObject *o, double &v) {
    if (PyFloat_CheckExact(o)) {
        v = PyFloat_AS_DOUBLE(o);
        return true;
    }
    int64_t i;
    if (!take(o, i)) return false;
    v = static_cast<double>(i);
    return true;
}

int activation_code(PyObject *o) {
    if (!PyUnicode_CheckExact(o)) return -1;
    const char *s = PyUnicode_AsUTF8(o);
    if (!s) {
        PyErr_Clear();
        return -1;
    }
    if (!strcmp(s, "relu")) return TH_ACT_RELU;
    if (!strcmp(s, "none")) return TH_ACT_NONE;
    if (!strcmp(s, "silu")) return TH_ACT_SILU;
    if (!strcmp(s, "relu2")) return TH_ACT_RELU2;
    return -1;
}

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return TH_F32;
        case at::kHalf: return TH_F16;
        case at::kBFloat16: return TH_BF16;
        default: return -1;
    }
}

Tensor empty_like_shape(c10::IntArrayRef sizes, at::ScalarType dtype, c10::Device device) {
    return Tensor(at::detail::empty_cuda(sizes, dtype, device, std::nullopt));
}

Tensor empty_same(const Tensor &t) { return t.defined() ? empty_like_shape(t.sizes(), t.scalar_type(), t.device()) : Tensor(); }

void *ptr(const Tensor &t) { return t.defined() ? t.data_ptr() : nullptr; }

void check(int code, const char *what) { TORCH_CHECK(code == 0, what, " failed with code ", code, ": ", th_last_error_string()); }

void *current_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// Rows of the last dimension, `width` wide, evenly strided with unit stride inside a row; copies when the layout asks for it.
struct Rows {
    Tensor keep;
    int64_t n = 0, stride = 0;
};

bool rows_of(const Tensor &t, int64_t width, Rows &r) {
    const auto sizes = t.sizes();
    const int64_t nd = t.dim();
    if (nd < 1 || sizes[nd - 1] != width) return false;
    r.n = width ? t.numel() / width : 0;
    if (t.is_contiguous()) {
        r.keep = t;
        r.stride = width;
        return true;
    }
    if (nd == 2 && t.stride(1) == 1 && t.stride(0) >= width) {
        r.keep = t;
        r.stride = r.n > 1 ? t.stride(0) : width;
        return true;
    }
    return false;
}

Rows rows_or_copy(const Tensor &t, int64_t width) {
    Rows r;
    if (!rows_of(t, width, r)) rows_of(t.contiguous(), width, r);
    return r;
}

template <typename N>
std::shared_ptr<N> make_node(torch::autograd::edge_list &&edges) {
    auto node = std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
    node->set_next_edges(std::move(edges));
    return node;
}

#define TH_NOT_MINE              \
    do {                         \
        Py_INCREF(Py_NotImplemented); \
        return Py_NotImplemented;     \
    } while (0)

struct NoGil {
    PyThreadState *state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};

// ---- level geometry and hash primes ----------------------------------------------------------------

struct Geometry {
    int levels = 0;
    int64_t total_rows = 0;
    int32_t res[TH_MAX_LEVELS];
    int64_t rows[TH_MAX_LEVELS], offsets[TH_MAX_LEVELS];
};

PyObject *g_geometry_source = nullptr;  // layers.hash_encoding.helpers.level_geometry
PyObject *g_primes_source = nullptr;    // layers.hash_encoding.kernel.host_primes

// Level layout of (levels, T, D, N_min, N_max) as the package's Python helper computes it, remembered.  Called
// with the interpreter lock held; null when the helper refuses the arguments (Python then raises its error).
std::shared_ptr<const Geometry> geometry(int64_t levels, int64_t cap, int64_t dims, int64_t min_res, int64_t max_res) {
    struct Key {
        int64_t v[5];
        bool operator==(const Key &o) const { return !memcmp(v, o.v, sizeof(v)); }
    };
    struct Hash {
        size_t operator()(const Key &k) const {
            size_t h = 0;
            for (int64_t x : k.v) h = h * 1000003u + static_cast<size_t>(x);
            return h;
        }
    };
    static std::unordered_map<Key, std::shared_ptr<const Geometry>, Hash> known;
    if (levels < 2 || levels > TH_MAX_LEVELS || (levels & (levels - 1)) || !g_geometry_source) return nullptr;
    const Key key{{levels, cap, dims, min_res, max_res}};
    const auto hit = known.find(key);
    if (hit != known.end()) return hit->second;
    PyObject *geo = PyObject_CallFunction(g_geometry_source, "LLLLL", levels, cap, dims, min_res, max_res);
    PyObject *res = geo ? PyObject_GetAttrString(geo, "resolutions") : nullptr;
    PyObject *rows = res ? PyObject_GetAttrString(geo, "rows") : nullptr;
    PyObject *offs = rows ? PyObject_GetAttrString(geo, "offsets") : nullptr;
    std::shared_ptr<Geometry> g;
    if (offs && PySequence_Size(res) == levels && PySequence_Size(rows) == levels && PySequence_Size(offs) == levels) {
        g = std::make_shared<Geometry>();
        g->levels = static_cast<int>(levels);
        auto item = [](PyObject *seq, Py_ssize_t i) {
            PyObject *o = PySequence_GetItem(seq, i);
            const int64_t v = o ? PyLong_AsLongLong(o) : -1;
            Py_XDECREF(o);
            return v;
        };
        for (Py_ssize_t l = 0; l < levels; ++l) {
            g->res[l] = static_cast<int32_t>(item(res, l));
            g->rows[l] = item(rows, l);
            g->offsets[l] = item(offs, l);
        }
        g->total_rows = g->offsets[levels - 1] + g->rows[levels - 1];
    }
    Py_XDECREF(offs);
    Py_XDECREF(rows);
    Py_XDECREF(res);
    Py_XDECREF(geo);
    if (PyErr_Occurred()) {
        PyErr_Clear();
        return nullptr;
    }
    if (!g) return nullptr;
    if (known.size() >= 1024) known.clear();
    known.emplace(key, g);
    return g;
}

struct Primes {
    int64_t v[TH_MAX_DIMS] = {1, 2654435761ll, 805459861ll};
};

// The first `dims` primes of a device tensor, read once per tensor and version (by the Python helper, which
// remembers them the same way); false when Python should look at the tensor itself.
bool primes_of(PyObject *o, const Tensor &pi, int64_t dims, Primes &out) {
    struct Seen {
        c10::weak_intrusive_ptr<c10::TensorImpl> tensor;
        uint32_t version;
        Primes primes;
        int64_t count;
    };
    static std::vector<Seen> seen;
    if (pi.dim() != 1 || pi.numel() < dims || pi.scalar_type() != at::kLong || pi.requires_grad() || pi.is_inference()) return false;
    const uint32_t version = static_cast<uint32_t>(pi._version());
    for (const Seen &s : seen) {
        if (s.tensor._unsafe_get_target() == pi.unsafeGetTensorImpl() && !s.tensor.expired() && s.version == version && s.count >= dims) {
            out = s.primes;
            return true;
        }
    }
    PyObject *values = g_primes_source ? PyObject_CallFunction(g_primes_source, "OL", o, dims) : nullptr;
    bool ok = values && PyTuple_Check(values) && PyTuple_GET_SIZE(values) == dims;
    for (int64_t d = 0; ok && d < dims; ++d) out.v[d] = PyLong_AsLongLong(PyTuple_GET_ITEM(values, d));
    Py_XDECREF(values);
    if (PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    if (!ok) return false;
    if (seen.size() >= 64) seen.clear();
    seen.push_back({c10::weak_intrusive_ptr<c10::TensorImpl>(pi.getIntrusivePtr()), version, out, dims});
    return true;
}

// ---- hash encoding ------------------------------------------------------------------------------------

// Everything about one encoding call that its backward pass needs again.
struct EncodeCall {
    std::shared_ptr<const Geometry> geo;
    Primes primes;
    int64_t dims = 0, feats = 0, n = 0;
    float scale = 1.f;
};

struct CoordArgs {
    Tensor keep;
    int64_t stride_n = 0, stride_d = 1;
};

// Coordinates (..., D) as rows with any strides (they are read element-wise when not packed).
CoordArgs coord_args(const Tensor &coords, int64_t dims) {
    CoordArgs a;
    a.keep = coords.dim() == 2 ? coords : coords.reshape({-1, dims});
    a.stride_n = a.keep.size(0) > 1 ? a.keep.stride(0) : dims;
    a.stride_d = a.keep.stride(1);
    return a;
}

// The batch along a space-filling curve, 16 bytes per point
Tensor point_order(const EncodeCall &c, const CoordArgs &x, void *stream) {
    Tensor order = empty_like_shape({c.n, 4}, at::kFloat, x.keep.device());
    const int64_t bytes = th_hash_order_scratch_bytes(c.n, static_cast<int>(c.dims));
    const Tensor scratch = empty_like_shape({bytes}, at::kByte, x.keep.device());
    check(th_hash_order(ptr(x.keep), x.stride_n, x.stride_d, dtype_code(x.keep.scalar_type()), c.n, static_cast<int>(c.dims), c.scale, ptr(order),
                        ptr(scratch), bytes, stream),
          "th_hash_order");
    return order;
}

// `order`: the batch's order, or an undefined tensor
void hash_forward(const EncodeCall &c, const CoordArgs &x, const Tensor &order, const Tensor &table, const Tensor &out, void *stream) {
    const Geometry &g = *c.geo;
    if (order.defined()) {
        check(th_hash_fwd_ordered(ptr(order), 0, ptr(table), dtype_code(table.scalar_type()), ptr(out), c.feats * g.levels, c.n,
                                  static_cast<int>(c.dims), static_cast<int>(c.feats), g.levels, g.res, g.rows, g.offsets, c.primes.v, 0, g.levels, stream),
              "th_hash_fwd_ordered");
        return;
    }
    check(th_hash_fwd(ptr(x.keep), x.stride_n, x.stride_d, dtype_code(x.keep.scalar_type()), ptr(table), dtype_code(table.scalar_type()),
                      ptr(out), c.feats * g.levels, c.n, static_cast<int>(c.dims), static_cast<int>(c.feats), g.levels, g.res, g.rows, g.offsets,
                      c.primes.v, c.scale, 0, g.levels, stream),
          "th_hash_fwd");
}

void hash_backward(const EncodeCall &c, const CoordArgs &x, const Tensor &order, const Rows &go, const Tensor &grad_table, void *stream) {
    const Geometry &g = *c.geo;
    if (order.defined()) {
        check(th_hash_bwd_ordered(ptr(order), 0, ptr(go.keep), go.stride, ptr(grad_table), dtype_code(grad_table.scalar_type()), c.n,
                                  static_cast<int>(c.dims), static_cast<int>(c.feats), g.levels, g.res, g.rows, g.offsets, c.primes.v, 0, g.levels, stream),
              "th_hash_bwd_ordered");
        return;
    }
    check(th_hash_bwd(ptr(x.keep), x.stride_n, x.stride_d, dtype_code(x.keep.scalar_type()), ptr(go.keep), go.stride, ptr(grad_table),
                      dtype_code(grad_table.scalar_type()), c.n, static_cast<int>(c.dims), static_cast<int>(c.feats), g.levels, g.res, g.rows,
                      g.offsets, c.primes.v, c.scale, 0, g.levels, stream),
          "th_hash_bwd");
}

struct HashEncodingNode : public Node {
    EncodeCall call;
    SavedVariable coords, table;
    Tensor order;

    std::string name() const override { return "HashEncodingBackward"; }
    void release_variables() override {
        order.reset();
        coords.reset_data();
        table.reset_data();
    }
    variable_list apply(variable_list &&grads) override {
        variable_list out(1);
        if (!grads[0].defined()) return out;
        const Tensor x = coords.unpack(), t = table.unpack();
        at::NoGradGuard no_grad;
        c10::cuda::CUDAGuard guard(t.device());
        Tensor go = grads[0];
        if (go.scalar_type() != t.scalar_type()) go = go.to(t.scalar_type());
        const Rows rows = rows_or_copy(go, call.feats * call.geo->levels);
        Tensor de = empty_like_shape(t.sizes(), t.scalar_type(), t.device());
        de.zero_();
        hash_backward(call, coord_args(x, call.dims), order, rows, de, current_stream());
        out[0] = std::move(de);
        return out;
    }
};

// Coordinates, table and geometry shared by the encoding and the fused encoding + MLP; false: not the usual call.
bool encode_call(EncodeCall &c, const Tensor &coords, const Tensor &table, PyObject *pi_object, PyObject *const *geometry_args, PyObject *levels_arg,
                 PyObject *scale_arg) {
    int64_t cap, min_res, max_res, levels;
    double scale;
    if (!plain(coords) || !plain(table) || coords.device() != table.device() || coords.requires_grad()) return false;
    if (dtype_code(coords.scalar_type()) < 0 || dtype_code(table.scalar_type()) < 0) return false;
    if (coords.dim() < 1 || table.dim() != 2 || !table.is_contiguous()) return false;
    if (!take(geometry_args[0], cap) || !take(geometry_args[1], min_res) || !take(geometry_args[2], max_res) || !take(levels_arg, levels) ||
        !take(scale_arg, scale))
        return false;
    c.dims = coords.size(-1);
    c.feats = table.size(1);
    if (c.dims < 1 || c.dims > TH_MAX_DIMS || (c.feats != 1 && c.feats != 2 && c.feats != 4 && c.feats != 8)) return false;
    c.n = coords.numel() / c.dims;
    c.scale = static_cast<float>(scale);
    if (pi_object != Py_None) {
        if (!THPVariable_Check(pi_object)) return false;
        const Tensor &pi = THPVariable_Unpack(pi_object);
        if (!plain(pi) || pi.device() != coords.device() || !primes_of(pi_object, pi, c.dims, c.primes)) return false;
    }
    c.geo = geometry(levels, cap, c.dims, min_res, max_res);
    return c.geo && table.size(0) >= c.geo->total_rows;
}

std::vector<int64_t> with_last(const Tensor &t, int64_t last) {
    std::vector<int64_t> sizes = t.sizes().vec();
    sizes.back() = last;
    return sizes;
}

// hash_encoding(coord, embeddings, features, pi, max_entries_per_level, min_res, max_res, levels, divider, bwd_divider, scale)
PyObject *py_hash_encoding(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (n_args != 11 || !usual_mode() || !THPVariable_Check(args[0]) || !THPVariable_Check(args[1]) || args[2] != Py_None ||
        args[8] != Py_None || args[9] != Py_None)
        TH_NOT_MINE;
    const Tensor coords = THPVariable_Unpack(args[0]), table = THPVariable_Unpack(args[1]);
    EncodeCall call;
    if (!encode_call(call, coords, table, args[3], args + 4, args[7], args[10])) TH_NOT_MINE;
    Tensor out;
    {
        NoGil release;
        const bool grad = torch::autograd::compute_requires_grad(table);
        std::shared_ptr<HashEncodingNode> node;
        if (grad) {
            node = make_node<HashEncodingNode>(torch::autograd::collect_next_edges(table));
            node->call = call;
            node->coords = SavedVariable(coords, false);
            node->table = SavedVariable(table, false);
        }
        {
            at::AutoDispatchBelowADInplaceOrView below;
            c10::cuda::CUDAGuard guard(coords.device());
            out = empty_like_shape(with_last(coords, call.feats * call.geo->levels), table.scalar_type(), table.device());
            const CoordArgs x = coord_args(coords, call.dims);
            void *stream = current_stream();
            Tensor order = th_hash_order_pays(call.n, static_cast<int>(call.dims), static_cast<int>(call.feats * table.element_size()), grad) ? point_order(call, x, stream) : Tensor();
            hash_forward(call, x, order, table, out, stream);
            if (grad) node->order = std::move(order);
        }
        if (grad) torch::autograd::set_history(out, node);
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// ---- fused MLP ---------------------------------------------------------------------------------------

struct MlpCall {
    int64_t batch = 0, length = 0;
    int d_in = 0, hidden = 0, d_out = 0, depth = 1, act = 0, dtype = TH_F16;
    int64_t x_stride = 0;

    int64_t rows() const { return batch * length; }
};

struct MlpTensors {
    Tensor w_in, b_in, w_out, b_out, w_hid, b_hid;
};

void mlp_forward(const MlpCall &c, const Tensor &x, const MlpTensors &p, const Tensor &out, void *stream) {
    check(th_mlp_fwd(ptr(x), c.x_stride, ptr(p.w_in), ptr(p.b_in), ptr(p.w_hid), ptr(p.b_hid), ptr(p.w_out), ptr(p.b_out), ptr(out), c.d_out,
                     c.rows(), c.d_in, c.hidden, c.d_out, c.depth, c.act, c.dtype, 0, stream),
          "th_mlp_fwd");
}

struct MlpNode : public Node {
    MlpCall call;
    SavedVariable x, w_in, b_in, w_out, b_out, w_hid, b_hid;
    bool has_bias = false;

    std::string name() const override { return "FullyFusedMLPBackward"; }
    void release_variables() override {
        for (SavedVariable *v : {&x, &w_in, &b_in, &w_out, &b_out, &w_hid, &b_hid}) v->reset_data();
    }
    variable_list apply(variable_list &&grads) override {
        variable_list out(7);
        if (!grads[0].defined()) return out;
        const bool hidden = call.depth > 1;
        const Tensor xs = x.unpack();
        MlpTensors p;
        p.w_in = w_in.unpack();
        p.w_out = w_out.unpack();
        if (hidden) p.w_hid = w_hid.unpack();
        if (has_bias) {
            p.b_in = b_in.unpack();
            p.b_out = b_out.unpack();
            if (hidden) p.b_hid = b_hid.unpack();
        }
        at::NoGradGuard no_grad;
        c10::cuda::CUDAGuard guard(xs.device());
        Tensor go = grads[0];
        if (go.scalar_type() != xs.scalar_type()) go = go.to(xs.scalar_type());
        const Rows g = rows_or_copy(go, call.d_out);
        const Tensor dx = task_should_compute_output(0) ? empty_like_shape({call.batch, call.length, call.d_in}, xs.scalar_type(), xs.device()) : Tensor();
        MlpTensors d;
        d.w_in = empty_same(p.w_in);
        d.b_in = empty_same(p.b_in);
        d.w_out = empty_same(p.w_out);
        d.b_out = empty_same(p.b_out);
        d.w_hid = empty_same(p.w_hid);
        d.b_hid = empty_same(p.b_hid);
        const int64_t bytes = th_mlp_workspace_bytes(call.d_in, call.hidden, call.d_out, call.depth);
        const Tensor workspace = empty_like_shape({bytes}, at::kByte, xs.device());
        check(th_mlp_bwd(ptr(xs), call.x_stride, ptr(p.w_in), ptr(p.b_in), ptr(p.w_hid), ptr(p.b_hid), ptr(p.w_out), ptr(p.b_out), ptr(g.keep), g.stride,
                         ptr(dx), call.d_in, ptr(d.w_in), ptr(d.b_in), ptr(d.w_hid), ptr(d.b_hid), ptr(d.w_out), ptr(d.b_out), ptr(workspace), bytes,
                         call.rows(), call.d_in, call.hidden, call.d_out, call.depth, call.act, call.dtype, 0, current_stream()),
              "th_mlp_bwd");
        out[0] = dx;
        out[1] = d.w_in;
        out[2] = d.b_in;
        out[3] = d.w_out;
        out[4] = d.b_out;
        out[5] = d.w_hid;
        out[6] = d.b_hid;
        return out;
    }
};

// A parameter of the layer: plain, contiguous, same dtype and device as the input.
bool parameter_like(const Tensor &t, const Tensor &x, c10::IntArrayRef sizes) {
    return plain(t) && t.is_contiguous() && t.scalar_type() == x.scalar_type() && t.device() == x.device() && t.sizes() == sizes;
}

bool mlp_call(MlpCall &c, const Tensor &x, MlpTensors &p, PyObject *activation) {
    if (!plain(x) || x.dim() != 3 || !plain(p.w_in) || p.w_in.dim() != 2 || !plain(p.w_out) || p.w_out.dim() != 2) return false;
    c.dtype = dtype_code(x.scalar_type());
    if (c.dtype != TH_F16 && c.dtype != TH_BF16) return false;
    const int64_t hidden = p.w_in.size(0), d_in = p.w_in.size(1), d_out = p.w_out.size(0);
    if (d_in < 1 || d_in > 64 || d_out < 1 || d_out > 64 || (hidden != 16 && hidden != 32 && hidden != 64)) return false;
    if (x.size(2) != d_in) return false;
    c.batch = x.size(0);
    c.length = x.size(1);
    c.act = activation_code(activation);
    if (c.act < 0) return false;
    int64_t depth = 1;
    if (p.w_hid.defined()) {
        if (p.w_hid.dim() != 2 || p.w_hid.numel() == 0) return false;
        depth += p.w_hid.size(0) / hidden;
        if (!parameter_like(p.w_hid, x, {(depth - 1) * hidden, hidden})) return false;
    }
    const bool bias = p.b_in.defined();
    if (p.b_out.defined() != bias || p.b_hid.defined() != (bias && depth > 1)) return false;
    if (!parameter_like(p.w_in, x, {hidden, d_in}) || !parameter_like(p.w_out, x, {d_out, hidden})) return false;
    if (bias && (!parameter_like(p.b_in, x, {hidden}) || !parameter_like(p.b_out, x, {d_out}) ||
                 (depth > 1 && !parameter_like(p.b_hid, x, {depth - 1, hidden}))))
        return false;
    // rows evenly strided over both leading dimensions
    if (x.stride(2) != 1 || (c.batch > 1 && x.stride(0) != c.length * x.stride(1)) || x.stride(1) < d_in) return false;
    c.x_stride = x.stride(1);
    c.d_in = static_cast<int>(d_in);
    c.hidden = static_cast<int>(hidden);
    c.d_out = static_cast<int>(d_out);
    c.depth = static_cast<int>(depth);
    return true;
}

// fully_fused_mlp(x, w_in, b_in, w_out, b_out, w_hid, b_hid, activation)
PyObject *py_fully_fused_mlp(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    Tensor x;
    MlpTensors p;
    if (n_args != 8 || !usual_mode() || !take(args[0], x) || !take(args[1], p.w_in) || !take(args[2], p.b_in) || !take(args[3], p.w_out) ||
        !take(args[4], p.b_out) || !take(args[5], p.w_hid) || !take(args[6], p.b_hid))
        TH_NOT_MINE;
    MlpCall call;
    if (!mlp_call(call, x, p, args[7])) TH_NOT_MINE;
    Tensor out;
    {
        NoGil release;
        const bool grad = torch::autograd::compute_requires_grad(x, p.w_in, p.b_in, p.w_out, p.b_out, p.w_hid, p.b_hid);
        std::shared_ptr<MlpNode> node;
        if (grad) {
            node = make_node<MlpNode>(torch::autograd::collect_next_edges(x, p.w_in, p.b_in, p.w_out, p.b_out, p.w_hid, p.b_hid));
            node->call = call;
            node->has_bias = p.b_in.defined();
            node->x = SavedVariable(x, false);
            node->w_in = SavedVariable(p.w_in, false);
            node->w_out = SavedVariable(p.w_out, false);
            if (p.w_hid.defined()) node->w_hid = SavedVariable(p.w_hid, false);
            if (p.b_in.defined()) node->b_in = SavedVariable(p.b_in, false);
            if (p.b_out.defined()) node->b_out = SavedVariable(p.b_out, false);
            if (p.b_hid.defined()) node->b_hid = SavedVariable(p.b_hid, false);
        }
        {
            at::AutoDispatchBelowADInplaceOrView below;
            c10::cuda::CUDAGuard guard(x.device());
            out = empty_like_shape({call.batch, call.length, call.d_out}, x.scalar_type(), x.device());
            mlp_forward(call, x, p, out, current_stream());
        }
        if (grad) torch::autograd::set_history(out, node);
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// ---- reversible MLP -------------------------------------------------------------------------------------

struct RevCall {
    int64_t rows = 0, x_stride = 0;
    int d_model = 0, hidden = 0, blocks = 0, act = 0, dtype = TH_F16;
};

struct ReversibleNode : public Node {
    RevCall call;
    SavedVariable y, w[4], b[4];
    bool has_bias = false;

    std::string name() const override { return "ReversibleMLPBackward"; }
    void release_variables() override {
        y.reset_data();
        for (int i = 0; i < 4; ++i) {
            w[i].reset_data();
            b[i].reset_data();
        }
    }
    variable_list apply(variable_list &&grads) override {
        variable_list out(9);
        if (!grads[0].defined()) return out;
        const Tensor ys = y.unpack(shared_from_this());
        Tensor ws[4], bs[4], dw[4], db[4];
        for (int i = 0; i < 4; ++i) {
            ws[i] = w[i].unpack();
            if (has_bias) bs[i] = b[i].unpack();
        }
        at::NoGradGuard no_grad;
        c10::cuda::CUDAGuard guard(ys.device());
        Tensor go = grads[0];
        if (go.scalar_type() != ys.scalar_type()) go = go.to(ys.scalar_type());
        Rows g = rows_or_copy(go, call.d_model);
        if (g.stride % 2 || reinterpret_cast<uintptr_t>(ptr(g.keep)) % 4) g = rows_or_copy(go.clone(at::MemoryFormat::Contiguous), call.d_model);
        for (int i = 0; i < 4; ++i) {
            dw[i] = empty_same(ws[i]);
            db[i] = empty_same(bs[i]);
        }
        const Tensor dx = empty_like_shape(ys.sizes(), ys.scalar_type(), ys.device());
        const int64_t bytes = th_rev_workspace_bytes(call.rows, call.d_model, call.hidden, call.blocks);
        const Tensor workspace = empty_like_shape({bytes}, at::kByte, ys.device());
        check(th_rev_bwd(ptr(ys), call.d_model, ptr(ws[0]), ptr(ws[1]), ptr(ws[2]), ptr(ws[3]), ptr(bs[0]), ptr(bs[1]), ptr(bs[2]), ptr(bs[3]),
                         ptr(g.keep), g.stride, ptr(dx), call.d_model, nullptr, call.d_model, ptr(dw[0]), ptr(dw[1]), ptr(dw[2]), ptr(dw[3]), ptr(db[0]),
                         ptr(db[1]), ptr(db[2]), ptr(db[3]), ptr(workspace), bytes, call.rows, call.d_model, call.hidden, call.blocks, call.act,
                         call.dtype, current_stream()),
              "th_rev_bwd");
        out[0] = dx;
        for (int i = 0; i < 4; ++i) {
            out[1 + i] = dw[i];
            out[5 + i] = db[i];
        }
        return out;
    }
};

// reversible_mlp(x, w_f1, w_f2, w_g1, w_g2, b_f1, b_f2, b_g1, b_g2, activation)
PyObject *py_reversible_mlp(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    Tensor x, w[4], b[4];
    if (n_args != 10 || !usual_mode() || !take(args[0], x)) TH_NOT_MINE;
    for (int i = 0; i < 4; ++i)
        if (!take(args[1 + i], w[i]) || !take(args[5 + i], b[i])) TH_NOT_MINE;
    RevCall call;
    call.act = activation_code(args[9]);
    if (call.act < 0 || !plain(x) || x.dim() < 1 || !plain(w[0]) || w[0].dim() != 2 || !plain(w[1]) || w[1].dim() != 2) TH_NOT_MINE;
    call.dtype = dtype_code(x.scalar_type());
    if (call.dtype != TH_F16 && call.dtype != TH_BF16) TH_NOT_MINE;
    const int64_t d_model = x.size(-1), half = d_model / 2, hidden = w[1].size(1);
    if (d_model % 32 || d_model < 32 || d_model > 128 || hidden % 16 || hidden < 16 || hidden > 64 || w[0].size(0) < hidden || w[0].size(0) % hidden)
        TH_NOT_MINE;
    const int64_t blocks = w[0].size(0) / hidden;
    const bool bias = b[0].defined();
    for (int i = 0; i < 4; ++i) {
        const int64_t rows = i % 2 ? half : hidden, cols = i % 2 ? hidden : half;
        if (!parameter_like(w[i], x, {blocks * rows, cols}) || b[i].defined() != bias || (bias && !parameter_like(b[i], x, {blocks, rows}))) TH_NOT_MINE;
    }
    Rows xr;
    if (!rows_of(x, d_model, xr) || xr.stride % 2 || reinterpret_cast<uintptr_t>(ptr(x)) % 4) TH_NOT_MINE;
    call.rows = xr.n;
    call.x_stride = xr.stride;
    call.d_model = static_cast<int>(d_model);
    call.hidden = static_cast<int>(hidden);
    call.blocks = static_cast<int>(blocks);
    Tensor out;
    {
        NoGil release;
        const bool grad = torch::autograd::compute_requires_grad(x, w[0], w[1], w[2], w[3], b[0], b[1], b[2], b[3]);
        std::shared_ptr<ReversibleNode> node;
        if (grad) {
            node = make_node<ReversibleNode>(torch::autograd::collect_next_edges(x, w[0], w[1], w[2], w[3], b[0], b[1], b[2], b[3]));
            node->call = call;
            node->has_bias = bias;
            for (int i = 0; i < 4; ++i) {
                node->w[i] = SavedVariable(w[i], false);
                if (bias) node->b[i] = SavedVariable(b[i], false);
            }
        }
        {
            at::AutoDispatchBelowADInplaceOrView below;
            c10::cuda::CUDAGuard guard(x.device());
            out = empty_like_shape(x.sizes(), x.scalar_type(), x.device());
            check(th_rev_fwd(ptr(x), call.x_stride, ptr(w[0]), ptr(w[1]), ptr(w[2]), ptr(w[3]), ptr(b[0]), ptr(b[1]), ptr(b[2]), ptr(b[3]), ptr(out),
                             d_model, call.rows, call.d_model, call.hidden, call.blocks, call.act, call.dtype, current_stream()),
                  "th_rev_fwd");
        }
        if (grad) {
            torch::autograd::set_history(out, node);
            // the OUTPUT is kept, not the input: backward reconstructs every intermediate from it
            node->y = SavedVariable(out, true);
        }
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// ---- hash encoding + MLP in one kernel per direction --------------------------------------------------------

struct FieldNode : public Node {
    EncodeCall call;
    MlpCall mlp;
    SavedVariable coords, table, w_in, w_out, w_hid;
    Tensor feats;

    std::string name() const override { return "HashEncodedMLPBackward"; }
    void release_variables() override {
        for (SavedVariable *v : {&coords, &table, &w_in, &w_out, &w_hid}) v->reset_data();
        feats.reset();
    }
    variable_list apply(variable_list &&grads) override {
        variable_list out(4);
        if (!grads[0].defined()) return out;
        const Tensor x = coords.unpack(), t = table.unpack(), wi = w_in.unpack(), wo = w_out.unpack();
        const Tensor wh = mlp.depth > 1 ? w_hid.unpack() : Tensor();
        at::NoGradGuard no_grad;
        c10::cuda::CUDAGuard guard(t.device());
        Tensor go = grads[0];
        if (go.scalar_type() != t.scalar_type()) go = go.to(t.scalar_type());
        const Rows g = rows_or_copy(go, mlp.d_out);
        Tensor de = empty_like_shape(t.sizes(), t.scalar_type(), t.device());
        de.zero_();
        const Geometry &geo = *call.geo;
        const int feat = static_cast<int>(call.feats), dims = static_cast<int>(call.dims);
        const int64_t bytes = th_field_workspace_bytes(geo.levels, feat, mlp.hidden, mlp.d_out, mlp.depth);
        const Tensor sums = empty_like_shape({bytes / 4}, at::kFloat, t.device());
        const CoordArgs c = coord_args(x, call.dims);
        void *stream = current_stream();
        check(th_field_bwd(ptr(c.keep), c.stride_n, c.stride_d, dtype_code(c.keep.scalar_type()), dims, feat, geo.levels, geo.res, geo.rows, geo.offsets,
                           call.primes.v, call.scale, ptr(wi), ptr(wh), ptr(wo), mlp.hidden, mlp.d_out, mlp.depth, mlp.act, ptr(feats), mlp.d_in,
                           ptr(g.keep), g.stride, ptr(de), nullptr, mlp.d_in, ptr(sums), bytes, call.n, dtype_code(t.scalar_type()), stream),
              "th_field_bwd");
        // float32 sums -> gradients in the parameter dtype: one rounding of the whole block, handed out as slices of it
        const int64_t n_in = wi.numel(), n_hid = wh.defined() ? wh.numel() : 0, n_out = wo.numel();
        const Tensor rounded = empty_like_shape({n_in + n_hid + n_out}, t.scalar_type(), t.device());
        check(th_scale_cast(sums.data_ptr<float>(), ptr(rounded), rounded.numel(), 1.f, mlp.dtype, stream), "th_scale_cast");
        out[0] = std::move(de);
        out[1] = rounded.narrow(0, 0, n_in).view(wi.sizes());
        out[2] = rounded.narrow(0, n_in + n_hid, n_out).view(wo.sizes());
        if (n_hid) out[3] = rounded.narrow(0, n_in, n_hid).view(wh.sizes());
        return out;
    }
};

// hash_encoded_mlp(coord, embeddings, w_in, w_out, w_hid, pi, max_entries_per_level, min_res, max_res, levels, activation, scale)
PyObject *py_hash_encoded_mlp(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (n_args != 12 || !usual_mode() || !THPVariable_Check(args[0]) || !THPVariable_Check(args[1])) TH_NOT_MINE;
    const Tensor coords = THPVariable_Unpack(args[0]), table = THPVariable_Unpack(args[1]);
    MlpTensors p;
    EncodeCall call;
    if (!take(args[2], p.w_in) || !take(args[3], p.w_out) || !take(args[4], p.w_hid) ||
        !encode_call(call, coords, table, args[5], args + 6, args[9], args[11]))
        TH_NOT_MINE;
    MlpCall mlp;
    mlp.act = activation_code(args[10]);
    mlp.dtype = dtype_code(table.scalar_type());
    if (mlp.act < 0 || mlp.dtype == TH_F32 || !plain(p.w_in) || p.w_in.dim() != 2 || !plain(p.w_out) || p.w_out.dim() != 2) TH_NOT_MINE;
    const int64_t hidden = p.w_in.size(0), d_in = p.w_in.size(1), d_out = p.w_out.size(0);
    int64_t depth = 1;
    if (p.w_hid.defined()) {
        if (p.w_hid.dim() != 2 || p.w_hid.numel() == 0 || hidden < 1) TH_NOT_MINE;
        depth += p.w_hid.size(0) / hidden;
        if (!parameter_like(p.w_hid, table, {(depth - 1) * hidden, hidden})) TH_NOT_MINE;
    }
    if (d_in != call.feats * call.geo->levels || !parameter_like(p.w_in, table, {hidden, d_in}) || !parameter_like(p.w_out, table, {d_out, hidden}))
        TH_NOT_MINE;
    mlp.d_in = static_cast<int>(d_in);
    mlp.hidden = static_cast<int>(hidden);
    mlp.d_out = static_cast<int>(d_out);
    mlp.depth = static_cast<int>(depth);
    Tensor out;
    {
        NoGil release;
        const bool grad = torch::autograd::compute_requires_grad(table, p.w_in, p.w_out, p.w_hid);
        std::shared_ptr<FieldNode> node;
        if (grad) {
            node = make_node<FieldNode>(torch::autograd::collect_next_edges(table, p.w_in, p.w_out, p.w_hid));
            node->call = call;
            node->mlp = mlp;
            node->coords = SavedVariable(coords, false);
            node->table = SavedVariable(table, false);
            node->w_in = SavedVariable(p.w_in, false);
            node->w_out = SavedVariable(p.w_out, false);
            if (p.w_hid.defined()) node->w_hid = SavedVariable(p.w_hid, false);
        }
        {
            at::AutoDispatchBelowADInplaceOrView below;
            c10::cuda::CUDAGuard guard(table.device());
            const Geometry &geo = *call.geo;
            const CoordArgs c = coord_args(coords, call.dims);
            Tensor feats = grad ? empty_like_shape({call.n, d_in}, table.scalar_type(), table.device()) : Tensor();
            out = empty_like_shape(with_last(coords, d_out), table.scalar_type(), table.device());
            const int rc = th_field_fwd(ptr(c.keep), c.stride_n, c.stride_d, dtype_code(c.keep.scalar_type()), ptr(table), static_cast<int>(call.dims),
                                        static_cast<int>(call.feats), geo.levels, geo.res, geo.rows, geo.offsets, call.primes.v, call.scale, ptr(p.w_in),
                                        nullptr, ptr(p.w_hid), nullptr, ptr(p.w_out), nullptr, mlp.hidden, mlp.d_out, mlp.depth, mlp.act, ptr(feats), d_in,
                                        ptr(out), d_out, nullptr, d_out, nullptr, d_out, nullptr, 1.f, call.n, mlp.dtype, current_stream());
            if (rc == TH_ERR_UNSUPPORTED) out.reset();  // nothing was launched: Python raises FieldUnsupported
            else check(rc, "th_field_fwd");
            if (grad) node->feats = std::move(feats);
        }
        if (grad && out.defined()) torch::autograd::set_history(out, node);
    }
    if (!out.defined()) TH_NOT_MINE;
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// ---- module -------------------------------------------------------------------------------------------------

// configure(level_geometry, host_primes): the package's Python helpers this module asks for geometry and primes
PyObject *py_configure(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    if (n_args != 2) {
        PyErr_SetString(PyExc_TypeError, "configure(level_geometry, host_primes)");
        return nullptr;
    }
    Py_INCREF(args[0]);
    Py_INCREF(args[1]);
    Py_XSETREF(g_geometry_source, args[0]);
    Py_XSETREF(g_primes_source, args[1]);
    Py_RETURN_NONE;
}

// defer(flag): while set, every function answers NotImplemented
PyObject *py_defer(PyObject *, PyObject *flag) {
    g_deferred.store(PyObject_IsTrue(flag) == 1, std::memory_order_relaxed);
    Py_RETURN_NONE;
}

#define TH_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {
    TH_FAST(hash_encoding), TH_FAST(fully_fused_mlp), TH_FAST(reversible_mlp), TH_FAST(hash_encoded_mlp), TH_FAST(configure),
    {"defer", py_defer, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&g_module); }
