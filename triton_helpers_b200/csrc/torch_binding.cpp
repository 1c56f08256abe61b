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
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <atomic>
#include <cstring>
#include <strings.h>
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
    // a dispatch or function mode, a functorch level or a torch.jit trace (which records the Python functions) shows up in the
    // thread's included keys
    using c10::DispatchKey;
    static const c10::DispatchKeySet modes({DispatchKey::Python, DispatchKey::PythonTLSSnapshot, DispatchKey::FuncTorchDynamicLayerFrontMode,
                                            DispatchKey::FuncTorchDynamicLayerBackMode, DispatchKey::Functionalize, DispatchKey::Tracer});
    return !g_deferred.load(std::memory_order_relaxed) && !at::autocast::is_autocast_enabled(at::kCUDA) &&
           !c10::impl::tls_local_dispatch_key_set().included_.has_any(modes) &&
           // inside a forward-mode level tensors may have tangents: the Python functions raise for lack of a derivative
           !torch::autograd::ForwardADLevel::try_get_by_idx(0);
}

// One optional tensor argument; false when it is neither None nor a tensor (or Parameter) itself: a subclass keeps its type through
// the Python functions.
bool take(PyObject *o, Tensor &t) {
    if (o == Py_None) return true;
    if (!THPVariable_CheckExact(o)) return false;
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

// A tensor that a node kept, checked to be what it was: a saved-tensor hook may hand back another one, with another layout, so
// no stride or pointer is remembered from the forward pass.
const Tensor &same(const Tensor &t, at::ScalarType type, int64_t numel) {
    TORCH_CHECK(t.defined() && t.is_cuda() && t.scalar_type() == type && t.numel() == numel,
                "a saved-tensor hook returned a tensor of another device, type or size than the one it was given");
    return t;
}

Tensor restored(const Tensor &t, at::ScalarType type, int64_t numel) { return same(t, type, numel).is_contiguous() ? t : t.contiguous(); }

// Three-dimensional rows evenly strided over both leading dimensions, unit stride inside a row
bool even_rows(const Tensor &x) {
    return x.stride(2) == 1 && (x.size(0) <= 1 || x.stride(0) == x.size(1) * x.stride(1)) && x.stride(1) >= x.size(2);
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
    int64_t dims = 0, feats = 0, n = 0, table_elems = 0;
    at::ScalarType table_type = at::kFloat;
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

bool order_pays(const EncodeCall &c, const Tensor &table, bool backward) {
    return th_hash_order_pays(c.n, static_cast<int>(c.dims), static_cast<int>(c.feats), c.geo->levels, static_cast<int>(c.feats * table.element_size()),
                              c.geo->total_rows, backward);
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
    SavedVariable coords, table, order;  // order: default-constructed where the batch was not ordered
    bool ordered = false;

    std::string name() const override { return "HashEncodingBackward"; }
    void release_variables() override {
        order.reset_data();
        coords.reset_data();
        table.reset_data();
    }
    variable_list apply(variable_list &&grads) override {
        variable_list out(1);
        if (!grads[0].defined()) return out;
        const Tensor x = coords.unpack(), t = table.unpack();
        Tensor o = ordered ? order.unpack() : Tensor();
        at::NoGradGuard no_grad;
        c10::cuda::CUDAGuard guard(t.device());
        same(x, x.scalar_type(), call.n * call.dims);
        same(t, call.table_type, call.table_elems);
        if (ordered) o = restored(o, at::kFloat, call.n * 4);
        Tensor go = grads[0];
        if (go.scalar_type() != t.scalar_type()) go = go.to(t.scalar_type());
        const Rows rows = rows_or_copy(go, call.feats * call.geo->levels);
        Tensor de = empty_like_shape(t.sizes(), t.scalar_type(), t.device());
        de.zero_();
        hash_backward(call, coord_args(x, call.dims), o, rows, de, current_stream());
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
    c.table_elems = table.numel();
    c.table_type = table.scalar_type();
    c.scale = static_cast<float>(scale);
    if (pi_object != Py_None) {
        if (!THPVariable_CheckExact(pi_object)) return false;
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
    if (n_args != 11 || !usual_mode() || !THPVariable_CheckExact(args[0]) || !THPVariable_CheckExact(args[1]) || args[2] != Py_None ||
        args[8] != Py_None || args[9] != Py_None)
        TH_NOT_MINE;
    const Tensor coords = THPVariable_Unpack(args[0]), table = THPVariable_Unpack(args[1]);
    EncodeCall call;
    if (!encode_call(call, coords, table, args[3], args + 4, args[7], args[10])) TH_NOT_MINE;
    Tensor out, order;
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
            if (order_pays(call, table, grad)) order = point_order(call, x, stream);
            hash_forward(call, x, order, table, out, stream);
        }
        if (grad) {
            node->ordered = order.defined();
            if (node->ordered) node->order = SavedVariable(order, false);
            torch::autograd::set_history(out, node);
        }
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
        const int64_t h = call.hidden, deep = call.depth - 1;
        Tensor xs = x.unpack();
        MlpTensors k;
        k.w_in = w_in.unpack();
        k.w_out = w_out.unpack();
        if (hidden) k.w_hid = w_hid.unpack();
        if (has_bias) {
            k.b_in = b_in.unpack();
            k.b_out = b_out.unpack();
            if (hidden) k.b_hid = b_hid.unpack();
        }
        at::NoGradGuard no_grad;
        const at::ScalarType type = call.dtype == TH_F16 ? at::kHalf : at::kBFloat16;
        same(xs, type, call.rows() * call.d_in);
        if (xs.dim() != 3 || xs.size(2) != call.d_in || !even_rows(xs)) xs = xs.contiguous().view({call.batch, call.length, call.d_in});
        MlpTensors p;
        p.w_in = restored(k.w_in, type, h * call.d_in);
        p.w_out = restored(k.w_out, type, call.d_out * h);
        if (hidden) p.w_hid = restored(k.w_hid, type, deep * h * h);
        if (has_bias) {
            p.b_in = restored(k.b_in, type, h);
            p.b_out = restored(k.b_out, type, call.d_out);
            if (hidden) p.b_hid = restored(k.b_hid, type, deep * h);
        }
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
        check(th_mlp_bwd(ptr(xs), xs.stride(1), ptr(p.w_in), ptr(p.b_in), ptr(p.w_hid), ptr(p.b_hid), ptr(p.w_out), ptr(p.b_out), ptr(g.keep), g.stride,
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

// float32 networks: every tensor is rounded to a 16-bit operand type, all of them in one launch and into one buffer; the
// results are cast back.  The backward pass keeps that buffer (as a saved tensor), not the float32 tensors, and hands out the
// float32 sums of the weight gradients as they are.
struct Float32Pack {
    Tensor buffer;          // 16-bit operands: x, w_in, b_in, w_out, b_out, w_hid, b_hid (where present)
    int64_t offset[7] = {-1, -1, -1, -1, -1, -1, -1};  // in elements; -1: absent

    void *part(int k, const Tensor &in) const { return offset[k] < 0 ? nullptr : static_cast<char *>(ptr(in)) + 2 * offset[k]; }
    void *part(int k) const { return part(k, buffer); }

    static at::ScalarType operands() {
        static const at::ScalarType type = [] {
            const char *v = getenv("TH_MLP_F32_OPERANDS");
            if (!v || !strcasecmp(v, "fp16") || !strcasecmp(v, "float16")) return at::kHalf;
            if (!strcasecmp(v, "bf16") || !strcasecmp(v, "bfloat16")) return at::kBFloat16;
            return at::kFloat;  // not a valid choice: Python says so
        }();
        return type;
    }

    void fill(const std::vector<Tensor> &tensors, void *stream) {
        int64_t total = 0, sizes[8];
        const void *src[8];
        void *dst[8];
        int n = 0;
        for (const Tensor &t : tensors) total += t.defined() ? (t.numel() + 15) / 16 * 16 : 0;
        buffer = empty_like_shape({total}, operands(), tensors[0].device());
        int64_t at = 0;
        for (size_t k = 0; k < tensors.size(); ++k) {
            if (!tensors[k].defined()) continue;
            offset[k] = at;
            dst[n] = part(static_cast<int>(k));
            src[n] = ptr(tensors[k]);
            sizes[n++] = tensors[k].numel();
            at += (tensors[k].numel() + 15) / 16 * 16;
        }
        check(th_cast(n, src, dst, sizes, TH_F32, dtype_code(operands()), stream), "th_cast");
    }
};

void cast_one(const Tensor &from, const Tensor &to, void *stream) {
    const void *src = ptr(from);
    void *dst = ptr(to);
    const int64_t n = from.numel();
    check(th_cast(1, &src, &dst, &n, dtype_code(from.scalar_type()), dtype_code(to.scalar_type()), stream), "th_cast");
}

struct Float32MlpNode : public Node {
    MlpCall call;
    Float32Pack pack;      // offsets; its buffer is in `saved`
    SavedVariable saved;
    int64_t saved_elems = 0;
    std::vector<int64_t> shapes[6];  // of w_in, b_in, w_out, b_out, w_hid, b_hid
    bool has_bias = false;

    std::string name() const override { return "FullyFusedMLPBackward"; }
    void release_variables() override { saved.reset_data(); }
    variable_list apply(variable_list &&grads) override {
        variable_list out(7);
        if (!grads[0].defined()) return out;
        Tensor buffer = saved.unpack();
        at::NoGradGuard no_grad;
        buffer = restored(buffer, Float32Pack::operands(), saved_elems);
        const c10::Device device = buffer.device();
        const at::ScalarType half = buffer.scalar_type();
        c10::cuda::CUDAGuard guard(device);
        auto part = [&](int k) { return pack.part(k, buffer); };
        void *stream = current_stream();
        const Tensor given = grads[0].contiguous();
        Tensor go = given;
        if (given.scalar_type() == at::kFloat) {
            go = empty_like_shape(given.sizes(), half, device);
            cast_one(given, go, stream);
        } else if (given.scalar_type() != half) {
            go = given.to(half);
        }
        const bool wants_dx = task_should_compute_output(0);
        const Tensor dx = wants_dx ? empty_like_shape({call.batch, call.length, call.d_in}, half, device) : Tensor();
        const int64_t bytes = th_mlp_workspace_bytes(call.d_in, call.hidden, call.d_out, call.depth);
        const Tensor sums = empty_like_shape({bytes / 4}, at::kFloat, device);
        check(th_mlp_bwd(part(0), call.d_in, part(1), part(2), part(5), part(6), part(3), part(4), ptr(go), call.d_out,
                         ptr(dx), call.d_in, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, ptr(sums), bytes, call.rows(), call.d_in, call.hidden,
                         call.d_out, call.depth, call.act, dtype_code(half), 0, stream),
              "th_mlp_bwd");
        if (wants_dx) {
            out[0] = empty_like_shape(dx.sizes(), at::kFloat, device);
            cast_one(dx, out[0], stream);
        }
        const int64_t h = call.hidden, n_in = h * call.d_in, n_hid = (call.depth - 1) * h * h, n_out = h * call.d_out;
        int64_t at = 0;
        auto slice = [&](int k, int64_t n) {  // the sums' layout: w_in, w_hid, w_out, b_in, b_hid, b_out
            out[1 + k] = sums.narrow(0, at, n).view(shapes[k]);
            at += n;
        };
        slice(0, n_in);
        if (n_hid) slice(4, n_hid);
        slice(2, n_out);
        if (has_bias) {
            slice(1, h);
            if (n_hid) slice(5, (call.depth - 1) * h);
            slice(3, call.d_out);
        }
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
    if (c.dtype < 0 || (c.dtype == TH_F32 && Float32Pack::operands() == at::kFloat)) return false;
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
    if (!even_rows(x)) return false;
    c.x_stride = x.stride(1);
    c.d_in = static_cast<int>(d_in);
    c.hidden = static_cast<int>(hidden);
    c.d_out = static_cast<int>(d_out);
    c.depth = static_cast<int>(depth);
    return true;
}

Tensor mlp_float32(const MlpCall &call, const Tensor &x, const MlpTensors &p, bool grad) {
    NoGil release;
    Tensor out;
    Float32Pack pack;
    std::shared_ptr<Float32MlpNode> node;
    if (grad) {
        node = make_node<Float32MlpNode>(torch::autograd::collect_next_edges(x, p.w_in, p.b_in, p.w_out, p.b_out, p.w_hid, p.b_hid));
        node->call = call;
        node->has_bias = p.b_in.defined();
        const Tensor *params[6] = {&p.w_in, &p.b_in, &p.w_out, &p.b_out, &p.w_hid, &p.b_hid};
        for (int k = 0; k < 6; ++k)
            if (params[k]->defined()) node->shapes[k] = params[k]->sizes().vec();
    }
    {
        at::AutoDispatchBelowADInplaceOrView below;
        c10::cuda::CUDAGuard guard(x.device());
        void *stream = current_stream();
        pack.fill({x.contiguous(), p.w_in, p.b_in, p.w_out, p.b_out, p.w_hid, p.b_hid}, stream);
        const Tensor half = empty_like_shape({call.batch, call.length, call.d_out}, pack.buffer.scalar_type(), x.device());
        check(th_mlp_fwd(pack.part(0), call.d_in, pack.part(1), pack.part(2), pack.part(5), pack.part(6), pack.part(3), pack.part(4), ptr(half), call.d_out,
                         call.rows(), call.d_in, call.hidden, call.d_out, call.depth, call.act, dtype_code(half.scalar_type()), 0, stream),
              "th_mlp_fwd");
        out = empty_like_shape(half.sizes(), at::kFloat, x.device());
        cast_one(half, out, stream);
    }
    if (grad) {
        node->saved_elems = pack.buffer.numel();
        node->saved = SavedVariable(std::move(pack.buffer), false);
        node->pack = pack;
        torch::autograd::set_history(out, node);
    }
    return out;
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
    const bool grad = torch::autograd::compute_requires_grad(x, p.w_in, p.b_in, p.w_out, p.b_out, p.w_hid, p.b_hid);
    if (call.dtype == TH_F32 && grad && call.depth >= 4) TH_NOT_MINE;  // its backward pass is refused, by the Python path
    if (call.dtype == TH_F32) return THPVariable_Wrap(mlp_float32(call, x, p, grad));
    Tensor out;
    {
        NoGil release;
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
        Tensor ys = y.unpack(shared_from_this());
        Tensor ws[4], bs[4], dw[4], db[4];
        for (int i = 0; i < 4; ++i) {
            ws[i] = w[i].unpack();
            if (has_bias) bs[i] = b[i].unpack();
        }
        at::NoGradGuard no_grad;
        const at::ScalarType type = call.dtype == TH_F16 ? at::kHalf : at::kBFloat16;
        ys = restored(ys, type, call.rows * call.d_model);
        for (int i = 0; i < 4; ++i) {
            ws[i] = restored(ws[i], type, static_cast<int64_t>(call.blocks) * call.hidden * (call.d_model / 2));
            if (has_bias) bs[i] = restored(bs[i], type, static_cast<int64_t>(call.blocks) * (i % 2 ? call.d_model / 2 : call.hidden));
        }
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

// ---- hash encoding + MLP --------------------------------------------------------------------------------------
//
// Up to six layers before the output (what the MLP backward holds at any width) the encoding's kernels and the MLP's run one after
// the other: each of them fills an SM by itself (the gathers and reductions want all its warps, the MLP its shared memory),
// large batches can be ordered in space, and together they are faster than the kernels that fuse the two (B200, 200 003 points in
// two dimensions, forward + backward, 192 -> 150 us; 2^21 points in three, forward 0.72 -> 0.47 ms).  Deeper networks take the fused
// kernels: without a gradient from here, with one from Python, whose FieldUnsupported says when the backward does not hold them.

// Unordered batches large enough to hide the host path, with 64 features and next to no network: the separate kernels write and read
// the features' gradient, 128 bytes a point, for a backward pass that takes no longer fused.  Forward + backward, separate over
// fused: 64 features, two dimensions, 2^19 .. 2^21 points, one layer 0.95-1.09, two layers of 16 1.02-1.08 (of 32 0.95-1.03,
// of 64 0.97-1.00), 2^18 0.85-0.97; three dimensions 2^18 0.96-1.05, 2^17 0.68-0.84; 32 features 0.72-1.03.
bool fused_pays(const EncodeCall &c, const MlpCall &m, bool ordered) {
    return !ordered && m.d_in == 64 && (m.depth == 1 || (m.depth == 2 && m.hidden == 16)) && c.n >= (c.dims == 2 ? 1 << 19 : 1 << 18);
}

// Forward alone, three dimensions, 16 levels, 64 -> 16 -> 16, time over the fused kernels' (tables of 2^14 .. 2^21 rows per level): from
// 2^20 points the order is worth it next to an MLP for 4-byte rows too (uniform points 0.68-0.88, clustered 0.91-1.03; without it
// 0.90-0.96 and 0.89-1.10).  Unordered batches of 2^19 points with 64 features stay fused (separate: 0.79-1.04 and 1.02-1.14).
bool field_ordered(const EncodeCall &c, const Tensor &table, bool grad) {
    return order_pays(c, table, grad) || (!grad && c.geo->levels >= 16 && c.n >= 1 << 20 && order_pays(c, table, true));
}

struct FieldNode : public Node {
    EncodeCall call;
    MlpCall mlp;
    SavedVariable coords, table, w_in, w_out, w_hid, feats, order;  // order: default-constructed where the batch was not ordered
    bool ordered = false;

    std::string name() const override { return "HashEncodedMLPBackward"; }
    void release_variables() override {
        for (SavedVariable *v : {&coords, &table, &w_in, &w_out, &w_hid, &feats, &order}) v->reset_data();
    }
    variable_list apply(variable_list &&grads) override {
        variable_list out(4);
        if (!grads[0].defined()) return out;
        const Tensor x = coords.unpack(), t = table.unpack();
        Tensor wi = w_in.unpack(), wo = w_out.unpack(), wh = mlp.depth > 1 ? w_hid.unpack() : Tensor();
        Tensor rows_in = feats.unpack(), o = ordered ? order.unpack() : Tensor();
        at::NoGradGuard no_grad;
        c10::cuda::CUDAGuard guard(t.device());
        same(x, x.scalar_type(), call.n * call.dims);
        same(t, call.table_type, call.table_elems);
        const int64_t width = mlp.hidden;
        wi = restored(wi, call.table_type, width * mlp.d_in);
        wo = restored(wo, call.table_type, mlp.d_out * width);
        if (mlp.depth > 1) wh = restored(wh, call.table_type, (mlp.depth - 1) * width * width);
        rows_in = restored(rows_in, call.table_type, call.n * mlp.d_in);
        if (ordered) o = restored(o, at::kFloat, call.n * 4);
        Tensor go = grads[0];
        if (go.scalar_type() != t.scalar_type()) go = go.to(t.scalar_type());
        const Rows g = rows_or_copy(go, mlp.d_out);
        Tensor de = empty_like_shape(t.sizes(), t.scalar_type(), t.device());
        de.zero_();
        const int64_t bytes = th_mlp_workspace_bytes(mlp.d_in, mlp.hidden, mlp.d_out, mlp.depth);
        const Tensor sums = empty_like_shape({bytes}, at::kByte, t.device()), grad_feats = empty_same(rows_in);
        out[1] = empty_same(wi);
        out[2] = empty_same(wo);
        if (wh.defined()) out[3] = empty_same(wh);
        void *stream = current_stream();
        check(th_mlp_bwd(ptr(rows_in), mlp.d_in, ptr(wi), nullptr, ptr(wh), nullptr, ptr(wo), nullptr, ptr(g.keep), g.stride, ptr(grad_feats), mlp.d_in,
                         ptr(out[1]), nullptr, ptr(out[3]), nullptr, ptr(out[2]), nullptr, ptr(sums), bytes, call.n, mlp.d_in, mlp.hidden, mlp.d_out,
                         mlp.depth, mlp.act, mlp.dtype, 0, stream),
              "th_mlp_bwd");
        Rows rows;
        rows_of(grad_feats, mlp.d_in, rows);
        hash_backward(call, coord_args(x, call.dims), o, rows, de, stream);
        out[0] = std::move(de);
        return out;
    }
};

// hash_encoded_mlp(coord, embeddings, w_in, w_out, w_hid, pi, max_entries_per_level, min_res, max_res, levels, activation, scale)
PyObject *py_hash_encoded_mlp(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (n_args != 12 || !usual_mode() || !THPVariable_CheckExact(args[0]) || !THPVariable_CheckExact(args[1])) TH_NOT_MINE;
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
    // what the fused kernels cover: anything else is Python's FieldUnsupported
    static const bool legacy = getenv("TH_MLP_LEGACY") && getenv("TH_MLP_LEGACY")[0] == '1';
    bool separate = !legacy && depth <= 6 && (call.dims == 2 || call.dims == 3) && (call.feats == 2 || call.feats == 4) &&
                          d_in % 16 == 0 && d_in <= 64 && (mlp.act == TH_ACT_RELU || mlp.act == TH_ACT_NONE) &&
                          (hidden == 16 || hidden == 32 || hidden == 64) && d_out >= 1 && d_out <= 64;
    const bool grad = torch::autograd::compute_requires_grad(table, p.w_in, p.w_out, p.w_hid);
    const bool ordered = separate && field_ordered(call, table, grad);
    if (grad && (!separate || fused_pays(call, mlp, ordered))) TH_NOT_MINE;
    if (!grad && separate && !ordered && d_in == 64 && call.dims == 3 && call.n >= 1 << 19) separate = false;
    Tensor out, feats, order;
    {
        NoGil release;
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
            if (separate) feats = empty_like_shape({call.n, d_in}, table.scalar_type(), table.device());
            out = empty_like_shape(with_last(coords, d_out), table.scalar_type(), table.device());
            int rc = 0;
            if (separate) {
                void *stream = current_stream();
                if (ordered) order = point_order(call, c, stream);
                hash_forward(call, c, order, table, feats, stream);
                check(th_mlp_fwd(ptr(feats), d_in, ptr(p.w_in), nullptr, ptr(p.w_hid), nullptr, ptr(p.w_out), nullptr, ptr(out), d_out, call.n, mlp.d_in,
                                 mlp.hidden, mlp.d_out, mlp.depth, mlp.act, mlp.dtype, 0, stream),
                      "th_mlp_fwd");
            } else {
                rc = th_field_fwd(ptr(c.keep), c.stride_n, c.stride_d, dtype_code(c.keep.scalar_type()), ptr(table), static_cast<int>(call.dims),
                                        static_cast<int>(call.feats), geo.levels, geo.res, geo.rows, geo.offsets, call.primes.v, call.scale, ptr(p.w_in),
                                        nullptr, ptr(p.w_hid), nullptr, ptr(p.w_out), nullptr, mlp.hidden, mlp.d_out, mlp.depth, mlp.act, ptr(feats), d_in,
                                        ptr(out), d_out, nullptr, d_out, nullptr, d_out, nullptr, 1.f, call.n, mlp.dtype, current_stream());
            }
            if (rc == TH_ERR_UNSUPPORTED) out.reset();  // nothing was launched: Python raises FieldUnsupported
            else check(rc, "th_field_fwd");
        }
        if (grad && out.defined()) {
            node->feats = SavedVariable(std::move(feats), false);
            node->ordered = order.defined();
            if (node->ordered) node->order = SavedVariable(std::move(order), false);
            torch::autograd::set_history(out, node);
        }
    }
    if (!out.defined()) TH_NOT_MINE;
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// ---- training step ------------------------------------------------------------------------------------------------

bool take_list(PyObject *o, std::vector<Tensor> &out) {
    if (!PyTuple_Check(o) && !PyList_Check(o)) return false;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(o);
    out.resize(n);
    for (Py_ssize_t k = 0; k < n; ++k)
        if (!take(PySequence_Fast_GET_ITEM(o, k), out[k])) return false;
    return true;
}

// adam_steps(params, grads, exp_avgs, exp_avg_sqs, grad_scales, zero_grad, lr, beta1, beta2, eps, step, skipped): sequences of
// one length (tensors of one dtype on one device); the update of all of them in one launch (16 tensors each)
PyObject *py_adam_steps(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    std::vector<Tensor> params, grads, m, v;
    double lr, beta1, beta2, eps;
    int64_t step;
    Tensor skipped;
    if (n_args != 12 || g_deferred.load(std::memory_order_relaxed) || !take_list(args[0], params) || !take_list(args[1], grads) || !take_list(args[2], m) ||
        !take_list(args[3], v) || !take(args[6], lr) || !take(args[7], beta1) || !take(args[8], beta2) || !take(args[9], eps) || !take(args[10], step) ||
        !take(args[11], skipped))
        TH_NOT_MINE;
    const size_t n = params.size();
    if (n == 0 || grads.size() != n || m.size() != n || v.size() != n || !PyTuple_Check(args[4]) || !PyTuple_Check(args[5]) ||
        PyTuple_GET_SIZE(args[4]) != static_cast<Py_ssize_t>(n) || PyTuple_GET_SIZE(args[5]) != static_cast<Py_ssize_t>(n))
        TH_NOT_MINE;
    const at::ScalarType type = params[0].scalar_type();
    std::vector<float> scales(n);
    std::vector<int> zero(n);
    auto aligned = [](const Tensor &t) { return reinterpret_cast<uintptr_t>(ptr(t)) % 32 == 0; };
    if (skipped.defined() && (!plain(skipped) || skipped.scalar_type() != at::kInt)) TH_NOT_MINE;
    for (size_t k = 0; k < n; ++k) {
        double scale;
        if (!take(PyTuple_GET_ITEM(args[4], k), scale)) TH_NOT_MINE;
        scales[k] = static_cast<float>(scale);
        zero[k] = PyObject_IsTrue(PyTuple_GET_ITEM(args[5], k)) == 1;
        for (const Tensor *t : {&params[k], &grads[k], &m[k], &v[k]})
            if (!plain(*t) || !t->is_contiguous() || t->device() != params[0].device() || t->numel() != params[k].numel() || !aligned(*t)) TH_NOT_MINE;
        if (params[k].scalar_type() != type || grads[k].scalar_type() != type || m[k].scalar_type() != at::kFloat || v[k].scalar_type() != at::kFloat)
            TH_NOT_MINE;
    }
    if (dtype_code(type) < 0) TH_NOT_MINE;
    {
        NoGil release;
        c10::cuda::CUDAGuard guard(params[0].device());
        void *stream = current_stream();
        for (size_t from = 0; from < n; from += 16) {
            const int count = static_cast<int>(n - from < 16 ? n - from : 16);
            void *pp[16], *gp[16];
            float *mp[16], *vp[16];
            int64_t sizes[16];
            for (int k = 0; k < count; ++k) {
                pp[k] = ptr(params[from + k]);
                gp[k] = ptr(grads[from + k]);
                mp[k] = m[from + k].data_ptr<float>();
                vp[k] = v[from + k].data_ptr<float>();
                sizes[k] = params[from + k].numel();
            }
            check(th_adam_steps(count, pp, gp, mp, vp, sizes, scales.data() + from, zero.data() + from, static_cast<float>(lr), static_cast<float>(beta1),
                                static_cast<float>(beta2), static_cast<float>(eps), static_cast<int>(step), dtype_code(type),
                                skipped.defined() ? skipped.data_ptr<int>() : nullptr, stream),
                  "th_adam_steps");
        }
    }
    // in-place updates that autograd has to know of
    for (const Tensor &t : params) t.unsafeGetTensorImpl()->bump_version();
    Py_RETURN_TRUE;
    END_HANDLE_TH_ERRORS
}

// train_gradients(coords, targets, table, table_grad, (w_in, b_in, w_hid, b_hid, w_out, b_out), sums, feats, grad_pred, grad_feats,
//                 mlp_grad, pi, max_entries_per_level, min_res, max_res, levels, activation, grad_scale, cast_scale)
//
// Forward, squared-error loss and backward of the encoding followed by the MLP, on the caller's buffers: table_grad (adds into it),
// sums (float32 sums of the MLP's gradients, laid out as th_mlp_bwd's workspace), feats / grad_pred / grad_feats (16-bit rows, scratch).
// 16-bit tables: sums * cast_scale are rounded into mlp_grad.  float32 tables: the MLP runs on 16-bit copies of its parameters,
// mlp_grad is None.  Large batches are ordered in space first; nothing in them is kept in the caller's row order.
// Returns the mean squared error (one float32 element); NotImplemented before anything has been launched that changes table_grad.
PyObject *py_train_gradients(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (n_args != 18 || !usual_mode()) TH_NOT_MINE;
    Tensor coords, targets, table, table_grad, sums, feats, grad_pred, grad_feats, mlp_grad;
    std::vector<Tensor> w;
    double grad_scale, cast_scale;
    if (!take(args[0], coords) || !take(args[1], targets) || !take(args[2], table) || !take(args[3], table_grad) || !take_list(args[4], w) || w.size() != 6 ||
        !take(args[5], sums) || !take(args[6], feats) || !take(args[7], grad_pred) || !take(args[8], grad_feats) || !take(args[9], mlp_grad) ||
        !take(args[16], grad_scale) || !take(args[17], cast_scale))
        TH_NOT_MINE;
    EncodeCall call;
    static PyObject *one = PyFloat_FromDouble(1.0);
    if (coords.dim() != 2 || !encode_call(call, coords, table, args[10], args + 11, args[14], one)) TH_NOT_MINE;
    const int act = activation_code(args[15]);
    const at::ScalarType type = table.scalar_type();
    const bool f32 = type == at::kFloat;
    if (act < 0 || !plain(w[0]) || w[0].dim() != 2 || !plain(w[4]) || w[4].dim() != 2) TH_NOT_MINE;
    const int64_t hidden = w[0].size(0), d_in = w[0].size(1), d_out = w[4].size(0), n = call.n;
    const bool bias = w[1].defined();
    int64_t depth = 1;
    if (w[2].defined()) {
        if (w[2].dim() != 2 || hidden < 1 || w[2].numel() == 0) TH_NOT_MINE;
        depth += w[2].size(0) / hidden;
        if (!parameter_like(w[2], table, {(depth - 1) * hidden, hidden})) TH_NOT_MINE;
    }
    if ((hidden != 16 && hidden != 32 && hidden != 64) || d_in > 64 || d_out > 64 || d_out % 8 || d_in != call.feats * call.geo->levels || n < 1) TH_NOT_MINE;
    if (!parameter_like(w[0], table, {hidden, d_in}) || !parameter_like(w[4], table, {d_out, hidden}) || w[5].defined() != bias ||
        w[3].defined() != (bias && depth > 1))
        TH_NOT_MINE;
    if (bias && (!parameter_like(w[1], table, {hidden}) || !parameter_like(w[5], table, {d_out}) ||
                 (depth > 1 && !parameter_like(w[3], table, {depth - 1, hidden}))))
        TH_NOT_MINE;
    const at::ScalarType half = f32 ? Float32Pack::operands() : type;
    if (half == at::kFloat) TH_NOT_MINE;
    const int64_t bytes = th_mlp_workspace_bytes(static_cast<int>(d_in), static_cast<int>(hidden), static_cast<int>(d_out), static_cast<int>(depth));
    auto buffer = [&](const Tensor &t, at::ScalarType st, int64_t numel) {
        return plain(t) && t.is_contiguous() && t.scalar_type() == st && t.numel() == numel && t.device() == table.device();
    };
    if (!buffer(table_grad, type, table.numel()) || !buffer(sums, at::kFloat, bytes / 4) || !buffer(feats, half, n * d_in) ||
        !buffer(grad_pred, half, n * d_out) || !buffer(grad_feats, half, n * d_in) || (!f32 && !buffer(mlp_grad, type, bytes / 4)))
        TH_NOT_MINE;
    if (!plain(targets) || targets.device() != table.device() || targets.dim() != 2 || targets.size(0) != n || targets.size(1) != d_out ||
        dtype_code(targets.scalar_type()) < 0 || targets.requires_grad())
        TH_NOT_MINE;
    const bool ordered = order_pays(call, table, true);
    if (f32 && (ordered || depth >= 4 || call.dims < 2 || (call.feats != 2 && call.feats != 4))) TH_NOT_MINE;
    Tensor loss;
    {
        NoGil release;
        at::NoGradGuard no_grad;
        c10::cuda::CUDAGuard guard(table.device());
        void *stream = current_stream();
        const Geometry &g = *call.geo;
        const int D = static_cast<int>(call.dims), F = static_cast<int>(call.feats), L = g.levels;
        const int code = dtype_code(half);
        const int ih = static_cast<int>(hidden), ii = static_cast<int>(d_in), io = static_cast<int>(d_out), id = static_cast<int>(depth);
        Tensor t = targets;
        if (!f32 && t.scalar_type() != type) t = t.to(type);
        if (f32 && t.scalar_type() != at::kFloat) t = t.to(at::kFloat);
        if (t.stride(1) != 1 || t.stride(0) < d_out || t.stride(0) % 8 || reinterpret_cast<uintptr_t>(ptr(t)) % 16) t = t.clone(at::MemoryFormat::Contiguous);
        loss = at::zeros({1}, sums.options());
        const CoordArgs x = coord_args(coords, call.dims);
        const int xcode = dtype_code(x.keep.scalar_type());
        Tensor order;
        const void *p[6];
        for (int k = 0; k < 6; ++k) p[k] = ptr(w[k]);
        Float32Pack pack;
        if (f32) {
            pack.fill(w, stream);
            for (int k = 0; k < 6; ++k) p[k] = pack.part(k);
            check(th_hash_fwd_cast(ptr(x.keep), x.stride_n, x.stride_d, xcode, table.data_ptr<float>(), ptr(feats), code, d_in, n, D, F, L, g.res, g.rows,
                                   g.offsets, call.primes.v, 1.f, stream),
                  "th_hash_fwd_cast");
        } else if (ordered) {
            order = point_order(call, x, stream);
            check(th_hash_fwd_ordered(ptr(order), 1, ptr(table), code, ptr(feats), d_in, n, D, F, L, g.res, g.rows, g.offsets, call.primes.v, 0, L, stream),
                  "th_hash_fwd_ordered");
        } else {
            check(th_hash_fwd(ptr(x.keep), x.stride_n, x.stride_d, xcode, ptr(table), code, ptr(feats), d_in, n, D, F, L, g.res, g.rows, g.offsets,
                              call.primes.v, 1.f, 0, L, stream),
                  "th_hash_fwd");
        }
        const int rc = th_mlp_fwd_mse_ordered(ptr(feats), d_in, p[0], p[1], p[2], p[3], p[4], p[5], ptr(t), t.stride(0), dtype_code(t.scalar_type()),
                                              ptr(order), ptr(grad_pred), d_out, loss.data_ptr<float>(), static_cast<float>(1.0 / (static_cast<double>(n) * d_out)),
                                              static_cast<float>(grad_scale), n, ii, ih, io, id, act, code, stream);
        if (rc == TH_ERR_UNSUPPORTED) {
            loss.reset();  // the caller takes another way; only feats was written
        } else {
            check(rc, "th_mlp_fwd_mse_ordered");
            check(th_mlp_bwd(ptr(feats), d_in, p[0], p[1], p[2], p[3], p[4], p[5], ptr(grad_pred), d_out, ptr(grad_feats), d_in, nullptr, nullptr, nullptr,
                             nullptr, nullptr, nullptr, ptr(sums), bytes, n, ii, ih, io, id, act, code, 0, stream),
                  "th_mlp_bwd");
            if (f32) {
                check(th_hash_bwd_cast(ptr(x.keep), x.stride_n, x.stride_d, xcode, ptr(grad_feats), code, d_in, table_grad.data_ptr<float>(), n, D, F, L, g.res,
                                       g.rows, g.offsets, call.primes.v, 1.f, stream),
                      "th_hash_bwd_cast");
            } else {
                check(th_scale_cast(sums.data_ptr<float>(), ptr(mlp_grad), mlp_grad.numel(), static_cast<float>(cast_scale), code, stream), "th_scale_cast");
                if (order.defined()) {
                    check(th_hash_bwd_ordered(ptr(order), 1, ptr(grad_feats), d_in, ptr(table_grad), code, n, D, F, L, g.res, g.rows, g.offsets, call.primes.v,
                                              0, L, stream),
                          "th_hash_bwd_ordered");
                } else {
                    check(th_hash_bwd(ptr(x.keep), x.stride_n, x.stride_d, xcode, ptr(grad_feats), d_in, ptr(table_grad), code, n, D, F, L, g.res, g.rows,
                                      g.offsets, call.primes.v, 1.f, 0, L, stream),
                          "th_hash_bwd");
                }
            }
        }
    }
    if (!loss.defined()) TH_NOT_MINE;
    return THPVariable_Wrap(std::move(loss));
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
    TH_FAST(hash_encoding), TH_FAST(fully_fused_mlp), TH_FAST(reversible_mlp), TH_FAST(hash_encoded_mlp), TH_FAST(adam_steps),
    TH_FAST(train_gradients), TH_FAST(configure),
    {"defer", py_defer, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&g_module); }
