// Host path of EPTQLinear calls: tensor checks, scratch lookup, output allocation and the C-ABI call in one
// native function per call.
//
// What bounds a small layer's call is this path, not the kernel: written in Python over ctypes it took 23 us per
// call (module attribute lookups of five buffers, two scratch-size calls, descriptor structures rebuilt for every
// grouped call) beside kernels of 3 to 10 us.  A LayerHandle keeps the EptqLayer descriptor of a module's device
// buffers; a call checks that the module still holds the same buffers, unchanged where the descriptor holds a value
// computed from them, and then only touches the ATen allocator and the library.
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/object_ptr.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <cstring>
#include <map>
#include <utility>
#include <vector>

#include "../../../include/eptq_b200.h"

namespace {

constexpr const char* kCapsule = "eptq_b200.LayerHandle";
// Every buffer the descriptor points into.  It also holds the maxima of h and S_group, so those may not change in place.
constexpr const char* kBufferNames[] = {"Q", "g", "h", "O_vals", "O_col", "O_row_ptr", "bias", "S_group", "crit_ptr", "crit_pos", "crit_O"};
constexpr int kBuffers = sizeof(kBufferNames) / sizeof(kBufferNames[0]);
constexpr int kOptionalFrom = 6;                                     // bias and what follows may be None
constexpr bool kHoldsValue[kBuffers] = {false, false, true, false, false, false, false, true, false, false, false};
constexpr int kTables = 2;                                           // the fp16 and the fp32 codebook
constexpr size_t kMinScratch = 1u << 20;
constexpr int kSmallRows = 16;

// A tensor as it was when the descriptor was made, or None.
struct Held {
    PyObject* obj = nullptr;            // owned
    const void* ptr = nullptr;
    int64_t numel = 0;
    int64_t version = 0;
};

struct LayerHandle {
    EptqLayer d;
    PyObject* keep;                     // tensors (and host tables) the descriptor points into
    PyObject* buffers;                  // the module's _buffers dict
    Held held[kBuffers];
    Held tables[kTables];
    int64_t in_features, out_features;
    size_t scratch[kSmallRows + 1];     // eptq_layer_workspace_bytes for small batches, 0 = not asked yet
};

void free_handle(PyObject* capsule) {
    auto* h = static_cast<LayerHandle*>(PyCapsule_GetPointer(capsule, kCapsule));
    if (h == nullptr) { PyErr_Clear(); return; }
    Py_XDECREF(h->keep);
    Py_XDECREF(h->buffers);
    for (const Held& t : h->held) Py_XDECREF(t.obj);
    for (const Held& t : h->tables) Py_XDECREF(t.obj);
    delete h;
}

LayerHandle* handle_of(PyObject* o) { return static_cast<LayerHandle*>(PyCapsule_GetPointer(o, kCapsule)); }

int64_t version_of(const at::Tensor& t) { return t.is_inference() ? 0 : static_cast<int64_t>(t._version()); }

void hold(Held& h, PyObject* o) {
    h.obj = Py_NewRef(o);
    if (o == Py_None) return;
    const at::Tensor& t = THPVariable_Unpack(o);
    h.ptr = t.const_data_ptr();
    h.numel = t.numel();
    h.version = version_of(t);
}

bool unchanged(const Held& h, bool value) {
    if (h.obj == Py_None) return true;
    const at::Tensor& t = THPVariable_Unpack(h.obj);
    return t.const_data_ptr() == h.ptr && t.numel() == h.numel && (!value || version_of(t) == h.version);
}

PyObject* const* buffer_keys() {
    static PyObject** keys = [] {
        auto** k = new PyObject*[kBuffers];
        for (int i = 0; i < kBuffers; ++i) k[i] = PyUnicode_InternFromString(kBufferNames[i]);
        return k;
    }();
    return keys;
}

// The descriptor still describes the module: the same buffers (replacing or moving one makes a new tensor or a new
// address), and unchanged values where it holds one: max|h|, max|S_group|, the codebooks' lattice scale and packed form.
bool is_current(const LayerHandle* h) {
    PyObject* const* keys = buffer_keys();
    for (int i = 0; i < kBuffers; ++i)
        if (PyDict_GetItem(h->buffers, keys[i]) != h->held[i].obj || !unchanged(h->held[i], kHoldsValue[i])) return false;
    for (const Held& t : h->tables)
        if (!unchanged(t, true)) return false;
    return true;
}

// One zero-filled scratch tensor per (device, stream), grown on demand; only touched with the GIL held.  A CUDA graph
// keeps the addresses it was captured with, so a tensor handed out during a capture is kept when a larger one
// replaces it.  A caller owns the tensor it gets until its launches are enqueued: the GIL is released for them, and
// another thread on the same stream may replace the map's tensor meanwhile.  Whether a graph is gone is not known here,
// so a kept tensor stays; its successor has at least twice its size, which bounds all that a stream keeps by the size of
// the scratch it has.
struct Scratch { at::Tensor t; bool captured = false; };
std::map<std::pair<int, int64_t>, Scratch>& scratch_map() {
    static auto* m = new std::map<std::pair<int, int64_t>, Scratch>();            // never destroyed: no CUDA calls at exit
    return *m;
}

std::vector<std::pair<int, at::Tensor>>& kept_scratch() {
    static auto* v = new std::vector<std::pair<int, at::Tensor>>();
    return *v;
}

at::Tensor scratch_for(int device, const c10::cuda::CUDAStream& stream, size_t bytes) {
    Scratch& s = scratch_map()[{device, static_cast<int64_t>(reinterpret_cast<intptr_t>(stream.stream()))}];
    if (!s.t.defined() || static_cast<size_t>(s.t.numel()) < bytes) {
        int64_t n = static_cast<int64_t>(bytes > kMinScratch ? bytes : kMinScratch);
        if (s.captured) {
            if (n < 2 * s.t.numel()) n = 2 * s.t.numel();
            kept_scratch().emplace_back(device, std::move(s.t));
        }
        s.t = at::zeros({n}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, static_cast<c10::DeviceIndex>(device)));
        s.captured = false;
    }
    if (!s.captured) {
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        s.captured = cudaStreamIsCapturing(stream.stream(), &st) == cudaSuccess && st != cudaStreamCaptureStatusNone;
    }
    return s.t;
}

bool fail(int status, const char* what) {
    PyErr_Format(PyExc_RuntimeError, "%s: %s (eptq status %d)", what, eptq_strerror(status), status);
    return false;
}

// x as contiguous fp16 rows of in_features; false with a Python error set if it cannot be.  With `reshape` its own
// dimensions do not matter (the output takes another input's), its values only have to fill whole rows.
bool as_rows(const LayerHandle* h, const at::Tensor& x, at::Tensor& rows, int64_t& n_rows, bool reshape = false) {
    if (!x.is_cuda()) {
        PyErr_SetString(PyExc_RuntimeError, "EPTQLinear runs on CUDA tensors only (there is no CPU path)");
        return false;
    }
    const bool whole = reshape && h->in_features > 0 && x.numel() % h->in_features == 0;
    if (!whole && (x.dim() < 1 || x.size(-1) != h->in_features)) {
        PyErr_Format(PyExc_RuntimeError, "EPTQLinear: the last dimension of the input must be %lld", (long long)h->in_features);
        return false;
    }
    rows = x.scalar_type() == at::kHalf ? x : x.to(at::kHalf);
    if (!rows.is_contiguous()) rows = rows.contiguous();
    n_rows = h->in_features > 0 ? rows.numel() / h->in_features : 0;
    return true;
}

at::Tensor new_output(const LayerHandle* h, const at::Tensor& x) {
    at::DimVector shape(x.sizes().begin(), x.sizes().end());
    shape.back() = h->out_features;
    return at::empty(shape, x.options().dtype(at::kHalf));
}

PyObject* wrap(at::Tensor y, at::ScalarType dtype) {
    return THPVariable_Wrap(dtype == at::kHalf ? std::move(y) : y.to(dtype));
}

// make_handle(descriptor bytes, keep, buffers dict, (fp16 codebook, fp32 codebook or None), in_features, out_features)
PyObject* make_handle(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 6 || !PyBytes_Check(a[0]) || PyBytes_GET_SIZE(a[0]) != static_cast<Py_ssize_t>(sizeof(EptqLayer)) ||
        !PyDict_Check(a[2]) || !PyTuple_Check(a[3]) || PyTuple_GET_SIZE(a[3]) != kTables) {
        PyErr_SetString(PyExc_TypeError, "make_handle(descriptor, keep, buffers, codebooks, in_features, out_features)");
        return nullptr;
    }
    const long long in = PyLong_AsLongLong(a[4]), out = PyLong_AsLongLong(a[5]);
    if (PyErr_Occurred()) return nullptr;
    PyObject* held[kBuffers];
    for (int i = 0; i < kBuffers; ++i) {
        held[i] = PyDict_GetItem(a[2], buffer_keys()[i]);
        if (held[i] == nullptr || !(THPVariable_Check(held[i]) || (i >= kOptionalFrom && held[i] == Py_None))) {
            PyErr_Format(PyExc_TypeError, "make_handle: buffer %s must be a tensor%s", kBufferNames[i], i >= kOptionalFrom ? " or None" : "");
            return nullptr;
        }
    }
    for (int i = 0; i < kTables; ++i) {
        PyObject* o = PyTuple_GET_ITEM(a[3], i);
        if (!THPVariable_Check(o) && o != Py_None) {
            PyErr_SetString(PyExc_TypeError, "make_handle: codebooks must be tensors or None");
            return nullptr;
        }
    }
    auto* h = new LayerHandle();
    h->keep = Py_NewRef(a[1]);
    h->buffers = Py_NewRef(a[2]);
    PyObject* c = PyCapsule_New(h, kCapsule, free_handle);               // owns h, also if what follows throws
    if (c == nullptr) {
        Py_DECREF(h->keep);
        Py_DECREF(h->buffers);
        delete h;
        return nullptr;
    }
    THPObjectPtr owner(c);
    std::memcpy(&h->d, PyBytes_AS_STRING(a[0]), sizeof(EptqLayer));
    for (int i = 0; i < kBuffers; ++i) hold(h->held[i], held[i]);
    for (int i = 0; i < kTables; ++i) hold(h->tables[i], PyTuple_GET_ITEM(a[3], i));
    h->in_features = in;
    h->out_features = out;
    return owner.release();
    END_HANDLE_TH_ERRORS
}

// forward(handle, x) -> y, or None if the module's buffers are no longer the descriptor's
PyObject* forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    LayerHandle* h = n == 2 ? handle_of(a[0]) : nullptr;
    if (h == nullptr || !THPVariable_Check(a[1])) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "forward(handle, tensor)");
        return nullptr;
    }
    if (!is_current(h)) Py_RETURN_NONE;
    const at::Tensor& x = THPVariable_Unpack(a[1]);
    at::Tensor rows;
    int64_t B = 0;
    if (!as_rows(h, x, rows, B)) return nullptr;
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    at::Tensor y = new_output(h, x);
    if (B == 0) return wrap(std::move(y), x.scalar_type());
    const auto stream = c10::cuda::getCurrentCUDAStream(x.device().index());
    size_t need = B <= kSmallRows ? h->scratch[B] : 0;
    if (need == 0) {
        need = eptq_layer_workspace_bytes(&h->d, static_cast<int>(B));
        if (B <= kSmallRows) h->scratch[B] = need;
    }
    const at::Tensor ws = scratch_for(x.device().index(), stream, need);
    void* const ws_ptr = ws.data_ptr();
    const size_t ws_bytes = static_cast<size_t>(ws.numel());
    const auto* xp = static_cast<const uint16_t*>(rows.const_data_ptr());
    auto* yp = static_cast<uint16_t*>(y.data_ptr());
    const EptqLayer d = h->d;
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = eptq_linear_forward(&d, xp, yp, static_cast<int>(B), ws_ptr, ws_bytes, stream.stream());
    Py_END_ALLOW_THREADS
    if (st != EPTQ_OK) { fail(st, "eptq linear forward"); return nullptr; }
    return wrap(std::move(y), x.scalar_type());
    END_HANDLE_TH_ERRORS
}

// forward_group(handles, xs) -> list of outputs, or None if some module's buffers have changed.  All outputs have
// the leading shape of the first input.
PyObject* forward_group(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (n_args != 2 || !PyList_Check(a[0]) || !PyList_Check(a[1]) || PyList_GET_SIZE(a[0]) != PyList_GET_SIZE(a[1]) ||
        PyList_GET_SIZE(a[0]) < 1) {
        PyErr_SetString(PyExc_TypeError, "forward_group(list of handles, list of as many tensors)");
        return nullptr;
    }
    const int n = static_cast<int>(PyList_GET_SIZE(a[0]));
    std::vector<EptqLayer> descs(n);
    std::vector<at::Tensor> rows(n), ys(n);
    std::vector<const uint16_t*> xp(n);
    std::vector<uint16_t*> yp(n);
    int64_t B = 0;
    c10::Device device(c10::kCPU);
    c10::cuda::OptionalCUDAGuard guard;
    at::DimVector lead;
    for (int i = 0; i < n; ++i) {
        LayerHandle* h = handle_of(PyList_GET_ITEM(a[0], i));
        PyObject* xo = PyList_GET_ITEM(a[1], i);
        if (h == nullptr || !THPVariable_Check(xo)) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "forward_group: handles and tensors expected");
            return nullptr;
        }
        if (!is_current(h)) Py_RETURN_NONE;
        const at::Tensor& x = THPVariable_Unpack(xo);
        int64_t b = 0;
        if (!as_rows(h, x, rows[i], b, i > 0)) return nullptr;
        if (i == 0) {
            B = b;
            device = x.device();
            guard.set_device(device);
            lead.assign(x.sizes().begin(), x.sizes().end());
        } else if (b != B || x.device() != device) {
            PyErr_SetString(PyExc_RuntimeError, "eptq_b200: grouped inputs need one row count and one device");
            return nullptr;
        }
        lead.back() = h->out_features;
        ys[i] = at::empty(lead, x.options().dtype(at::kHalf));
        descs[i] = h->d;
        xp[i] = static_cast<const uint16_t*>(rows[i].const_data_ptr());
        yp[i] = static_cast<uint16_t*>(ys[i].data_ptr());
    }
    const size_t need = eptq_group_workspace_bytes(descs.data(), n, static_cast<int>(B));
    if (need == 0) {
        PyErr_SetString(PyExc_RuntimeError, "eptq_b200: this set of layers cannot run as one group launch");
        return nullptr;
    }
    const auto stream = c10::cuda::getCurrentCUDAStream(device.index());
    const at::Tensor ws = scratch_for(device.index(), stream, need);
    void* const ws_ptr = ws.data_ptr();
    const size_t ws_bytes = static_cast<size_t>(ws.numel());
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = eptq_linear_forward_group(descs.data(), n, xp.data(), yp.data(), static_cast<int>(B), ws_ptr, ws_bytes, stream.stream());
    Py_END_ALLOW_THREADS
    if (st != EPTQ_OK) { fail(st, "eptq group forward"); return nullptr; }
    PyObject* out = PyList_New(n);
    if (out == nullptr) return nullptr;
    for (int i = 0; i < n; ++i)
        PyList_SET_ITEM(out, i, wrap(std::move(ys[i]), THPVariable_Unpack(PyList_GET_ITEM(a[1], i)).scalar_type()));
    return out;
    END_HANDLE_TH_ERRORS
}

// dequantize(handle) -> fp16 (out, in) weight, or None if the module's buffers have changed
PyObject* dequantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    LayerHandle* h = n == 1 ? handle_of(a[0]) : nullptr;
    if (h == nullptr) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "dequantize(handle)");
        return nullptr;
    }
    if (!is_current(h)) Py_RETURN_NONE;
    const at::Tensor& q = THPVariable_Unpack(h->held[0].obj);
    if (!q.is_cuda()) {
        PyErr_SetString(PyExc_RuntimeError, "eptq_b200: `Q` must be a CUDA tensor (no CPU path exists)");
        return nullptr;
    }
    const c10::cuda::OptionalCUDAGuard guard(q.device());
    at::Tensor w = at::empty({h->out_features, h->in_features}, q.options().dtype(at::kHalf));
    const auto stream = c10::cuda::getCurrentCUDAStream(q.device().index());
    auto* wp = static_cast<uint16_t*>(w.data_ptr());
    const EptqLayer d = h->d;
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = eptq_dequantize(&d, wp, stream.stream());
    Py_END_ALLOW_THREADS
    if (st != EPTQ_OK) { fail(st, "eptq dequantize"); return nullptr; }
    return THPVariable_Wrap(std::move(w));
    END_HANDLE_TH_ERRORS
}

// scratch(device index, bytes) -> the scratch tensor of the current stream
PyObject* scratch(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 2) { PyErr_SetString(PyExc_TypeError, "scratch(device index, bytes)"); return nullptr; }
    const long device = PyLong_AsLong(a[0]);
    const size_t bytes = PyLong_AsSize_t(a[1]);
    if (PyErr_Occurred()) return nullptr;
    const c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(device)));
    return THPVariable_Wrap(scratch_for(static_cast<int>(device), c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)), bytes));
    END_HANDLE_TH_ERRORS
}

// scratch_of_device(device index) -> list of all its scratch tensors (one per stream that ran the kernels)
PyObject* scratch_of_device(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 1) { PyErr_SetString(PyExc_TypeError, "scratch_of_device(device index)"); return nullptr; }
    const long device = PyLong_AsLong(a[0]);
    if (PyErr_Occurred()) return nullptr;
    PyObject* out = PyList_New(0);
    if (out == nullptr) return nullptr;
    std::vector<at::Tensor> all;
    for (const auto& kv : scratch_map())
        if (kv.first.first == device) all.push_back(kv.second.t);
    for (const auto& kv : kept_scratch())
        if (kv.first == device) all.push_back(kv.second);
    for (const at::Tensor& s : all) {
        PyObject* t = THPVariable_Wrap(s);
        if (t == nullptr || PyList_Append(out, t) != 0) { Py_XDECREF(t); Py_DECREF(out); return nullptr; }
        Py_DECREF(t);
    }
    return out;
    END_HANDLE_TH_ERRORS
}

#define METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {METHOD(make_handle), METHOD(forward), METHOD(forward_group), METHOD(dequantize),
                         METHOD(scratch), METHOD(scratch_of_device), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_eptq_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__eptq_host(void) { return PyModule_Create(&module); }
