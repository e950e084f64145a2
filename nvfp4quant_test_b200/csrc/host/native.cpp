// Host half of the Python entry points: argument checks, output allocation, current stream and launch in one C call.
//
// What bounds a small call is the host, not the GPU: a decode-sized quantization runs 2-3 us on the device, while the
// same checks, two torch.empty, a dtype view and a 15-argument ctypes call cost 13-15 us of interpreter time.  Every
// function here does the whole common case and returns None for anything else (a wrong shape, a CPU tensor, a strided
// or misaligned operand, a tensor subclass, a stream under capture where scratch words are needed, a failed launch); the
// Python entry point then takes its own path, which holds the conversions and all error messages, so that there is one
// place that decides what an error of a caller is.
//
// The kernels are reached through the C ABI of include/nvfp4_b200.h, like from any other caller.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/core/CachingHostAllocator.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/zeros.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/autograd/python_variable.h>

#include <list>
#include <memory>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "nvfp4_b200.h"

namespace {

using at::Tensor;

PyTypeObject* g_parameter_type = nullptr;   // torch.nn.Parameter: the one subclass that behaves like a plain tensor

inline int64_t round_up(int64_t x, int64_t y) { return (x + y - 1) / y * y; }

// The tensor behind a plain torch.Tensor or Parameter, NULL for everything else.
inline const Tensor* tensor_of(PyObject* o) {
    if (Py_TYPE(o) != reinterpret_cast<PyTypeObject*>(THPVariableClass) && Py_TYPE(o) != g_parameter_type) return nullptr;
    return &THPVariable_Unpack(o);
}

inline bool plain_cuda(const Tensor& t) { return t.is_cuda() && t.layout() == at::kStrided; }
inline uintptr_t address(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.const_data_ptr()); }
inline bool aligned(const Tensor& t, uintptr_t to) { return (address(t) & (to - 1)) == 0; }

inline int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kBFloat16: return NVFP4_DT_BF16;
        case at::kHalf: return NVFP4_DT_F16;
        case at::kFloat: return NVFP4_DT_F32;
        default: return -1;
    }
}

inline cudaStream_t current_stream(c10::DeviceIndex device) { return c10::cuda::getCurrentCUDAStream(device).stream(); }

// Runs `launch` with the tensor's device current and without the interpreter lock (a full launch queue blocks the caller).
template <class F>
inline int launch_on(c10::DeviceIndex device, F&& launch) {
    c10::cuda::OptionalCUDAGuard guard;
    if (c10::cuda::current_device() != device) guard.set_index(device);
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = launch();
    Py_END_ALLOW_THREADS
    return st;
}

inline Tensor empty(at::IntArrayRef sizes, at::ScalarType dtype, c10::DeviceIndex device) {
    return at::detail::empty_cuda(sizes, dtype, c10::Device(c10::kCUDA, device), std::nullopt);
}

// 0-dim view of element `index` of a contiguous float vector, without a trip through the dispatcher.
inline Tensor scalar_view(const Tensor& v, int64_t index) {
    Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(v.storage()), v.key_set(), v.dtype());
    t.unsafeGetTensorImpl()->set_storage_offset(v.storage_offset() + index);
    t.unsafeGetTensorImpl()->set_sizes_contiguous({});
    return t;
}

inline PyObject* none() { Py_RETURN_NONE; }
inline PyObject* truth() { Py_RETURN_TRUE; }

// None or an int; false when it is neither.
inline bool int_or_none(PyObject* o, int64_t if_none, int64_t* out) {
    if (o == Py_None) {
        *out = if_none;
        return true;
    }
    if (!PyLong_CheckExact(o)) return false;
    *out = PyLong_AsLongLong(o);
    if (*out == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}
inline bool as_float(PyObject* o, float* out) {
    if (!PyFloat_CheckExact(o) && !PyLong_CheckExact(o)) return false;
    const double d = PyFloat_AsDouble(o);
    if (d == -1.0 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    *out = static_cast<float>(d);
    return true;
}
// An int of the candidate window; false for anything else and for what does not fit.
inline bool window_int(PyObject* o, int* out) {
    int overflow = 0;
    const long v = PyLong_CheckExact(o) ? PyLong_AsLongAndOverflow(o, &overflow) : 0;
    *out = static_cast<int>(v);
    return PyLong_CheckExact(o) && overflow == 0 && *out == v;
}
inline int small_int(PyObject* o) { return static_cast<int>(PyLong_AsLong(o)); }   // a constant of the package's own

PyObject* pack(std::initializer_list<Tensor> ts) {
    PyObject* t = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
    if (!t) return nullptr;
    Py_ssize_t i = 0;
    for (const Tensor& x : ts) {
        PyObject* o = THPVariable_Wrap(x);
        if (!o) {
            Py_DECREF(t);
            return nullptr;
        }
        PyTuple_SET_ITEM(t, i++, o);
    }
    return t;
}

// Any C++ exception (a torch check, an allocation failure) becomes "not the common case": the Python path repeats the
// call and reports it in its own words.
template <class F>
inline PyObject* guarded(F&& f) {
    try {
        return f();
    } catch (...) {
        PyErr_Clear();
        return none();
    }
}

// ---- scratch words of the global-scale kernel -----------------------------------------------------------------------
// Two zeroed words for each of up to 16 tensors per (device, stream), left zeroed by every launch; at most 32 streams, least recently used dropped (the
// block goes back to torch's allocator, which hands it out again in stream order).  Under capture the caller takes the
// Python path, which keeps a scratch per capture.  Guarded by the interpreter lock, which every caller holds.
struct ScratchKey {
    c10::DeviceIndex device;
    cudaStream_t stream;
    bool operator==(const ScratchKey& o) const { return device == o.device && stream == o.stream; }
};
struct ScratchHash {
    size_t operator()(const ScratchKey& k) const { return reinterpret_cast<size_t>(k.stream) * 31 + static_cast<size_t>(k.device); }
};
constexpr size_t kScratchStreams = 32;
std::list<std::pair<ScratchKey, Tensor>>& scratch_list() {
    static auto* l = new std::list<std::pair<ScratchKey, Tensor>>();   // never destroyed: the CUDA context may be gone by then
    return *l;
}
std::unordered_map<ScratchKey, std::list<std::pair<ScratchKey, Tensor>>::iterator, ScratchHash>& scratch_map() {
    static auto* m = new std::unordered_map<ScratchKey, std::list<std::pair<ScratchKey, Tensor>>::iterator, ScratchHash>();
    return *m;
}

// Undefined where the caller takes the Python path.  The caller keeps the tensor until its launch is queued: it gives up the
// interpreter lock for that, and other threads may drop the block from the list meanwhile.
Tensor scratch_words(c10::DeviceIndex device, cudaStream_t stream) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) {
        cudaGetLastError();   // e.g. the legacy stream while another stream captures: the Python path decides
        return Tensor();
    }
    if (status != cudaStreamCaptureStatusNone) return Tensor();
    auto& l = scratch_list();
    auto& m = scratch_map();
    const ScratchKey key{device, stream};
    auto it = m.find(key);
    if (it != m.end()) {
        if (it->second != l.begin()) l.splice(l.begin(), l, it->second);
    } else {
        Tensor words = at::zeros({32}, at::TensorOptions().dtype(at::kInt).device(c10::Device(c10::kCUDA, device)));
        l.emplace_front(key, words);
        m[key] = l.begin();
        if (l.size() > kScratchStreams) {
            m.erase(l.back().first);
            l.pop_back();
        }
    }
    return l.front().second;
}
inline uint32_t* words_of(const Tensor& scratch) { return static_cast<uint32_t*>(scratch.mutable_data_ptr()); }

// ---- quantizers -----------------------------------------------------------------------------------------------------

struct QuantIn {
    const Tensor* x;
    const float* importance;
    int64_t m, n;
    int dtype;
    c10::DeviceIndex device;
};

// The input (and, for the weighted variant, the importance row) as every quantizer entry takes it.
bool quant_input(PyObject* input, PyObject* importance, QuantIn* q) {
    const Tensor* x = tensor_of(input);
    if (!x || !plain_cuda(*x) || x->dim() != 2 || !x->is_contiguous()) return false;
    q->x = x;
    q->m = x->size(0);
    q->n = x->size(1);
    q->dtype = dtype_code(x->scalar_type());
    q->device = x->device().index();
    q->importance = nullptr;
    if (q->dtype < 0 || q->m <= 0 || q->n <= 0 || q->n % 16 || !aligned(*x, 16)) return false;
    if (importance != Py_None) {
        const Tensor* w = tensor_of(importance);
        if (!w || !plain_cuda(*w) || w->device() != x->device() || w->scalar_type() != at::kFloat || w->dim() != 2 ||
            w->size(0) != 1 || w->size(1) != q->n || !w->is_contiguous() || !aligned(*w, 16))
            return false;
        q->importance = static_cast<const float*>(w->const_data_ptr());
    }
    return true;
}

bool scalar_input(PyObject* o, c10::DeviceIndex device, const float** out) {
    const Tensor* s = tensor_of(o);
    if (!s || !plain_cuda(*s) || s->device().index() != device || s->scalar_type() != at::kFloat || s->numel() < 1) return false;
    *out = static_cast<const float*>(s->const_data_ptr());
    return true;
}

// Shapes of vllm's create_fp4_output_tensors, the scale buffer typed float8_e4m3fn as the entry points return it.
inline Tensor empty_scales(int64_t m, int64_t padded_n, bool tiled, c10::DeviceIndex device) {
    if (tiled) return empty({round_up(m, 128), round_up(padded_n / 16, 4)}, at::kFloat8_e4m3fn, device);
    return empty({m, padded_n / 16}, at::kFloat8_e4m3fn, device);
}

// quant_impl(variant, input, importance | None, input_scale, tiled, padded_n | None, lower, upper) -> (codes, scales)
PyObject* quant_impl(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 8) return none();
        QuantIn q;
        const float* gs_inv;
        int64_t padded_n;
        int lower, upper;
        if (!quant_input(a[1], a[2], &q) || !scalar_input(a[3], q.device, &gs_inv) || !PyBool_Check(a[4]) ||
            !int_or_none(a[5], q.n, &padded_n) || padded_n < q.n || padded_n % 16 || !window_int(a[6], &lower) || !window_int(a[7], &upper))
            return none();
        const int variant = small_int(a[0]);
        const bool tiled = a[4] == Py_True;
        Tensor codes = empty({q.m, padded_n / 2}, at::kByte, q.device);
        Tensor scales = empty_scales(q.m, padded_n, tiled, q.device);
        const cudaStream_t s = current_stream(q.device);
        const int st = launch_on(q.device, [&] {
            return nvfp4_quant_launch(variant, q.x->const_data_ptr(), q.dtype, q.importance, gs_inv,
                                      static_cast<uint8_t*>(codes.mutable_data_ptr()), static_cast<uint8_t*>(scales.mutable_data_ptr()),
                                      q.m, q.n, padded_n, lower, upper, tiled ? 1 : 0, s);
        });
        return st == NVFP4_OK ? pack({codes, scales}) : none();
    });
}

// quant_out(variant, input, importance | None, input_scale, tiled, output, output_scale, lower, upper) -> True; the caller's buffers
// may be a prepared weight's
PyObject* quant_out(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 9) return none();
        QuantIn q;
        const float* gs_inv;
        int lower, upper;
        if (!quant_input(a[1], a[2], &q) || !scalar_input(a[3], q.device, &gs_inv) || !PyBool_Check(a[4]) || !window_int(a[7], &lower) ||
            !window_int(a[8], &upper))
            return none();
        const Tensor *codes = tensor_of(a[5]), *scales = tensor_of(a[6]);
        if (!codes || !scales || !plain_cuda(*codes) || !plain_cuda(*scales) || codes->device() != q.x->device() ||
            scales->device() != q.x->device() || codes->scalar_type() != at::kByte || codes->dim() != 2 || codes->size(0) != q.m ||
            !codes->is_contiguous() || !scales->is_contiguous())
            return none();
        const int64_t padded_n = codes->size(1) * 2;
        if (padded_n % 16 || padded_n < q.n) return none();
        const bool tiled = a[4] == Py_True;
        const int64_t need = tiled ? round_up(q.m, 128) * round_up(padded_n / 16, 4) : q.m * (padded_n / 16);
        if (static_cast<int64_t>(scales->nbytes()) < need) return none();
        const int variant = small_int(a[0]);
        const cudaStream_t s = current_stream(q.device);
        const int st = launch_on(q.device, [&] {
            return nvfp4_quant_launch_in_place(variant, q.x->const_data_ptr(), q.dtype, q.importance, gs_inv,
                                               static_cast<uint8_t*>(codes->mutable_data_ptr()), static_cast<uint8_t*>(scales->mutable_data_ptr()),
                                               q.m, q.n, padded_n, lower, upper, tiled ? 1 : 0, s);
        });
        return st == NVFP4_OK ? truth() : none();
    });
}

// global_scale(x, fp8_max, out | None) -> (global_scale, 1 / global_scale), 0-dim views of one pair
PyObject* global_scale(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 3) return none();
        const Tensor* x = tensor_of(a[0]);
        float fp8_max;
        if (!x || !plain_cuda(*x) || !x->is_contiguous() || x->numel() == 0 || !aligned(*x, 16) || !as_float(a[1], &fp8_max)) return none();
        const int dt = dtype_code(x->scalar_type());
        if (dt < 0) return none();
        const c10::DeviceIndex dev = x->device().index();
        Tensor out;
        if (a[2] == Py_None) {
            out = empty({2}, at::kFloat, dev);
        } else {
            const Tensor* o = tensor_of(a[2]);
            if (!o || o->device() != x->device() || o->scalar_type() != at::kFloat || o->dim() != 1 || o->size(0) != 2 || !o->is_contiguous())
                return none();
            out = *o;
        }
        const cudaStream_t s = current_stream(dev);
        const Tensor scratch = scratch_words(dev, s);
        if (!scratch.defined()) return none();
        const int st = launch_on(dev, [&] {
            return nvfp4_global_scale_launch(x->const_data_ptr(), dt, x->numel(), fp8_max, static_cast<float*>(out.mutable_data_ptr()), words_of(scratch), s);
        });
        return st == NVFP4_OK ? pack({scalar_view(out, 0), scalar_view(out, 1)}) : none();
    });
}

// quant_dynamic(variant, input, importance | None, fp8_max, tiled, padded_n | None, lower, upper)
//   -> (codes, scales, global_scale, 1 / global_scale): the global scale and the quantizer that reads it, two dependent
// launches from one call
PyObject* quant_dynamic(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 8) return none();
        QuantIn q;
        float fp8_max;
        int64_t padded_n;
        int lower, upper;
        if (!quant_input(a[1], a[2], &q) || !as_float(a[3], &fp8_max) || !PyBool_Check(a[4]) || !int_or_none(a[5], q.n, &padded_n) ||
            padded_n < q.n || padded_n % 16 || !window_int(a[6], &lower) || !window_int(a[7], &upper))
            return none();
        const int variant = small_int(a[0]);
        const bool tiled = a[4] == Py_True;
        const cudaStream_t s = current_stream(q.device);
        const Tensor scratch = scratch_words(q.device, s);
        if (!scratch.defined()) return none();
        Tensor codes = empty({q.m, padded_n / 2}, at::kByte, q.device);
        Tensor scales = empty_scales(q.m, padded_n, tiled, q.device);
        Tensor gs = empty({2}, at::kFloat, q.device);
        const int st = launch_on(q.device, [&] {
            return nvfp4_quant_chain_launch(variant, q.x->const_data_ptr(), q.dtype, q.importance, fp8_max,
                                            static_cast<float*>(gs.mutable_data_ptr()), words_of(scratch), static_cast<uint8_t*>(codes.mutable_data_ptr()),
                                            static_cast<uint8_t*>(scales.mutable_data_ptr()), q.m, q.n, padded_n, lower, upper, tiled ? 1 : 0, s);
        });
        return st == NVFP4_OK ? pack({codes, scales, scalar_view(gs, 0), scalar_view(gs, 1)}) : none();
    });
}

// quant_dynamic_multi(variant, [input], fp8_max, lower, upper) -> [(codes, scales, global_scale, 1 / global_scale)], tiled scales,
// no padding: quant_dynamic over several unweighted tensors, sharing their launches
PyObject* quant_dynamic_multi(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        float fp8_max;
        int lower, upper;
        if (nargs != 5 || !PyList_CheckExact(a[1]) || !as_float(a[2], &fp8_max) || !window_int(a[3], &lower) || !window_int(a[4], &upper)) return none();
        const Py_ssize_t n = PyList_GET_SIZE(a[1]);
        constexpr Py_ssize_t kMost = 16;
        if (n < 1 || n > kMost) return none();
        QuantIn q[kMost];
        for (Py_ssize_t i = 0; i < n; ++i)
            if (!quant_input(PyList_GET_ITEM(a[1], i), Py_None, &q[i]) || q[i].device != q[0].device || q[i].dtype != q[0].dtype) return none();
        const c10::DeviceIndex dev = q[0].device;
        const cudaStream_t s = current_stream(dev);
        const Tensor scratch = scratch_words(dev, s);
        if (!scratch.defined()) return none();
        nvfp4_chain_item items[kMost];
        Tensor codes[kMost], scales[kMost], gs[kMost];
        for (Py_ssize_t i = 0; i < n; ++i) {
            codes[i] = empty({q[i].m, q[i].n / 2}, at::kByte, dev);
            scales[i] = empty_scales(q[i].m, q[i].n, true, dev);
            gs[i] = empty({2}, at::kFloat, dev);
            items[i] = {q[i].x->const_data_ptr(), nullptr, static_cast<float*>(gs[i].mutable_data_ptr()), words_of(scratch) + 2 * i,
                        static_cast<uint8_t*>(codes[i].mutable_data_ptr()), static_cast<uint8_t*>(scales[i].mutable_data_ptr()), q[i].m, q[i].n, q[i].n};
        }
        const int variant = small_int(a[0]);
        const int st = launch_on(dev, [&] {
            return nvfp4_quant_chain_multi_launch(variant, q[0].dtype, fp8_max, items, static_cast<int>(n), lower, upper, 1, s);
        });
        if (st != NVFP4_OK) return none();
        PyObject* l = PyList_New(n);
        for (Py_ssize_t i = 0; l && i < n; ++i) {
            PyObject* t = pack({codes[i], scales[i], scalar_view(gs[i], 0), scalar_view(gs[i], 1)});
            if (!t) {
                Py_DECREF(l);
                return nullptr;
            }
            PyList_SET_ITEM(l, i, t);
        }
        return l;
    });
}

// channel_square_norm(x, out | None) -> float32 [1, dim]
PyObject* channel_square_norm(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 2) return none();
        const Tensor* x = tensor_of(a[0]);
        if (!x || !plain_cuda(*x) || x->dim() != 2 || x->size(1) % 4 || x->size(1) == 0 || !aligned(*x, 16)) return none();
        const int dt = dtype_code(x->scalar_type());
        const int64_t m = x->size(0), n = x->size(1);
        // a column slice of a wider batch is read in place through its row pitch
        const int64_t ld = m > 1 ? x->stride(0) : n;
        if (dt < 0 || x->stride(1) != 1 || (m > 1 && (ld < n || ld % 4))) return none();
        const c10::DeviceIndex dev = x->device().index();
        Tensor out;
        if (a[1] == Py_None) {
            out = empty({1, n}, at::kFloat, dev);
        } else {
            const Tensor* o = tensor_of(a[1]);
            if (!o || o->device() != x->device() || o->scalar_type() != at::kFloat || o->dim() != 2 || o->size(0) != 1 || o->size(1) != n ||
                !o->is_contiguous())
                return none();
            out = *o;
        }
        const cudaStream_t s = current_stream(dev);
        const int st = launch_on(dev, [&] {
            return nvfp4_channel_sqnorm_launch_strided(x->const_data_ptr(), dt, m, n, ld, static_cast<float*>(out.mutable_data_ptr()), s);
        });
        if (st != NVFP4_OK) return none();
        if (a[1] != Py_None) {
            Py_INCREF(a[1]);
            return a[1];
        }
        return THPVariable_Wrap(out);
    });
}

// The dequantizer and the scale layouts are torch operations anywhere but here, so what torch does beside computing them has to
// go on: a tracer or a dispatch mode sees the operations, gradients and forward-mode tangents flow through them, a lazily negated
// scale is read as its value.  (Inside torch.func transforms a wrapped tensor has no data to point at and falls out by itself.)
inline bool observed() { return c10::impl::dispatch_mode_enabled() || c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Tracer); }
inline bool plain_value(const Tensor& t) { return !(c10::GradMode::is_enabled() && t.requires_grad()) && !t._fw_grad(0).defined() && !t.is_neg(); }

// dequant(codes, block scales | None, global scale | None) -> float32 [m, n]
PyObject* dequant(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 3 || observed()) return none();
        const Tensor* q = tensor_of(a[0]);
        if (!q || !plain_cuda(*q) || q->dim() != 2 || q->scalar_type() != at::kByte || !q->is_contiguous() || !aligned(*q, 4)) return none();
        const int64_t m = q->size(0), n = q->size(1) * 2;
        const c10::DeviceIndex dev = q->device().index();
        const uint8_t* scales = nullptr;
        const float* gs = nullptr;
        if (m == 0 || n == 0) return none();
        if (a[1] == Py_None) {
            if (n % 8) return none();
        } else {
            const Tensor *s = tensor_of(a[1]), *g = tensor_of(a[2]);
            if (!s || !g || s->device() != q->device() || s->scalar_type() != at::kFloat8_e4m3fn || s->dim() != 2 || s->size(0) != m ||
                s->size(1) * 16 != n || !s->is_contiguous() || g->numel() != 1 || g->dim() > 2 || !plain_value(*s) || !plain_value(*g) || !scalar_input(a[2], dev, &gs))
                return none();
            scales = static_cast<const uint8_t*>(s->const_data_ptr());
        }
        Tensor out = empty({m, n}, at::kFloat, dev);
        const cudaStream_t st = current_stream(dev);
        const int rc = launch_on(dev, [&] {
            return nvfp4_dequant_launch(static_cast<const uint8_t*>(q->const_data_ptr()), scales, gs, static_cast<float*>(out.mutable_data_ptr()),
                                        m, n, st);
        });
        return rc == NVFP4_OK ? THPVariable_Wrap(out) : none();
    });
}

// scale_layout(scales, m, k, to_tiled): row-major [m, k] -> flat tiled buffer, or a tiled buffer of any shape -> [m, k]
PyObject* scale_layout(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        int64_t m, k;
        if (nargs != 4 || observed() || !int_or_none(a[1], 0, &m) || !int_or_none(a[2], 0, &k) || m <= 0 || k <= 0) return none();
        const bool to_tiled = a[3] == Py_True;
        const Tensor* s = tensor_of(a[0]);
        const int64_t padded = round_up(m, 128) * round_up(k, 4);
        if (!s || !plain_cuda(*s) || s->element_size() != 1 || !s->is_contiguous() || s->numel() != (to_tiled ? m * k : padded)) return none();
        const c10::DeviceIndex dev = s->device().index();
        Tensor out = to_tiled ? empty({padded}, s->scalar_type(), dev) : empty({m, k}, s->scalar_type(), dev);
        const cudaStream_t st = current_stream(dev);
        const int rc = launch_on(dev, [&] {
            return nvfp4_scale_layout_launch(static_cast<const uint8_t*>(s->const_data_ptr()), static_cast<uint8_t*>(out.mutable_data_ptr()), m, k,
                                             to_tiled ? 1 : 0, st);
        });
        return rc == NVFP4_OK ? THPVariable_Wrap(out) : none();
    });
}

// ---- GEMM -----------------------------------------------------------------------------------------------------------

inline int64_t scale_bytes(int64_t rows, int64_t k) { return round_up(rows, 128) * round_up(k / 16, 4); }

// Codes uint8 [rows, k/2] and their tiled scales, both contiguous.
bool quantized_operand(PyObject* codes, PyObject* scales, const Tensor** c, const Tensor** s) {
    *c = tensor_of(codes);
    *s = tensor_of(scales);
    if (!*c || !*s || !plain_cuda(**c) || !plain_cuda(**s) || (*c)->dim() != 2 || (*c)->scalar_type() != at::kByte || !(*c)->is_contiguous() ||
        !(*s)->is_contiguous() || (*s)->device() != (*c)->device())
        return false;
    return static_cast<int64_t>((*s)->nbytes()) >= scale_bytes((*c)->size(0), (*c)->size(1) * 2);
}

// The caller's output or a fresh one; false when the caller's does not fit.
bool output_matrix(PyObject* o, int64_t m, int64_t n, c10::DeviceIndex dev, Tensor* out) {
    if (o == Py_None) {
        *out = empty({m, n}, at::kBFloat16, dev);
        return true;
    }
    const Tensor* t = tensor_of(o);
    if (!t || !plain_cuda(*t) || t->device().index() != dev || t->scalar_type() != at::kBFloat16 || t->dim() != 2 || t->size(0) != m ||
        t->size(1) != n || !t->is_contiguous())
        return false;
    *out = *t;
    return true;
}

PyObject* output_object(PyObject* given, const Tensor& out) {
    if (given != Py_None) {
        Py_INCREF(given);
        return given;
    }
    return THPVariable_Wrap(out);
}

// scaled_mm(a, b, block_scale_a, block_scale_b, alpha, out | None) -> bf16 [m, n]
PyObject* scaled_mm(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 6) return none();
        const Tensor *qa, *qb, *sa, *sb;
        const float* alpha;
        if (!quantized_operand(a[0], a[2], &qa, &sa) || !quantized_operand(a[1], a[3], &qb, &sb) || qa->device() != qb->device()) return none();
        const c10::DeviceIndex dev = qa->device().index();
        const int64_t m = qa->size(0), n = qb->size(0), k = qa->size(1) * 2;
        Tensor out;
        if (qb->size(1) * 2 != k || k % 64 || m == 0 || n == 0 || !scalar_input(a[4], dev, &alpha) || !output_matrix(a[5], m, n, dev, &out))
            return none();
        const cudaStream_t s = current_stream(dev);
        const int st = launch_on(dev, [&] {
            return nvfp4_gemm_launch(static_cast<const uint8_t*>(qa->const_data_ptr()), static_cast<const uint8_t*>(qb->const_data_ptr()),
                                     static_cast<const uint8_t*>(sa->const_data_ptr()), static_cast<const uint8_t*>(sb->const_data_ptr()), alpha,
                                     out.mutable_data_ptr(), m, n, k, nullptr, 0, s);
        });
        return st == NVFP4_OK ? output_object(a[5], out) : none();
    });
}

// A prepared weight as the Python object keeps it for these calls: (handle, n, k, device index).
struct Weight {
    void* handle;
    int64_t n, k;
    c10::DeviceIndex device;
};
bool weight_of(PyObject* t, Weight* w) {
    if (!PyTuple_CheckExact(t) || PyTuple_GET_SIZE(t) != 4) return false;
    w->handle = PyLong_AsVoidPtr(PyTuple_GET_ITEM(t, 0));
    w->n = PyLong_AsLongLong(PyTuple_GET_ITEM(t, 1));
    w->k = PyLong_AsLongLong(PyTuple_GET_ITEM(t, 2));
    w->device = static_cast<c10::DeviceIndex>(PyLong_AsLong(PyTuple_GET_ITEM(t, 3)));
    return w->handle != nullptr && !PyErr_Occurred();
}

// scaled_mm_prepared(a, block_scale_a, alpha, weight, out | None) -> bf16 [m, n]
PyObject* scaled_mm_prepared(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 5) return none();
        const Tensor *qa, *sa;
        const float* alpha;
        Weight w;
        if (!weight_of(a[3], &w) || !quantized_operand(a[0], a[1], &qa, &sa)) {
            PyErr_Clear();
            return none();
        }
        const c10::DeviceIndex dev = qa->device().index();
        const int64_t m = qa->size(0);
        Tensor out;
        if (w.device != dev || qa->size(1) * 2 != w.k || m == 0 || !scalar_input(a[2], dev, &alpha) || !output_matrix(a[4], m, w.n, dev, &out))
            return none();
        const cudaStream_t s = current_stream(dev);
        const int st = launch_on(dev, [&] {
            return nvfp4_gemm_launch_prepared(w.handle, static_cast<const uint8_t*>(qa->const_data_ptr()),
                                              static_cast<const uint8_t*>(sa->const_data_ptr()), alpha, out.mutable_data_ptr(), m, nullptr, 0, s);
        });
        return st == NVFP4_OK ? output_object(a[4], out) : none();
    });
}

PyObject* tensor_list(const std::vector<Tensor>& ts) {
    PyObject* l = PyList_New(static_cast<Py_ssize_t>(ts.size()));
    for (size_t i = 0; l && i < ts.size(); ++i) {
        PyObject* o = THPVariable_Wrap(ts[i]);
        if (!o) {
            Py_DECREF(l);
            return nullptr;
        }
        PyList_SET_ITEM(l, static_cast<Py_ssize_t>(i), o);
    }
    return l;
}

// scaled_mm_grouped(a, block_scale_a, alpha_a | None, [weight], [alpha_w], [out] | None) -> [bf16 [m, n_i]]
PyObject* scaled_mm_grouped(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 6 || !PyList_CheckExact(a[3]) || !PyList_CheckExact(a[4]) || (a[5] != Py_None && !PyList_CheckExact(a[5]))) return none();
        const Py_ssize_t count = PyList_GET_SIZE(a[3]);
        if (count < 1 || count > 64 || PyList_GET_SIZE(a[4]) != count || (a[5] != Py_None && PyList_GET_SIZE(a[5]) != count)) return none();
        const Tensor *qa, *sa;
        if (!quantized_operand(a[0], a[1], &qa, &sa)) return none();
        const c10::DeviceIndex dev = qa->device().index();
        const int64_t m = qa->size(0), k = qa->size(1) * 2;
        const float* alpha_a = nullptr;
        if (m == 0 || (a[2] != Py_None && !scalar_input(a[2], dev, &alpha_a))) return none();
        void *handles[64], *outs[64];
        const float* alphas[64];
        std::vector<Tensor> out(static_cast<size_t>(count));
        for (Py_ssize_t i = 0; i < count; ++i) {
            Weight w;
            if (!weight_of(PyList_GET_ITEM(a[3], i), &w) || w.device != dev || w.k != k ||
                !scalar_input(PyList_GET_ITEM(a[4], i), dev, &alphas[i]) ||
                !output_matrix(a[5] == Py_None ? Py_None : PyList_GET_ITEM(a[5], i), m, w.n, dev, &out[i])) {
                PyErr_Clear();
                return none();
            }
            handles[i] = w.handle;
            outs[i] = out[i].mutable_data_ptr();
        }
        const cudaStream_t s = current_stream(dev);
        const int st = launch_on(dev, [&] {
            return nvfp4_gemm_launch_grouped(handles, static_cast<int>(count), static_cast<const uint8_t*>(qa->const_data_ptr()),
                                             static_cast<const uint8_t*>(sa->const_data_ptr()), alpha_a, alphas, outs, m, s);
        });
        if (st != NVFP4_OK) return none();
        if (a[5] != Py_None) {
            Py_INCREF(a[5]);
            return a[5];
        }
        return tensor_list(out);
    });
}

// scaled_mm_multi([a], [block_scale_a], [alpha_a | None], [weight], [alpha_w]) -> [bf16 [m, n_i]]
PyObject* scaled_mm_multi(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 5) return none();
        for (int i = 0; i < 5; ++i)
            if (!PyList_CheckExact(a[i]) || PyList_GET_SIZE(a[i]) != PyList_GET_SIZE(a[0])) return none();
        const Py_ssize_t count = PyList_GET_SIZE(a[0]);
        if (count < 1 || count > 64) return none();
        nvfp4_gemm_item items[64];
        std::vector<Tensor> out(static_cast<size_t>(count));
        int64_t m = 0;
        c10::DeviceIndex dev = 0;
        for (Py_ssize_t i = 0; i < count; ++i) {
            const Tensor *qa, *sa;
            Weight w;
            nvfp4_gemm_item& it = items[i];
            it.alpha_a = nullptr;
            if (!weight_of(PyList_GET_ITEM(a[3], i), &w) || !quantized_operand(PyList_GET_ITEM(a[0], i), PyList_GET_ITEM(a[1], i), &qa, &sa)) {
                PyErr_Clear();
                return none();
            }
            if (i == 0) {
                m = qa->size(0);
                dev = qa->device().index();
            }
            PyObject* alpha_a = PyList_GET_ITEM(a[2], i);
            if (m == 0 || qa->size(0) != m || qa->device().index() != dev || w.device != dev || qa->size(1) * 2 != w.k ||
                (alpha_a != Py_None && !scalar_input(alpha_a, dev, &it.alpha_a)) || !scalar_input(PyList_GET_ITEM(a[4], i), dev, &it.alpha_w))
                return none();
            out[i] = empty({m, w.n}, at::kBFloat16, dev);
            it.weight = w.handle;
            it.a = static_cast<const uint8_t*>(qa->const_data_ptr());
            it.sfa = static_cast<const uint8_t*>(sa->const_data_ptr());
            it.out_bf16 = out[i].mutable_data_ptr();
        }
        const cudaStream_t s = current_stream(dev);
        const int st = launch_on(dev, [&] { return nvfp4_gemm_launch_multi(items, static_cast<int>(count), m, s); });
        return st == NVFP4_OK ? tensor_list(out) : none();
    });
}

// linear_multi(variant, [x], fp8_max, lower, upper, [index of x], [weight], [vector of weight scales], [slot in it])
//   -> [bf16 [m, n_i]]: every activation quantized with its own global scale, then every product with it; codes, scales and
// global scales stay inside, in one workspace
PyObject* linear_multi(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        constexpr Py_ssize_t kMostActs = 16, kMost = 64;
        float fp8_max;
        int lower, upper;
        if (nargs != 9 || !PyList_CheckExact(a[1]) || !as_float(a[2], &fp8_max) || !window_int(a[3], &lower) || !window_int(a[4], &upper)) return none();
        for (int i = 5; i < 9; ++i)
            if (!PyList_CheckExact(a[i]) || PyList_GET_SIZE(a[i]) != PyList_GET_SIZE(a[5])) return none();
        const Py_ssize_t acts = PyList_GET_SIZE(a[1]), count = PyList_GET_SIZE(a[5]);
        if (acts < 1 || acts > kMostActs || count < 1 || count > kMost) return none();
        QuantIn q[kMostActs];
        int64_t at[kMostActs][2], bytes = 0;
        for (Py_ssize_t i = 0; i < acts; ++i) {
            if (!quant_input(PyList_GET_ITEM(a[1], i), Py_None, &q[i]) || q[i].device != q[0].device || q[i].dtype != q[0].dtype || q[i].m != q[0].m)
                return none();
            at[i][0] = bytes;
            at[i][1] = bytes += round_up(q[i].m * q[i].n / 2, 256);
            bytes += round_up(scale_bytes(q[i].m, q[i].n), 256);
        }
        const int64_t gs_at = bytes;
        const c10::DeviceIndex dev = q[0].device;
        const cudaStream_t s = current_stream(dev);
        const Tensor scratch = scratch_words(dev, s);
        if (!scratch.defined()) return none();
        nvfp4_gemm_item items[kMost];
        std::vector<Tensor> out(static_cast<size_t>(count));
        Tensor work = empty({gs_at + 256}, at::kByte, dev);
        uint8_t* base = static_cast<uint8_t*>(work.mutable_data_ptr());
        float* gs = reinterpret_cast<float*>(base + gs_at);
        for (Py_ssize_t i = 0; i < count; ++i) {
            int64_t x, slot;
            Weight w;
            const Tensor* vec = tensor_of(PyList_GET_ITEM(a[7], i));
            if (!int_or_none(PyList_GET_ITEM(a[5], i), -1, &x) || !int_or_none(PyList_GET_ITEM(a[8], i), -1, &slot) || x < 0 || x >= acts ||
                !weight_of(PyList_GET_ITEM(a[6], i), &w) || w.device != dev || w.k != q[x].n || w.k % 64 || !vec || !plain_cuda(*vec) ||
                vec->device().index() != dev || vec->scalar_type() != at::kFloat || !vec->is_contiguous() || slot < 0 || slot >= vec->numel()) {
                PyErr_Clear();
                return none();
            }
            out[i] = empty({q[0].m, w.n}, at::kBFloat16, dev);
            items[i] = {w.handle, base + at[x][0], base + at[x][1], gs + 2 * x, static_cast<const float*>(vec->const_data_ptr()) + slot,
                        out[i].mutable_data_ptr()};
        }
        nvfp4_chain_item chain[kMostActs];
        for (Py_ssize_t i = 0; i < acts; ++i)
            chain[i] = {q[i].x->const_data_ptr(), nullptr, gs + 2 * i, words_of(scratch) + 2 * i, base + at[i][0], base + at[i][1], q[i].m, q[i].n, q[i].n};
        const int variant = small_int(a[0]);
        const int st = launch_on(dev, [&] {
            const int c = nvfp4_quant_chain_multi_launch(variant, q[0].dtype, fp8_max, chain, static_cast<int>(acts), lower, upper, 1, s);
            return c != NVFP4_OK ? c : nvfp4_gemm_launch_multi(items, static_cast<int>(count), q[0].m, s);
        });
        return st == NVFP4_OK ? tensor_list(out) : none();
    });
}

// ---- preallocated decode blocks -------------------------------------------------------------------------------------
// What kernels/linear.py checks and builds once: addresses and sizes of buffers that the Python object owns and keeps.

struct Chain {   // global scale -> quantizer of an activation [m, n]
    int dtype, variant, lower, upper;
    c10::DeviceIndex device;
    float fp8_max;
    float* gs;
    uint32_t* scratch;
    uint8_t *codes, *scales;
    int64_t m, n;
};
struct Group {   // one activation against several prepared weights
    c10::DeviceIndex device;
    int64_t m, k;
    std::vector<void*> handles, outs;
    std::vector<const float*> alphas;
};
constexpr const char* kChainName = "nvfp4.chain";
constexpr const char* kGroupName = "nvfp4.group";

void free_chain(PyObject* c) { delete static_cast<Chain*>(PyCapsule_GetPointer(c, kChainName)); }
void free_group(PyObject* c) { delete static_cast<Group*>(PyCapsule_GetPointer(c, kGroupName)); }

// make_chain(dtype code, variant, device index, fp8_max, gs ptr, scratch ptr, codes ptr, scales ptr, m, n, lower, upper)
PyObject* make_chain(PyObject*, PyObject* args) {
    Chain c;
    int dev;
    Py_ssize_t gs, scratch, codes, scales, m, n;
    if (!PyArg_ParseTuple(args, "iiifnnnnnnii", &c.dtype, &c.variant, &dev, &c.fp8_max, &gs, &scratch, &codes, &scales, &m, &n, &c.lower, &c.upper))
        return nullptr;
    c.device = static_cast<c10::DeviceIndex>(dev);
    c.gs = reinterpret_cast<float*>(gs);
    c.scratch = reinterpret_cast<uint32_t*>(scratch);
    c.codes = reinterpret_cast<uint8_t*>(codes);
    c.scales = reinterpret_cast<uint8_t*>(scales);
    c.m = m;
    c.n = n;
    return PyCapsule_New(new Chain(c), kChainName, free_chain);
}

// make_group(device index, m, k, (handle, ...), (alpha ptr, ...), (out ptr, ...))
PyObject* make_group(PyObject*, PyObject* args) {
    int dev;
    Py_ssize_t m, k;
    PyObject *handles, *alphas, *outs;
    if (!PyArg_ParseTuple(args, "innO!O!O!", &dev, &m, &k, &PyTuple_Type, &handles, &PyTuple_Type, &alphas, &PyTuple_Type, &outs)) return nullptr;
    const Py_ssize_t n = PyTuple_GET_SIZE(handles);
    if (PyTuple_GET_SIZE(alphas) != n || PyTuple_GET_SIZE(outs) != n) {
        PyErr_SetString(PyExc_ValueError, "handles, alphas and outs must have the same length");
        return nullptr;
    }
    Group* g = new Group();
    g->device = static_cast<c10::DeviceIndex>(dev);
    g->m = m;
    g->k = k;
    for (Py_ssize_t i = 0; i < n; ++i) {
        g->handles.push_back(PyLong_AsVoidPtr(PyTuple_GET_ITEM(handles, i)));
        g->alphas.push_back(static_cast<const float*>(PyLong_AsVoidPtr(PyTuple_GET_ITEM(alphas, i))));
        g->outs.push_back(PyLong_AsVoidPtr(PyTuple_GET_ITEM(outs, i)));
    }
    if (PyErr_Occurred()) {
        delete g;
        return nullptr;
    }
    return PyCapsule_New(g, kGroupName, free_group);
}

bool chain_input(const Chain& c, const Tensor& x) {
    return plain_cuda(x) && x.device().index() == c.device && dtype_code(x.scalar_type()) == c.dtype && x.dim() == 2 && x.size(0) == c.m &&
           x.size(1) == c.n && x.is_contiguous() && aligned(x, 16);
}

// chain_call(chain, x) -> True
PyObject* chain_call(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 2) return none();
        const Chain* c = static_cast<const Chain*>(PyCapsule_GetPointer(a[0], kChainName));
        const Tensor* x = tensor_of(a[1]);
        if (!c || !x || !chain_input(*c, *x)) {
            PyErr_Clear();
            return none();
        }
        const cudaStream_t s = current_stream(c->device);
        const nvfp4_chain_item item = {x->const_data_ptr(), nullptr, c->gs, c->scratch, c->codes, c->scales, c->m, c->n, c->n};
        const int st = launch_on(c->device, [&] {   // products follow: the layer's form, see quant.cu
            return nvfp4_quant_chain_multi_launch(c->variant, c->dtype, c->fp8_max, &item, 1, c->lower, c->upper, 1, s);
        });
        return st == NVFP4_OK ? truth() : none();
    });
}

// group_call(group, codes, scales, alpha_a | None) -> True
PyObject* group_call(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        if (nargs != 4) return none();
        const Group* g = static_cast<const Group*>(PyCapsule_GetPointer(a[0], kGroupName));
        const Tensor *qa, *sa;
        const float* alpha_a = nullptr;
        if (!g || !quantized_operand(a[1], a[2], &qa, &sa) || qa->device().index() != g->device || qa->size(0) != g->m ||
            qa->size(1) * 2 != g->k || (a[3] != Py_None && !scalar_input(a[3], g->device, &alpha_a))) {
            PyErr_Clear();
            return none();
        }
        const cudaStream_t s = current_stream(g->device);
        const int st = launch_on(g->device, [&] {
            return nvfp4_gemm_launch_grouped(g->handles.data(), static_cast<int>(g->handles.size()), static_cast<const uint8_t*>(qa->const_data_ptr()),
                                             static_cast<const uint8_t*>(sa->const_data_ptr()), alpha_a, g->alphas.data(), g->outs.data(), g->m, s);
        });
        return st == NVFP4_OK ? truth() : none();
    });
}

// A layer whose activations are all at hand: their chains and every product, two to three launches from one call.
struct Program {
    std::vector<const Chain*> chains;
    std::vector<nvfp4_gemm_item> products;
    int64_t m;
};
constexpr const char* kProgramName = "nvfp4.program";
void free_program(PyObject* c) { delete static_cast<Program*>(PyCapsule_GetPointer(c, kProgramName)); }

// make_program((chain, ...), (index of the activation, ...), (group, ...)): the chains and groups stay the caller's and outlive it
PyObject* make_program(PyObject*, PyObject* args) {
    PyObject *chains, *index, *groups;
    if (!PyArg_ParseTuple(args, "O!O!O!", &PyTuple_Type, &chains, &PyTuple_Type, &index, &PyTuple_Type, &groups)) return nullptr;
    Program* p = new Program();
    bool ok = PyTuple_GET_SIZE(chains) > 0 && PyTuple_GET_SIZE(chains) <= 64 && PyTuple_GET_SIZE(index) == PyTuple_GET_SIZE(groups);
    for (Py_ssize_t i = 0; ok && i < PyTuple_GET_SIZE(chains); ++i) {
        const Chain* c = static_cast<const Chain*>(PyCapsule_GetPointer(PyTuple_GET_ITEM(chains, i), kChainName));
        const Chain* f = i > 0 ? p->chains[0] : c;
        ok = c && c->dtype == f->dtype && c->variant == f->variant && c->lower == f->lower && c->upper == f->upper && c->device == f->device &&
             c->fp8_max == f->fp8_max && c->m == f->m;
        p->chains.push_back(c);
    }
    for (Py_ssize_t i = 0; ok && i < PyTuple_GET_SIZE(groups); ++i) {
        const Group* g = static_cast<const Group*>(PyCapsule_GetPointer(PyTuple_GET_ITEM(groups, i), kGroupName));
        const Py_ssize_t at = PyLong_AsSsize_t(PyTuple_GET_ITEM(index, i));
        ok = g && at >= 0 && at < static_cast<Py_ssize_t>(p->chains.size()) && g->m == p->chains[at]->m && g->k == p->chains[at]->n &&
             g->device == p->chains[at]->device;
        for (size_t j = 0; ok && j < g->handles.size(); ++j)
            p->products.push_back({g->handles[j], p->chains[at]->codes, p->chains[at]->scales, p->chains[at]->gs, g->alphas[j], g->outs[j]});
    }
    if (!ok || p->products.empty() || p->products.size() > 64) {
        PyErr_Clear();
        delete p;
        return none();
    }
    p->m = p->chains[0]->m;
    return PyCapsule_New(p, kProgramName, free_program);
}

// program_call(program, x0, x1, ...) -> True
PyObject* program_call(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        const Program* p = nargs > 0 ? static_cast<const Program*>(PyCapsule_GetPointer(a[0], kProgramName)) : nullptr;
        if (!p || nargs != 1 + static_cast<Py_ssize_t>(p->chains.size())) {
            PyErr_Clear();
            return none();
        }
        nvfp4_chain_item items[64];
        const int n = static_cast<int>(p->chains.size());
        for (int i = 0; i < n; ++i) {
            const Chain* c = p->chains[i];
            const Tensor* x = tensor_of(a[1 + i]);
            if (!x || !chain_input(*c, *x)) return none();
            items[i] = {x->const_data_ptr(), nullptr, c->gs, c->scratch, c->codes, c->scales, c->m, c->n, c->n};
        }
        const Chain* c = p->chains[0];
        const cudaStream_t s = current_stream(c->device);
        const int st = launch_on(c->device, [&] {
            const int q = nvfp4_quant_chain_multi_launch(c->variant, c->dtype, c->fp8_max, items, n, c->lower, c->upper, 1, s);
            return q != NVFP4_OK ? q : nvfp4_gemm_launch_multi(p->products.data(), static_cast<int>(p->products.size()), p->m, s);
        });
        return st == NVFP4_OK ? truth() : none();
    });
}

// ---- pinned host memory in and out ----------------------------------------------------------------------------------
// What host_pipeline.HostQuantizer lays out once: row chunks, staging buffers and streams (the Python object's), and the
// events that order them (this object's).
struct HostPipe {
    c10::DeviceIndex device;
    int dtype, variant, lower, upper;
    int64_t rows, dim;
    std::vector<std::pair<int64_t, int64_t>> plan;
    std::vector<void*> in, codes, scales;      // `depth` staging slots
    cudaStream_t up, run, down;
    std::vector<cudaEvent_t> ev_up, ev_run, ev_down;
    std::vector<bool> used;                    // slot j's events have been recorded, by this call or an earlier one
    cudaEvent_t begin = nullptr, end_run = nullptr, end_down = nullptr;
    std::mutex mutex;                          // one call at a time: `used` and the events, which are queued without the interpreter lock
    ~HostPipe() {
        for (auto* v : {&ev_up, &ev_run, &ev_down})
            for (cudaEvent_t e : *v) cudaEventDestroy(e);
        for (cudaEvent_t e : {begin, end_run, end_down})
            if (e) cudaEventDestroy(e);
    }
};
constexpr const char* kHostPipeName = "nvfp4.host_pipe";
void free_host_pipe(PyObject* c) { delete static_cast<HostPipe*>(PyCapsule_GetPointer(c, kHostPipeName)); }

bool pointers(PyObject* t, std::vector<void*>* out) {
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(t); ++i) out->push_back(PyLong_AsVoidPtr(PyTuple_GET_ITEM(t, i)));
    return !PyErr_Occurred();
}

// make_host_pipe(device, dtype code, variant, lower, upper, rows, dim, (start, stop, start, stop, ...), (in ptr, ...),
//                (codes ptr, ...), (scales ptr, ...), up, run, down)
PyObject* make_host_pipe(PyObject*, PyObject* args) {
    int dev;
    Py_ssize_t rows, dim, up, run, down;
    PyObject *plan, *in, *codes, *scales;
    auto p = std::make_unique<HostPipe>();
    if (!PyArg_ParseTuple(args, "iiiiinnO!O!O!O!nnn", &dev, &p->dtype, &p->variant, &p->lower, &p->upper, &rows, &dim, &PyTuple_Type, &plan,
                          &PyTuple_Type, &in, &PyTuple_Type, &codes, &PyTuple_Type, &scales, &up, &run, &down))
        return nullptr;
    p->device = static_cast<c10::DeviceIndex>(dev);
    p->rows = rows;
    p->dim = dim;
    for (Py_ssize_t i = 0; i + 1 < PyTuple_GET_SIZE(plan); i += 2)
        p->plan.emplace_back(PyLong_AsLongLong(PyTuple_GET_ITEM(plan, i)), PyLong_AsLongLong(PyTuple_GET_ITEM(plan, i + 1)));
    if (!pointers(in, &p->in) || !pointers(codes, &p->codes) || !pointers(scales, &p->scales)) return nullptr;
    p->up = reinterpret_cast<cudaStream_t>(up);
    p->run = reinterpret_cast<cudaStream_t>(run);
    p->down = reinterpret_cast<cudaStream_t>(down);
    p->used.assign(p->in.size(), false);
    c10::cuda::CUDAGuard guard(p->device);
    auto event = [](cudaEvent_t* e) { return cudaEventCreateWithFlags(e, cudaEventDisableTiming) == cudaSuccess; };
    bool ok = event(&p->begin) && event(&p->end_run) && event(&p->end_down);
    for (auto* v : {&p->ev_up, &p->ev_run, &p->ev_down})
        for (size_t i = 0; ok && i < p->in.size(); ++i) {
            cudaEvent_t e = nullptr;
            ok = event(&e);
            if (ok) v->push_back(e);
        }
    if (!ok) {
        PyErr_SetString(PyExc_RuntimeError, "cudaEventCreate failed");
        return nullptr;
    }
    return PyCapsule_New(p.release(), kHostPipeName, free_host_pipe);
}

// Keeps a pinned block of torch's host allocator from being handed out again before `stream` is done with it.
inline void keep_pinned(const Tensor& t, cudaStream_t stream, c10::DeviceIndex device) {
    if (t.is_cuda() || !t.is_pinned()) return;
    at::getHostAllocator(at::kCUDA)->record_event(const_cast<void*>(t.const_data_ptr()), t.storage().data_ptr().get_context(),
                                                  c10::cuda::getStreamFromExternal(stream, device).unwrap());
}

cudaError_t host_pipe_run(HostPipe& p, const char* x, const float* gs_inv, const float* importance, char* codes, char* scales, cudaStream_t cur,
                          int* status) {
    const int64_t row_in = p.dim * (p.dtype == NVFP4_DT_F32 ? 4 : 2), row_codes = p.dim / 2, scale_row = round_up(p.dim / 16, 4);
    const size_t depth = p.in.size();
    cudaError_t e = cudaSuccess;
    auto ok = [&](cudaError_t r) {
        if (e == cudaSuccess) e = r;
        return e == cudaSuccess;
    };
    // One chunk has nothing to overlap: everything in order on the caller's stream, without the round trips between streams.
    const bool one = p.plan.size() == 1;
    const cudaStream_t up = one ? cur : p.up, run = one ? cur : p.run, down = one ? cur : p.down;
    if (!one && ok(cudaEventRecord(p.begin, cur)))
        for (cudaStream_t s : {up, run, down}) ok(cudaStreamWaitEvent(s, p.begin, 0));
    for (size_t i = 0; e == cudaSuccess && *status == NVFP4_OK && i < p.plan.size(); ++i) {
        const size_t j = i % depth;
        const int64_t a = p.plan[i].first, n = p.plan[i].second - a;
        if (p.used[j]) ok(cudaStreamWaitEvent(up, p.ev_run[j], 0));          // staging input free once its kernel ran
        ok(cudaMemcpyAsync(p.in[j], x + a * row_in, static_cast<size_t>(n * row_in), cudaMemcpyDefault, up));
        if (!one && ok(cudaEventRecord(p.ev_up[j], up))) ok(cudaStreamWaitEvent(run, p.ev_up[j], 0));
        if (p.used[j]) ok(cudaStreamWaitEvent(run, p.ev_down[j], 0));        // staging outputs free once downloaded
        if (e != cudaSuccess) break;
        *status = nvfp4_quant_launch(p.variant, p.in[j], p.dtype, importance, gs_inv, static_cast<uint8_t*>(p.codes[j]),
                                     static_cast<uint8_t*>(p.scales[j]), n, p.dim, p.dim, p.lower, p.upper, 1, run);
        if (*status != NVFP4_OK) break;
        if (ok(cudaEventRecord(p.ev_run[j], run)) && !one) ok(cudaStreamWaitEvent(down, p.ev_run[j], 0));
        ok(cudaMemcpyAsync(codes + a * row_codes, p.codes[j], static_cast<size_t>(n * row_codes), cudaMemcpyDefault, down));
        ok(cudaMemcpyAsync(scales + a * scale_row, p.scales[j], static_cast<size_t>(round_up(n, 128) * scale_row), cudaMemcpyDefault, down));
        ok(cudaEventRecord(p.ev_down[j], down));
        p.used[j] = true;
    }
    if (!one) {
        if (ok(cudaEventRecord(p.end_run, run))) ok(cudaStreamWaitEvent(cur, p.end_run, 0));
        if (ok(cudaEventRecord(p.end_down, down))) ok(cudaStreamWaitEvent(cur, p.end_down, 0));
    }
    return e;
}

// host_pipe_call(pipe, x, gs_inv, codes, scales, importance | None) -> True; the operands are checked by the caller except
// for what their addresses need
PyObject* host_pipe_call(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        HostPipe* p = nargs == 6 ? static_cast<HostPipe*>(PyCapsule_GetPointer(a[0], kHostPipeName)) : nullptr;
        const Tensor *x = tensor_of(a[1]), *codes = tensor_of(a[3]), *scales = tensor_of(a[4]);
        const float *gs_inv = nullptr, *importance = nullptr;
        if (!p || !x || !codes || !scales || !scalar_input(a[2], p->device, &gs_inv)) {
            PyErr_Clear();
            return none();
        }
        if (x->dim() != 2 || x->size(0) != p->rows || x->size(1) != p->dim || dtype_code(x->scalar_type()) != p->dtype || !x->is_contiguous() ||
            codes->scalar_type() != at::kByte || codes->dim() != 2 || codes->size(0) != p->rows || codes->size(1) != p->dim / 2 || !codes->is_contiguous() || !scales->is_contiguous() ||
            static_cast<int64_t>(scales->nbytes()) < round_up(p->rows, 128) * round_up(p->dim / 16, 4))
            return none();
        if (a[5] != Py_None) {
            const Tensor* w = tensor_of(a[5]);
            if (!w || !plain_cuda(*w) || w->device().index() != p->device || w->scalar_type() != at::kFloat || w->numel() != p->dim ||
                !w->is_contiguous() || !aligned(*w, 16))
                return none();
            importance = static_cast<const float*>(w->const_data_ptr());
        } else if (p->variant == NVFP4_VARIANT_WEIGHTED) {
            return none();
        }
        const cudaStream_t cur = current_stream(p->device);
        const bool one = p->plan.size() == 1;
        int status = NVFP4_OK;
        const int e = launch_on(p->device, [&] {
            const std::lock_guard<std::mutex> one_call(p->mutex);
            return static_cast<int>(host_pipe_run(*p, static_cast<const char*>(x->const_data_ptr()), gs_inv, importance,
                                                  static_cast<char*>(codes->mutable_data_ptr()), static_cast<char*>(scales->mutable_data_ptr()), cur, &status));
        });
        keep_pinned(*x, one ? cur : p->up, p->device);
        keep_pinned(*codes, one ? cur : p->down, p->device);
        keep_pinned(*scales, one ? cur : p->down, p->device);
        if (e != cudaSuccess || status != NVFP4_OK) {
            PyErr_Format(PyExc_RuntimeError, "host pipeline: %s", e != cudaSuccess ? cudaGetErrorString(static_cast<cudaError_t>(e)) : nvfp4_status_string(status));
            return nullptr;
        }
        return truth();
    });
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(name)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {
    FAST(quant_impl),
    FAST(quant_out),
    FAST(quant_dynamic),
    FAST(quant_dynamic_multi),
    FAST(global_scale),
    FAST(channel_square_norm),
    FAST(dequant),
    FAST(scale_layout),
    FAST(scaled_mm),
    FAST(scaled_mm_prepared),
    FAST(scaled_mm_grouped),
    FAST(scaled_mm_multi),
    FAST(linear_multi),
    FAST(chain_call),
    FAST(group_call),
    FAST(program_call),
    FAST(host_pipe_call),
    {"make_chain", make_chain, METH_VARARGS, nullptr},
    {"make_group", make_group, METH_VARARGS, nullptr},
    {"make_program", make_program, METH_VARARGS, nullptr},
    {"make_host_pipe", make_host_pipe, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
#undef FAST

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", "Host half of the entry points (None = not the common case).", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
    PyObject* nn = PyImport_ImportModule("torch.nn");
    if (!nn) return nullptr;
    PyObject* parameter = PyObject_GetAttrString(nn, "Parameter");
    Py_DECREF(nn);
    if (!parameter) return nullptr;
    g_parameter_type = reinterpret_cast<PyTypeObject*>(parameter);   // kept for the life of the process
    return PyModule_Create(&kModule);
}
