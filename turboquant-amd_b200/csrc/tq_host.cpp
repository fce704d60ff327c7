// Host path of the eager calls: argument checks, output allocation and launch in one native call.
//
// A decode step calls the library twice per layer with kernels of 5 to 15 us; the same work in Python (custom-op
// dispatch, a dozen tensor property reads, ctypes conversion) took 25 to 50 us per call and set the pace of every small
// launch.  Each function here takes the arguments of one entry point, checks them, and either launches and returns
// the result, or returns None ("declined") without having done anything.  The Python caller then takes its general
// path: the torch custom op, which is also what tracing, tensor subclasses, dispatch modes and autograd go through,
// and whose checks raise the errors.  So a condition below decides speed only, never results.
//
// The kernels stay in the C library; its launchers are looked up in the very file that Python loaded (bind()).
#include <Python.h>
#include <dlfcn.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/TracerMode.h>
#include <ATen/core/grad_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/tq_b200.h"

namespace {

struct Library {
    decltype(&tq_page_bytes) page_bytes;
    decltype(&tq_compress_paged) compress_paged;
    decltype(&tq_decode_workspace_bytes) decode_workspace_bytes;
    decltype(&tq_decode_auto_workspace_bytes) decode_auto_workspace_bytes;
    decltype(&tq_decode_paged) decode_paged;
    decltype(&tq_wht_rows) wht_rows;
    decltype(&tq_compress_k) compress_k;
    decltype(&tq_compress_v) compress_v;
    decltype(&tq_polarquant_compress) polarquant;
    decltype(&tq_packed_attention_workspace_bytes) attention_workspace_bytes;
    decltype(&tq_packed_attention) packed_attention;
};
Library L = {};

constexpr int kMaxDevices = 64;
int32_t* g_status[kMaxDevices] = {};   // device status words; the tensors are owned by the Python module for good

PyObject* declined() { Py_RETURN_NONE; }

// Inside torch.func transforms, __torch_dispatch__ and __torch_function__ modes and torch.jit.trace an operator call has to be
// seen by the dispatcher.
bool plain_eager() {
    if (c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled() || at::tracer::impl::is_dispatch_enabled())
        return false;
    return !c10::impl::tls_local_dispatch_key_set().included_.has_any(
        c10::DispatchKeySet({c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::Python}));
}

// The tensor behind obj when it is an ordinary dense CUDA tensor, else null.
const at::Tensor* cuda_tensor(PyObject* obj) {
    if (!THPVariable_CheckExact(obj)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(obj);
    if (!t.defined() || !t.is_cuda() || t.layout() != c10::kStrided || t.is_conj() || t.is_neg()) return nullptr;
    if (t.key_set().has(c10::DispatchKey::FuncTorchBatched) || t.key_set().has(c10::DispatchKey::FuncTorchGradWrapper)) return nullptr;
    return &t;
}

// N tensors at args[0 .. N), all on one device; false when one of them does not qualify.
template <int N>
bool tensors_on_one_device(PyObject* const* args, const at::Tensor* (&t)[N]) {
    bool grad = false;
    for (int i = 0; i < N; ++i) {
        t[i] = cuda_tensor(args[i]);
        if (!t[i] || t[i]->get_device() != t[0]->get_device()) return false;
        grad |= t[i]->requires_grad();
    }
    return !(grad && at::GradMode::is_enabled());
}

int dtype_code(const at::Tensor& t) {
    switch (t.scalar_type()) {
        case at::kHalf: return TQ_DTYPE_F16;
        case at::kBFloat16: return TQ_DTYPE_BF16;
        case at::kFloat: return TQ_DTYPE_F32;
        default: return -1;
    }
}

bool is_codebook(const at::Tensor& t, int64_t n) { return t.scalar_type() == at::kFloat && t.numel() == n && t.is_contiguous(); }

bool ints(PyObject* const* args, int n, long long* out) {
    for (int i = 0; i < n; ++i) {
        out[i] = PyLong_AsLongLong(args[i]);   // True and False included
        if (out[i] == -1 && PyErr_Occurred()) {
            PyErr_Clear();
            return false;
        }
    }
    return true;
}

bool floats(PyObject* const* args, int n, float* out) {
    for (int i = 0; i < n; ++i) {
        const double v = PyFloat_AsDouble(args[i]);
        if (v == -1.0 && PyErr_Occurred()) {
            PyErr_Clear();
            return false;
        }
        out[i] = static_cast<float>(v);
    }
    return true;
}

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const at::Device& dev) {
    return at::detail::empty_cuda(sizes, type, dev, std::nullopt);
}

tq_stream_t stream_of(const at::Device& dev) {
    return reinterpret_cast<tq_stream_t>(c10::cuda::getCurrentCUDAStream(dev.index()).stream());
}

// The launch itself runs without the interpreter lock: it blocks when the stream's launch queue is full.
template <typename F>
int launch(F f) {
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f();
    Py_END_ALLOW_THREADS
    return rc;
}

PyObject* failed(const char* what, int rc) {
    const char* why = rc == TQ_ERR_ARG ? "bad argument" : rc == TQ_ERR_UNSUPPORTED ? "unsupported configuration"
                    : rc == TQ_ERR_LAUNCH ? "CUDA launch failed" : rc == TQ_ERR_WORKSPACE ? "workspace too small" : "error";
    PyErr_Format(PyExc_RuntimeError, "%s failed: %s (status %d)", what, why, rc);
    return nullptr;
}

// decode(q, cache, block_tables, seq_lens, kc, vc, q_proj | None, out | None, skip_stats | None,
//        sm_scale, corr_scale, sparse_thresh, block_size, k_bits, v_bits, use_qjl, chunk_pages, io_flags, max_seq_len) -> out
PyObject* decode(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    const at::Tensor* t[6];
    float scale[3];
    long long v[7];
    if (nargs != 19 || !plain_eager() || !tensors_on_one_device(args, t) || !floats(args + 9, 3, scale) || !ints(args + 12, 7, v))
        return declined();
    const at::Tensor &cache = *t[1], &tables = *t[2], &lens = *t[3], &kc = *t[4], &vc = *t[5];
    const long long block_size = v[0], kb = v[1], vb = v[2], qjl = v[3] != 0, flags = v[5], max_len = v[6];
    const long long chunk = std::max(v[4], 0ll);
    const int dev = cache.get_device();
    if (dev >= kMaxDevices || !g_status[dev]) return declined();
    if (t[0]->dim() != 3 || t[0]->size(2) != 128 || t[0]->size(0) == 0) return declined();
    const int dtype = dtype_code(*t[0]);
    if (dtype != TQ_DTYPE_F16 && dtype != TQ_DTYPE_BF16) return declined();
    if (kb < 2 || kb > 4 || vb < 2 || vb > 4 || block_size < 16 || block_size % 16) return declined();
    const int64_t ns = t[0]->size(0), hq = t[0]->size(1), sub = block_size / 16;
    if (cache.scalar_type() != at::kByte || cache.dim() != 3 || !cache.is_contiguous()) return declined();
    const int64_t hkv = cache.size(1);
    if (hkv == 0 || hq == 0 || hq % hkv || cache.size(2) != sub * L.page_bytes(int(kb), int(vb), int(qjl))) return declined();
    if (tables.scalar_type() != at::kInt || tables.dim() != 2 || tables.size(0) < ns || tables.size(1) == 0 || tables.stride(1) != 1)
        return declined();
    if (lens.scalar_type() != at::kInt || !lens.is_contiguous() || lens.numel() < ns) return declined();
    if (!is_codebook(kc, 1ll << kb) || !is_codebook(vc, 1ll << vb)) return declined();
    const void *proj = nullptr, *stats = nullptr;
    void* out_ptr = nullptr;
    auto like_q = [&](PyObject* obj, void*& ptr) {
        const at::Tensor* x = cuda_tensor(obj);
        if (!x || x->get_device() != dev || x->sizes() != t[0]->sizes() || x->scalar_type() != t[0]->scalar_type() || !x->is_contiguous())
            return false;
        ptr = x->data_ptr();
        return true;
    };
    void* tmp = nullptr;
    if (args[6] != Py_None) {
        if (!like_q(args[6], tmp) || (at::GradMode::is_enabled() && THPVariable_Unpack(args[6]).requires_grad())) return declined();
        proj = tmp;
    }
    if (args[7] != Py_None && !like_q(args[7], out_ptr)) return declined();
    if (args[8] != Py_None) {
        const at::Tensor* x = cuda_tensor(args[8]);
        if (!x || x->get_device() != dev || x->element_size() != 4 || x->numel() < 2 || !x->is_contiguous()) return declined();
        stats = x->data_ptr();
    }
    int64_t pages = tables.size(1) * sub;
    if (max_len > 0) pages = std::min<int64_t>(pages, (max_len + 15) / 16);
    if (pages > INT32_MAX || ns > INT32_MAX) return declined();

    const at::Device device = cache.device();
    const c10::cuda::CUDAGuard guard(device);
    const at::Tensor q = t[0]->is_contiguous() ? *t[0] : t[0]->contiguous();
    at::Tensor out;
    if (!out_ptr) {
        out = empty(q.sizes(), q.scalar_type(), device);
        out_ptr = out.data_ptr();
    }
    // Split-K partials: a block of the caching allocator, held for this call only.  Its reuse is ordered by the
    // stream, so calls on other streams and threads never share it.
    const int64_t bytes = chunk > 0 ? L.decode_workspace_bytes(int(ns), int(hq), int(hkv), int(pages), int(chunk))
                                    : L.decode_auto_workspace_bytes(int(ns), int(hq), int(hkv), int(pages));
    if (bytes < 0) return failed("tq_decode_paged", int(bytes));
    at::DataPtr workspace = c10::cuda::CUDACachingAllocator::get()->allocate(bytes);
    const tq_stream_t stream = stream_of(device);
    const int rc = launch([&] {
        return L.decode_paged(out_ptr, q.data_ptr(), proj, dtype | int(flags), cache.data_ptr(), cache.size(0), int(block_size),
                              tables.data_ptr<int32_t>(), tables.stride(0), lens.data_ptr<int32_t>(), kc.data_ptr<float>(),
                              vc.data_ptr<float>(), scale[0], scale[1], scale[2], workspace.get(), bytes, g_status[dev],
                              static_cast<uint32_t*>(const_cast<void*>(stats)), int(ns), int(hq), int(hkv), int(pages), int(kb),
                              int(vb), int(qjl), int(chunk), stream);
    });
    if (rc != TQ_OK) return failed("tq_decode_paged", rc);
    if (out.defined()) return THPVariable_Wrap(std::move(out));
    Py_INCREF(args[7]);
    return args[7];
    END_HANDLE_TH_ERRORS
}

// compress_paged(key, value, cache, slot_mapping, kc, kb, vb, block_size, k_bits, v_bits, use_qjl, rotation_flags) -> True
PyObject* compress_paged(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    const at::Tensor* t[7];
    long long v[5];
    if (nargs != 12 || !plain_eager() || !tensors_on_one_device(args, t) || !ints(args + 7, 5, v)) return declined();
    const at::Tensor &key = *t[0], &value = *t[1], &cache = *t[2], &slots = *t[3];
    const long long block_size = v[0], kb = v[1], vb = v[2], qjl = v[3] != 0, flags = v[4];
    const int dev = key.get_device();
    if (dev >= kMaxDevices || !g_status[dev]) return declined();
    const int dtype = dtype_code(key);
    if (dtype < 0 || value.scalar_type() != key.scalar_type() || key.dim() != 3 || key.size(2) != 128 || value.sizes() != key.sizes() ||
        key.stride(2) != 1 || value.stride(2) != 1)
        return declined();
    if (kb < 2 || kb > 4 || vb < 2 || vb > 4 || block_size < 16 || block_size % 16) return declined();
    const int64_t T = key.size(0), H = key.size(1);
    if (T > INT32_MAX || H == 0) return declined();
    if (cache.scalar_type() != at::kByte || cache.dim() != 3 || !cache.is_contiguous() || cache.size(1) != H ||
        cache.size(2) != block_size / 16 * L.page_bytes(int(kb), int(vb), int(qjl)))
        return declined();
    if (slots.scalar_type() != at::kLong || slots.numel() < T || !slots.is_contiguous()) return declined();
    if (!is_codebook(*t[4], 1ll << kb) || !is_codebook(*t[5], (1ll << kb) - 1) || !is_codebook(*t[6], (1ll << vb) - 1)) return declined();
    const c10::cuda::CUDAGuard guard(key.device());
    const tq_stream_t stream = stream_of(key.device());
    const int rc = launch([&] {
        return L.compress_paged(key.data_ptr(), value.data_ptr(), dtype, key.stride(0), key.stride(1), value.stride(0), value.stride(1),
                                cache.data_ptr(), cache.size(0), int(block_size), slots.data_ptr<int64_t>(), t[4]->data_ptr<float>(),
                                t[5]->data_ptr<float>(), nullptr, t[6]->data_ptr<float>(), int(T), int(H), int(kb), int(vb), int(qjl),
                                int(flags), g_status[dev], stream);
    });
    if (rc != TQ_OK) return failed("tq_compress_paged", rc);
    if (!cache.is_inference()) cache.unsafeGetTensorImpl()->bump_version();   // written to, as the custom op's schema says
    Py_RETURN_TRUE;
    END_HANDLE_TH_ERRORS
}

// wht_rows(x, scale) -> x @ H * scale
PyObject* wht_rows(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    const at::Tensor* t[1];
    float scale[1];
    if (nargs != 2 || !plain_eager() || !tensors_on_one_device(args, t) || !floats(args + 1, 1, scale)) return declined();
    const int dtype = dtype_code(*t[0]);
    if (dtype < 0 || t[0]->dim() < 1 || t[0]->size(-1) != 128 || !t[0]->is_contiguous()) return declined();
    const c10::cuda::CUDAGuard guard(t[0]->device());
    at::Tensor out = empty(t[0]->sizes(), t[0]->scalar_type(), t[0]->device());
    const tq_stream_t stream = stream_of(t[0]->device());
    const int rc = launch([&] { return L.wht_rows(t[0]->data_ptr(), out.data_ptr(), dtype, out.numel() / 128, scale[0], stream); });
    if (rc != TQ_OK) return failed("tq_wht_rows", rc);
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// Rows [n, 128] and a codebook at args[0 .. 2]: (x, centroids, boundaries).  Returns the index width, or 0.
int rows_and_codebook(PyObject* const* args, const at::Tensor* (&t)[3]) {
    if (!plain_eager() || !tensors_on_one_device(args, t)) return 0;
    if (dtype_code(*t[0]) < 0 || t[0]->dim() != 2 || t[0]->size(1) != 128 || !t[0]->is_contiguous()) return 0;
    const int64_t n = t[1]->numel();
    const int bits = n == 4 ? 2 : n == 8 ? 3 : n == 16 ? 4 : 0;
    return bits && is_codebook(*t[1], n) && is_codebook(*t[2], n - 1) ? bits : 0;
}

// compress_k(K, centroids, boundaries, rotate, permute) -> (k_idx, k_signs, k_rnorm, k_norm)
PyObject* compress_k(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    const at::Tensor* t[3];
    long long v[2];
    int bits;
    if (nargs != 5 || !(bits = rows_and_codebook(args, t)) || !ints(args + 3, 2, v)) return declined();
    const at::Device dev = t[0]->device();
    const c10::cuda::CUDAGuard guard(dev);
    const int64_t n = t[0]->size(0);
    at::Tensor idx = empty({n, 16 * bits}, at::kByte, dev), signs = empty({n, 16}, at::kByte, dev);
    at::Tensor rnorm = empty({n}, at::kHalf, dev), norm = empty({n}, at::kHalf, dev);
    const tq_stream_t stream = stream_of(dev);
    const int rc = launch([&] {
        return L.compress_k(t[0]->data_ptr(), dtype_code(*t[0]), n, t[1]->data_ptr<float>(), t[2]->data_ptr<float>(), bits, !v[0],
                            v[1] != 0, idx.data_ptr<uint8_t>(), signs.data_ptr<uint8_t>(), rnorm.data_ptr(), norm.data_ptr(), stream);
    });
    if (rc != TQ_OK) return failed("tq_compress_k", rc);
    return Py_BuildValue("(NNNN)", THPVariable_Wrap(std::move(idx)), THPVariable_Wrap(std::move(signs)),
                         THPVariable_Wrap(std::move(rnorm)), THPVariable_Wrap(std::move(norm)));
    END_HANDLE_TH_ERRORS
}

// compress_v(V, centroids, boundaries, rotate) -> (v_idx, v_norm)
PyObject* compress_v(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    const at::Tensor* t[3];
    long long v[1];
    int bits;
    if (nargs != 4 || !(bits = rows_and_codebook(args, t)) || !ints(args + 3, 1, v)) return declined();
    const at::Device dev = t[0]->device();
    const c10::cuda::CUDAGuard guard(dev);
    const int64_t n = t[0]->size(0);
    at::Tensor idx = empty({n, 16 * bits}, at::kByte, dev), norm = empty({n}, at::kHalf, dev);
    const tq_stream_t stream = stream_of(dev);
    const int rc = launch([&] {
        return L.compress_v(t[0]->data_ptr(), dtype_code(*t[0]), n, t[2]->data_ptr<float>(), bits, !v[0], idx.data_ptr<uint8_t>(),
                            norm.data_ptr(), stream);
    });
    if (rc != TQ_OK) return failed("tq_compress_v", rc);
    return Py_BuildValue("(NN)", THPVariable_Wrap(std::move(idx)), THPVariable_Wrap(std::move(norm)));
    END_HANDLE_TH_ERRORS
}

// polarquant(x [n, 128], centroids, boundaries, bits, use_qjl, rotate)
//   -> (indices, norms, k_mse_rot) or, with use_qjl, (..., signs, rnorm)
PyObject* polarquant(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    const at::Tensor* t[3];
    long long v[3];
    if (nargs != 6 || !ints(args + 3, 3, v)) return declined();
    const int bits = rows_and_codebook(args, t);
    if (!bits || bits != v[0]) return declined();
    const bool qjl = v[1] != 0;
    const at::Device dev = t[0]->device();
    const c10::cuda::CUDAGuard guard(dev);
    const int64_t n = t[0]->size(0);
    at::Tensor indices = empty({n, 128}, at::kLong, dev), norms = empty({n}, at::kFloat, dev), mse = empty({n, 128}, at::kFloat, dev);
    at::Tensor signs, rnorm;
    if (qjl) {
        signs = empty({n, 128}, at::kFloat, dev);
        rnorm = empty({n}, at::kFloat, dev);
    }
    const tq_stream_t stream = stream_of(dev);
    const int rc = launch([&] {
        return L.polarquant(t[0]->data_ptr(), dtype_code(*t[0]), n, t[1]->data_ptr<float>(), t[2]->data_ptr<float>(), bits, qjl, !v[2],
                            indices.data_ptr<int64_t>(), norms.data_ptr<float>(), mse.data_ptr<float>(),
                            qjl ? signs.data_ptr<float>() : nullptr, qjl ? rnorm.data_ptr<float>() : nullptr, stream);
    });
    if (rc != TQ_OK) return failed("tq_polarquant_compress", rc);
    if (!qjl)
        return Py_BuildValue("(NNN)", THPVariable_Wrap(std::move(indices)), THPVariable_Wrap(std::move(norms)), THPVariable_Wrap(std::move(mse)));
    return Py_BuildValue("(NNNNN)", THPVariable_Wrap(std::move(indices)), THPVariable_Wrap(std::move(norms)), THPVariable_Wrap(std::move(mse)),
                         THPVariable_Wrap(std::move(signs)), THPVariable_Wrap(std::move(rnorm)));
    END_HANDLE_TH_ERRORS
}

// packed_attention(Q, Q_proj, k_idx, k_signs, k_rnorm, k_norm, v_idx, v_norm, centroids, corr_scale, num_splits) -> out
PyObject* packed_attention(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    const at::Tensor* t[9];
    float corr[1];
    long long splits;
    if (nargs != 11 || !plain_eager() || !tensors_on_one_device(args, t) || !floats(args + 9, 1, corr) || !ints(args + 10, 1, &splits))
        return declined();
    if (t[0]->dim() != 2 || t[0]->size(1) != 128 || t[4]->dim() != 2) return declined();
    const int64_t BH = t[0]->size(0), Sk = t[4]->size(1), n = t[8]->numel();
    const int bits = n == 4 ? 2 : n == 8 ? 3 : n == 16 ? 4 : 0;
    if (!bits || !is_codebook(*t[8], n) || BH == 0 || Sk == 0 || BH > INT32_MAX || Sk > INT32_MAX) return declined();
    const int64_t width[8] = {128, 128, 16 * bits, 16, 0, 0, 16 * bits, 0};
    for (int i = 0; i < 8; ++i) {
        const at::Tensor& x = *t[i];
        const bool bytes = i == 2 || i == 3 || i == 6;
        if (x.scalar_type() != (bytes ? at::kByte : at::kHalf) || !x.is_contiguous()) return declined();
        const bool fits = i < 2 ? x.dim() == 2 && x.size(0) == BH && x.size(1) == 128
                        : bytes ? x.dim() == 3 && x.size(0) == BH && x.size(1) == Sk && x.size(2) == width[i]
                                : x.dim() == 2 && x.size(0) == BH && x.size(1) == Sk;
        if (!fits) return declined();
        if (i == 0 && reinterpret_cast<uintptr_t>(x.const_data_ptr()) % 16) return declined();   // read 16 bytes at a time: to be copied
    }
    const at::Device dev = t[0]->device();
    const c10::cuda::CUDAGuard guard(dev);
    splits = std::max<long long>(0, std::min<long long>(splits, Sk));   // 0: the library shares the work out
    const int64_t bytes = L.attention_workspace_bytes(int(BH), int(splits));
    at::DataPtr workspace = c10::cuda::CUDACachingAllocator::get()->allocate(std::max<int64_t>(bytes, 16));   // this call's only
    at::Tensor out = empty({BH, 128}, at::kHalf, dev);
    const tq_stream_t stream = stream_of(dev);
    const int rc = launch([&] {
        return L.packed_attention(t[0]->data_ptr(), t[1]->data_ptr(), t[2]->data_ptr<uint8_t>(), t[3]->data_ptr<uint8_t>(), t[4]->data_ptr(),
                                  t[5]->data_ptr(), t[6]->data_ptr<uint8_t>(), t[7]->data_ptr(), t[8]->data_ptr<float>(), corr[0], int(BH),
                                  int(Sk), bits, int(splits), workspace.get(), std::max<int64_t>(bytes, 16), out.data_ptr(), stream);
    });
    if (rc != TQ_OK) return failed("tq_packed_attention", rc);
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// set_status(device index, int32 tensor that lives as long as the process)
PyObject* set_status(PyObject*, PyObject* args) {
    HANDLE_TH_ERRORS
    int dev;
    PyObject* obj;
    if (!PyArg_ParseTuple(args, "iO", &dev, &obj)) return nullptr;
    const at::Tensor* t = cuda_tensor(obj);
    if (!t || t->scalar_type() != at::kInt || dev < 0 || t->get_device() != dev) {
        PyErr_SetString(PyExc_ValueError, "set_status: int32 CUDA tensor on that device");
        return nullptr;
    }
    if (dev < kMaxDevices) g_status[dev] = t->data_ptr<int32_t>();
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// bind(path): take the launchers from the library at path (already loaded by the caller)
PyObject* bind(PyObject*, PyObject* args) {
    const char* path;
    if (!PyArg_ParseTuple(args, "s", &path)) return nullptr;
    void* h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
    if (!h) {
        PyErr_SetString(PyExc_RuntimeError, dlerror());
        return nullptr;
    }
    bool ok = true;
    auto take = [&](auto& f, const char* name) {
        f = reinterpret_cast<std::remove_reference_t<decltype(f)>>(dlsym(h, name));
        ok = ok && f;
    };
    take(L.page_bytes, "tq_page_bytes");
    take(L.compress_paged, "tq_compress_paged");
    take(L.decode_workspace_bytes, "tq_decode_workspace_bytes");
    take(L.decode_auto_workspace_bytes, "tq_decode_auto_workspace_bytes");
    take(L.decode_paged, "tq_decode_paged");
    take(L.wht_rows, "tq_wht_rows");
    take(L.compress_k, "tq_compress_k");
    take(L.compress_v, "tq_compress_v");
    take(L.polarquant, "tq_polarquant_compress");
    take(L.attention_workspace_bytes, "tq_packed_attention_workspace_bytes");
    take(L.packed_attention, "tq_packed_attention");
    if (!ok) {
        PyErr_Format(PyExc_RuntimeError, "%s lacks a tq_* entry point", path);
        return nullptr;
    }
    Py_RETURN_NONE;
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyCFunction fast() { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(F)); }

PyMethodDef kMethods[] = {
    {"decode", fast<decode>(), METH_FASTCALL, nullptr},
    {"compress_paged", fast<compress_paged>(), METH_FASTCALL, nullptr},
    {"wht_rows", fast<wht_rows>(), METH_FASTCALL, nullptr},
    {"compress_k", fast<compress_k>(), METH_FASTCALL, nullptr},
    {"compress_v", fast<compress_v>(), METH_FASTCALL, nullptr},
    {"polarquant", fast<polarquant>(), METH_FASTCALL, nullptr},
    {"packed_attention", fast<packed_attention>(), METH_FASTCALL, nullptr},
    {"set_status", set_status, METH_VARARGS, nullptr},
    {"bind", bind, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_tq_host", "Native host path of the eager TurboQuant calls.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__tq_host(void) { return PyModule_Create(&kModule); }
