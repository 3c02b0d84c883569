// Python binding of the calls a serving loop makes once per layer and step (module _fp8host).
//
// The kernels stay behind the C ABI (include/fp8lin.h); this file only replaces the interpreter work around it.  A
// decode-sized linear runs 4 to 20 us on the GPU, and the same call made through ctypes from Python (shape and type
// checks, allocation, two foreign calls with a dozen converted arguments each) kept the host busy for 28 us, so an
// eager decode loop was bound by the interpreter.  Here a call checks its tensors through their TensorImpl, takes the
// result from torch's caching allocator, looks the stream's scratch up and launches; the interpreter lock is released
// around the launch, as ctypes does, because a launch may block on a full queue.
//
// Functions take positional arguments only (METH_FASTCALL) and None for an absent tensor.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdio>
#include <map>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/fp8lin.h"

namespace {

struct ValueError : std::runtime_error { using std::runtime_error::runtime_error; };

// ---- arguments ---------------------------------------------------------------------------------------------------

const at::Tensor& tensor(PyObject* o, const char* what) {
    if (!THPVariable_Check(o)) throw ValueError(std::string(what) + " must be a tensor");
    return THPVariable_Unpack(o);
}

// nullptr for None
const at::Tensor* optional_tensor(PyObject* o, const char* what) {
    return o == Py_None ? nullptr : &tensor(o, what);
}

void need_cuda(const at::Tensor& t) {
    if (!t.is_cuda()) throw ValueError("fp8lin kernels need CUDA tensors (there is no CPU path)");
}

// ---- scratch: one zero-initialised buffer per (device, stream), grown on demand ------------------------------------
// An outgrown buffer is kept (a captured CUDA graph has its address baked in) until release().
// Every buffer of a stream names the same pinned word, where a kernel that gives up a wait leaves its code: the next call on
// the stream sees it and raises, at the cost of a load from host memory.

struct StreamScratch {
    at::Tensor buffer;
    at::Tensor gave_up;          // pinned int
    volatile int* word = nullptr;        // ... its address
};
struct Scratch {
    std::mutex lock;
    std::map<std::pair<int, void*>, StreamScratch> live;
    std::vector<at::Tensor> retired;
};
constexpr int64_t kHostWordAt = 8;           // byte of the header that names the host's word
Scratch& scratch() { static Scratch* s = new Scratch; return *s; }      // (outlives the CUDA context's teardown)

// A kernel of an earlier call on this stream gave up a wait: forgets it and raises.
[[noreturn]] void raise_given_up(StreamScratch& e) {
    const int code = *e.word;
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None) {
        *e.word = 0;
        const c10::InferenceMode any_tensor(true);      // (the buffer may have been made in inference mode)
        e.buffer.narrow(0, 0, (int64_t)sizeof(int)).zero_();
    }
    char hex[16];
    snprintf(hex, sizeof(hex), "0x%x", code);
    throw std::runtime_error(std::string("a kernel of an earlier call on this stream gave up a bounded wait (device status ") + hex +
                             "): the result of that call is not valid");
}

at::Tensor workspace(c10::cuda::CUDAStream stream, size_t nbytes, bool raise = true) {
    Scratch& s = scratch();
    const auto key = std::make_pair((int)stream.device_index(), (void*)stream.stream());
    std::lock_guard<std::mutex> guard(s.lock);
    auto it = s.live.find(key);
    if (it != s.live.end()) {
        if (raise && *it->second.word != 0) raise_given_up(it->second);
        if ((size_t)it->second.buffer.numel() >= nbytes) return it->second.buffer;
    }
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None)
        throw std::runtime_error("fp8lin scratch for this stream must grow to " + std::to_string(nbytes) +
                                 " bytes during a CUDA graph capture; run the shape once (or call reserve_workspace) on "
                                 "the capturing stream before the capture");
    size_t size = nbytes < (size_t)FP8LIN_WS_HEADER_BYTES ? (size_t)FP8LIN_WS_HEADER_BYTES : nbytes;
    if (it != s.live.end()) {
        const size_t old = (size_t)it->second.buffer.numel();
        if (size < 2 * old) size = 2 * old;
    }
    StreamScratch fresh;
    fresh.buffer = at::zeros({(int64_t)size}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, stream.device_index()));
    fresh.gave_up = it != s.live.end() ? it->second.gave_up : at::zeros({1}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    fresh.word = fresh.gave_up.mutable_data_ptr<int>();
    fresh.buffer.narrow(0, kHostWordAt, (int64_t)sizeof(int64_t)).view(at::kLong).fill_((int64_t)(intptr_t)fresh.word);
    if (it != s.live.end()) s.retired.push_back(it->second.buffer);
    s.live[key] = fresh;
    return fresh.buffer;
}

// ---- running one call of the library ---------------------------------------------------------------------------------

void check(int rc, const char* what) {
    if (rc == FP8LIN_OK) return;
    const std::string msg = std::string(what) + ": " + fp8lin_last_error() + " (fp8lin status " + std::to_string(rc) + ")";
    if (rc == FP8LIN_ERR_NULL || rc == FP8LIN_ERR_SHAPE || rc == FP8LIN_ERR_ALIGN || rc == FP8LIN_ERR_ARG) throw ValueError(msg);
    throw std::runtime_error(msg);
}

template <class F>
int unlocked(F&& f) {
    PyThreadState* st = PyEval_SaveThread();
    const int rc = f();
    PyEval_RestoreThread(st);
    return rc;
}

PyObject* g_out_of_memory = nullptr;         // torch.OutOfMemoryError

template <class F>
PyObject* guarded(F&& f) {
    try {
        return f();
    } catch (const ValueError& e) {
        PyErr_SetString(PyExc_ValueError, e.what());
    } catch (const c10::OutOfMemoryError& e) {
        PyErr_SetString(g_out_of_memory ? g_out_of_memory : PyExc_RuntimeError, e.what_without_backtrace());
    } catch (const c10::Error& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

// Rows of a [.., K] tensor as a matrix with one row pitch: a view where the strides allow it, else a copy.
struct Rows {
    at::Tensor t;           // owner
    int64_t m, k, ld;
};
Rows rows_of(const at::Tensor& x) {
    const int64_t d = x.dim();
    if (d == 2 && x.stride(1) == 1) return {x, x.size(0), x.size(1), x.stride(0)};
    if (d < 1) throw ValueError("activations need at least one dimension");
    const int64_t k = x.size(d - 1);
    at::Tensor t = x.is_contiguous() ? x : x.reshape({-1, k});
    if (!x.is_contiguous()) {
        if (t.stride(1) != 1) t = t.contiguous();
        return {t, t.size(0), k, t.stride(0)};
    }
    int64_t m = 1;
    for (int64_t i = 0; i + 1 < d; ++i) m *= x.size(i);
    return {t, m, k, k};
}

// A result tensor straight from the CUDA allocator (the dispatcher's way to the same function costs half a microsecond).
at::Tensor empty(at::IntArrayRef shape, at::ScalarType dtype, c10::Device device) {
    return at::detail::empty_cuda(shape, dtype, device, c10::nullopt);
}

at::Tensor empty_like_rows(const at::Tensor& x, int64_t n, at::ScalarType dtype) {
    if (x.dim() == 2) {
        const int64_t shape[2] = {x.size(0), n};
        return empty(shape, dtype, x.device());
    }
    std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = n;
    return empty(shape, dtype, x.device());
}

void check_weight(const at::Tensor& w, const at::Tensor& w_scale, const at::Tensor* bias, int64_t k) {
    need_cuda(w);
    need_cuda(w_scale);
    if (w.scalar_type() != at::kByte || w.dim() != 1 || !w.is_contiguous())
        throw ValueError("w_packed must be the flat uint8 buffer made by prepack_weight / pack_weight_nk");
    if (w_scale.scalar_type() != at::kFloat || w_scale.dim() != 1)
        throw ValueError("weight_scale must be float32 with one value per output channel");
    const int64_t n = w_scale.numel();
    if (k % 16 != 0 || (size_t)w.numel() != fp8lin_packed_bytes(k, n))
        throw ValueError("x has K=" + std::to_string(k) + ", weight_scale has N=" + std::to_string(n) + ", but the packed weight holds " +
                         std::to_string(w.numel()) + " bytes (expected " +
                         (k % 16 == 0 ? std::to_string(fp8lin_packed_bytes(k, n)) : std::string("K % 16 == 0")) + ")");
    if (bias) {
        need_cuda(*bias);
        if (bias->scalar_type() != at::kBFloat16 || bias->numel() != n) throw ValueError("bias must be bfloat16 [N]");
    }
}

void check_scale(const at::Tensor& s, const char* what) {
    need_cuda(s);
    if (s.scalar_type() != at::kFloat || s.numel() != 1) throw ValueError(std::string(what) + " must be one float32 value on the device");
}

inline const void* ptr(const at::Tensor* t) { return t ? t->const_data_ptr() : nullptr; }

void need_args(Py_ssize_t got, Py_ssize_t want, const char* fn) {
    if (got != want) throw std::runtime_error(std::string(fn) + ": wrong number of arguments");
}

struct Out {
    at::Tensor t;
    int64_t ld;
};
// The caller's output matrix, or a new tensor with x's leading dimensions.
Out output_for(const at::Tensor& x, int64_t m, int64_t n, const at::Tensor* out) {
    if (!out) return {empty_like_rows(x, n, at::kBFloat16), n};
    need_cuda(*out);
    if (out->scalar_type() != at::kBFloat16 || out->dim() != 2 || out->size(0) != m || out->size(1) != n || (n > 1 && out->stride(1) != 1))
        throw ValueError("out must be a bfloat16 matrix [M, N] with contiguous rows");
    return {*out, m > 1 ? out->stride(0) : (out->stride(0) > n ? out->stride(0) : n)};
}

// ---- module functions -------------------------------------------------------------------------------------------------

// linear(scheme, x, w_packed, weight_scale, input_scale | None, bias | None, out | None) -> y [.., N]
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&]() -> PyObject* {
        need_args(na, 7, "linear");
        const long scheme = PyLong_AsLong(a[0]);
        const at::Tensor& x0 = tensor(a[1], "x");
        const at::Tensor& w = tensor(a[2], "w_packed");
        const at::Tensor& ws = tensor(a[3], "weight_scale");
        const at::Tensor* is = optional_tensor(a[4], "input_scale");
        const at::Tensor* bias = optional_tensor(a[5], "bias");
        const at::Tensor* out = optional_tensor(a[6], "out");
        need_cuda(x0);
        const bool bf16 = x0.scalar_type() == at::kBFloat16;
        const at::Tensor xb = bf16 ? x0 : x0.to(at::kBFloat16);
        at::Tensor bias_bf16;
        if (bias && bias->scalar_type() != at::kBFloat16) {
            bias_bf16 = bias->to(at::kBFloat16);
            bias = &bias_bf16;
        }
        const Rows r = rows_of(xb);
        check_weight(w, ws, bias, r.k);
        const int64_t n = ws.numel();
        const bool w8a8 = scheme == FP8LIN_W8A8_STATIC;
        if (w8a8) {
            if (!is) throw ValueError("input_scale must be one float32 value on the device");
            check_scale(*is, "input_scale");
        }
        const c10::cuda::CUDAGuard device(x0.device());
        const Out y = output_for(xb, r.m, n, out);
        const auto stream = c10::cuda::getCurrentCUDAStream();
        const at::Tensor scr = workspace(stream, fp8lin_workspace_bytes((int)scheme, r.m, r.k, n));
        const int rc = unlocked([&] {
            return w8a8 ? fp8lin_w8a8(r.t.const_data_ptr(), r.ld, w.const_data_ptr(), (const float*)ws.const_data_ptr(),
                                      (const float*)is->const_data_ptr(), ptr(bias), y.t.mutable_data_ptr(), y.ld, r.m, r.k, n,
                                      scr.mutable_data_ptr(), (size_t)scr.numel(), stream.stream())
                        : fp8lin_w8a16(r.t.const_data_ptr(), r.ld, w.const_data_ptr(), (const float*)ws.const_data_ptr(), ptr(bias),
                                       y.t.mutable_data_ptr(), y.ld, r.m, r.k, n, scr.mutable_data_ptr(), (size_t)scr.numel(),
                                       stream.stream());
        });
        check(rc, w8a8 ? "fp8lin_w8a8" : "fp8lin_w8a16");
        if (!bf16 && !out) return THPVariable_Wrap(y.t.to(x0.scalar_type()));
        return THPVariable_Wrap(y.t);
    });
}

// linear_codes(xq, w_packed, weight_scale, input_scale, bias | None, out | None) -> y [.., N]
PyObject* py_linear_codes(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&]() -> PyObject* {
        need_args(na, 6, "linear_codes");
        const at::Tensor& xq = tensor(a[0], "xq");
        const at::Tensor& w = tensor(a[1], "w_packed");
        const at::Tensor& ws = tensor(a[2], "weight_scale");
        const at::Tensor& is = tensor(a[3], "input_scale");
        const at::Tensor* bias = optional_tensor(a[4], "bias");
        const at::Tensor* out = optional_tensor(a[5], "out");
        need_cuda(xq);
        if (xq.scalar_type() != at::kByte || xq.dim() < 1 || !xq.is_contiguous())
            throw ValueError("xq must be a contiguous 2-D uint8 tensor of e4m3 codes [M, K]");
        at::Tensor bias_bf16;
        if (bias && bias->scalar_type() != at::kBFloat16) {
            bias_bf16 = bias->to(at::kBFloat16);
            bias = &bias_bf16;
        }
        const Rows r = rows_of(xq);
        check_weight(w, ws, bias, r.k);
        check_scale(is, "input_scale");
        const int64_t n = ws.numel();
        const c10::cuda::CUDAGuard device(xq.device());
        const Out y = output_for(xq, r.m, n, out);
        const auto stream = c10::cuda::getCurrentCUDAStream();
        const at::Tensor scr = workspace(stream, fp8lin_workspace_bytes(FP8LIN_W8A8_STATIC, r.m, r.k, n));
        const int rc = unlocked([&] {
            return fp8lin_w8a8_preq(r.t.const_data_ptr(), w.const_data_ptr(), (const float*)ws.const_data_ptr(),
                                    (const float*)is.const_data_ptr(), ptr(bias), y.t.mutable_data_ptr(), y.ld, r.m, r.k, n,
                                    scr.mutable_data_ptr(), (size_t)scr.numel(), stream.stream());
        });
        check(rc, "fp8lin_w8a8_preq");
        return THPVariable_Wrap(y.t);
    });
}

// rmsnorm_quant(x, weight, eps, input_scale | None, residual | None, want_bf16, xq_out | None, y_out | None) -> (xq | None, y | None)
PyObject* py_rmsnorm_quant(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&]() -> PyObject* {
        need_args(na, 8, "rmsnorm_quant");
        const at::Tensor& x = tensor(a[0], "x");
        const at::Tensor& w0 = tensor(a[1], "weight");
        const double eps = PyFloat_AsDouble(a[2]);
        const at::Tensor* is = optional_tensor(a[3], "input_scale");
        const at::Tensor* res = optional_tensor(a[4], "residual");
        const bool want_bf16 = a[5] == Py_True;
        const at::Tensor* xq_out = optional_tensor(a[6], "xq_out");
        const at::Tensor* y_out = optional_tensor(a[7], "y_out");
        need_cuda(x);
        if (x.scalar_type() != at::kBFloat16) throw ValueError("x must be a 2-D bfloat16 tensor and weight a bfloat16 vector");
        if (is) need_cuda(*is);
        const Rows r = rows_of(x);
        at::Tensor w = w0;
        if (w.scalar_type() != at::kBFloat16 || w.device() != x.device()) w = w.detach().to(x.device(), at::kBFloat16);
        if (!w.is_contiguous()) w = w.contiguous();
        if (w.numel() != r.k) throw ValueError("weight must be a contiguous vector of H elements");
        int64_t ld_res = 0;
        if (res) {
            need_cuda(*res);
            const int64_t d = res->dim();
            if (res->scalar_type() != at::kBFloat16 || res->sizes() != x.sizes() || (res->stride(d - 1) != 1 && r.k > 1) ||
                (d != 2 && !res->is_contiguous()))
                throw ValueError("residual must be a bfloat16 tensor of x's shape with contiguous rows (it is updated in place)");
            ld_res = d == 2 ? res->stride(0) : r.k;
        }
        const c10::cuda::CUDAGuard device(x.device());
        at::Tensor xq, y;
        int64_t ldy = 0;
        if (is) xq = xq_out ? *xq_out : empty_like_rows(x, r.k, at::kByte);
        if (want_bf16 || !is) {
            y = y_out ? *y_out : empty_like_rows(x, r.k, at::kBFloat16);
            ldy = y.dim() == 2 ? y.stride(0) : r.k;
        }
        const auto stream = c10::cuda::getCurrentCUDAStream();
        const int rc = unlocked([&] {
            return fp8lin_rmsnorm_quant(r.t.const_data_ptr(), r.ld, res ? res->mutable_data_ptr() : nullptr, ld_res, w.const_data_ptr(),
                                        (float)eps, (const float*)ptr(is), xq.defined() ? xq.mutable_data_ptr() : nullptr,
                                        y.defined() ? y.mutable_data_ptr() : nullptr, ldy, r.m, r.k, stream.stream());
        });
        check(rc, "fp8lin_rmsnorm_quant");
        PyObject* t = PyTuple_New(2);
        if (!t) return nullptr;
        PyTuple_SET_ITEM(t, 0, xq.defined() ? THPVariable_Wrap(xq) : Py_NewRef(Py_None));
        PyTuple_SET_ITEM(t, 1, y.defined() ? THPVariable_Wrap(y) : Py_NewRef(Py_None));
        return t;
    });
}

// mlp(x bf16 or codes, w_gate_up, gate_up_scale, gate_up_input_scale, gate_up_bias | None, w_down, down_scale, down_input_scale,
//     down_bias | None, out | None) -> y [.., N]
PyObject* py_mlp(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&]() -> PyObject* {
        need_args(na, 10, "mlp");
        const at::Tensor& x = tensor(a[0], "x");
        const at::Tensor& wg = tensor(a[1], "w_gate_up");
        const at::Tensor& gs = tensor(a[2], "gate_up_scale");
        const at::Tensor& gi = tensor(a[3], "gate_up_input_scale");
        const at::Tensor* gb = optional_tensor(a[4], "gate_up_bias");
        const at::Tensor& wd = tensor(a[5], "w_down");
        const at::Tensor& ds = tensor(a[6], "down_scale");
        const at::Tensor& di = tensor(a[7], "down_input_scale");
        const at::Tensor* db = optional_tensor(a[8], "down_bias");
        const at::Tensor* out = optional_tensor(a[9], "out");
        need_cuda(x);
        const bool codes = x.scalar_type() == at::kByte;
        if (codes && !x.is_contiguous()) throw ValueError("pre-quantised activations must be a contiguous 2-D uint8 CUDA tensor");
        if (!codes && x.scalar_type() != at::kBFloat16) throw ValueError("x must be a 2-D bfloat16 tensor [M, K]");
        const Rows r = rows_of(x);
        check_weight(wg, gs, gb, r.k);
        const int64_t inter = gs.numel() / 2, n = ds.numel();
        need_cuda(wd);
        need_cuda(ds);
        check_scale(gi, "gate_up_input_scale");
        check_scale(di, "down_input_scale");
        if ((size_t)wd.numel() != fp8lin_packed_bytes(inter, n)) throw ValueError("w_down does not match the intermediate size of the gate_up weight");
        if (db && (db->scalar_type() != at::kBFloat16 || db->numel() != n)) throw ValueError("down_bias must be bf16 [N]");
        const c10::cuda::CUDAGuard device(x.device());
        const Out y = output_for(x, r.m, n, out);
        const auto stream = c10::cuda::getCurrentCUDAStream();
        const at::Tensor scr = workspace(stream, fp8lin_mlp_workspace_bytes(r.m, r.k, inter, n));
        const int rc = unlocked([&] {
            if (codes)
                return fp8lin_mlp_w8a8_preq(r.t.const_data_ptr(), wg.const_data_ptr(), (const float*)gs.const_data_ptr(),
                                            (const float*)gi.const_data_ptr(), ptr(gb), wd.const_data_ptr(),
                                            (const float*)ds.const_data_ptr(), (const float*)di.const_data_ptr(), ptr(db),
                                            y.t.mutable_data_ptr(), y.ld, r.m, r.k, inter, n, scr.mutable_data_ptr(),
                                            (size_t)scr.numel(), stream.stream());
            return fp8lin_mlp_w8a8(r.t.const_data_ptr(), r.ld, wg.const_data_ptr(), (const float*)gs.const_data_ptr(),
                                   (const float*)gi.const_data_ptr(), ptr(gb), wd.const_data_ptr(), (const float*)ds.const_data_ptr(),
                                   (const float*)di.const_data_ptr(), ptr(db), y.t.mutable_data_ptr(), y.ld, r.m, r.k, inter, n,
                                   scr.mutable_data_ptr(), (size_t)scr.numel(), stream.stream());
        });
        check(rc, codes ? "fp8lin_mlp_w8a8_preq" : "fp8lin_mlp_w8a8");
        return THPVariable_Wrap(y.t);
    });
}

// moe_route(logits, top_k, renormalize) -> (weights f32 [T, k], ids i64 [T, k])
PyObject* py_moe_route(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&]() -> PyObject* {
        need_args(na, 3, "moe_route");
        const at::Tensor& l0 = tensor(a[0], "router_logits");
        const int64_t k = PyLong_AsLongLong(a[1]);
        const int renormalize = PyObject_IsTrue(a[2]);
        if (!l0.is_cuda()) throw ValueError("the router kernel needs CUDA tensors (there is no CPU path)");
        if (l0.dim() != 2 || (l0.scalar_type() != at::kFloat && l0.scalar_type() != at::kBFloat16))
            throw ValueError("router_logits must be [T, E] float32 or bfloat16");
        const at::Tensor l = l0.stride(1) == 1 ? l0 : l0.contiguous();
        const int64_t t = l.size(0), e = l.size(1);
        const c10::cuda::CUDAGuard device(l.device());
        const at::Tensor w = empty({t, k}, at::kFloat, l.device());
        const at::Tensor ids = empty({t, k}, at::kLong, l.device());
        const auto stream = c10::cuda::getCurrentCUDAStream();
        const int rc = unlocked([&] {
            return fp8lin_moe_route_i64(l.const_data_ptr(), l.scalar_type() == at::kBFloat16 ? 1 : 0, l.stride(0), t, (int)e, (int)k, renormalize,
                                        (float*)w.mutable_data_ptr(), (int64_t*)ids.mutable_data_ptr(), stream.stream());
        });
        check(rc, "fp8lin_moe_route");
        PyObject* r = PyTuple_New(2);
        if (!r) return nullptr;
        PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(w));
        PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(ids));
        return r;
    });
}

// moe_block(x, topk_weights [T, k], topk_ids [T, k], w13, w13_scale, w13_input_scale, w2, w2_scale, w2_input_scale, experts, inter) -> y [T, H]
PyObject* py_moe_block(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&]() -> PyObject* {
        need_args(na, 11, "moe_block");
        const at::Tensor& x = tensor(a[0], "x");
        const at::Tensor& w0 = tensor(a[1], "topk_weights");
        const at::Tensor& i0 = tensor(a[2], "topk_ids");
        const at::Tensor* wt[6];
        for (int i = 0; i < 6; ++i) { wt[i] = &tensor(a[3 + i], "expert weights"); need_cuda(*wt[i]); }
        const int64_t experts = PyLong_AsLongLong(a[9]), inter = PyLong_AsLongLong(a[10]);
        if (!x.is_cuda()) throw ValueError("the expert kernels need CUDA tensors (there is no CPU path)");
        if (x.scalar_type() != at::kBFloat16 || x.dim() != 2) throw ValueError("x must be a bfloat16 matrix [T, H]");
        need_cuda(w0);
        need_cuda(i0);
        const Rows r = rows_of(x);
        if (i0.dim() != 2 || i0.size(0) != r.m || w0.sizes() != i0.sizes()) throw ValueError("topk_weights and topk_ids must be [T, k]");
        const int64_t k = i0.size(1);
        const bool i64 = i0.scalar_type() == at::kLong;
        const at::Tensor ids = i64 ? i0.contiguous() : i0.to(at::kInt).contiguous();
        const at::Tensor w = w0.to(at::kFloat).contiguous();
        if ((size_t)wt[0]->numel() != (size_t)experts * fp8lin_packed_bytes(r.k, 2 * inter) ||
            (size_t)wt[3]->numel() != (size_t)experts * fp8lin_packed_bytes(inter, r.k))
            throw ValueError("the packed expert weights do not match the number of experts, x's width and the intermediate size");
        const c10::cuda::CUDAGuard device(x.device());
        const at::Tensor y = empty({r.m, r.k}, at::kBFloat16, x.device());
        const auto stream = c10::cuda::getCurrentCUDAStream();
        const at::Tensor scr = workspace(stream, fp8lin_moe_block_workspace_bytes(r.m, (int)k, (int)experts, r.k, inter));
        auto f = [&](int i) { return (const float*)wt[i]->const_data_ptr(); };
        const int rc = unlocked([&] {
            return fp8lin_moe_block_w8a8(r.t.const_data_ptr(), r.ld, ids.const_data_ptr(), i64 ? 1 : 0, (const float*)w.const_data_ptr(), r.m, (int)k,
                                         wt[0]->const_data_ptr(), f(1), f(2), wt[3]->const_data_ptr(), f(4), f(5), (int)experts, r.k, inter,
                                         y.mutable_data_ptr(), r.k, scr.mutable_data_ptr(), (size_t)scr.numel(), stream.stream());
        });
        check(rc, "fp8lin_moe_block_w8a8");
        return THPVariable_Wrap(y);
    });
}

// workspace(device_index, stream_handle, nbytes, for_status) -> the stream's scratch tensor.  for_status: to read the status
// word, so a wait that was given up is not raised here, and the host's copy of its code is forgotten.
PyObject* py_workspace(PyObject*, PyObject* const* a, Py_ssize_t na) {
    return guarded([&]() -> PyObject* {
        need_args(na, 4, "workspace");
        const long device = PyLong_AsLong(a[0]);
        void* handle = PyLong_AsVoidPtr(a[1]);
        const size_t nbytes = PyLong_AsSize_t(a[2]);
        const bool for_status = a[3] == Py_True;
        if (PyErr_Occurred()) return nullptr;
        const c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
        const auto stream = c10::cuda::getCurrentCUDAStream();
        if ((void*)stream.stream() != handle) throw std::runtime_error("workspace: the stream is not the current one");
        const at::Tensor t = workspace(stream, nbytes, !for_status);
        if (for_status) {
            stream.synchronize();
            Scratch& s = scratch();
            std::lock_guard<std::mutex> lock(s.lock);
            *s.live.at(std::make_pair((int)stream.device_index(), (void*)stream.stream())).word = 0;
        }
        return THPVariable_Wrap(t);
    });
}

PyObject* py_release_workspaces(PyObject*, PyObject*) {
    Scratch& s = scratch();
    std::lock_guard<std::mutex> guard(s.lock);
    s.live.clear();
    s.retired.clear();
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"linear", (PyCFunction)(void (*)(void))py_linear, METH_FASTCALL, nullptr},
    {"linear_codes", (PyCFunction)(void (*)(void))py_linear_codes, METH_FASTCALL, nullptr},
    {"rmsnorm_quant", (PyCFunction)(void (*)(void))py_rmsnorm_quant, METH_FASTCALL, nullptr},
    {"mlp", (PyCFunction)(void (*)(void))py_mlp, METH_FASTCALL, nullptr},
    {"moe_route", (PyCFunction)(void (*)(void))py_moe_route, METH_FASTCALL, nullptr},
    {"moe_block", (PyCFunction)(void (*)(void))py_moe_block, METH_FASTCALL, nullptr},
    {"workspace", (PyCFunction)(void (*)(void))py_workspace, METH_FASTCALL, nullptr},
    {"release_workspaces", py_release_workspaces, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_fp8host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fp8host(void) {
    PyObject* torch = PyImport_ImportModule("torch");
    if (!torch) return nullptr;
    g_out_of_memory = PyObject_GetAttrString(torch, "OutOfMemoryError");
    if (!g_out_of_memory) PyErr_Clear();
    Py_DECREF(torch);
    return PyModule_Create(&kModule);
}
