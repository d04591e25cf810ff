// Native host side of the per-forward entry points.
//
// An HSA forward is three or four launches of 5..100 us, and a layer makes half a dozen such calls: with the checks,
// the descriptors and the workspace look-up done in Python through ctypes a call took 60..80 us to enqueue, more than
// the small shapes take to run.  Here a call is one C function: it reads the tensors' sizes and strides itself, takes
// its output from PyTorch's caching allocator, keeps the workspace of each stream, and calls the C ABI of libwa_b200.so.
// The functions of that library are handed over by address (`bind`), so this module does not care which file they
// come from.
#include <torch/extension.h>

#include <ATen/core/CachingHostAllocator.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <list>
#include <string>
#include <unordered_map>

#include "../../../include/worldattention_b200.h"

namespace {

using at::Tensor;

// ---- the C ABI, by address ---------------------------------------------------------------------
decltype(&wa_last_error) f_last_error;
decltype(&wa_hsa_workspace_bytes) f_workspace_bytes;
decltype(&wa_hsa_forward) f_forward;
decltype(&wa_hsa_status) f_status;
decltype(&wa_qk_norm_rope) f_rope;
decltype(&wa_qk_norm_rope_at) f_rope_at;
decltype(&wa_kv_append_workspace_bytes) f_append_bytes;
decltype(&wa_kv_append_compress) f_append;
decltype(&wa_ln_modulate) f_ln;
decltype(&wa_gated_residual) f_residual;
PyObject *py_out_of_memory = nullptr;                                 // torch.OutOfMemoryError
PyObject *py_status_word = nullptr, *py_raise_if_failed = nullptr;   // _lib.status_word(index) -> address, _lib.raise_if_failed(index)

constexpr int MAX_DEVICES = 64;
volatile int *status_words[MAX_DEVICES] = {nullptr};

struct PyFailure {};   // a Python exception is set

[[noreturn]] void fail(PyObject *type, const std::string &msg) {
    PyErr_SetString(type, msg.c_str());
    throw PyFailure();
}

void check(int rc) {
    if (rc == 0) return;
    const std::string msg = f_last_error();
    if (rc == WA_ERR_ARG || rc == WA_ERR_ALIGN || rc == WA_ERR_WORKSPACE) fail(PyExc_ValueError, msg);
    if (rc == WA_ERR_UNSUPPORTED) fail(PyExc_NotImplementedError, msg);
    fail(PyExc_RuntimeError, "CUDA error " + std::to_string(rc) + ": " + msg);
}

// ---- arguments ---------------------------------------------------------------------------------
const Tensor *tensor_or_null(PyObject *o, const char *name) {
    if (o == Py_None) return nullptr;
    if (!THPVariable_Check(o)) fail(PyExc_TypeError, std::string(name) + " must be a tensor");
    return &THPVariable_Unpack(o);
}
const Tensor &tensor(PyObject *o, const char *name) {
    const Tensor *t = tensor_or_null(o, name);
    if (!t) fail(PyExc_TypeError, std::string(name) + " must be a tensor");
    return *t;
}
long long integer(PyObject *o) {
    if (!PyLong_Check(o)) {
        PyObject *as_int = PyNumber_Long(o);
        if (!as_int) throw PyFailure();
        const long long v = PyLong_AsLongLong(as_int);
        Py_DECREF(as_int);
        if (v == -1 && PyErr_Occurred()) throw PyFailure();
        return v;
    }
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw PyFailure();
    return v;
}
double real(PyObject *o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw PyFailure();
    return v;
}
void expect_args(Py_ssize_t got, Py_ssize_t want) {
    if (got != want) fail(PyExc_TypeError, "expected " + std::to_string(want) + " arguments, got " + std::to_string(got));
}

std::string shape_of(const Tensor &t) {
    std::string s = "(";
    for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
    return s + (t.dim() == 1 ? ",)" : ")");
}

void require_cuda(const Tensor &t, c10::Device &dev, bool &seen) {
    if (!t.is_cuda())
        fail(PyExc_RuntimeError, "worldattention_b200 runs on CUDA tensors only (there is no CPU path); got a tensor on " + t.device().str());
    if (!seen) {
        dev = t.device();
        seen = true;
    } else if (t.device() != dev) {
        fail(PyExc_ValueError, "tensors live on different devices: " + dev.str() + " and " + t.device().str());
    }
}

int dtype_code(at::ScalarType t) {
    if (t == at::kFloat) return WA_F32;
    if (t == at::kBFloat16) return WA_BF16;
    fail(PyExc_ValueError, std::string("worldattention_b200 kernels take float32 or bfloat16 tensors, got ") +
                               (t == at::kHalf ? "torch.float16" : t == at::kDouble ? "torch.float64" : c10::toString(t)));
}

// `[B, L, H, D]` descriptor; `keep` holds a re-laid-out copy for the duration of the call where one is needed
wa_tensor4 view4(const Tensor &t, Tensor &keep) {
    if (t.dim() != 4) fail(PyExc_ValueError, "expected a [B, L, H, D] tensor, got shape " + shape_of(t));
    const Tensor *x = &t;
    if (t.stride(3) != 1 && t.size(3) != 1) {
        keep = t.contiguous();
        x = &keep;
    }
    return wa_tensor4{x->data_ptr(), dtype_code(x->scalar_type()), 0, x->stride(0), x->stride(1), x->stride(2)};
}

// a parameter as the kernels take it: on the device, contiguous, optionally in another tensor's dtype
const Tensor &plain(const Tensor &t, c10::Device dev, Tensor &keep, at::ScalarType dtype) {
    if (t.device() == dev && t.is_contiguous() && t.scalar_type() == dtype) return t;
    keep = t.detach().to(dev, dtype).contiguous();
    return keep;
}
const Tensor &plain(const Tensor &t, c10::Device dev, Tensor &keep) { return plain(t, dev, keep, t.scalar_type()); }

volatile int *status_word(int dev) {
    if (dev < 0 || dev >= MAX_DEVICES) fail(PyExc_RuntimeError, "device index out of range");
    if (!status_words[dev]) {
        PyObject *r = PyObject_CallFunction(py_status_word, "i", dev);
        if (!r) throw PyFailure();
        status_words[dev] = reinterpret_cast<volatile int *>(PyLong_AsVoidPtr(r));
        Py_DECREF(r);
        if (PyErr_Occurred()) throw PyFailure();
    }
    return status_words[dev];
}
void raise_if_failed(int dev) {
    if (*status_word(dev) == 0) return;
    PyObject *r = PyObject_CallFunction(py_raise_if_failed, "i", dev);
    if (!r) throw PyFailure();
    Py_DECREF(r);
}

// ---- workspaces: one growing buffer per (kind, device, stream), the least recently used dropped beyond a bound ----
// A buffer is only handed out and its launches only enqueued while the interpreter lock is held, so two threads on one
// stream cannot interleave the launches that share it.  A dropped buffer goes back to the caching allocator, which
// recycles it in the order of the stream it was taken on.  A call that is being captured into a graph takes a buffer of
// its own (from the graph's memory pool): the graph outlives any bookkeeping here.
struct Slot {
    int kind, dev;
    cudaStream_t stream;
    Tensor buf;
};
std::list<Slot> &slots = *new std::list<Slot>;   // never destroyed: at exit the CUDA context may be gone before static objects
constexpr size_t MAX_SLOTS = 32;

Tensor workspace(int kind, c10::Device dev, cudaStream_t stream, size_t bytes, bool zeroed) {
    const auto opt = at::TensorOptions().dtype(at::kByte).device(dev);
    auto fresh = [&](size_t n) { return zeroed ? at::zeros({(int64_t)n}, opt) : at::empty({(int64_t)n}, opt); };
    if (at::cuda::currentStreamCaptureStatusMayInitCtx() != at::cuda::CaptureStatus::None) return fresh(bytes);
    for (auto it = slots.begin(); it != slots.end(); ++it)
        if (it->kind == kind && it->dev == dev.index() && it->stream == stream) {
            if (it != slots.begin()) slots.splice(slots.begin(), slots, it);
            if ((size_t)it->buf.numel() < bytes) {
                it->buf = Tensor();
                it->buf = fresh(bytes);
            }
            return it->buf;
        }
    if (slots.size() >= MAX_SLOTS) slots.pop_back();
    slots.push_front(Slot{kind, dev.index(), stream, fresh(std::max<size_t>(bytes, 1 << 20))});
    return slots.front().buf;
}

// ---- hsa_attention (wan/modules/hsa/attention.py:153-259) ---------------------------------------
// q, k, v, k_coarse|None, v_coarse|None, k_proj, v_proj, gate_w|None, gate_b|None, topk|None, block, tau_min, tau_max,
// segment, flags, k_pooled|None, k_pooled_valid, want_routing, check_status
//   -> out, or (out, index, num, thresholds, used_tuned) with want_routing
PyObject *hsa_forward(PyObject *const *a, Py_ssize_t n) {
    expect_args(n, 19);
    const Tensor &q = tensor(a[0], "q"), &k = tensor(a[1], "k"), &v0 = tensor(a[2], "v");
    const Tensor *kc = tensor_or_null(a[3], "k_coarse"), *vc = tensor_or_null(a[4], "v_coarse");
    const Tensor *gw = tensor_or_null(a[7], "gate weight"), *gb = tensor_or_null(a[8], "gate bias"), *topk = tensor_or_null(a[9], "topk_per_head");
    const Tensor *pooled = tensor_or_null(a[15], "k_pooled_cache");
    const bool want_routing = a[17] == Py_True, check_status = a[18] == Py_True;

    if (q.dim() != 4 || k.dim() != 4 || v0.dim() != 4) fail(PyExc_ValueError, "q, k and v must be [B, L, H, D] tensors");
    const int64_t B = q.size(0), Lq = q.size(1), H = q.size(2), D = q.size(3), Lkv = k.size(1);
    if (Lq <= 0 || Lkv <= 0) fail(PyExc_ValueError, "q_len and kv_len must be positive");
    c10::Device dev(c10::kCUDA, 0);
    bool seen = false;
    for (const Tensor *t : {&q, &k, &v0, kc, vc})
        if (t) require_cuda(*t, dev, seen);
    raise_if_failed(dev.index());
    c10::cuda::CUDAGuard guard(dev);
    cudaStream_t stream = at::cuda::getCurrentCUDAStream(dev.index()).stream();

    Tensor keep[12];
    wa_hsa_params p{};
    const long long block = integer(a[10]);
    if (block <= 0 || block > INT_MAX) fail(PyExc_ValueError, "block_size must be positive, got " + std::to_string(block));   // divided by below
    p.B = (int)B; p.H = (int)H; p.D = (int)D; p.Lq = (int)Lq; p.Lkv = (int)Lkv;
    p.block_size = (int)block;
    p.tau_min = real(a[11]);
    p.tau_max = real(a[12]);
    p.flags = (int)integer(a[14]);
    p.status_mirror = const_cast<int *>(status_word(dev.index()));
    const Tensor *v = &v0;
    if (v0.scalar_type() != k.scalar_type()) {
        keep[0] = v0.to(k.scalar_type());
        v = &keep[0];
    }
    p.q = view4(q, keep[1]);
    p.k = view4(k, keep[2]);
    p.v = view4(*v, keep[3]);
    if (pooled) {
        const int64_t blocks = (Lkv + block - 1) / block;
        if (pooled->scalar_type() != at::kFloat || pooled->sizes() != at::IntArrayRef({B, H, blocks, D}) || !pooled->is_contiguous() ||
            pooled->device() != dev)
            fail(PyExc_ValueError, "expected k_pooled_cache: contiguous float32 [" + std::to_string(B) + ", " + std::to_string(H) + ", " +
                                       std::to_string(blocks) + ", " + std::to_string(D) + "] on " + dev.str());
        const long long valid = integer(a[16]);
        if (valid < 0 || valid > blocks)
            fail(PyExc_ValueError, "k_pooled_valid must be in [0, " + std::to_string(blocks) + "], got " + std::to_string(valid));
        p.k_pooled = pooled->data_ptr<float>();
        p.k_pooled_valid = (int)valid;
    }
    if (kc) {
        if (kc->dim() != 4 || kc->size(0) != B || kc->size(2) != H || kc->size(3) != D)
            fail(PyExc_ValueError, "expected k_coarse shaped [B, Lc, " + std::to_string(H) + ", " + std::to_string(D) + "], got " + shape_of(*kc));
        if (vc->sizes() != kc->sizes()) fail(PyExc_ValueError, "v_coarse must have the same shape as k_coarse");
        if (kc->scalar_type() != vc->scalar_type()) {
            keep[4] = kc->to(vc->scalar_type());
            kc = &keep[4];
        }
        p.Lc = (int)kc->size(1);
        p.k_coarse = view4(*kc, keep[5]);
        p.v_coarse = view4(*vc, keep[6]);
    } else {
        const Tensor &kp = tensor(a[5], "k_proj_mat"), &vp = tensor(a[6], "v_proj_mat");
        if (kp.sizes() != vp.sizes())
            fail(PyExc_ValueError, "k_proj_mat and v_proj_mat must have the same shape, got " + shape_of(kp) + " and " + shape_of(vp));
        const long long asked = integer(a[13]), seg = asked > 0 ? asked : Lkv;
        if (std::min<long long>(seg, Lkv) > kp.size(1))
            fail(PyExc_ValueError, "segment length " + std::to_string(std::min<long long>(seg, Lkv)) + " exceeds projection length " +
                                       std::to_string(kp.size(1)) + "; increase proj_segment_len");
        const Tensor &pk = plain(kp, dev, keep[4]);
        const Tensor &pv = plain(vp, dev, keep[5], pk.scalar_type());
        p.proj_segment_len = (int)seg;
        p.proj_rank = (int)pk.size(0);
        p.proj_cols = (int)pk.size(1);
        p.proj_dtype = dtype_code(pk.scalar_type());
        p.k_proj = pk.data_ptr();
        p.v_proj = pv.data_ptr();
    }
    if (gw) {
        const Tensor &w = plain(*gw, dev, keep[7]);
        p.gate_dtype = dtype_code(w.scalar_type());
        p.gate_w = w.data_ptr();
        if (gb) p.gate_b = plain(*gb, dev, keep[8], w.scalar_type()).data_ptr();
    }
    if (topk) {
        const Tensor &counts = plain(*topk, dev, keep[9], at::kInt);
        if (counts.numel() != H) fail(PyExc_ValueError, "topk_per_head must have " + std::to_string(H) + " entries");
        p.topk_per_head = counts.data_ptr<int32_t>();
    }
    Tensor out = at::empty({B, Lq, H, D}, q.options().requires_grad(false));
    p.out = wa_tensor4{out.data_ptr(), dtype_code(out.scalar_type()), 0, Lq * H * D, H * D, D};
    Tensor index, num, thresholds;
    if (want_routing) {
        const int64_t nq = (Lq + block - 1) / block, nkv = (Lkv + block - 1) / block;
        const auto opt = at::TensorOptions().device(dev).dtype(at::kInt);
        index = at::empty({B, H, nq, nkv}, opt);
        num = at::empty({B, H, nq}, opt);
        thresholds = at::empty({H}, opt.dtype(at::kFloat));
        p.index_out = index.data_ptr<int32_t>();
        p.num_out = num.data_ptr<int32_t>();
        p.thresholds_out = thresholds.data_ptr<float>();
    }
    // A call that waits for its own status lets other threads run meanwhile, so its workspace is nobody else's.
    const size_t ws_bytes = f_workspace_bytes(&p);
    const Tensor ws = check_status ? at::empty({(int64_t)ws_bytes}, at::TensorOptions().dtype(at::kByte).device(dev))
                                   : workspace(0, dev, stream, ws_bytes, false);
    p.workspace = ws.data_ptr();
    p.workspace_bytes = (size_t)ws.numel();
    int used = 0;
    check(f_forward(&p, &used, stream));
    if (check_status && used) {
        int status = 0, rc = 0;
        Py_BEGIN_ALLOW_THREADS          // waits for the stream: other threads may be what it waits for
        rc = f_status(&p, &status, stream);
        Py_END_ALLOW_THREADS
        check(rc);
        if (status) {
            *status_word(dev.index()) = 0;
            fail(PyExc_RuntimeError, "tcgen05 HSA kernel gave up at wait site " + std::to_string(status) + "; its output is invalid");
        }
    }
    if (!want_routing) return THPVariable_Wrap(std::move(out));
    return Py_BuildValue("(NNNNO)", THPVariable_Wrap(out), THPVariable_Wrap(index), THPVariable_Wrap(num), THPVariable_Wrap(thresholds),
                         used ? Py_True : Py_False);
}

// ---- run_forward: address of a wa_hsa_params (workspace unset), device index -> used_tuned, or None ----------------
// For callers that fill the parameters themselves (partial outputs of a key shard): the stream's kept workspace and the
// launches, under the interpreter lock as above.  None: the call asked for the tcgen05 kernel, which does not cover it.
PyObject *run_forward(PyObject *const *a, Py_ssize_t n) {
    expect_args(n, 2);
    wa_hsa_params *p = reinterpret_cast<wa_hsa_params *>(PyLong_AsVoidPtr(a[0]));
    if (PyErr_Occurred()) throw PyFailure();
    if (!p) fail(PyExc_ValueError, "null parameters");
    const c10::Device dev(c10::kCUDA, (c10::DeviceIndex)integer(a[1]));
    c10::cuda::CUDAGuard guard(dev);
    cudaStream_t stream = at::cuda::getCurrentCUDAStream(dev.index()).stream();
    const Tensor ws = workspace(0, dev, stream, f_workspace_bytes(p), false);
    p->workspace = ws.data_ptr();
    p->workspace_bytes = (size_t)ws.numel();
    int used = 0;
    const int rc = f_forward(p, &used, stream);
    if (rc == WA_ERR_UNSUPPORTED && (p->flags & WA_HSA_REQUIRE_TUNED)) Py_RETURN_NONE;
    check(rc);
    return PyBool_FromLong(used);
}

// ---- qk_norm_rope: x [B, L, H, D], weight|None, eps, table|None, start_frame (int or int32 device tensor), grid_h, grid_w -> out ----
PyObject *qk_norm_rope(PyObject *const *a, Py_ssize_t n) {
    expect_args(n, 7);
    const Tensor &x = tensor(a[0], "x");
    c10::Device dev(c10::kCUDA, 0);
    bool seen = false;
    require_cuda(x, dev, seen);
    c10::cuda::CUDAGuard guard(dev);
    cudaStream_t stream = at::cuda::getCurrentCUDAStream(dev.index()).stream();
    Tensor keep[2];
    const wa_tensor4 xv = view4(x, keep[0]);
    Tensor out = at::empty(x.sizes(), x.options().requires_grad(false).memory_format(at::MemoryFormat::Contiguous));
    const int64_t L = x.size(1), H = x.size(2), D = x.size(3);
    const wa_tensor4 ov{out.data_ptr(), xv.dtype, 0, L * H * D, H * D, D};
    const Tensor *weight = tensor_or_null(a[1], "norm_weight"), *table = tensor_or_null(a[3], "table");
    const void *wp = nullptr;
    int wdt = 0;
    if (weight) {
        const Tensor &w = plain(*weight, dev, keep[1]);
        wp = w.data_ptr();
        wdt = dtype_code(w.scalar_type());
    }
    const double *freqs = table ? table->data_ptr<double>() : nullptr;
    const int rows = table ? (int)table->size(0) : 0, gh = (int)integer(a[5]), gw = (int)integer(a[6]);
    const float eps = (float)real(a[2]);
    if (THPVariable_Check(a[4])) {
        const Tensor &at_frame = THPVariable_Unpack(a[4]);
        if (at_frame.scalar_type() != at::kInt || at_frame.numel() != 1 || at_frame.device() != dev)
            fail(PyExc_ValueError, "a device-resident start_frame must be one int32 on the tensors' device");
        check(f_rope_at(&xv, &ov, (int)x.size(0), (int)L, (int)H, (int)D, wp, wdt, eps, freqs, rows, at_frame.data_ptr<int32_t>(), gh, gw, stream));
    } else {
        check(f_rope(&xv, &ov, (int)x.size(0), (int)L, (int)H, (int)D, wp, wdt, eps, freqs, rows, (int)integer(a[4]), gh, gw, stream));
    }
    return THPVariable_Wrap(std::move(out));
}

// ---- append_kv: k_new, v_new, k_cache, v_cache, k_coarse, v_coarse, position, segment, k_proj, v_proj, block -> bool ----
// False: the fused kernel does not cover the shape or the layout (nothing was launched).
PyObject *append_kv(PyObject *const *a, Py_ssize_t n) {
    expect_args(n, 11);
    static const char *names[6] = {"k_new", "v_new", "k_cache", "v_cache", "k_coarse", "v_coarse"};
    c10::Device dev(c10::kCUDA, 0);
    bool seen = false;
    Tensor keep[8];
    wa_tensor4 t[6];
    for (int i = 0; i < 6; ++i) require_cuda(tensor(a[i], names[i]), dev, seen);
    const Tensor &k_new = THPVariable_Unpack(a[0]);
    if (k_new.dim() != 4) fail(PyExc_ValueError, "expected [B, L, H, D] tensors");
    const long long position = integer(a[6]), seg = integer(a[7]), block = integer(a[10]);
    if (seg <= 0 || position % seg)
        fail(PyExc_ValueError, "rows are appended at segment boundaries, got position=" + std::to_string(position) + ", segment_len=" + std::to_string(seg));
    if (position + k_new.size(1) > THPVariable_Unpack(a[2]).size(1)) fail(PyExc_ValueError, "the rows do not fit the cache");
    if (seg > INT_MAX || block <= 0 || block > INT_MAX) fail(PyExc_ValueError, "segment_len and block_size must be positive");
    // what the kernels write, addressed from here on: rows in both caches, `rank` slots per whole segment in both tiers
    const int64_t rank_rows = tensor(a[8], "k_proj_mat").dim() == 2 ? THPVariable_Unpack(a[8]).size(0) : 0;
    const int64_t n_new = k_new.size(1), whole = n_new / seg, tail = n_new % seg;
    const int64_t stride = std::min<int64_t>(rank_rows, (seg + block - 1) / block);
    const int64_t slots = (position / seg + whole) * stride + std::min<int64_t>(rank_rows, (tail + block - 1) / block);
    for (int i = 1; i < 6; ++i) {
        const Tensor &x = THPVariable_Unpack(a[i]);
        const int64_t rows = i == 1 ? n_new : i < 4 ? position + n_new : slots;
        if (x.dim() != 4 || x.size(0) < k_new.size(0) || x.size(1) < rows || x.size(2) < k_new.size(2) || x.size(3) < k_new.size(3))
            fail(PyExc_ValueError, std::string(names[i]) + " of shape " + shape_of(x) + " does not hold the rows of k_new " + shape_of(k_new) +
                                       " (" + std::to_string(rows) + " of them are needed)");
    }
    for (int i = 2; i < 6; ++i) {      // written in place: a re-laid-out copy would take the rows
        const Tensor &dst = THPVariable_Unpack(a[i]);
        if (dst.dim() == 4 && dst.stride(3) != 1 && dst.size(3) != 1) Py_RETURN_FALSE;
    }
    for (int i = 0; i < 6; ++i) t[i] = view4(THPVariable_Unpack(a[i]), keep[i]);
    c10::cuda::CUDAGuard guard(dev);
    cudaStream_t stream = at::cuda::getCurrentCUDAStream(dev.index()).stream();
    const Tensor &pk = plain(tensor(a[8], "k_proj_mat"), dev, keep[6]);
    const Tensor &pv = plain(tensor(a[9], "v_proj_mat"), dev, keep[7], pk.scalar_type());
    const int B = (int)k_new.size(0), N = (int)k_new.size(1), H = (int)k_new.size(2), D = (int)k_new.size(3), rank = (int)pk.size(0);
    auto call = [&](void *ws, size_t bytes) {
        return f_append(&t[0], &t[1], &t[2], &t[3], &t[4], &t[5], B, N, (int)position, H, D, (int)seg, (int)block, pk.data_ptr(), pv.data_ptr(),
                        dtype_code(pk.scalar_type()), rank, (int)pk.size(1), ws, bytes, stream);
    };
    int rc = call(nullptr, 0);                                     // the tensor-core stream needs no workspace
    if (rc == WA_ERR_WORKSPACE) {
        const Tensor ws = workspace(1, dev, stream, f_append_bytes(B, N, H, D, (int)seg, (int)block, rank), true);   // zeroed once; every call leaves the counters zeroed
        rc = call(ws.data_ptr(), (size_t)ws.numel());
    }
    if (rc == WA_ERR_UNSUPPORTED) Py_RETURN_FALSE;
    check(rc);
    Py_RETURN_TRUE;
}

// ---- the element-wise steps of a block (causal_dit.py) ------------------------------------------
// `[B, F, 1, C]` or `[B, F, C]` modulation view -> (pointer, elements between consecutive frames); it must step uniformly
// over (b, f) and hold a vector for every `tokens` of the `rows` rows: the kernels take the vector of row / tokens
const void *frame_vectors(const Tensor *e, int64_t rows, int64_t tokens, int64_t dim, Tensor &keep, long long &stride) {
    if (!e) return nullptr;
    const Tensor *t = e;
    if (e->dim() < 3 || e->size(-1) < dim) fail(PyExc_ValueError, "expected a [B, F, 1, C] or [B, F, C] modulation, got shape " + shape_of(*e));
    const int64_t b = e->size(0), f = e->size(1);
    if (tokens > 0 && (rows + tokens - 1) / tokens > b * f)
        fail(PyExc_ValueError, std::to_string(rows) + " rows of " + std::to_string(tokens) + " tokens per frame need more than the modulation's " +
                                   std::to_string(b * f) + " frames");
    if (e->stride(-1) != 1 || (b > 1 && e->stride(0) != f * e->stride(1))) {
        keep = e->contiguous();
        t = &keep;
    }
    stride = t->stride(1);
    return t->data_ptr();
}

const Tensor &rows_bf16(const Tensor &t, Tensor &keep) {
    if (t.scalar_type() != at::kBFloat16) fail(PyExc_NotImplementedError, "the fused block glue is bf16 only");
    if (t.is_contiguous()) return t;
    keep = t.contiguous();
    return keep;
}

// x, eps, weight|None, bias|None, scale|None, shift|None, tokens_per_frame -> out
PyObject *ln_modulate(PyObject *const *a, Py_ssize_t n) {
    expect_args(n, 7);
    c10::Device dev(c10::kCUDA, 0);
    bool seen = false;
    require_cuda(tensor(a[0], "x"), dev, seen);
    Tensor keep[3];
    const Tensor &x = rows_bf16(THPVariable_Unpack(a[0]), keep[0]);
    c10::cuda::CUDAGuard guard(dev);
    cudaStream_t stream = at::cuda::getCurrentCUDAStream(dev.index()).stream();
    Tensor out = at::empty(x.sizes(), x.options().requires_grad(false));
    const int64_t c = x.size(-1);
    const Tensor *w = tensor_or_null(a[2], "weight"), *b = tensor_or_null(a[3], "bias");
    const Tensor *scale = tensor_or_null(a[4], "scale"), *shift = tensor_or_null(a[5], "shift");
    long long ss = 0, hs = 0;
    const int64_t rows = c ? x.numel() / c : 0, tokens = (int)integer(a[6]);
    const void *sp = frame_vectors(scale, rows, tokens, c, keep[1], ss), *hp = frame_vectors(shift, rows, tokens, c, keep[2], hs);
    if (sp && hp && ss != hs) fail(PyExc_ValueError, "scale and shift must share a layout");
    check(f_ln(x.data_ptr(), out.data_ptr(), rows, (int)c, (float)real(a[1]), w ? w->data_ptr() : nullptr, b ? b->data_ptr() : nullptr,
               sp, hp, ss ? ss : hs, (int)tokens, stream));
    return THPVariable_Wrap(std::move(out));
}

// x, y, gate|None, tokens_per_frame -> out
PyObject *gated_residual(PyObject *const *a, Py_ssize_t n) {
    expect_args(n, 4);
    c10::Device dev(c10::kCUDA, 0);
    bool seen = false;
    require_cuda(tensor(a[0], "x"), dev, seen);
    Tensor keep[3];
    const Tensor &x = rows_bf16(THPVariable_Unpack(a[0]), keep[0]), &y = rows_bf16(tensor(a[1], "y"), keep[1]);
    c10::cuda::CUDAGuard guard(dev);
    cudaStream_t stream = at::cuda::getCurrentCUDAStream(dev.index()).stream();
    Tensor out = at::empty(x.sizes(), x.options().requires_grad(false));
    const int64_t c = x.size(-1);
    long long gs = 0;
    const int64_t rows = c ? x.numel() / c : 0, tokens = (int)integer(a[3]);
    const void *gp = frame_vectors(tensor_or_null(a[2], "gate"), rows, tokens, c, keep[2], gs);
    check(f_residual(x.data_ptr(), y.data_ptr(), out.data_ptr(), rows, (int)c, gp, gs, (int)tokens, stream));
    return THPVariable_Wrap(std::move(out));
}

// ---- tensor_table(tensors) -> bytes: twelve int64 per tensor -------------------------------------
// address, device index (-1: host), scalar type, dimensions, the first four sizes, the first four strides.  A prompt switch looks
// at some hundred tensors; asked for one attribute at a time from Python that took longer than the copies.
PyObject *tensor_table(PyObject *const *a, Py_ssize_t n) {
    expect_args(n, 1);
    PyObject *seq = PySequence_Fast(a[0], "expected a sequence of tensors");
    if (!seq) throw PyFailure();
    const Py_ssize_t count = PySequence_Fast_GET_SIZE(seq);
    PyObject *out = PyBytes_FromStringAndSize(nullptr, count * 12 * (Py_ssize_t)sizeof(int64_t));
    if (!out) {
        Py_DECREF(seq);
        throw PyFailure();
    }
    int64_t *row = reinterpret_cast<int64_t *>(PyBytes_AS_STRING(out));
    try {
        for (Py_ssize_t i = 0; i < count; ++i, row += 12) {
            const Tensor &t = tensor(PySequence_Fast_GET_ITEM(seq, i), "every element");
            row[0] = reinterpret_cast<int64_t>(t.data_ptr());
            row[1] = t.is_cuda() ? t.device().index() : -1;
            row[2] = (int64_t)t.scalar_type();
            row[3] = t.dim();
            for (int d = 0; d < 4; ++d) {
                row[4 + d] = d < t.dim() ? t.size(d) : 1;
                row[8 + d] = d < t.dim() ? t.stride(d) : 0;
            }
        }
    } catch (...) {
        Py_DECREF(seq);
        Py_DECREF(out);
        throw;
    }
    Py_DECREF(seq);
    return out;
}

// ---- read_on_stream(tensors, stream_id, device_index) -> bool -------------------------------------
// Tells PyTorch's allocator of page-locked memory that the stream reads these host tensors, so that it keeps their memory from the
// next allocation until what the stream carries by then is done, whoever drops them and when: its own copies say so, a copy
// queued by this library does not.  False: some are page-locked by another hand, and only the caller can keep them.
PyObject *read_on_stream(PyObject *const *a, Py_ssize_t n) {
    expect_args(n, 3);
    const c10::Stream stream = c10::Stream::unpack3(integer(a[1]), (c10::DeviceIndex)integer(a[2]), c10::DeviceType::CUDA);
    PyObject *seq = PySequence_Fast(a[0], "expected a sequence of tensors");
    if (!seq) throw PyFailure();
    bool all = true;
    try {
        at::HostAllocator *allocator = at::getHostAllocator(at::kCUDA);
        for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); ++i) {
            const Tensor &t = tensor(PySequence_Fast_GET_ITEM(seq, i), "every element");
            const c10::DataPtr &memory = t.storage().data_ptr();
            if (t.numel() && !allocator->record_event(memory.get(), memory.get_context(), stream) && t.is_pinned()) all = false;
        }
    } catch (...) {
        Py_DECREF(seq);
        throw;
    }
    Py_DECREF(seq);
    return PyBool_FromLong(all);
}

// ---- bind(addresses: dict name -> int, status_word, raise_if_failed) ----------------------------
PyObject *bind(PyObject *const *a, Py_ssize_t n) {
    expect_args(n, 3);
    auto get = [&](const char *name, auto &fn) {
        PyObject *o = PyDict_GetItemString(a[0], name);
        if (!o) fail(PyExc_KeyError, name);
        fn = reinterpret_cast<std::decay_t<decltype(fn)>>(PyLong_AsVoidPtr(o));
    };
    get("wa_last_error", f_last_error);
    get("wa_hsa_workspace_bytes", f_workspace_bytes);
    get("wa_hsa_forward", f_forward);
    get("wa_hsa_status", f_status);
    get("wa_qk_norm_rope", f_rope);
    get("wa_qk_norm_rope_at", f_rope_at);
    get("wa_kv_append_workspace_bytes", f_append_bytes);
    get("wa_kv_append_compress", f_append);
    get("wa_ln_modulate", f_ln);
    get("wa_gated_residual", f_residual);
    if (PyErr_Occurred()) throw PyFailure();
    PyObject *torch_module = PyImport_ImportModule("torch");
    py_out_of_memory = torch_module ? PyObject_GetAttrString(torch_module, "OutOfMemoryError") : nullptr;
    Py_XDECREF(torch_module);
    if (!py_out_of_memory) throw PyFailure();
    Py_INCREF(a[1]);
    Py_INCREF(a[2]);
    py_status_word = a[1];
    py_raise_if_failed = a[2];
    Py_RETURN_NONE;
}

template <PyObject *(*F)(PyObject *const *, Py_ssize_t)>
PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n) {
    try {
        return F(args, n);
    } catch (const PyFailure &) {
        return nullptr;
    } catch (const c10::OutOfMemoryError &e) {
        PyErr_SetString(py_out_of_memory, e.what_without_backtrace());
        return nullptr;
    } catch (const c10::Error &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
        return nullptr;
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

#define WA_ENTRY(name) {#name, (PyCFunction)(void (*)(void))entry<name>, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {WA_ENTRY(bind), WA_ENTRY(hsa_forward), WA_ENTRY(run_forward), WA_ENTRY(qk_norm_rope), WA_ENTRY(append_kv), WA_ENTRY(ln_modulate),
                         WA_ENTRY(gated_residual), WA_ENTRY(tensor_table), WA_ENTRY(read_on_stream), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }
