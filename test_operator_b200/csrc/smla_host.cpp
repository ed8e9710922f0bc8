// Host side of the two operator calls as a small CPython module: one look at the tensors, the outputs' allocation and the C ABI
// call (include/smla_bwd.h) without a trip through the interpreter for each.  It holds no kernels: the library that op.py has
// loaded hands its entry points over (init).
//
// Why: the smallest calls keep the GPU busy for 15 - 20 us, and a call's way through Python took the host as long.  Host time of a
// call, through Python / so: backward of 64 queries x 16 heads x top-k 64 (three launches) 23.7 / 12.4 us, forward of eight tokens x 128
// heads (two) 17.0 / 8.0; from an idle GPU to the result 46.1 / 34.9 and 42.0 / 33.3.
//
// It takes what nearly every call passes and answers None (or a size of 0) for anything else - other argument types, tensor
// subclasses, wrapped tensors, wrong shapes - which op.py then handles itself, error messages included.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <condition_variable>
#include <cstring>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "../../include/smla_bwd.h"
#include "smla_host_delta.h"

namespace {

decltype(&smla_fwd_run) g_fwd_run = nullptr;
decltype(&smla_fwd_workspace_size) g_fwd_size = nullptr;
decltype(&smla_bwd_run_stages) g_bwd_run = nullptr;
decltype(&smla_bwd_workspace_size) g_bwd_size = nullptr;

// A plain strided CUDA tensor with memory of its own, contiguous, of this type; null for anything else.
const at::Tensor* plain(PyObject* o, at::ScalarType dtype) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    static const c10::DispatchKeySet wrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                              c10::DispatchKey::Functionalize, c10::DispatchKey::FuncTorchBatchedDecomposition});
    if (!t.defined() || t.layout() != at::kStrided || t.key_set().has_any(wrapped) || !t.has_storage() || !t.is_cuda() ||
        t.scalar_type() != dtype || t.numel() == 0 || !t.is_contiguous())
        return nullptr;
    return &t;
}

// sm_scale (None or a number) and q_start_index_s (None or an int) as the C ABI has them; false: not plainly that.
bool scalars(PyObject* scale, PyObject* start, float* sm_scale, int32_t* q_start) {
    *sm_scale = 0.f;
    if (PyFloat_CheckExact(scale)) *sm_scale = static_cast<float>(PyFloat_AS_DOUBLE(scale));
    else if (scale != Py_None) return false;
    *q_start = SMLA_NO_CAUSAL;
    if (start == Py_None) return true;
    if (!PyLong_CheckExact(start)) return false;
    int overflow = 0;
    const long long v = PyLong_AsLongLongAndOverflow(start, &overflow);
    if (overflow || v < INT32_MIN || v > INT32_MAX) return false;
    *q_start = static_cast<int32_t>(v);
    return true;
}

// kv [s_kv, 576] or [s_kv, 1, 576]; indices [s_q, topk] or [s_q, 1, topk]; q [s_q, h_q, 576]: the sizes, or false.
struct Sizes { int64_t s_q, h_q, s_kv, topk; };
bool sizes(const at::Tensor& q, const at::Tensor& kv, const at::Tensor& idx, Sizes* s) {
    if (q.dim() != 3 || q.size(2) != SMLA_D_QK || kv.dim() < 2 || kv.dim() > 3 || idx.dim() < 2 || idx.dim() > 3) return false;
    if (kv.size(-1) != SMLA_D_QK || (kv.dim() == 3 && kv.size(1) != 1) || (idx.dim() == 3 && idx.size(1) != 1)) return false;
    *s = Sizes{q.size(0), q.size(1), kv.size(0), idx.size(-1)};
    return idx.size(0) == s->s_q && s->h_q <= 128 && s->h_q % 8 == 0 && s->s_q <= INT32_MAX && s->s_kv <= INT32_MAX && s->topk <= INT32_MAX &&
           kv.get_device() == q.get_device() && idx.get_device() == q.get_device();
}
bool same_heads(const at::Tensor& t, const at::Tensor& q, int64_t d) {
    return t.dim() == (d ? 3 : 2) && t.size(0) == q.size(0) && t.size(1) == q.size(1) && (!d || t.size(2) == d) && t.get_device() == q.get_device();
}

struct BwdIn {
    const at::Tensor *q, *kv, *dO, *lse, *O, *idx;
    Sizes s;
};
bool bwd_inputs(PyObject* const* a, BwdIn* in) {
    *in = BwdIn{plain(a[0], at::kBFloat16), plain(a[1], at::kBFloat16), plain(a[2], at::kBFloat16), plain(a[3], at::kFloat),
                plain(a[4], at::kBFloat16), plain(a[5], at::kInt), {}};
    return in->q && in->kv && in->dO && in->lse && in->O && in->idx && sizes(*in->q, *in->kv, *in->idx, &in->s) &&
           same_heads(*in->dO, *in->q, SMLA_D_V) && same_heads(*in->O, *in->q, SMLA_D_V) && same_heads(*in->lse, *in->q, 0);
}

// bwd_need(q, kv, dO, lse, O, indices) -> bytes of workspace, 0 where the call is not one for this module
PyObject* bwd_need(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    BwdIn in;
    if (n != 6 || !g_bwd_size || !bwd_inputs(a, &in)) return PyLong_FromLong(0);
    smla_bwd_params p{};
    p.s_q = static_cast<int32_t>(in.s.s_q);
    p.s_kv = static_cast<int32_t>(in.s.s_kv);
    p.h_q = static_cast<int32_t>(in.s.h_q);
    p.topk = static_cast<int32_t>(in.s.topk);
    return PyLong_FromSize_t(g_bwd_size(&p, 0));
    END_HANDLE_TH_ERRORS
}

at::Tensor empty(at::IntArrayRef shape, at::ScalarType dtype, const at::Tensor& like) {
    return at::empty(shape, at::TensorOptions().dtype(dtype).device(like.device()));
}

// bwd(q, kv, dO, lse, O, indices, sm_scale, q_start_index_s, lse_is_base2, dQ or None, dKV or None, query_meta or None, workspace
// pointer, workspace bytes, stages) -> (dQ, dKV), a status, or None.  The given outputs and the table have been checked.
PyObject* bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    BwdIn in;
    smla_bwd_params p{};
    if (n != 15 || !g_bwd_run || !bwd_inputs(a, &in) || !scalars(a[6], a[7], &p.sm_scale, &p.q_start_index_s)) Py_RETURN_NONE;
    for (int i = 9; i < 12; ++i)
        if (a[i] != Py_None && !THPVariable_Check(a[i])) Py_RETURN_NONE;
    void* ws = PyLong_AsVoidPtr(a[12]);
    const size_t ws_bytes = PyLong_AsSize_t(a[13]);
    const long stages = PyLong_AsLong(a[14]), base2 = PyLong_AsLong(a[8]);
    if (PyErr_Occurred()) return nullptr;
    const c10::cuda::CUDAGuard guard(in.q->device());
    const at::Tensor dQ = a[9] != Py_None ? THPVariable_Unpack(a[9]) : empty(in.q->sizes(), at::kBFloat16, *in.q);
    const at::Tensor dKV = a[10] != Py_None ? THPVariable_Unpack(a[10]) : empty(in.kv->sizes(), at::kFloat, *in.q);
    p.q = in.q->data_ptr();
    p.kv = in.kv->data_ptr();
    p.dO = in.dO->data_ptr();
    p.lse = static_cast<const float*>(in.lse->data_ptr());
    p.O = in.O->data_ptr();
    p.indices = static_cast<const int32_t*>(in.idx->data_ptr());
    p.dQ = dQ.data_ptr();
    p.dKV = static_cast<float*>(dKV.data_ptr());
    p.s_q = static_cast<int32_t>(in.s.s_q);
    p.s_kv = static_cast<int32_t>(in.s.s_kv);
    p.h_q = static_cast<int32_t>(in.s.h_q);
    p.topk = static_cast<int32_t>(in.s.topk);
    p.lse_is_base2 = base2 ? 1 : 0;
    if (a[11] != Py_None) p.query_meta = static_cast<const int32_t*>(THPVariable_Unpack(a[11]).data_ptr());
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(in.q->get_device()).stream();
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = g_bwd_run(&p, ws, ws_bytes, stream, static_cast<int>(stages));
    Py_END_ALLOW_THREADS
    if (st != SMLA_OK) return PyLong_FromLong(st);
    return PyTuple_Pack(2, py::reinterpret_steal<py::object>(THPVariable_Wrap(dQ)).ptr(), py::reinterpret_steal<py::object>(THPVariable_Wrap(dKV)).ptr());
    END_HANDLE_TH_ERRORS
}

// fwd(q, kv, indices, sm_scale, q_start_index_s, lse_is_base2) -> (o, lse), a status, or None.  The scratch is
// allocated per call: the allocator keeps it apart from other threads' calls and gives it to a captured graph's pool.
PyObject* fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    smla_fwd_params p{};
    Sizes s;
    if (n != 6 || !g_fwd_run || !g_fwd_size || !scalars(a[3], a[4], &p.sm_scale, &p.q_start_index_s)) Py_RETURN_NONE;
    const at::Tensor *q = plain(a[0], at::kBFloat16), *kv = plain(a[1], at::kBFloat16), *idx = plain(a[2], at::kInt);
    if (!q || !kv || !idx || !sizes(*q, *kv, *idx, &s)) Py_RETURN_NONE;
    const long base2 = PyLong_AsLong(a[5]);
    if (PyErr_Occurred()) return nullptr;
    p.s_q = static_cast<int32_t>(s.s_q);
    p.s_kv = static_cast<int32_t>(s.s_kv);
    p.h_q = static_cast<int32_t>(s.h_q);
    p.topk = static_cast<int32_t>(s.topk);
    const size_t need = g_fwd_size(&p, 0);
    if (!need) Py_RETURN_NONE;
    const c10::cuda::CUDAGuard guard(q->device());
    const at::Tensor o = empty({s.s_q, s.h_q, SMLA_D_V}, at::kBFloat16, *q), lse = empty({s.s_q, s.h_q}, at::kFloat, *q);
    const at::Tensor ws = empty({static_cast<int64_t>(need)}, at::kByte, *q);
    p.q = q->data_ptr();
    p.kv = kv->data_ptr();
    p.indices = static_cast<const int32_t*>(idx->data_ptr());
    p.o = o.data_ptr();
    p.lse = static_cast<float*>(lse.data_ptr());
    p.lse_is_base2 = base2 ? 1 : 0;
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(q->get_device()).stream();
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = g_fwd_run(&p, ws.data_ptr(), need, stream);
    Py_END_ALLOW_THREADS
    if (st != SMLA_OK) return PyLong_FromLong(st);
    return PyTuple_Pack(2, py::reinterpret_steal<py::object>(THPVariable_Wrap(o)).ptr(), py::reinterpret_steal<py::object>(THPVariable_Wrap(lse)).ptr());
    END_HANDLE_TH_ERRORS
}

// ---- Delta = rowsum(O * dO) on the host, for inputs that lie there (smla_host_delta.h) ------------------------------------------
// O is needed for Delta alone, and Delta is 256 times smaller: found here, O does not have to cross PCIe (29 % of the input bytes of 128
// heads x 512 columns).  Bound by reading O and dO from the host's memory.

// Threads of its own go through the rows in order, a piece at a time; they end with the rows, and at the latest with the object.
class DeltaJob {
public:
    DeltaJob(const at::Tensor& o, const at::Tensor& g, const at::Tensor& out, int threads)
        : o_(o), g_(g), out_(out), rows_(out.numel()), done_((rows_ + kPiece - 1) / kPiece, 0) {
        try {
            for (int i = 0; i < threads; ++i) workers_.emplace_back([this] { work(); });
        } catch (const std::system_error&) {       // fewer threads than asked for, or none: wait() does what is left
        }
    }
    ~DeltaJob() {
        next_.store(static_cast<int64_t>(done_.size()));
        for (auto& t : workers_) t.join();
    }
    // Whether the first `rows` rows are there; `block`: waits for them.
    bool wait(int64_t rows, bool block) {
        if (block && workers_.empty()) work();
        std::unique_lock<std::mutex> lock(mu_);
        const auto there = [&] { return std::min(ready_ * kPiece, rows_) >= std::min(rows, rows_); };
        if (block) cv_.wait(lock, there);
        return there();
    }

private:
    static constexpr int64_t kPiece = 128;         // rows: 256 KB of inputs
    void work() {
        const auto* o = static_cast<const uint16_t*>(o_.data_ptr());
        const auto* g = static_cast<const uint16_t*>(g_.data_ptr());
        auto* out = static_cast<float*>(out_.data_ptr());
        const auto pieces = static_cast<int64_t>(done_.size());
        for (int64_t i; (i = next_.fetch_add(1)) < pieces;) {
            const int64_t r = i * kPiece;
            delta_rows_host(o + r * SMLA_D_V, g + r * SMLA_D_V, out + r, std::min(kPiece, rows_ - r));
            std::lock_guard<std::mutex> lock(mu_);
            done_[i] = 1;
            const int64_t before = ready_;
            while (ready_ < pieces && done_[ready_]) ++ready_;
            if (ready_ != before) cv_.notify_all();
        }
    }
    const at::Tensor o_, g_, out_;
    const int64_t rows_;
    std::atomic<int64_t> next_{0};
    std::mutex mu_;
    std::condition_variable cv_;
    std::vector<char> done_;
    int64_t ready_ = 0;
    std::vector<std::thread> workers_;
};
constexpr const char* kDeltaJob = "smla_delta_job";
void free_delta_job(PyObject* c) {
    auto* job = static_cast<DeltaJob*>(PyCapsule_GetPointer(c, kDeltaJob));
    Py_BEGIN_ALLOW_THREADS
    delete job;
    Py_END_ALLOW_THREADS
}
const at::Tensor* plain_host(PyObject* o, at::ScalarType dtype) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    return t.defined() && t.layout() == at::kStrided && t.device().is_cpu() && t.has_storage() && t.scalar_type() == dtype && t.numel() > 0 &&
           t.is_contiguous() && !t.is_neg() ? &t : nullptr;
}
// delta_start(O, dO, out, threads) -> the job, or None; delta_wait(job, rows, block) -> whether the first `rows` rows of out are there, after
// waiting for them if `block`
PyObject* delta_start(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 4) Py_RETURN_NONE;
    const at::Tensor *o = plain_host(a[0], at::kBFloat16), *g = plain_host(a[1], at::kBFloat16), *out = plain_host(a[2], at::kFloat);
    const long threads = PyLong_AsLong(a[3]);
    if (PyErr_Occurred()) return nullptr;
    if (!o || !g || !out || o->numel() != out->numel() * SMLA_D_V || g->numel() != o->numel() || threads < 1 || threads > 256) Py_RETURN_NONE;
    auto job = std::make_unique<DeltaJob>(*o, *g, *out, static_cast<int>(threads));
    PyObject* c = PyCapsule_New(job.get(), kDeltaJob, free_delta_job);
    if (c) job.release();
    return c;
    END_HANDLE_TH_ERRORS
}
PyObject* delta_wait(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    auto* job = n == 3 ? static_cast<DeltaJob*>(PyCapsule_GetPointer(a[0], kDeltaJob)) : nullptr;
    const long long rows = job ? PyLong_AsLongLong(a[1]) : 0;
    if (PyErr_Occurred()) return nullptr;
    if (!job) {
        PyErr_SetString(PyExc_TypeError, "delta_wait takes a job, a number of rows and whether to wait");
        return nullptr;
    }
    const bool block = a[2] == Py_True;
    bool there;
    Py_BEGIN_ALLOW_THREADS
    there = job->wait(rows, block);
    Py_END_ALLOW_THREADS
    return PyBool_FromLong(there);
    END_HANDLE_TH_ERRORS
}

// init(addresses of smla_fwd_run, smla_fwd_workspace_size, smla_bwd_run_stages, smla_bwd_workspace_size)
PyObject* init(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void* f[4];
    if (n != 4) {
        PyErr_SetString(PyExc_TypeError, "init takes four addresses");
        return nullptr;
    }
    for (int i = 0; i < 4; ++i) f[i] = PyLong_AsVoidPtr(a[i]);
    if (PyErr_Occurred()) return nullptr;
    g_fwd_run = reinterpret_cast<decltype(g_fwd_run)>(f[0]);
    g_fwd_size = reinterpret_cast<decltype(g_fwd_size)>(f[1]);
    g_bwd_run = reinterpret_cast<decltype(g_bwd_run)>(f[2]);
    g_bwd_size = reinterpret_cast<decltype(g_bwd_size)>(f[3]);
    Py_RETURN_NONE;
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)> PyCFunction fast() { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(F)); }
PyMethodDef g_methods[] = {{"init", fast<init>(), METH_FASTCALL, nullptr},
                           {"fwd", fast<fwd>(), METH_FASTCALL, nullptr},
                           {"bwd_need", fast<bwd_need>(), METH_FASTCALL, nullptr},
                           {"bwd", fast<bwd>(), METH_FASTCALL, nullptr},
                           {"delta_start", fast<delta_start>(), METH_FASTCALL, nullptr},
                           {"delta_wait", fast<delta_wait>(), METH_FASTCALL, nullptr},
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_smla_host", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__smla_host() { return PyModule_Create(&g_module); }
