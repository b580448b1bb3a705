// The host side of flashkda_b200.fwd as a CPython extension: the argument checks of the reference operator
// (csrc/flash_kda.cpp:44-174), the scratch allocation and the call of the C ABI, in one native function.
//
// A decode step runs for a few microseconds on the GPU, so what a call costs on the host is what such a step costs: the
// same checks written in Python (some ninety attribute reads through the interpreter, a ctypes structure, two device
// contexts) took 25 us per call; here they are plain C++ reads of the tensors' metadata.  Tensors are unwrapped in
// place (no copies, no reference counts), the scratch comes straight from PyTorch's caching allocator on the current
// stream and goes back to it in stream order when the call returns, and the device is switched only when the
// tensors are not on the current one.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <optional>
#include <string>

#include "../../include/flashkda_b200.h"

namespace {

struct Refused : std::runtime_error {
    using std::runtime_error::runtime_error;
};
inline void check(bool ok, const char* msg) {
    if (!ok) throw Refused(msg);
}
inline void check_named(bool ok, const char* name, const char* msg) {
    if (!ok) throw Refused(std::string(name) + msg);
}

const at::Tensor& tensor_arg(PyObject* o, const char* name) {
    if (!THPVariable_Check(o)) throw Refused(std::string(name) + " must be a torch.Tensor");
    return THPVariable_Unpack(o);
}
const at::Tensor* optional_tensor_arg(PyObject* o, const char* name) { return o == Py_None ? nullptr : &tensor_arg(o, name); }

// Whatever float() takes: numpy scalars, one-element tensors, strings.
double number_arg(PyObject* o) {
    if (PyFloat_Check(o)) return PyFloat_AS_DOUBLE(o);
    PyObject* f = PyNumber_Float(o);
    if (f == nullptr) throw std::bad_cast();
    const double x = PyFloat_AS_DOUBLE(f);
    Py_DECREF(f);
    return x;
}
// Whatever int() takes.
long integer_arg(PyObject* o) {
    if (PyLong_Check(o)) {
        const long x = PyLong_AsLong(o);
        if (x == -1 && PyErr_Occurred()) throw std::bad_cast();
        return x;
    }
    PyObject* i = PyNumber_Long(o);
    if (i == nullptr) throw std::bad_cast();
    const long x = PyLong_AsLong(i);
    Py_DECREF(i);
    if (x == -1 && PyErr_Occurred()) throw std::bad_cast();
    return x;
}

int algo_arg(PyObject* o) {
    const int given = PyObject_IsTrue(o);
    if (given < 0) throw std::bad_cast();
    if (given && !PyUnicode_Check(o)) {
        PyErr_SetObject(PyExc_KeyError, o);
        throw std::bad_cast();
    }
    const char* s = given ? PyUnicode_AsUTF8(o) : std::getenv("FLASHKDA_B200_ALGO");
    if (given && s == nullptr) throw std::bad_cast();
    if (s == nullptr) return FKDA_ALGO_AUTO;
    if (std::strcmp(s, "auto") == 0) return FKDA_ALGO_AUTO;
    if (std::strcmp(s, "twopass") == 0) return FKDA_ALGO_TWOPASS;
    if (std::strcmp(s, "tc") == 0) return FKDA_ALGO_TC;
    PyErr_SetString(PyExc_KeyError, s);
    throw std::bad_cast();
}

bool shape_is(const at::Tensor& t, std::initializer_list<int64_t> want) {
    const auto s = t.sizes();
    return s.size() == want.size() && std::equal(want.begin(), want.end(), s.begin());
}

// Whether the allocator can hand out a scratch of `bytes`, up to a gigabyte, that a call can do without, and nobody else pays for it.
// The device (or what a limit on this process leaves of it) has to have that much unused even if no cached block serves the call:
// otherwise the allocator would first give every cached block back, synchronising the device, on each such call (2.5 to 3.2 ms of
// host time).  And twice as much before the first block is cached, so that what made room once makes room again.  The device is
// asked (68 us) when something has been given back to it since the last time that there was room, or when less is cached than
// the call takes.  Not under capture: a graph would keep the block for as long as it lives.
bool spare_memory(c10::DeviceIndex dev, size_t bytes, cudaStream_t stream) {
    static std::atomic<int64_t> room_since[64];   // per device: blocks given back when there last was room, plus one
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    auto ok = [](cudaError_t e) { return e == cudaSuccess || (cudaGetLastError(), false); };   // (a refusal here is not the call's)
    if (dev < 0 || dev >= 64 || !ok(cudaStreamIsCapturing(stream, &capture)) || capture != cudaStreamCaptureStatusNone) return false;
    try {
        auto* allocator = c10::cuda::CUDACachingAllocator::get();
        const auto stats = allocator->getDeviceStats(dev);
        const size_t all = static_cast<size_t>(c10::CachingAllocator::StatType::AGGREGATE);
        const double reserved = (double)stats.reserved_bytes[all].current;
        const double cached = std::min(reserved - (double)stats.allocated_bytes[all].current, (double)bytes);
        const int64_t given_back = stats.num_device_free + 1;
        if (cached >= (double)bytes && room_since[dev].load(std::memory_order_relaxed) == given_back) return true;
        size_t unused = 0, total = 0;
        {
            c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);   // (another thread may be capturing)
            if (!ok(cudaMemGetInfo(&unused, &total))) return false;
        }
        const double allowed = allocator->getMemoryFraction(dev) * (double)total - reserved;
        if (std::min((double)unused, allowed) + cached < 2.0 * (double)bytes) return false;
        room_since[dev].store(given_back, std::memory_order_relaxed);
        return true;
    } catch (const c10::Error&) {   // (an allocator that keeps no such figures)
        return false;
    }
}

// fwd(q, k, v, g, beta, scale, out, A_log, dt_bias, lower_bound, initial_state, final_state, cu_seqlens, algo, workspace,
//     phase_mask, flags, chunk_states, chunk_states_every)
void fwd_checked(PyObject* const* a) {
    static const char* const big_names[6] = {"q", "k", "v", "g", "beta", "out"};
    static const int big_at[6] = {0, 1, 2, 3, 4, 6};
    const at::Tensor* big[6];
    for (int i = 0; i < 6; ++i) big[i] = &tensor_arg(a[big_at[i]], big_names[i]);
    const at::Tensor &q = *big[0], &k = *big[1], &v = *big[2], &g = *big[3], &beta = *big[4], &out = *big[5];
    for (int i = 0; i < 6; ++i) check(big[i]->is_cuda(), "all tensors must be on CUDA");
    for (int i = 0; i < 6; ++i) check(big[i]->is_contiguous(), "all tensors must be contiguous");
    for (int i = 0; i < 6; ++i) check_named(big[i]->scalar_type() == at::kBFloat16, big_names[i], " must be bfloat16");
    const at::Tensor* h0 = optional_tensor_arg(a[10], "initial_state");
    const at::Tensor* hT = optional_tensor_arg(a[11], "final_state");
    bool state_fp32 = false;
    auto check_state = [&](const at::Tensor* s, const char* name) {
        if (s == nullptr) return;
        check_named(s->is_cuda() && s->is_contiguous(), name, " must be contiguous CUDA tensor");
        check_named(s->scalar_type() == at::kBFloat16 || s->scalar_type() == at::kFloat, name, " must be bfloat16 or float32");
        state_fp32 |= s->scalar_type() == at::kFloat;
    };
    check_state(h0, "initial_state");
    check_state(hT, "final_state");
    if (h0 != nullptr && hT != nullptr)
        check(h0->scalar_type() == hT->scalar_type(), "initial_state and final_state must have the same dtype");
    const at::Tensor &A_log = tensor_arg(a[7], "A_log"), &dt_bias = tensor_arg(a[8], "dt_bias");
    check(A_log.is_cuda() && A_log.is_contiguous(), "A_log must be contiguous CUDA tensor");
    check(A_log.scalar_type() == at::kFloat, "A_log must be float32");
    check(dt_bias.is_cuda() && dt_bias.is_contiguous(), "dt_bias must be contiguous CUDA tensor");
    check(dt_bias.scalar_type() == at::kFloat, "dt_bias must be float32");
    for (int i = 0; i < 4; ++i) check_named(big[i]->dim() == 4, big_names[i], " must be [B, T, H, D]");
    check(beta.dim() == 3, "beta must be [B, T, H]");
    check(out.dim() == 4, "out must be [B, T, H, D]");
    const int64_t B = q.size(0), T = q.size(1), H = q.size(2), D = q.size(3);
    check(k.sizes() == q.sizes(), "k must match q shape");
    check(v.sizes() == q.sizes(), "v must match q shape");
    check(g.sizes() == q.sizes(), "g must match q shape");
    check(out.sizes() == q.sizes(), "out must match q shape");
    check(shape_is(beta, {B, T, H}), "beta must be [B, T, H] matching q");
    check(shape_is(A_log, {H}), "A_log must be [H]");
    check(shape_is(dt_bias, {H, D}), "dt_bias must be [H, D]");
    check(D == FKDA_HEAD_DIM, "currently only supports D == 128");
    const double lower_bound = number_arg(a[9]);
    check(-5.0 <= lower_bound && lower_bound <= 0.0, "lower_bound must be in [-5.0, 0]");
    const c10::Device dev = q.device();
    check(k.device() == dev && v.device() == dev && g.device() == dev && beta.device() == dev && out.device() == dev &&
              A_log.device() == dev && dt_bias.device() == dev,
          "all tensors must be on the same device");
    int64_t N = B;
    const at::Tensor* cu = optional_tensor_arg(a[12], "cu_seqlens");
    if (cu != nullptr) {
        check(B == 1, "B must be 1 when cu_seqlens is provided");
        check(cu->is_cuda(), "cu_seqlens must be on CUDA");
        check(cu->scalar_type() == at::kLong, "cu_seqlens must be int64");
        check(cu->dim() == 1, "cu_seqlens must be 1D");
        N = cu->numel() - 1;
        check(N > 0, "cu_seqlens must have at least 2 elements");
        check(cu->is_contiguous(), "cu_seqlens must be contiguous");
    }
    auto check_state_shape = [&](const at::Tensor* s, const char* name) {
        if (s == nullptr) return;
        check_named(shape_is(*s, {N, H, FKDA_HEAD_DIM, FKDA_HEAD_DIM}), name, " must be [N, H, D, D]");
        check_named(s->device() == dev, name, " must be on the same device as q");
    };
    check_state_shape(h0, "initial_state");
    check_state_shape(hT, "final_state");
    const at::Tensor* cs = optional_tensor_arg(a[17], "chunk_states");
    long every = 0;
    if (cs != nullptr) {
        check(cs->is_cuda() && cs->is_contiguous() && cs->scalar_type() == at::kBFloat16,
              "chunk_states must be a contiguous CUDA bfloat16 tensor");
        every = integer_arg(a[18]);
        check(every >= 1, "chunk_states_every must be >= 1");
        const int64_t group = 16 * (int64_t)every;
        check(cu != nullptr || cs->numel() == B * ((T + group - 1) / group) * H * FKDA_HEAD_DIM * FKDA_HEAD_DIM,
              "chunk_states must hold B * ceil(T / (16 * every)) slots of [H, 128, 128]");
    }
    fkda_fwd_params p;
    std::memset(&p, 0, sizeof(p));
    p.algo = algo_arg(a[13]);
    if (B * T == 0 && hT == nullptr) return;
    auto ptr = [](const at::Tensor* t) { return t == nullptr ? nullptr : t->data_ptr(); };
    p.q = q.data_ptr(); p.k = k.data_ptr(); p.v = v.data_ptr(); p.g = g.data_ptr(); p.beta = beta.data_ptr();
    p.out = out.data_ptr();
    p.A_log = static_cast<const float*>(A_log.data_ptr());
    p.dt_bias = static_cast<const float*>(dt_bias.data_ptr());
    p.initial_state = ptr(h0);
    p.final_state = ptr(hT);
    p.state_dtype = state_fp32 ? FKDA_STATE_FP32 : FKDA_STATE_BF16;
    p.cu_seqlens = static_cast<const int64_t*>(ptr(cu));
    p.B = B; p.T = T; p.H = H; p.N = N;
    p.token_stride = H * FKDA_HEAD_DIM;
    p.beta_token_stride = H;
    p.scale = (float)number_arg(a[5]);
    p.lower_bound = lower_bound;
    p.phase_mask = (int32_t)integer_arg(a[15]);
    p.flags = (int32_t)integer_arg(a[16]);
    p.chunk_states = ptr(cs);
    p.chunk_states_every = (int32_t)every;
    c10::cuda::OptionalCUDAGuard guard;
    if (c10::cuda::current_device() != dev.index()) guard.set_index(dev.index());
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const size_t need = fkda_workspace_bytes_for(&p);   // what this call's path needs (a decode step: nothing)
    const at::Tensor* ws = optional_tensor_arg(a[14], "workspace");
    c10::DataPtr scratch;   // given back when it goes out of scope; the allocator reuses it in stream order
    if (ws != nullptr) {
        // (also where none is needed, one that is given has room for the header: the status word goes there)
        check(ws->is_cuda() && ws->is_contiguous() && ws->scalar_type() == at::kByte && (size_t)ws->numel() >= need && ws->numel() >= 256,
              "workspace must be a contiguous CUDA uint8 tensor of sufficient size");
        p.workspace = ws->data_ptr();
        p.workspace_bytes = (size_t)ws->numel();
    } else if (need > 0) {
        p.workspace_bytes = fkda_workspace_bytes_wanted(&p);   // more than the path needs only makes it faster
        if (p.workspace_bytes > need && !spare_memory(dev.index(), p.workspace_bytes, stream)) p.workspace_bytes = need;
        if (p.workspace_bytes > need) {
            try {
                scratch = c10::cuda::CUDACachingAllocator::get()->allocate(p.workspace_bytes);
            } catch (const c10::OutOfMemoryError&) {   // (another thread was faster)
                p.workspace_bytes = need;
            }
        }
        if (scratch.get() == nullptr) scratch = c10::cuda::CUDACachingAllocator::get()->allocate(need);
        p.workspace = scratch.get();
    }
    int rc;
    Py_BEGIN_ALLOW_THREADS   // (a launch may wait for room in the stream's queue; the caller holds the tensors)
    rc = fkda_fwd(&p, stream);
    Py_END_ALLOW_THREADS
    if (rc != 0)
        throw Refused(std::string("fkda_fwd failed: ") + fkda_status_string(rc) + " (status " + std::to_string(rc) + ")");
}

PyObject* host_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 19) {
        PyErr_SetString(PyExc_TypeError, "fwd takes 19 arguments");
        return nullptr;
    }
    try {
        fwd_checked(args);
    } catch (const std::bad_cast&) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "fwd: an argument has the wrong type");
        return nullptr;
    } catch (const c10::OutOfMemoryError& e) {
        PyObject* torch = PyImport_ImportModule("torch");
        PyObject* cls = torch != nullptr ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
        PyErr_SetString(cls != nullptr ? cls : PyExc_RuntimeError, e.what_without_backtrace());
        Py_XDECREF(cls);
        Py_XDECREF(torch);
        return nullptr;
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"fwd", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(host_fwd)), METH_FASTCALL,
     "Checks the arguments of one forward call and enqueues it (see flashkda_b200.fwd)."},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "Native host side of flashkda_b200.fwd.", -1, methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module_def); }
