// The torch front end of the C ABI in native code: one CPython function per operation, tensors in, freshly allocated
// tensors out, everything enqueued on torch's current stream of the tensors' device, nothing synchronised.
//
// What bounds it: a step through the module API is 20 to 40 operations whose kernels take 2 to 30 us each, so the host
// must need less than that per operation or the GPU idles.  The same wrappers in Python over ctypes (argument
// conversion of 20 to 35 values, two to four torch.empty calls, stream and device look-ups) took 25-30 us per operation
// on the B200 boxes' hosts; METH_FASTCALL functions that read the tensors' fields directly, allocate from the caching
// allocator without going through the dispatcher and call the C ABI take 4-8 us, most of it the launches.
// The GIL is released while memory is allocated and kernels are launched (a full launch queue blocks there).
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <ATen/core/CachingHostAllocator.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <array>
#include <mutex>
#include <string>

#include "../../include/niti_b200.h"

namespace {

using at::Tensor;

PyObject* g_error = nullptr;  // niti_b200._lib.NitiError, for non-zero status codes

struct StatusError : std::exception {
    int code; const char* what_op;
    StatusError(int c, const char* w) : code(c), what_op(w) {}
};
struct AssertError : std::exception {};
void check(int code, const char* op) { if (code != NITI_OK) throw StatusError(code, op); }
void require(bool ok) { if (!ok) throw AssertError(); }

// ---------------------------------------------------------------------------------------------- arguments
struct Args {
    PyObject* const* v; Py_ssize_t n; Py_ssize_t i = 0;
    PyObject* next() {
        TORCH_CHECK_TYPE(i < n, "niti_b200: too few arguments");
        return v[i++];
    }
    const Tensor& tensor() {
        PyObject* o = next();
        TORCH_CHECK_TYPE(THPVariable_Check(o), "niti_b200: a tensor was expected as argument ", i);
        return THPVariable_Unpack(o);
    }
    // null for None
    const Tensor* maybe() {
        PyObject* o = next();
        if (o == Py_None) return nullptr;
        TORCH_CHECK_TYPE(THPVariable_Check(o), "niti_b200: a tensor or None was expected as argument ", i);
        return &THPVariable_Unpack(o);
    }
    int64_t integer() {
        const long long r = PyLong_AsLongLong(next());
        if (r == -1 && PyErr_Occurred()) throw python_error();
        return r;
    }
    uint64_t u64() {
        const unsigned long long r = PyLong_AsUnsignedLongLongMask(next());
        if (r == static_cast<unsigned long long>(-1) && PyErr_Occurred()) throw python_error();
        return r;
    }
    uint32_t u32() { return static_cast<uint32_t>(u64()); }
    int i32() { return static_cast<int>(integer()); }
    bool flag() {
        const int r = PyObject_IsTrue(next());
        if (r < 0) throw python_error();
        return r != 0;
    }
};

void need_cuda(std::initializer_list<const Tensor*> ts) {
    for (const Tensor* t : ts)
        if (t != nullptr && !(t->is_cuda() && t->is_contiguous()))
            throw c10::Error({__func__, __FILE__, __LINE__}, "niti_b200 ops need contiguous CUDA tensors (there is no CPU path)");
}
template <class T = void> const T* cptr(const Tensor* t) { return t == nullptr ? nullptr : static_cast<const T*>(t->const_data_ptr()); }
template <class T = void> const T* cptr(const Tensor& t) { return static_cast<const T*>(t.const_data_ptr()); }
template <class T = void> T* mptr(const Tensor& t) { return static_cast<T*>(t.mutable_data_ptr()); }
template <class T = void> T* mptr(const Tensor* t) { return t == nullptr ? nullptr : static_cast<T*>(t->mutable_data_ptr()); }

// Everything an operation needs of the device its first tensor lives on, with the GIL released while it exists.
std::mutex g_status_mutex;
std::array<Tensor, 64> g_status;
int32_t* status_ptr(const c10::Device& dev) {
    std::lock_guard<std::mutex> lock(g_status_mutex);
    Tensor& t = g_status.at(static_cast<size_t>(dev.index()));
    if (!t.defined()) t = at::zeros({4}, at::TensorOptions().dtype(at::kInt).device(dev));
    return t.mutable_data_ptr<int32_t>();
}
struct Launch {
    PyThreadState* gil;
    c10::Device dev;
    c10::cuda::OptionalCUDAGuard guard;
    void* stream;
    explicit Launch(const Tensor& t) : gil(PyEval_SaveThread()), dev(t.device()) {
        try {
            guard.set_device(dev);
            stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
        } catch (...) { PyEval_RestoreThread(gil); throw; }
    }
    ~Launch() { PyEval_RestoreThread(gil); }
    int32_t* status() const { return status_ptr(dev); }
    Tensor empty(at::IntArrayRef shape, at::ScalarType type) const {
        return at::detail::empty_cuda(shape, type, dev, std::nullopt);
    }
    Tensor bytes(size_t n) const { return empty({static_cast<int64_t>(n)}, at::kByte); }
};

// ---------------------------------------------------------------------------------------------- results
PyObject* wrap(const Tensor& t) {
    if (!t.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(t);
}
template <class... Ts> PyObject* tuple(const Ts&... ts) {
    PyObject* r = PyTuple_New(sizeof...(Ts));
    if (r == nullptr) throw python_error();
    Py_ssize_t i = 0;
    (PyTuple_SET_ITEM(r, i++, wrap(ts)), ...);
    return r;
}

using Impl = PyObject* (*)(Args&);
template <Impl F> PyObject* entry(PyObject*, PyObject* const* v, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    try {
        Args a{v, n};
        return F(a);
    } catch (const StatusError& e) {
        std::string text = std::string(e.what_op) + " failed with status " + std::to_string(e.code) + ": " + niti_strerror(e.code);
        if (e.code == NITI_ERR_CUDA) text += std::string(": ") + niti_last_cuda_error();
        PyErr_SetString(g_error != nullptr ? g_error : PyExc_RuntimeError, text.c_str());
        return nullptr;
    } catch (const AssertError&) {
        PyErr_SetNone(PyExc_AssertionError);
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

PyObject* set_error_type(Args& a) {
    PyObject* o = a.next();
    Py_INCREF(o);
    Py_XDECREF(g_error);
    g_error = o;
    Py_RETURN_NONE;
}
PyObject* status_word(Args& a) {
    const c10::Device dev(c10::kCUDA, static_cast<c10::DeviceIndex>(a.i32()));
    status_ptr(dev);
    return wrap(g_status.at(static_cast<size_t>(dev.index())));
}

struct Conv { int N, H, W, C, K, R, S; };
Conv conv_shape(const Tensor& x, const Tensor& w) {  // x [N,H,W,C], w [K,R,S,C]
    require(x.dim() == 4 && w.dim() == 4);
    const auto xs = x.sizes(), ws = w.sizes();
    return {int(xs[0]), int(xs[1]), int(xs[2]), int(xs[3]), int(ws[0]), int(ws[1]), int(ws[2])};
}

// ---------------------------------------------------------------------------------------------- what serves a shape
template <int COUNT> std::array<int, COUNT> ints(Args& a) {
    std::array<int, COUNT> r;
    for (int& x : r) x = a.i32();
    return r;
}
PyObject* conv_fprop_fused_supported(Args& a) {
    const auto v = ints<5>(a);
    return PyBool_FromLong(niti_conv_fprop_requant_supported(v[0], v[1], v[2], v[3], v[4]));
}
PyObject* conv_dgrad_fused_supported(Args& a) {
    const auto v = ints<5>(a);
    return PyBool_FromLong(niti_conv_dgrad_requant_supported(v[0], v[1], v[2], v[3], v[4]));
}
PyObject* conv_wgrad_accumulate_supported(Args& a) {
    const auto v = ints<5>(a);
    return PyBool_FromLong(niti_conv_wgrad_accumulate_supported(v[0], v[1], v[2], v[3], v[4]));
}
PyObject* conv_wgrad_update_supported(Args& a) {
    const auto v = ints<5>(a);
    return PyBool_FromLong(niti_conv_wgrad_update_elems(v[0], v[1], v[2], v[3], v[4]) != 0);
}
PyObject* conv_fprop_pool_fused_supported(Args& a) {
    const auto v = ints<8>(a);
    return PyBool_FromLong(niti_conv_fprop_requant_pool_supported(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]));
}
PyObject* conv_fprop_scratch_bytes(Args& a) {
    const auto v = ints<7>(a);
    return PyLong_FromSize_t(niti_conv_fprop_scratch_bytes(v[0], v[1], v[2], v[3], v[4], v[5], v[6]));
}
PyObject* conv_dgrad_side_bytes(Args& a) {
    const auto v = ints<8>(a);
    return PyLong_FromSize_t(niti_conv_dgrad_requant_side_bytes(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]));
}

// ---------------------------------------------------------------------------------------------- contractions
PyObject* conv_fprop_acc(Args& a) {
    const Tensor &x = a.tensor(), &w = a.tensor();
    const int pad = a.i32(), stride = a.i32();
    const bool want_max = a.flag();
    need_cuda({&x, &w});
    const Conv s = conv_shape(x, w);
    require(w.size(3) == s.C && x.scalar_type() == at::kChar && w.scalar_type() == at::kChar);
    Tensor y32, mx, sc;
    {
        Launch l(x);
        y32 = l.empty({s.N, s.H + 2 * pad - s.R + 1, s.W + 2 * pad - s.S + 1, s.K}, at::kInt);
        if (want_max) mx = l.empty({1}, at::kInt);
        const size_t nb = niti_conv_fprop_scratch_bytes(s.N, s.H, s.W, s.C, s.K, s.R, s.S);
        if (nb) sc = l.bytes(nb);
        check(niti_conv_fprop_i8(cptr<int8_t>(x), cptr<int8_t>(w), mptr<int32_t>(y32), want_max ? mptr<uint32_t>(mx) : nullptr, nb ? mptr(sc) : nullptr, nb,
                                 s.N, s.H, s.W, s.C, s.K, s.R, s.S, pad, stride, l.status(), l.stream), "niti_conv_fprop_i8");
    }
    return tuple(y32, mx);
}

// the arguments all fused convolutions share, in the order of the Python functions
struct Narrow {
    int pad, mode; const Tensor* seed; uint32_t rng_stream; uint64_t rng_offset;
    explicit Narrow(Args& a) : pad(a.i32()), mode(a.i32()), seed(a.maybe()), rng_stream(a.u32()),
                               rng_offset(a.u64()) {}
};
// two int32 words as two 0-dim tensors over one allocation
std::pair<Tensor, Tensor> two_words(const Launch& l) {
    Tensor both = l.empty({2}, at::kInt);
    auto word = [&](int64_t at_) {
        Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(both.storage()), both.key_set(), both.dtype());
        t.unsafeGetTensorImpl()->set_storage_offset(at_);
        t.unsafeGetTensorImpl()->set_sizes_contiguous({});
        return t;
    };
    return {word(0), word(1)};
}

PyObject* conv_fprop_fused(Args& a) {
    const Tensor &x = a.tensor(), &w = a.tensor(), &state = a.tensor();
    const Narrow n(a);
    const bool relu = a.flag();
    const Tensor *ea = a.maybe(), *eb = a.maybe(), *scratch = a.maybe();
    need_cuda({&x, &w, &state, scratch});
    const Conv s = conv_shape(x, w);
    Tensor y8, sc; std::pair<Tensor, Tensor> e;
    {
        Launch l(x);
        y8 = l.empty({s.N, s.H, s.W, s.K}, at::kChar);
        e = two_words(l);
        size_t nb = niti_conv_fprop_scratch_bytes(s.N, s.H, s.W, s.C, s.K, s.R, s.S);
        if (nb && scratch == nullptr) sc = l.bytes(nb);
        if (nb && scratch != nullptr) { sc = *scratch; nb = static_cast<size_t>(scratch->numel()); }
        check(niti_conv_fprop_requant_i8(cptr<int8_t>(x), cptr<int8_t>(w), mptr<int8_t>(y8), mptr<int32_t>(state), nb ? mptr(sc) : nullptr, nb,
                                         s.N, s.H, s.W, s.C, s.K, s.R, s.S, n.pad, n.mode, cptr<uint64_t>(n.seed), n.rng_stream, n.rng_offset,
                                         relu, cptr<int32_t>(ea), cptr<int32_t>(eb), mptr<int32_t>(e.first), mptr<int32_t>(e.second),
                                         l.status(), l.stream), "niti_conv_fprop_requant_i8");
    }
    return tuple(y8, e.first, e.second);
}

PyObject* conv_fprop_pool_fused(Args& a) {
    const Tensor &x = a.tensor(), &w = a.tensor(), &state = a.tensor();
    const Narrow n(a);
    const bool relu = a.flag();
    const Tensor *ea = a.maybe(), *eb = a.maybe();
    need_cuda({&x, &w, &state});
    const Conv s = conv_shape(x, w);
    Tensor y8, yp; std::pair<Tensor, Tensor> e;
    {
        Launch l(x);
        y8 = l.empty({s.N, s.H, s.W, s.K}, at::kChar);
        yp = l.empty({s.N, s.H / 2, s.W / 2, s.K}, at::kChar);
        e = two_words(l);
        check(niti_conv_fprop_requant_pool_i8(cptr<int8_t>(x), cptr<int8_t>(w), mptr<int8_t>(y8), mptr<int8_t>(yp), mptr<int32_t>(state),
                                              s.N, s.H, s.W, s.C, s.K, s.R, s.S, n.pad, n.mode, cptr<uint64_t>(n.seed), n.rng_stream,
                                              n.rng_offset, relu, cptr<int32_t>(ea), cptr<int32_t>(eb), mptr<int32_t>(e.first),
                                              mptr<int32_t>(e.second), l.status(), l.stream), "niti_conv_fprop_requant_pool_i8");
    }
    return tuple(y8, yp, e.first, e.second);
}

PyObject* conv_dgrad_fused(Args& a) {
    const Tensor &err = a.tensor(), &w = a.tensor(), &state = a.tensor();
    const Narrow n(a);
    const Tensor *ea = a.maybe(), *eb = a.maybe(), *mask = a.maybe(), *side = a.maybe();
    need_cuda({&err, &w, &state, mask, side});
    require(err.dim() == 4 && w.dim() == 4);
    const int N = err.size(0), H = err.size(1), W = err.size(2), K = err.size(3), R = w.size(1), S = w.size(2), C = w.size(3);
    Tensor e8; std::pair<Tensor, Tensor> e;
    {
        Launch l(err);
        e8 = l.empty({N, H, W, C}, at::kChar);
        e = two_words(l);
        check(niti_conv_dgrad_requant_side_i8(cptr<int8_t>(err), cptr<int8_t>(w), mptr<int8_t>(e8), mptr<int32_t>(state), mptr(side),
                                              side ? static_cast<size_t>(side->numel()) : 0, N, H, W, C, K, R, S, n.pad, n.mode,
                                              cptr<uint64_t>(n.seed), n.rng_stream, n.rng_offset, cptr<int32_t>(ea), cptr<int32_t>(eb),
                                              mptr<int32_t>(e.first), mptr<int32_t>(e.second), cptr<int8_t>(mask), l.status(), l.stream),
              "niti_conv_dgrad_requant_i8");
    }
    return tuple(e8, e.first, e.second);
}

PyObject* conv_dgrad_acc(Args& a) {
    const Tensor &err = a.tensor(), &w = a.tensor();
    const int pad = a.i32();
    need_cuda({&err, &w});
    require(err.dim() == 4 && w.dim() == 4 && err.size(3) == w.size(0));
    const int N = err.size(0), H = err.size(1), W = err.size(2), K = err.size(3), R = w.size(1), S = w.size(2), C = w.size(3);
    Tensor e32, mx;
    {
        Launch l(err);
        e32 = l.empty({N, H, W, C}, at::kInt);
        mx = l.empty({1}, at::kInt);
        check(niti_conv_dgrad_i8(cptr<int8_t>(err), cptr<int8_t>(w), mptr<int32_t>(e32), mptr<uint32_t>(mx), N, H, W, C, K, R, S, pad,
                                 l.status(), l.stream), "niti_conv_dgrad_i8");
    }
    return tuple(e32, mx);
}

PyObject* conv_wgrad_acc(Args& a) {
    const Tensor &x = a.tensor(), &err = a.tensor();
    const int R = a.i32(), S = a.i32(), pad = a.i32();
    const Tensor* out = a.maybe();
    const bool want_max = a.flag();
    need_cuda({&x, &err, out});
    require(x.dim() == 4 && err.dim() == 4);
    const int N = x.size(0), H = x.size(1), W = x.size(2), C = x.size(3), K = err.size(3);
    Tensor g32, mx;
    {
        Launch l(x);
        g32 = out ? *out : l.empty({K, R, S, C}, at::kInt);
        if (want_max) mx = l.empty({1}, at::kInt);
        const size_t nb = niti_conv_wgrad_scratch_bytes(N, H, W, C, K, R, S);
        const Tensor sc = l.bytes(nb);
        check(niti_conv_wgrad_i8(cptr<int8_t>(x), cptr<int8_t>(err), mptr<int32_t>(g32), want_max ? mptr<uint32_t>(mx) : nullptr, mptr(sc), nb,
                                 N, H, W, C, K, R, S, pad, l.status(), l.stream), "niti_conv_wgrad_i8");
    }
    return tuple(g32, mx);
}

// gradient [K,R,S,C] and its maximum, views of one allocation; w is updated in place
PyObject* conv_wgrad_update(Args& a) {
    const Tensor &x = a.tensor(), &err = a.tensor(), &w = a.tensor();
    const int pad = a.i32(), mu = a.i32(), mode = a.i32();
    const Tensor* seed = a.maybe();
    const uint32_t stream = a.u32();
    const Tensor* state = a.maybe();
    need_cuda({&x, &err, &w, state});
    require(x.dim() == 4 && err.dim() == 4 && w.scalar_type() == at::kChar);
    require(state == nullptr || (state->scalar_type() == at::kInt && state->numel() >= 4));
    const Conv s = conv_shape(x, w);
    require(w.size(3) == s.C && err.size(3) == s.K && err.size(0) == s.N && err.size(1) == s.H && err.size(2) == s.W);
    Tensor g32, mx;
    {
        Launch l(x);
        const int64_t elems = static_cast<int64_t>(niti_conv_wgrad_update_elems(s.C, s.K, s.R, s.S, pad));
        const Tensor both = l.empty({elems}, at::kInt);
        if (state != nullptr)
            check(niti_conv_wgrad_update_state_i8(cptr<int8_t>(x), cptr<int8_t>(err), mptr<int32_t>(both), mptr<int8_t>(w), mptr<int32_t>(state), s.N,
                                                  s.H, s.W, s.C, s.K, s.R, s.S, pad, mu, mode, cptr<uint64_t>(seed), stream, l.status(), l.stream),
                  "niti_conv_wgrad_update_state_i8");
        else
            check(niti_conv_wgrad_update_i8(cptr<int8_t>(x), cptr<int8_t>(err), mptr<int32_t>(both), mptr<int8_t>(w), s.N, s.H, s.W, s.C, s.K, s.R,
                                            s.S, pad, mu, mode, cptr<uint64_t>(seed), stream, l.status(), l.stream), "niti_conv_wgrad_update_i8");
        auto view = [&](int64_t at_, at::IntArrayRef shape) {
            Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(both.storage()), both.key_set(), both.dtype());
            t.unsafeGetTensorImpl()->set_storage_offset(at_);
            t.unsafeGetTensorImpl()->set_sizes_contiguous(shape);
            return t;
        };
        g32 = view(0, {s.K, s.R, s.S, s.C});
        mx = view((static_cast<int64_t>(s.K) * s.R * s.S * s.C + 3) / 4 * 4, {1});
    }
    return tuple(g32, mx);
}
PyObject* conv_wgrad_batch_inner_supported(Args& a) {
    const auto v = ints<6>(a);
    return PyBool_FromLong(niti_conv_wgrad_batch_inner_supported(v[0], v[1], v[2], v[3], v[4], v[5]));
}
PyObject* conv_wgrad_batch_inner(Args& a) {
    const Tensor &x = a.tensor(), &err = a.tensor();
    const int R = a.i32(), S = a.i32(), pad = a.i32();
    need_cuda({&x, &err});
    require(x.dim() == 4 && err.dim() == 4 && x.size(1) == err.size(1) && x.size(2) == err.size(2) && x.size(3) == err.size(3));
    const int C = x.size(0), H = x.size(1), W = x.size(2), N = x.size(3), K = err.size(0);
    Tensor out;
    {
        Launch l(x);
        out = l.empty({C, R, S, K}, at::kInt);
        check(niti_conv_wgrad_batch_inner_i8(cptr<int8_t>(x), cptr<int8_t>(err), mptr<int32_t>(out), N, H, W, C, K, R, S, pad, l.status(),
                                             l.stream), "niti_conv_wgrad_batch_inner_i8");
    }
    return wrap(out);
}

PyObject* conv_wgrad_from_patches(Args& a) {
    const Tensor &patches = a.tensor(), &err = a.tensor();
    const int C = a.i32(), R = a.i32(), S = a.i32();
    const Tensor* out = a.maybe();
    const bool want_max = a.flag();
    need_cuda({&patches, &err, out});
    require(err.dim() == 4);
    const int N = err.size(0), H = err.size(1), W = err.size(2), K = err.size(3);
    Tensor g32, mx;
    {
        Launch l(err);
        g32 = out ? *out : l.empty({K, R, S, C}, at::kInt);
        if (want_max) mx = l.empty({1}, at::kInt);
        const size_t nb = niti_conv_wgrad_patches_scratch_bytes(N, H, W, C, K, R, S);
        const Tensor sc = l.bytes(nb);
        check(niti_conv_wgrad_patches_i8(cptr<int8_t>(patches), cptr<int8_t>(err), mptr<int32_t>(g32), want_max ? mptr<uint32_t>(mx) : nullptr,
                                         mptr(sc), nb, N, H, W, C, K, R, S, l.status(), l.stream), "niti_conv_wgrad_patches_i8");
    }
    return tuple(g32, mx);
}

PyObject* conv_wgrad_accumulate(Args& a) {
    const Tensor &x = a.tensor(), &err = a.tensor(), &g32 = a.tensor();
    const int R = a.i32(), S = a.i32(), pad = a.i32();
    need_cuda({&x, &err, &g32});
    require(x.dim() == 4 && err.dim() == 4);
    const int N = x.size(0), H = x.size(1), W = x.size(2), C = x.size(3), K = err.size(3);
    require(g32.scalar_type() == at::kInt && g32.numel() == static_cast<int64_t>(K) * R * S * C);
    {
        Launch l(x);
        check(niti_conv_wgrad_accumulate_i8(cptr<int8_t>(x), cptr<int8_t>(err), mptr<int32_t>(g32), N, H, W, C, K, R, S, pad, l.status(),
                                            l.stream), "niti_conv_wgrad_accumulate_i8");
    }
    return wrap(g32);
}

// result, maximum, and how many launches besides the product the call made (row copies around a padded product)
PyObject* gemm_acc(Args& a) {
    const Tensor &A = a.tensor(), &B = a.tensor();
    const bool ta = a.flag(), tb = a.flag();
    const Tensor* out = a.maybe();
    const bool want_max = a.flag();
    need_cuda({&A, &B, out});
    require(A.dim() == 2 && B.dim() == 2);
    const int M = A.size(ta ? 1 : 0), K = A.size(ta ? 0 : 1), N = B.size(tb ? 0 : 1);
    require(B.size(tb ? 1 : 0) == K);
    Tensor c32, mx;
    size_t nb = 0;
    {
        Launch l(A);
        c32 = out ? *out : l.empty({M, N}, at::kInt);
        if (want_max) mx = l.empty({1}, at::kInt);
        nb = niti_gemm_scratch_bytes(M, N, K, ta, tb);
        Tensor sc;
        if (nb) sc = l.bytes(nb);
        check(niti_gemm_scratch_i8(cptr<int8_t>(A), cptr<int8_t>(B), mptr<int32_t>(c32), want_max ? mptr<uint32_t>(mx) : nullptr,
                                   nb ? mptr(sc) : nullptr, nb, M, N, K, ta, tb, l.status(), l.stream), "niti_gemm_i8");
    }
    const auto aligned = [](const Tensor& t) { return reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0; };
    const bool padded = nb != 0 && aligned(A) && aligned(B) && aligned(c32);
    PyObject* r = PyTuple_New(3);
    if (r == nullptr) throw python_error();
    PyTuple_SET_ITEM(r, 0, wrap(c32));
    PyTuple_SET_ITEM(r, 1, wrap(mx));
    PyTuple_SET_ITEM(r, 2, PyLong_FromLong(padded ? ((ta ? M : K) % 16 != 0) + (N % 4 != 0) : 0));
    return r;
}

// ---------------------------------------------------------------------------------------------- requantisation, memory-bound layers
PyObject* requant(Args& a) {
    const Tensor &acc = a.tensor(), &maxabs = a.tensor();
    const int kind = a.i32(), bits = a.i32(), mode = a.i32();
    const Tensor* seed = a.maybe();
    const uint32_t stream = a.u32();
    const uint64_t offset = a.u64();
    const bool relu = a.flag();
    const Tensor *ea = a.maybe(), *eb = a.maybe();
    const bool want_shift = a.flag();
    need_cuda({&acc, &maxabs});
    Tensor out; std::pair<Tensor, Tensor> e;
    {
        Launch l(acc);
        out = l.empty(acc.sizes(), at::kChar);
        e = two_words(l);
        check(niti_requant_i8(cptr<int32_t>(acc), mptr<int8_t>(out), cptr<uint32_t>(maxabs), acc.numel(), kind, bits, mode, cptr<uint64_t>(seed),
                              stream, offset, relu, cptr<int32_t>(ea), cptr<int32_t>(eb), mptr<int32_t>(e.first),
                              want_shift ? mptr<int32_t>(e.second) : nullptr, l.stream), "niti_requant_i8");
    }
    return want_shift ? tuple(out, e.first, e.second) : tuple(out, e.first, Tensor());
}

PyObject* absmax(Args& a) {
    const Tensor& acc = a.tensor();
    need_cuda({&acc});
    Tensor mx;
    {
        Launch l(acc);
        mx = l.empty({1}, at::kInt);
        check(niti_absmax_i32(cptr<int32_t>(acc), acc.numel(), mptr<uint32_t>(mx), l.stream), "niti_absmax_i32");
    }
    return wrap(mx);
}

PyObject* maxpool_fwd(Args& a) {
    const Tensor& x = a.tensor();
    const int k = a.i32(), stride = a.i32();
    need_cuda({&x});
    require(x.dim() == 4 && stride > 0);
    const int N = x.size(0), H = x.size(1), W = x.size(2), C = x.size(3);
    Tensor y;
    {
        Launch l(x);
        y = l.empty({N, (H - k) / stride + 1, (W - k) / stride + 1, C}, at::kChar);
        check(niti_maxpool_fwd_i8(cptr<int8_t>(x), mptr<int8_t>(y), N, H, W, C, k, stride, l.stream), "niti_maxpool_fwd_i8");
    }
    return wrap(y);
}
PyObject* maxpool_bwd(Args& a) {
    const Tensor &x = a.tensor(), &dy = a.tensor();
    const int k = a.i32(), stride = a.i32();
    const bool mask = a.flag();
    need_cuda({&x, &dy});
    require(x.dim() == 4);
    const int N = x.size(0), H = x.size(1), W = x.size(2), C = x.size(3);
    Tensor dx;
    {
        Launch l(x);
        dx = l.empty(x.sizes(), x.scalar_type());
        check(niti_maxpool_bwd_i8(cptr<int8_t>(x), cptr<int8_t>(dy), mptr<int8_t>(dx), N, H, W, C, k, stride, mask, l.stream), "niti_maxpool_bwd_i8");
    }
    return wrap(dx);
}
PyObject* maxpool_bwd_f16(Args& a) {
    const Tensor &x = a.tensor(), &dy = a.tensor();
    const int k = a.i32(), stride = a.i32();
    need_cuda({&x, &dy});
    require(x.dim() == 4 && x.scalar_type() == at::kHalf && dy.scalar_type() == at::kHalf);
    const int N = x.size(0), H = x.size(1), W = x.size(2), C = x.size(3);
    Tensor dx;
    {
        Launch l(x);
        dx = l.empty(x.sizes(), at::kHalf);
        check(niti_maxpool_bwd_f16(cptr(x), cptr(dy), mptr(dx), N, H, W, C, k, stride, l.stream), "niti_maxpool_bwd_f16");
    }
    return wrap(dx);
}
PyObject* relu_fwd(Args& a) {
    const Tensor& x = a.tensor();
    need_cuda({&x});
    Tensor y;
    {
        Launch l(x);
        y = l.empty(x.sizes(), x.scalar_type());
        check(niti_relu_fwd_i8(cptr<int8_t>(x), mptr<int8_t>(y), x.numel(), l.stream), "niti_relu_fwd_i8");
    }
    return wrap(y);
}
PyObject* relu_bwd(Args& a) {
    const Tensor &act = a.tensor(), &err = a.tensor();
    need_cuda({&act, &err});
    Tensor out;
    {
        Launch l(err);
        out = l.empty(err.sizes(), err.scalar_type());
        check(niti_relu_bwd_i8(cptr<int8_t>(act), cptr<int8_t>(err), mptr<int8_t>(out), err.numel(), l.stream), "niti_relu_bwd_i8");
    }
    return wrap(out);
}
PyObject* dropout(Args& a) {
    const Tensor &x = a.tensor(), &seed = a.tensor();
    const uint32_t stream = a.u32();
    need_cuda({&x, &seed});
    require(x.dim() >= 1 && x.size(0) > 0);
    Tensor y;
    {
        Launch l(x);
        y = l.empty(x.sizes(), x.scalar_type());
        check(niti_dropout_i8(cptr<int8_t>(x), mptr<int8_t>(y), x.size(0), x.numel() / x.size(0), cptr<uint64_t>(seed), stream, l.stream),
              "niti_dropout_i8");
    }
    return wrap(y);
}
PyObject* loss_err(Args& a) {
    const Tensor &out8 = a.tensor(), &out_exp = a.tensor(), &target = a.tensor(), &seed = a.tensor();
    const uint32_t stream = a.u32();
    const uint64_t offset = a.u64();
    need_cuda({&out8, &out_exp, &target, &seed});
    require(out8.dim() == 2 && target.scalar_type() == at::kLong && out_exp.scalar_type() == at::kInt);
    Tensor err;
    {
        Launch l(out8);
        err = l.empty(out8.sizes(), out8.scalar_type());
        check(niti_loss_i8(cptr<int8_t>(out8), cptr<int32_t>(out_exp), cptr<int64_t>(target), mptr<int8_t>(err), out8.size(0), out8.size(1),
                           cptr<uint64_t>(seed), stream, offset, l.stream), "niti_loss_i8");
    }
    return wrap(err);
}
PyObject* update(Args& a) {
    const Tensor &w = a.tensor(), &g32 = a.tensor(), &maxabs = a.tensor();
    const int mu = a.i32(), mode = a.i32();
    const Tensor* seed = a.maybe();
    const uint32_t stream = a.u32();
    need_cuda({&w, &g32, &maxabs});
    {
        Launch l(w);
        check(niti_update_i8(mptr<int8_t>(w), cptr<int32_t>(g32), cptr<uint32_t>(maxabs), w.numel(), mu, mode, cptr<uint64_t>(seed), stream,
                             l.stream), "niti_update_i8");
    }
    Py_RETURN_NONE;
}
PyObject* quantize_input(Args& a) {
    const Tensor& x = a.tensor();
    need_cuda({&x});
    require(x.dim() == 4 && x.scalar_type() == at::kFloat);
    const int N = x.size(0), C = x.size(1), H = x.size(2), W = x.size(3);
    Tensor x8; std::pair<Tensor, Tensor> e;
    {
        Launch l(x);
        x8 = l.empty({N, H, W, C}, at::kChar);
        e = two_words(l);
        check(niti_quantize_input_f32(cptr<float>(x), mptr<int8_t>(x8), mptr<int32_t>(e.first), mptr<uint32_t>(e.second), N, C, H, W, l.stream),
              "niti_quantize_input_f32");
    }
    return tuple(x8, e.first);
}

// A step's results into pinned host tensors, on the device and the stream of `out`: a replayed step runs there whatever device is
// current, and the event behind the launch is recorded there.
PyObject* publish_step(Args& a) {
    const Tensor &out = a.tensor(), &exp = a.tensor(), &status = a.tensor(), &host_out = a.tensor(), &host_exp = a.tensor(), &host_status = a.tensor();
    // the kernel stores through the host addresses: one exponent, four status words, as many logits as there are
    for (const Tensor* t : {&host_out, &host_exp, &host_status})
        if (!(t->is_cpu() && t->is_contiguous() && t->is_pinned()))
            throw c10::Error({__func__, __FILE__, __LINE__}, "niti_publish_step writes to contiguous pinned host tensors");
    require(host_out.scalar_type() == at::kChar && host_out.sizes() == out.sizes() && host_exp.scalar_type() == at::kInt && host_exp.numel() == 1 &&
            host_status.scalar_type() == at::kInt && host_status.numel() >= 4);
    need_cuda({&out, &exp, &status});
    require(out.scalar_type() == at::kChar && exp.scalar_type() == at::kInt && exp.numel() == 1 && status.scalar_type() == at::kInt &&
            status.numel() >= 4 && out.device() == exp.device() && out.device() == status.device());
    {
        Launch l(out);
        check(niti_publish_step(cptr<int8_t>(out), out.numel(), cptr<int32_t>(exp), cptr<int32_t>(status), mptr<int8_t>(host_out),
                                mptr<int32_t>(host_exp), mptr<int32_t>(host_status), l.stream), "niti_publish_step");
        // as a copy does: whoever drops a host tensor before the kernel has run does not free memory that is still to be written
        const c10::Stream used = c10::cuda::getCurrentCUDAStream(l.dev.index()).unwrap();
        for (const Tensor* t : {&host_out, &host_exp, &host_status}) {
            const c10::DataPtr& p = t->storage().data_ptr();
            at::getHostAllocator(at::kCUDA)->record_event(p.get(), p.get_context(), used);
        }
    }
    Py_RETURN_NONE;
}

#define NITI_ENTRY(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<&name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    NITI_ENTRY(set_error_type), NITI_ENTRY(status_word), NITI_ENTRY(conv_fprop_fused_supported),
    NITI_ENTRY(conv_dgrad_fused_supported), NITI_ENTRY(conv_wgrad_accumulate_supported), NITI_ENTRY(conv_wgrad_update_supported), NITI_ENTRY(conv_fprop_pool_fused_supported),
    NITI_ENTRY(conv_fprop_scratch_bytes), NITI_ENTRY(conv_dgrad_side_bytes),
    NITI_ENTRY(conv_fprop_acc), NITI_ENTRY(conv_fprop_fused),
    NITI_ENTRY(conv_fprop_pool_fused), NITI_ENTRY(conv_dgrad_fused), NITI_ENTRY(conv_dgrad_acc), NITI_ENTRY(conv_wgrad_acc),
    NITI_ENTRY(conv_wgrad_batch_inner_supported), NITI_ENTRY(conv_wgrad_batch_inner), NITI_ENTRY(maxpool_bwd_f16),
    NITI_ENTRY(conv_wgrad_from_patches), NITI_ENTRY(conv_wgrad_update), NITI_ENTRY(conv_wgrad_accumulate), NITI_ENTRY(gemm_acc), NITI_ENTRY(requant),
    NITI_ENTRY(absmax), NITI_ENTRY(maxpool_fwd), NITI_ENTRY(maxpool_bwd), NITI_ENTRY(relu_fwd), NITI_ENTRY(relu_bwd),
    NITI_ENTRY(dropout), NITI_ENTRY(loss_err), NITI_ENTRY(update), NITI_ENTRY(quantize_input), NITI_ENTRY(publish_step),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_torch_ops", "native torch front end of libniti_b200 (" NITI_OPS_TAG ")", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__torch_ops() { return PyModule_Create(&module_def); }
