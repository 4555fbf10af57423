// Native half of kaio_b200/ops.py: one function per C-ABI entry point that unpacks the Python
// arguments, checks every tensor and calls libkaio_b200.so.
//
// Why it exists: a decode step is a few microseconds of GPU work per call.  The ctypes route cost
// 12-16 us of host time per call (a wrapper object per argument, two device-guard context switches,
// a stream query through three Python layers), so every small call was bound by the host, not by
// its kernel.  Here a call is one vectorcall, a pass over the argument array and one C call.
//
// A binding is a list of argument kinds, each of which turns one Python object into the C
// arguments it stands for: Buf<T> (a contiguous CUDA tensor of type T -> pointer, element count),
// Ptr (an address), Ptrs (a sequence of addresses -> an array), U32, I32, SZ, F32.  The stream comes
// last, from the KaioDevice.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <tuple>
#include <utility>

#include "../../include/kaio_b200.h"

namespace {

PyObject* g_from_code = nullptr;  // kaio_b200.errors.from_code
PyObject* g_device_type = nullptr;  // kaio_b200.ops.KaioDevice
PyObject *g_ordinal = nullptr, *g_stream = nullptr, *g_cuda_stream = nullptr, *g_stream_handle = nullptr;  // names

struct ArgError {};  // a Python exception has been set

const char* dtype_name(c10::ScalarType t)
{
    switch (t) {
    case c10::kChar: return "torch.int8";
    case c10::kInt: return "torch.int32";
    case c10::kHalf: return "torch.float16";
    case c10::kFloat: return "torch.float32";
    case c10::kDouble: return "torch.float64";
    case c10::kBFloat16: return "torch.bfloat16";
    case c10::kByte: return "torch.uint8";
    case c10::kShort: return "torch.int16";
    case c10::kLong: return "torch.int64";
    case c10::kBool: return "torch.bool";
    default: return c10::toString(t);
    }
}

// ---------------------------------------------------------------- argument kinds
struct Data {
    void* ptr;
    size_t numel;
};

Data unpack_tensor(PyObject* o, c10::ScalarType dtype, const char* what)
{
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "%s: expected a torch.Tensor, got %s", what, Py_TYPE(o)->tp_name);
        throw ArgError();
    }
    const at::Tensor& t = THPVariable_Unpack(o);
    if (t.scalar_type() != dtype) {
        PyErr_Format(PyExc_TypeError, "%s: expected dtype %s, got %s", what, dtype_name(dtype),
                     dtype_name(t.scalar_type()));
        throw ArgError();
    }
    if (!t.is_cuda()) {
        PyErr_Format(PyExc_TypeError, "%s: expected a CUDA tensor (there is no CPU fallback)", what);
        throw ArgError();
    }
    if (!t.is_contiguous()) {
        PyErr_Format(PyExc_TypeError, "%s: expected a contiguous tensor", what);
        throw ArgError();
    }
    return {t.data_ptr(), (size_t)t.numel()};
}

struct S8 { using type = int8_t; static constexpr auto dtype = c10::kChar; };
struct S32 { using type = int32_t; static constexpr auto dtype = c10::kInt; };
struct U32w { using type = uint32_t; static constexpr auto dtype = c10::kInt; };  // u32 words in an int32 tensor
struct F16 { using type = kaio_f16; static constexpr auto dtype = c10::kHalf; };
struct F32t { using type = float; static constexpr auto dtype = c10::kFloat; };

template <class T>
struct Buf {
    static auto get(PyObject* o, const char* what)
    {
        const Data d = unpack_tensor(o, T::dtype, what);
        return std::make_tuple(static_cast<typename T::type*>(d.ptr), d.numel);
    }
};

// A buffer without its length (the op takes one length for several buffers).
template <class T>
struct BufPtr {
    static auto get(PyObject* o, const char* what)
    {
        return std::make_tuple(static_cast<typename T::type*>(unpack_tensor(o, T::dtype, what).ptr));
    }
};

// None stands for "no buffer".
template <class T>
struct OptBuf {
    static auto get(PyObject* o, const char* what)
    {
        if (o == Py_None)
            return std::make_tuple(static_cast<typename T::type*>(nullptr), (size_t)0);
        return Buf<T>::get(o, what);
    }
};

struct AnyBuf {  // f16 or f32, as void*
    static auto get(PyObject* o, const char* what)
    {
        const bool half = THPVariable_Check(o) && THPVariable_Unpack(o).scalar_type() == c10::kHalf;
        const Data d = unpack_tensor(o, half ? c10::kHalf : c10::kFloat, what);
        return std::make_tuple(d.ptr, d.numel);
    }
};

// An int or whatever stands for one (a numpy integer, an integer tensor of one element), modulo 2^64.
unsigned long long unpack_int(PyObject* o, const char* what)
{
    PyObject* i = PyNumber_Index(o);
    if (!i) {
        if (PyErr_ExceptionMatches(PyExc_TypeError))
            PyErr_Format(PyExc_TypeError, "%s: expected an int, got %s", what, Py_TYPE(o)->tp_name);
        throw ArgError();
    }
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(i);
    Py_DECREF(i);
    return v;
}

struct U32 { static auto get(PyObject* o, const char* w) { return std::make_tuple((uint32_t)unpack_int(o, w)); } };
struct I32 { static auto get(PyObject* o, const char* w) { return std::make_tuple((int32_t)unpack_int(o, w)); } };
struct SZ { static auto get(PyObject* o, const char* w) { return std::make_tuple((size_t)unpack_int(o, w)); } };

template <class T>
struct Ptr { static auto get(PyObject* o, const char* w) { return std::make_tuple(reinterpret_cast<T*>(unpack_int(o, w))); } };

struct F32 {
    static auto get(PyObject* o, const char*)
    {
        const double v = PyFloat_AsDouble(o);
        if (v == -1.0 && PyErr_Occurred())
            throw ArgError();
        return std::make_tuple((float)v);
    }
};

struct PtrArray {
    void* p[8] = {};
    operator void* const*() const { return p; }
};
struct Ptrs {  // up to eight addresses; the C side rejects a world / num_out above eight before it reads them
    static auto get(PyObject* o, const char* what)
    {
        PtrArray a;
        PyObject* seq = PySequence_Fast(o, "expected a sequence of device addresses");
        if (!seq)
            throw ArgError();
        const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
        try {
            for (Py_ssize_t i = 0; i < n && i < 8; ++i)
                a.p[i] = reinterpret_cast<void*>(unpack_int(PySequence_Fast_GET_ITEM(seq, i), what));
        } catch (ArgError&) {
            Py_DECREF(seq);
            throw;
        }
        Py_DECREF(seq);
        return std::make_tuple(a);
    }
};

// ---------------------------------------------------------------- the call
// Makes the KaioDevice's device current for the call (restored when it was another one) and finds
// its stream: the one it was created with, else torch's current stream of that device.  Another type
// of device is asked for its stream_handle().
struct DeviceScope {
    c10::DeviceIndex before, mine;
    void* stream = nullptr;

    explicit DeviceScope(PyObject* dev)
    {
        PyObject* o = attribute(dev, g_ordinal);
        const long ord = PyLong_AsLong(o);
        Py_DECREF(o);
        if (ord == -1 && PyErr_Occurred())
            throw ArgError();
        mine = (c10::DeviceIndex)ord;
        PyObject* handle = nullptr;
        if (reinterpret_cast<PyObject*>(Py_TYPE(dev)) == g_device_type) {
            PyObject* s = attribute(dev, g_stream);
            if (s == Py_None)
                stream = c10::cuda::getCurrentCUDAStream(mine).stream();
            else
                handle = PyObject_GetAttr(s, g_cuda_stream);
            Py_DECREF(s);
        } else {
            handle = PyObject_CallMethodNoArgs(dev, g_stream_handle);
        }
        if (handle) {
            stream = reinterpret_cast<void*>(PyLong_AsUnsignedLongLongMask(handle));
            Py_DECREF(handle);
        }
        if (PyErr_Occurred())
            throw ArgError();
        before = c10::cuda::current_device();
        if (before != mine)
            c10::cuda::set_device(mine);
    }
    ~DeviceScope()
    {
        if (before != mine)
            (void)c10::cuda::MaybeSetDevice(before);  // set_device would throw, out of a destructor
    }

    static PyObject* attribute(PyObject* o, PyObject* name)
    {
        PyObject* v = PyObject_GetAttr(o, name);
        if (!v)
            throw ArgError();
        return v;
    }
};

// Held again at the end of the scope, whichever way it is left: what the library throws (memory) is
// turned into a Python exception further up.
struct WithoutGil {
    PyThreadState* state = PyEval_SaveThread();
    ~WithoutGil() { PyEval_RestoreThread(state); }
};

PyObject* raise_code(int32_t code)
{
    const char* text = kaio_b200_last_error();
    PyObject* message = PyUnicode_DecodeUTF8(text, (Py_ssize_t)strlen(text), "replace");  // it may be cut anywhere
    PyObject* e = message ? PyObject_CallFunction(g_from_code, "iO", (int)code, message) : nullptr;
    Py_XDECREF(message);
    if (e) {
        PyErr_SetObject(reinterpret_cast<PyObject*>(Py_TYPE(e)), e);
        Py_DECREF(e);
    }
    return nullptr;
}

template <class... Kinds, class Fn, size_t... I>
PyObject* call(Fn fn, const char* const* names, PyObject* const* args, Py_ssize_t n, std::index_sequence<I...>)
{
    if (n != (Py_ssize_t)sizeof...(Kinds) + 1) {
        PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", (Py_ssize_t)sizeof...(Kinds) + 1, n);
        return nullptr;
    }
    try {
        // braces: from left to right, so that the first argument that is wrong is the one reported
        std::tuple<decltype(Kinds::get(args[I + 1], names[I]))...> each{Kinds::get(args[I + 1], names[I])...};
        auto c_args = std::apply([](const auto&... a) { return std::tuple_cat(a...); }, each);
        int32_t code;
        {
            DeviceScope scope(args[0]);
            WithoutGil nogil;
            code = std::apply([&](const auto&... a) { return fn(a..., scope.stream); }, c_args);
        }
        if (code != 0)
            return raise_code(code);
    } catch (ArgError&) {
        return nullptr;
    } catch (const std::exception& e) {
        if (!PyErr_Occurred())
            PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
    Py_RETURN_NONE;
}

// BIND(python name, C function, names of the arguments for error texts, kinds...)
#define L(...) ({__VA_ARGS__})
#define UNPAREN(...) __VA_ARGS__
#define BIND(py, cfn, names, ...)                                                                    \
    PyObject* py_##py(PyObject*, PyObject* const* args, Py_ssize_t n)                                \
    {                                                                                                \
        static const char* const w[] = UNPAREN names;                                                \
        return call_of<__VA_ARGS__>(cfn, w, args, n);                                                \
    }

template <class... Kinds, class Fn>
PyObject* call_of(Fn fn, const char* const* names, PyObject* const* args, Py_ssize_t n)
{
    return call<Kinds...>(fn, names, args, n, std::index_sequence_for<Kinds...>());
}

BIND(matmul_int8, kaio_b200_matmul_int8, L("a", "b", "c", "scale", "m", "n", "k"),
     Buf<S8>, Buf<S8>, Buf<F32t>, F32, U32, U32, U32)
BIND(matmul_int8_scaled, kaio_b200_matmul_int8_scaled, L("a", "b", "c", "a_scale", "w_scale", "m", "n", "k"),
     Buf<S8>, Buf<S8>, Buf<F32t>, Buf<F32t>, Buf<F32t>, U32, U32, U32)
BIND(matmul_int8_acc, kaio_b200_matmul_int8_acc, L("a", "b", "acc", "m", "n", "k"),
     Buf<S8>, Buf<S8>, Buf<S32>, U32, U32, U32)
BIND(matmul_tc, kaio_b200_matmul_tc, L("a", "b", "c", "m", "n", "k"),
     Buf<F16>, Buf<F16>, Buf<F32t>, U32, U32, U32)
BIND(matmul_tc_async, kaio_b200_matmul_tc_async, L("a", "b", "c", "m", "n", "k"),
     Buf<F16>, Buf<F16>, Buf<F32t>, U32, U32, U32)
BIND(matmul_tc_f16out, kaio_b200_matmul_tc_f16out, L("a", "b", "c", "m", "n", "k"),
     Buf<F16>, Buf<F16>, Buf<F16>, U32, U32, U32)
BIND(dequantize_int4, kaio_b200_dequantize_int4, L("b_packed", "scales", "w", "k", "n", "group_size"),
     Buf<U32w>, Buf<F16>, Buf<F16>, U32, U32, U32)
BIND(matmul_int4, kaio_b200_matmul_int4, L("a", "b_packed", "scales", "c", "m", "n", "k", "group_size"),
     Buf<F16>, Buf<U32w>, Buf<F16>, Buf<F32t>, U32, U32, U32, U32)
BIND(matmul_int4_f16out, kaio_b200_matmul_int4_f16out,
     L("a", "b_packed", "scales", "c", "m", "n", "k", "group_size"),
     Buf<F16>, Buf<U32w>, Buf<F16>, Buf<F16>, U32, U32, U32, U32)
BIND(matmul_int4_allgather, kaio_b200_matmul_int4_allgather,
     L("a", "b_packed_shard", "scales_shard", "out_ptrs", "out_numel", "world", "rank", "m", "n_total", "k",
       "group_size"),
     Buf<F16>, Buf<U32w>, Buf<F16>, Ptrs, SZ, U32, U32, U32, U32, U32, U32)
BIND(matmul_int4_allgather_multicast, kaio_b200_matmul_int4_allgather_multicast,
     L("a", "b_packed_shard", "scales_shard", "out_ptrs", "out_numel", "multicast_out", "world", "rank", "m",
       "n_total", "k", "group_size"),
     Buf<F16>, Buf<U32w>, Buf<F16>, Ptrs, SZ, Ptr<void>, U32, U32, U32, U32, U32, U32)
BIND(allgather_cols, kaio_b200_allgather_cols,
     L("shard", "out", "m", "n_total", "elem_bytes", "world", "nccl_comm"),
     AnyBuf, AnyBuf, U32, U32, U32, U32, Ptr<void>)
BIND(matmul_int4_peer_partials, kaio_b200_matmul_int4_peer_partials,
     L("a", "b_packed", "scales", "slot_ptrs", "slot_numel", "world", "rank", "scatter", "m", "n", "k",
       "group_size"),
     Buf<F16>, Buf<U32w>, Buf<F16>, Ptrs, SZ, U32, U32, I32, U32, U32, U32, U32)
BIND(sum_partials_f32, kaio_b200_sum_partials_f32,
     L("slots", "world", "rows", "cols", "out_ptrs", "num_out", "out_numel", "out_ld", "out_col0"),
     Buf<F32t>, U32, U32, U32, Ptrs, U32, SZ, U32, U32)
BIND(sum_partials_f32_multicast, kaio_b200_sum_partials_f32_multicast,
     L("slots", "world", "rows", "cols", "multicast_out", "out_numel", "out_ld", "out_col0"),
     Buf<F32t>, U32, U32, U32, Ptr<void>, SZ, U32, U32)
BIND(matmul_int4_silu_gate, kaio_b200_matmul_int4_silu_gate,
     L("x", "b_packed", "scales", "act", "gu_scratch", "m", "cols", "k", "group_size"),
     Buf<F16>, Buf<U32w>, Buf<F16>, Buf<F16>, OptBuf<F16>, U32, U32, U32, U32)
BIND(allreduce_multimem_f32, kaio_b200_allreduce_multimem_f32,
     L("multicast_in", "multicast_out", "numel", "rows", "cols", "ld", "col0"),
     Ptr<const void>, Ptr<void>, SZ, U32, U32, U32, U32)
BIND(qkv_project_int8, kaio_b200_qkv_project_int8,
     L("x", "w_q", "w_k", "w_v", "scale_q", "scale_k", "scale_v", "q_out", "k_out", "v_out", "m", "n", "k"),
     Buf<F16>, Buf<S8>, Buf<S8>, Buf<S8>, F32, F32, F32, Buf<F16>, Buf<F16>, Buf<F16>, U32, U32, U32)
BIND(qkv_project_int8_colscale, kaio_b200_qkv_project_int8_colscale,
     L("x", "w_q", "w_k", "w_v", "scale_q", "scale_k", "scale_v", "scale_len", "q_out", "k_out", "v_out", "m",
       "n", "k"),
     Buf<F16>, Buf<S8>, Buf<S8>, Buf<S8>, BufPtr<F32t>, BufPtr<F32t>, BufPtr<F32t>, SZ, Buf<F16>, Buf<F16>,
     Buf<F16>, U32, U32, U32)
BIND(qkv_project_w8a8, kaio_b200_qkv_project_w8a8,
     L("x", "w_q", "w_k", "w_v", "scale_q", "scale_k", "scale_v", "scale_len", "q_out", "k_out", "v_out", "m",
       "n", "k"),
     Buf<F16>, Buf<S8>, Buf<S8>, Buf<S8>, BufPtr<F32t>, BufPtr<F32t>, BufPtr<F32t>, SZ, Buf<F16>, Buf<F16>,
     Buf<F16>, U32, U32, U32)
BIND(qkv_project_int4, kaio_b200_qkv_project_int4,
     L("x", "w_q_packed", "w_k_packed", "w_v_packed", "scales_q", "scales_k", "scales_v", "q_out", "k_out",
       "v_out", "m", "n", "k", "group_size"),
     Buf<F16>, Buf<U32w>, Buf<U32w>, Buf<U32w>, Buf<F16>, Buf<F16>, Buf<F16>, Buf<F16>, Buf<F16>, Buf<F16>,
     U32, U32, U32, U32)
BIND(quantize_rows_int8, kaio_b200_quantize_rows_int8, L("x", "q", "scale", "m", "k"),
     Buf<F32t>, Buf<S8>, Buf<F32t>, U32, U32)
BIND(quantize_pack_int4, kaio_b200_quantize_pack_int4, L("w", "packed", "scales", "k", "n", "group_size"),
     Buf<F32t>, Buf<U32w>, Buf<F16>, U32, U32, U32)
BIND(silu_gate_f32, kaio_b200_silu_gate_f32, L("x", "gate", "out", "n"),
     Buf<F32t>, Buf<F32t>, Buf<F32t>, U32)
BIND(silu_gate_f16, kaio_b200_silu_gate_f16,
     L("x", "gate", "out", "rows", "cols", "x_ld", "gate_ld", "out_ld"),
     Buf<F16>, Buf<F16>, Buf<F16>, U32, U32, U32, U32, U32)
BIND(attention_tc, kaio_b200_attention_tc,
     L("q", "k", "v", "out", "seq_q", "seq_k", "d_k", "d_v", "causal"),
     Buf<F16>, Buf<F16>, Buf<F16>, Buf<F32t>, U32, U32, U32, U32, I32)
BIND(attention_mha_f16, kaio_b200_attention_mha_f16,
     L("q", "k", "v", "out", "batch", "heads", "seq_q", "seq_k", "head_dim", "row_stride", "causal"),
     Buf<F16>, Buf<F16>, Buf<F16>, Buf<F16>, U32, U32, U32, U32, U32, U32, I32)
BIND(selftest_bounded_wait, kaio_b200_selftest_bounded_wait, L("budget_us"), U32)

#define ENTRY(py) {#py, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##py)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {
    ENTRY(matmul_int8), ENTRY(matmul_int8_scaled), ENTRY(matmul_int8_acc), ENTRY(matmul_tc),
    ENTRY(matmul_tc_async), ENTRY(matmul_tc_f16out), ENTRY(dequantize_int4), ENTRY(matmul_int4),
    ENTRY(matmul_int4_f16out), ENTRY(matmul_int4_allgather), ENTRY(matmul_int4_allgather_multicast),
    ENTRY(allgather_cols), ENTRY(matmul_int4_peer_partials), ENTRY(sum_partials_f32),
    ENTRY(sum_partials_f32_multicast), ENTRY(matmul_int4_silu_gate), ENTRY(allreduce_multimem_f32),
    ENTRY(qkv_project_int8), ENTRY(qkv_project_int8_colscale), ENTRY(qkv_project_w8a8),
    ENTRY(qkv_project_int4), ENTRY(quantize_rows_int8), ENTRY(quantize_pack_int4), ENTRY(silu_gate_f32),
    ENTRY(silu_gate_f16), ENTRY(attention_tc), ENTRY(attention_mha_f16), ENTRY(selftest_bounded_wait),
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native()
{
    // compiled against one torch's C++ headers; another's tensors may be laid out differently
    PyObject* torch = PyImport_ImportModule("torch");
    PyObject* version = torch ? PyObject_GetAttrString(torch, "__version__") : nullptr;
    PyObject* text = version ? PyObject_Str(version) : nullptr;
    Py_XDECREF(torch);
    Py_XDECREF(version);
    if (!text)
        return nullptr;
    const bool same = PyUnicode_CompareWithASCIIString(text, KAIO_TORCH_VERSION) == 0;
    if (!same)
        PyErr_Format(PyExc_ImportError, "built for torch %s, this is torch %U", KAIO_TORCH_VERSION, text);
    Py_DECREF(text);
    if (!same)
        return nullptr;
    PyObject* errors = PyImport_ImportModule("kaio_b200.errors");
    if (!errors)
        return nullptr;
    g_from_code = PyObject_GetAttrString(errors, "from_code");
    Py_DECREF(errors);
    g_ordinal = PyUnicode_InternFromString("ordinal");
    g_stream = PyUnicode_InternFromString("_stream");
    g_cuda_stream = PyUnicode_InternFromString("cuda_stream");
    g_stream_handle = PyUnicode_InternFromString("stream_handle");
    PyObject* ops = PyImport_ImportModule("kaio_b200.ops");
    if (!ops)
        return nullptr;
    g_device_type = PyObject_GetAttrString(ops, "KaioDevice");
    Py_DECREF(ops);
    if (!g_from_code || !g_device_type || !g_ordinal || !g_stream || !g_cuda_stream || !g_stream_handle)
        return nullptr;
    return PyModule_Create(&g_module);
}
