// calls.cc - the launchers of libcai_kernels.so as Python functions (module _calls).
//
// An op on small tensors is bound by its host path, not by its kernel: of some 11 us a call of the 17 arguments of a product through ctypes takes
// 2.4 us, here 0.4. Each function takes its launcher's arguments in order (pointers as integers or None) and returns its result; the
// interpreter's lock is given up meanwhile, as by ctypes: a launch waits when the stream's queue is full.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <tuple>
#include <type_traits>
#include <utility>

#include "../comm/moe.h"
#include "../kernels/cai_kernels.h"

namespace {

// Like ctypes: integers are taken modulo their C type, None is a null pointer, a float parameter takes any real number.
template <typename T>
bool take(PyObject* o, T& out) {
    if constexpr (std::is_pointer_v<T>) {
        if (o == Py_None) {
            out = nullptr;
            return true;
        }
        const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
        out = reinterpret_cast<T>(static_cast<uintptr_t>(v));
    } else if constexpr (std::is_floating_point_v<T>) {
        out = static_cast<T>(PyFloat_AsDouble(o));
    } else {
        out = static_cast<T>(PyLong_AsUnsignedLongLongMask(o));
    }
    return !PyErr_Occurred();
}

template <auto kFunction> struct Call;
template <typename... Args, int (*kFunction)(Args...)> struct Call<kFunction> {
    static PyObject* run(PyObject*, PyObject* const* args, Py_ssize_t n) {
        if (n != static_cast<Py_ssize_t>(sizeof...(Args))) {
            PyErr_Format(PyExc_TypeError, "%zu arguments are wanted, %zd given", sizeof...(Args), n);
            return nullptr;
        }
        return go(args, std::index_sequence_for<Args...>());
    }
    template <size_t... I>
    static PyObject* go(PyObject* const* args, std::index_sequence<I...>) {
        std::tuple<Args...> v;
        if (!(take(args[I], std::get<I>(v)) && ...)) return nullptr;
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = kFunction(std::get<I>(v)...);
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(rc);
    }
};

#define CAI_CALL(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&Call<&f>::run)), METH_FASTCALL, nullptr}
PyMethodDef functions[] = {
    CAI_CALL(cai_gemm_bf16), CAI_CALL(cai_gemm_bf16_seg), CAI_CALL(cai_gemm_bf16_grouped),
    CAI_CALL(cai_gemm_fp8_blockscaled), CAI_CALL(cai_quant_rows_1x128), CAI_CALL(cai_quant_blocks_128x128),
    CAI_CALL(cai_moe_route_fwd), CAI_CALL(cai_moe_route_bwd),
    CAI_CALL(cai_rmsnorm_fwd), CAI_CALL(cai_rmsnorm_bwd_parts), CAI_CALL(cai_rmsnorm_bwd),
    CAI_CALL(cai_rope_table), CAI_CALL(cai_rope_apply), CAI_CALL(cai_swiglu_fwd), CAI_CALL(cai_swiglu_bwd),
    CAI_CALL(cai_embed_fwd), CAI_CALL(cai_embed_bwd), CAI_CALL(cai_cross_entropy), CAI_CALL(cai_adamw),
    CAI_CALL(cai_flash_attn_fwd_variant), CAI_CALL(cai_flash_attn_bwd_parts),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, functions, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() { return PyModule_Create(&module); }
