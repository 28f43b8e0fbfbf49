// The grouped GEMM's call as a CPython function: reading six tensors' types, shapes and strides through the interpreter and
// converting twenty arguments for ctypes takes longer than a decode kernel runs (a decode call of 16 tokens,
// 32 of 256 experts, N = 1024, K = 2048: 11.5 us among others by the general way, 6.1 with this function, which then is the kernels'
// time, each overlapping the next).
//
// It takes ordinary calls only -- plain CUDA tensors of the current device, shapes and types that fit -- and answers None to
// anything else, tensors without storage included; _C.py then goes through its conditions one by one and names the one
// that does not hold.  The C ABI's entry point comes from the caller (bind), so that nothing here is linked to it.
#include <torch/csrc/autograd/python_variable.h>

#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include <algorithm>

#include "../../include/nvfp4_b200.h"

namespace {

decltype(&nvfp4_grouped_gemm_contiguous) g_gemm = nullptr;

// A torch.Tensor or Parameter whose memory is on a CUDA device, else nullptr.  dim < 0: any number of dimensions.
const at::Tensor* plain(PyObject* o, at::ScalarType type, int64_t dim)
{
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    return t.is_cuda() && t.layout() == at::kStrided && t.has_storage() && t.scalar_type() == type && (dim < 0 || t.dim() == dim) ? &t : nullptr;
}

// The interpreter goes on while the library launches, as it does under ctypes.
struct Unlocked {
    PyThreadState* state = PyEval_SaveThread();
    ~Unlocked() { PyEval_RestoreThread(state); }
};

PyObject* bind(PyObject*, PyObject* address)
{
    void* p = PyLong_AsVoidPtr(address);
    if (p == nullptr && PyErr_Occurred()) return nullptr;
    g_gemm = reinterpret_cast<decltype(g_gemm)>(p);
    Py_RETURN_NONE;
}

// contiguous(a, b, sfb, gw, d, m_indices, policy code, residual pass, orientation, m_alignment) -> error code, or None
PyObject* contiguous(PyObject*, PyObject* const* args, Py_ssize_t count)
{
    if (count != 10) { PyErr_SetString(PyExc_TypeError, "contiguous() takes ten arguments"); return nullptr; }
    int option[4];
    for (int i = 0; i < 4; ++i) {
        const long value = PyLong_Check(args[6 + i]) ? PyLong_AsLong(args[6 + i]) : -1;
        if (PyErr_Occurred()) PyErr_Clear();
        if (value < 0 || value > INT32_MAX) Py_RETURN_NONE;
        option[i] = static_cast<int>(value);
    }
    try {
        const at::Tensor* a = plain(args[0], at::kBFloat16, 2);
        const at::Tensor* b = plain(args[1], at::kChar, 2);
        const at::Tensor* sfb = plain(args[2], at::kInt, 2);
        const at::Tensor* gw = plain(args[3], at::kFloat, -1);
        const at::Tensor* d = plain(args[4], at::kBFloat16, 2);
        const at::Tensor* m_indices = plain(args[5], at::kInt, 1);
        if (g_gemm == nullptr || a == nullptr || b == nullptr || sfb == nullptr || gw == nullptr || d == nullptr || m_indices == nullptr)
            Py_RETURN_NONE;
        const int64_t m = a->size(0), k = a->size(1), n = d->size(1), e = gw->numel();
        if (m > INT32_MAX || k > INT32_MAX || n > INT32_MAX || e > INT32_MAX || d->size(0) != m || m_indices->size(0) != m || b->size(0) != e * n ||
            b->size(1) != k / 2 || sfb->size(0) != e * (k / 64) || sfb->size(1) != n || a->stride(1) != 1 || d->stride(1) != 1 ||
            !b->is_contiguous() || !sfb->is_contiguous() || !gw->is_contiguous() || !m_indices->is_contiguous())
            Py_RETURN_NONE;
        const auto device = a->get_device();
        if (b->get_device() != device || sfb->get_device() != device || gw->get_device() != device || d->get_device() != device ||
            m_indices->get_device() != device || c10::cuda::current_device() != device)
            Py_RETURN_NONE;
        // the stride of a single row is not used, and may be anything
        const int64_t lda = m > 1 ? a->stride(0) : std::max<int64_t>(a->stride(0), k), ldd = m > 1 ? d->stride(0) : std::max<int64_t>(d->stride(0), n);
        const void *pa = a->data_ptr(), *pb = b->data_ptr(), *psfb = sfb->data_ptr(), *pm = m_indices->data_ptr();
        const float* pgw = static_cast<const float*>(gw->data_ptr());
        void* pd = d->data_ptr();
        cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device).stream();
        int rc = 0;
        {
            Unlocked unlocked;
            rc = g_gemm(pa, lda, pb, psfb, pgw, pd, ldd, static_cast<const int32_t*>(pm), static_cast<int>(m), static_cast<int>(n),
                        static_cast<int>(k), static_cast<int>(e), option[0], option[1], option[2], option[3], nullptr, nullptr, stream);
        }
        return PyLong_FromLong(rc);
    } catch (const std::exception&) {       // a tensor that has no memory to point at: the general path says so
        Py_RETURN_NONE;
    }
}

PyMethodDef kMethods[] = {
    {"bind", bind, METH_O, nullptr},
    {"contiguous", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(contiguous)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding() { return PyModule_Create(&kModule); }
