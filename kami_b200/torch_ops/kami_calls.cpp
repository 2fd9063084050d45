// kami_calls.cpp -- api.gemm_batched, api.spmm and api.spgemm as CPython
// functions over the C ABI of libkami_b200.so.
//
// A call of api.gemm_batched cost 11.3 us of host time (attribute reads and
// checks of each tensor, torch.empty, the ctypes conversion of 27 arguments),
// 3 us of them the launch: more than the kernel of a small batch takes.  Here
// the same checks and the same call take 3.5 us (1024 x 32^3 FP64, back to
// back: 11.7 us a call before, 8.2 after).  api.spgemm, whose host waits for the
// number of C tiles, saves the same on each of its calls (n = 16384 at 1 %: 83 us
// before, 71 after).
//
// Each function takes the calls it can make as they are and returns what the
// Python function returns; a failed call returns its status, for the caller to
// raise; anything else (another type, layout, device or argument than expected)
// returns NotImplemented, and the Python code runs, with its own checks and
// errors.  The entry points' addresses come from the loader (bind), so the
// calls go to the library that Python uses.  The interpreter lock is released
// around them, as ctypes does.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <climits>
#include <optional>

#include "kami.h"

namespace {

using at::Tensor;

decltype(&kami_gemm_batched) g_gemm = nullptr;
decltype(&kami_spmm_bsr) g_spmm = nullptr;
decltype(&kami_spgemm_bsr_symbolic) g_symbolic = nullptr;
decltype(&kami_spgemm_bsr_fill_numeric) g_fill_numeric = nullptr;

// What Python has to look at itself.
struct Decline
{
};

int type_of(at::ScalarType t)
{
    switch (t)
    {
    case at::kHalf: return KAMI_F16;
    case at::kBFloat16: return KAMI_BF16;
    case at::kDouble: return KAMI_F64;
    case at::kFloat: return KAMI_F32;
    default: throw Decline();
    }
}

const Tensor &tensor_of(PyObject *o)
{
    if (!THPVariable_CheckExact(o))
        throw Decline();
    const Tensor &t = THPVariable_Unpack(o);
    if (!t.is_cuda() || !t.has_storage())
        throw Decline();
    return t;
}

int to_int(int64_t v)
{
    if (v < INT_MIN || v > INT_MAX)
        throw Decline();
    return (int)v;
}

int int_of(PyObject *o)
{
    if (!PyLong_CheckExact(o))
        throw Decline();
    int over = 0;
    const long v = PyLong_AsLongAndOverflow(o, &over);
    if (over)
        throw Decline();
    return to_int(v);
}

double float_of(PyObject *o)
{
    if (PyFloat_CheckExact(o))
        return PyFloat_AS_DOUBLE(o);
    return int_of(o);
}

at::ScalarType dtype_of(PyObject *o)
{
    if (!THPDtype_Check(o))
        throw Decline();
    return reinterpret_cast<THPDtype *>(o)->scalar_type;
}

void same_device(const Tensor &a, const Tensor &b)
{
    if (a.device() != b.device())
        throw Decline();
}

// A [batch, rows, cols] operand; 2-D is a batch of one.
struct Operand
{
    const Tensor &t;
    int64_t batch, rows, cols, ld, stride;
    explicit Operand(const Tensor &x) : t(x)
    {
        const int64_t d = x.dim();
        if (d != 2 && d != 3)
            throw Decline();
        batch = d == 3 ? x.size(0) : 1;
        rows = x.size(d - 2);
        cols = x.size(d - 1);
        if (cols > 1 && x.stride(d - 1) != 1)
            throw Decline();
        ld = rows > 1 ? x.stride(d - 2) : cols;
        stride = batch > 1 ? x.stride(0) : 0;
    }
};

void *entries(const Tensor &t) { return t.numel() ? t.data_ptr() : nullptr; }

// Calls f without the interpreter lock, and holds it again however f ends: what
// catches an exception needs it.
template <class F> int unlocked(F &&f)
{
    struct Unlock
    {
        PyThreadState *const state = PyEval_SaveThread();
        ~Unlock() { PyEval_RestoreThread(state); }
    } unlock;
    return f();
}

// Runs f: a tensor (or tuple) object, or a status, or NotImplemented.
template <class F> PyObject *guarded(F &&f)
{
    try
    {
        if (at::impl::torch_function_mode_enabled())
            throw Decline();
        return f();
    }
    catch (const std::exception &)
    {
    }
    catch (const Decline &)
    {
    }
    PyErr_Clear();
    Py_RETURN_NOTIMPLEMENTED;
}

// gemm_batched(A, B, C | None, out_dtype | None, a_layout, b_layout, partition, variant, P, alloc_warps, num_iter,
//              alpha, beta)
PyObject *gemm_batched(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return guarded([&]() -> PyObject * {
        if (n != 13)
            throw Decline();
        const Operand A(tensor_of(a[0])), B(tensor_of(a[1]));
        if (A.t.scalar_type() != B.t.scalar_type())
            throw Decline();
        same_device(A.t, B.t);
        const int al = int_of(a[4]), bl = int_of(a[5]);
        const int M = to_int(al == KAMI_A_ROW_MK ? A.rows : A.cols), K = to_int(al == KAMI_A_ROW_MK ? A.cols : A.rows);
        const int N = to_int(bl == KAMI_B_REF_NK ? B.rows : B.cols);
        const int in = type_of(A.t.scalar_type());
        const int part = int_of(a[6]), variant = int_of(a[7]), P = int_of(a[8]), alloc = int_of(a[9]),
                  iters = int_of(a[10]);
        const double alpha = float_of(a[11]), beta = float_of(a[12]);
        const c10::cuda::CUDAGuard guard(A.t.device());
        Tensor made;
        if (a[2] == Py_None)
        {
            const at::ScalarType o = a[3] != Py_None ? dtype_of(a[3]) : in == KAMI_F64 ? at::kDouble : at::kFloat;
            type_of(o);
            made = at::empty({A.batch, M, N}, A.t.options().dtype(o).requires_grad(false));
        }
        const Tensor &Ct = a[2] == Py_None ? made : tensor_of(a[2]);
        same_device(A.t, Ct);
        const Operand C(Ct);
        const int out = type_of(Ct.scalar_type());
        const void *pa = A.t.data_ptr(), *pb = B.t.data_ptr();
        void *pc = Ct.data_ptr();
        void *stream = c10::cuda::getCurrentCUDAStream(A.t.device().index()).stream();
        const int st = unlocked([&] {
            return g_gemm((kami_dtype_t)in, (kami_dtype_t)out, (kami_partition_t)part, (kami_variant_t)variant, M, N, K, P,
                          alloc, A.batch, pa, A.ld, A.stride, (kami_a_layout_t)al, pb, B.ld, B.stride,
                          (kami_b_layout_t)bl, pc, C.ld, C.stride, alpha, beta, iters, nullptr, 0, stream);
        });
        if (st != KAMI_OK)
            return PyLong_FromLong(st);
        if (a[2] != Py_None)
            return Py_NewRef(a[2]);
        return THPVariable_Wrap(A.t.dim() == 2 ? made.select(0, 0) : made);
    });
}

// spmm(row_ptr, col_idx, values, block_rows, block_cols, B, C | None, out_dtype, b_layout, num_iter, alpha, beta)
PyObject *spmm(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return guarded([&]() -> PyObject * {
        if (n != 12)
            throw Decline();
        const Tensor &rp = tensor_of(a[0]), &ci = tensor_of(a[1]), &va = tensor_of(a[2]);
        const int mb = int_of(a[3]), kb = int_of(a[4]), bl = int_of(a[8]), iters = int_of(a[9]);
        const double alpha = float_of(a[10]), beta = float_of(a[11]);
        const Tensor &Bt = tensor_of(a[5]);
        if (Bt.dim() != 2 || Bt.stride(1) != 1)
            throw Decline();
        const int64_t K = (int64_t)kb * 16;
        const int N = to_int(bl == KAMI_B_ROW_KN ? Bt.size(1) : Bt.size(0));
        if ((bl == KAMI_B_ROW_KN ? Bt.size(0) : Bt.size(1)) != K)
            throw Decline();
        same_device(Bt, rp);
        same_device(Bt, ci);
        same_device(Bt, va);
        const c10::cuda::CUDAGuard guard(Bt.device());
        const Operand B(Bt);
        Tensor made;
        if (a[6] == Py_None)
            made = at::empty({(int64_t)mb * 16, N}, Bt.options().dtype(dtype_of(a[7])).requires_grad(false));
        const Tensor &C = a[6] == Py_None ? made : tensor_of(a[6]);
        same_device(Bt, C);
        if (C.dim() != 2)
            throw Decline();
        const int64_t ldc = C.size(0) > 1 ? C.stride(0) : C.size(1);
        const int in = type_of(va.scalar_type()), out = type_of(C.scalar_type());
        const int *prp = static_cast<const int *>(rp.data_ptr()), *pci = static_cast<const int *>(entries(ci));
        const void *pv = entries(va), *pb = Bt.data_ptr();
        void *pc = C.data_ptr();
        void *stream = c10::cuda::getCurrentCUDAStream(Bt.device().index()).stream();
        const int st = unlocked([&] {
            return g_spmm((kami_dtype_t)in, (kami_dtype_t)out, 16, mb, kb, N, 1, prp, pci, 0, 0, pv, 0, pb, B.ld, 0,
                          (kami_b_layout_t)bl, pc, ldc, 0, alpha, beta, iters, stream);
        });
        if (st != KAMI_OK)
            return PyLong_FromLong(st);
        return a[6] != Py_None ? Py_NewRef(a[6]) : THPVariable_Wrap(made);
    });
}

// spgemm(row_ptr_a, col_idx_a, values_a, block_rows_a, block_cols_a, row_ptr_b, col_idx_b, values_b, block_cols_b,
//        out_dtype, num_iter, variant): (row_ptr_c, col_idx_c, values_c)
PyObject *spgemm(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    return guarded([&]() -> PyObject * {
        if (n != 12)
            throw Decline();
        const Tensor &ra = tensor_of(a[0]), &ca = tensor_of(a[1]), &va = tensor_of(a[2]);
        const Tensor &rb = tensor_of(a[5]), &cb = tensor_of(a[6]), &vb = tensor_of(a[7]);
        for (const Tensor *t : {&ca, &va, &rb, &cb, &vb})
            same_device(ra, *t);
        const int mb = int_of(a[3]), kb = int_of(a[4]), nb = int_of(a[8]), iters = int_of(a[10]), variant = int_of(a[11]);
        if (mb < 0)
            throw Decline();
        const int in = type_of(va.scalar_type());
        const at::ScalarType o = dtype_of(a[9]);
        const int out = type_of(o);
        const c10::cuda::CUDAGuard guard(ra.device());
        const at::TensorOptions ints = at::TensorOptions().dtype(at::kInt).device(ra.device());
        const Tensor rc = at::empty({(int64_t)mb + 1}, ints);
        const int *pra = static_cast<const int *>(ra.data_ptr()), *pca = static_cast<const int *>(entries(ca));
        const int *prb = static_cast<const int *>(rb.data_ptr()), *pcb = static_cast<const int *>(entries(cb));
        const void *pva = entries(va), *pvb = entries(vb);
        int *prc = static_cast<int *>(rc.data_ptr());
        void *stream = c10::cuda::getCurrentCUDAStream(ra.device().index()).stream();
        // page-locked, so that its copy is one transfer (torch keeps and reuses the block)
        const Tensor count = at::empty({1}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
        int *pn = static_cast<int *>(count.data_ptr());
        int st = unlocked([&] { return g_symbolic(16, mb, kb, nb, pra, pca, prb, pcb, prc, pn, stream); });
        if (st != KAMI_OK)
            return PyLong_FromLong(st);
        const int nnz = *pn;
        const int64_t room = nnz > 0 ? nnz : 1;
        const Tensor cc = at::empty({room}, ints);
        int *pcc = static_cast<int *>(cc.data_ptr());
        const Tensor vc = at::empty({room, 16, 16}, ints.dtype(o));
        void *pvc = vc.data_ptr();
        int *pcn = nnz > 0 ? pcc : nullptr;
        if (nnz <= 0)
            pvc = nullptr;
        st = unlocked([&] {
            return g_fill_numeric((kami_variant_t)variant, (kami_dtype_t)in, (kami_dtype_t)out, 16, mb, kb, nb, pra, pca, pva,
                             prb, pcb, pvb, prc, pcn, pvc, nnz, 1.0, 0.0, iters, stream);
        });
        if (st != KAMI_OK)
            return PyLong_FromLong(st);
        PyObject *r = PyTuple_New(3);
        if (!r)
            return nullptr;
        PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(rc));
        PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(cc.slice(0, 0, nnz)));
        PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(vc.slice(0, 0, nnz)));
        return r;
    });
}

// bind(kami_gemm_batched, kami_spmm_bsr, kami_spgemm_bsr_symbolic, kami_spgemm_bsr_fill_numeric): their addresses
// in the loaded library
PyObject *bind(PyObject *, PyObject *args)
{
    unsigned long long p[4];
    if (!PyArg_ParseTuple(args, "KKKK", &p[0], &p[1], &p[2], &p[3]))
        return nullptr;
    g_gemm = reinterpret_cast<decltype(g_gemm)>(p[0]);
    g_spmm = reinterpret_cast<decltype(g_spmm)>(p[1]);
    g_symbolic = reinterpret_cast<decltype(g_symbolic)>(p[2]);
    g_fill_numeric = reinterpret_cast<decltype(g_fill_numeric)>(p[3]);
    Py_RETURN_NONE;
}

PyMethodDef g_methods[] = {
    {"bind", bind, METH_VARARGS, nullptr},
    {"gemm_batched", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(gemm_batched)), METH_FASTCALL, nullptr},
    {"spmm", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(spmm)), METH_FASTCALL, nullptr},
    {"spgemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(spgemm)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "kami_calls", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit_kami_calls(void) { return PyModule_Create(&g_module); }
