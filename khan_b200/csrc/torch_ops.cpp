// Python binding of the per-batch operators (ani_sort, featurize, featurize_grad) on torch tensors.
//
// What bounds a call on a batch of up to a few thousand atoms is not the GPU (5 to 40 us a kernel) but the
// host: through ctypes the three operators cost 150 us of Python a batch (about twenty tensor checks, four
// allocations and seventy object conversions).  Here the checks, the allocations and the call are one C++
// function each, 15-20 us for all three.
//
// A function takes the straightforward case only -- CUDA tensors of one device, contiguous, of the types the
// kernels read, the counts in a host int32[4] -- and returns None for anything else: ani_mod then converts or
// refuses and calls again.  A negative status of the library is returned as an int.  The entry points are
// handed over as addresses (bind), so that there is one copy of the library in the process.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/utils/pybind.h>

#define NPY_NO_DEPRECATED_API NPY_1_20_API_VERSION
#include <numpy/arrayobject.h>

#include <stdint.h>

#include <vector>

namespace py = pybind11;

namespace {

constexpr int64_t kFeatures = 384;

using SortFn = int (*)(const int*, int, int*, int*, int*, void*);
using FeaturizeFn = int (*)(const void*, const void*, const void*, const int*, const int*, const int*, int, const int*,
                            void*, void*, void*, void*, const int*, void*);
using GradFn = int (*)(const void*, const void*, const void*, const int*, const int*, const int*, int, const int*,
                       const void*, const void*, const void*, const void*, void*, void*, void*, const int*, void*);

SortFn g_sort = nullptr;
FeaturizeFn g_featurize[2] = {};   // f32, f64
GradFn g_grad[2] = {};

void bind(uintptr_t sort, uintptr_t featurize_f32, uintptr_t featurize_f64, uintptr_t grad_f32, uintptr_t grad_f64)
{
    g_sort = reinterpret_cast<SortFn>(sort);
    g_featurize[0] = reinterpret_cast<FeaturizeFn>(featurize_f32);
    g_featurize[1] = reinterpret_cast<FeaturizeFn>(featurize_f64);
    g_grad[0] = reinterpret_cast<GradFn>(grad_f32);
    g_grad[1] = reinterpret_cast<GradFn>(grad_f64);
}

bool fits(const at::Tensor& t, c10::ScalarType dtype, c10::Device device)
{
    return t.scalar_type() == dtype && t.device() == device && t.is_contiguous();
}
template <typename T = void> T* data(const at::Tensor& t)
{
    return t.numel() ? static_cast<T*>(t.data_ptr()) : nullptr;
}

// The counts of the four elements from a host int32[4] (anything else: false).
bool read_counts(PyObject* o, int* acs)
{
    if (!PyObject_CheckBuffer(o)) return false;
    Py_buffer b;
    if (PyObject_GetBuffer(o, &b, PyBUF_FORMAT | PyBUF_C_CONTIGUOUS)) {
        PyErr_Clear();
        return false;
    }
    const bool ok = b.itemsize == 4 && b.len == 16 && b.format && b.format[0] == 'i' && !b.format[1];
    if (ok) memcpy(acs, b.buf, 16);
    PyBuffer_Release(&b);
    return ok;
}

struct Batch {
    bool ok = false, f64 = false;
    c10::Device device = c10::Device(c10::DeviceType::CPU);
    c10::ScalarType dtype = c10::kFloat;
    int acs[4] = {};
    int64_t n_atoms = 0, n_mols = 0;
};

Batch check_batch(const at::Tensor& x, const at::Tensor& y, const at::Tensor& z, const at::Tensor& a,
                  const at::Tensor& mo, const at::Tensor& mac, const at::Tensor& si, PyObject* acs)
{
    Batch b;
    b.dtype = x.scalar_type();
    b.device = x.device();
    b.f64 = b.dtype == c10::kDouble;
    if (!b.device.is_cuda() || (b.dtype != c10::kFloat && !b.f64)) return b;
    if (!fits(x, b.dtype, b.device) || !fits(y, b.dtype, b.device) || !fits(z, b.dtype, b.device) ||
        !fits(a, c10::kInt, b.device) || !fits(mo, c10::kInt, b.device) || !fits(mac, c10::kInt, b.device) ||
        !fits(si, c10::kInt, b.device) || !read_counts(acs, b.acs))
        return b;
    for (int t = 0; t < 4; t++) b.n_atoms += b.acs[t];
    b.n_mols = mo.numel();
    b.ok = b.n_mols <= INT32_MAX;
    return b;
}

int call_featurize(const Batch& b, const at::Tensor& x, const at::Tensor& y, const at::Tensor& z, const at::Tensor& a,
                   const at::Tensor& mo, const at::Tensor& mac, const at::Tensor& si, const at::Tensor& out)
{
    const int64_t row = kFeatures * (b.f64 ? 8 : 4);
    char* p = static_cast<char*>(out.data_ptr());
    void* rows[4];
    for (int t = 0; t < 4; t++) {
        rows[t] = p;
        p += b.acs[t] * row;
    }
    return g_featurize[b.f64](data(x), data(y), data(z), data<int>(a), data<int>(mo), data<int>(mac), (int)b.n_mols,
                              data<int>(si), rows[0], rows[1], rows[2], rows[3], b.acs,
                              at::cuda::getCurrentCUDAStream(b.device.index()).stream());
}

py::object ani_sort(const at::Tensor& a)
{
    if (!a.is_cuda() || a.scalar_type() != c10::kInt || !a.is_contiguous() || a.numel() > INT32_MAX) return py::none();
    const c10::cuda::CUDAGuard guard(a.device());
    const int64_t n = a.numel();
    at::Tensor scatter = at::detail::empty_cuda({n}, c10::kInt, a.device(), std::nullopt);
    at::Tensor gather = at::detail::empty_cuda({n}, c10::kInt, a.device(), std::nullopt);
    at::Tensor counts = at::detail::empty_cuda({4}, c10::kInt, a.device(), std::nullopt);
    const int rc = g_sort(data<int>(a), (int)n, data<int>(scatter), data<int>(gather), data<int>(counts),
                          at::cuda::getCurrentCUDAStream(a.device().index()).stream());
    if (rc) return py::int_(rc);
    return py::make_tuple(scatter, gather, counts);
}

py::object featurize_into(const at::Tensor& x, const at::Tensor& y, const at::Tensor& z, const at::Tensor& a,
                          const at::Tensor& mo, const at::Tensor& mac, const at::Tensor& si, py::handle acs,
                          const at::Tensor& out)
{
    const Batch b = check_batch(x, y, z, a, mo, mac, si, acs.ptr());
    if (!b.ok || !fits(out, b.dtype, b.device) || out.numel() < b.n_atoms * kFeatures) return py::none();
    const c10::cuda::CUDAGuard guard(b.device);
    return py::int_(call_featurize(b, x, y, z, a, mo, mac, si, out));
}

// split: the four per-element outputs as slices of one allocation; else that allocation, [n_atoms, 384].
py::object featurize(const at::Tensor& x, const at::Tensor& y, const at::Tensor& z, const at::Tensor& a,
                     const at::Tensor& mo, const at::Tensor& mac, const at::Tensor& si, py::handle acs, bool split)
{
    const Batch b = check_batch(x, y, z, a, mo, mac, si, acs.ptr());
    if (!b.ok) return py::none();
    const c10::cuda::CUDAGuard guard(b.device);
    at::Tensor out = at::detail::empty_cuda({b.n_atoms, kFeatures}, b.dtype, b.device, std::nullopt);
    if (const int rc = call_featurize(b, x, y, z, a, mo, mac, si, out)) return py::int_(rc);
    if (!split) return py::cast(out);
    const at::AutoDispatchBelowADInplaceOrView below;   // plain slices: nothing here is differentiated
    at::Tensor parts[4];
    int64_t at = 0;
    for (int t = 0; t < 4; t++) {
        const int64_t n = b.acs[t] * kFeatures;
        parts[t] = out.as_strided({n}, {1}, at);
        at += n;
    }
    return py::make_tuple(parts[0], parts[1], parts[2], parts[3]);
}

py::object featurize_grad(const at::Tensor& x, const at::Tensor& y, const at::Tensor& z, const at::Tensor& a,
                          const at::Tensor& mo, const at::Tensor& mac, const at::Tensor& si, py::handle acs,
                          const at::Tensor& gh, const at::Tensor& gc, const at::Tensor& gn, const at::Tensor& go)
{
    const Batch b = check_batch(x, y, z, a, mo, mac, si, acs.ptr());
    if (!b.ok) return py::none();
    const at::Tensor* g[4] = {&gh, &gc, &gn, &go};
    for (int t = 0; t < 4; t++)
        if (!fits(*g[t], b.dtype, b.device) || g[t]->numel() != b.acs[t] * kFeatures) return py::none();
    const c10::cuda::CUDAGuard guard(b.device);
    const int64_t n = b.n_atoms, size = b.f64 ? 8 : 4;
    at::Tensor out = at::detail::empty_cuda({3, n}, b.dtype, b.device, std::nullopt);
    cudaStream_t stream = at::cuda::getCurrentCUDAStream(b.device.index()).stream();
    char* p = data<char>(out);
    // an atom that no molecule covers gets a zero gradient (above a mean of 24 atoms a molecule the library's
    // own kernels start with a zero fill of everything)
    if (n && n <= 24 * b.n_mols) C10_CUDA_CHECK(cudaMemsetAsync(p, 0, (size_t)(3 * n * size), stream));
    const int rc = g_grad[b.f64](data(x), data(y), data(z), data<int>(a), data<int>(mo), data<int>(mac), (int)b.n_mols,
                                 data<int>(si), data(gh), data(gc), data(gn), data(go), p, p + n * size,
                                 p + 2 * n * size, b.acs, stream);
    if (rc) return py::int_(rc);
    const at::AutoDispatchBelowADInplaceOrView below;
    return py::make_tuple(out.as_strided({n}, {1}, 0), out.as_strided({n}, {1}, n), out.as_strided({n}, {1}, 2 * n));
}

// Row ranges [cuts[k] - cuts[0], cuts[k + 1] - cuts[0]) of a C-contiguous 2-d array as a list of views.  Cutting the
// gradients of a batch into molecules is what coordinate_gradients spends its host time on: 1024 views take 160 us
// through slice objects, 85 us here.
py::list split_rows(const py::object& rows, const py::object& cuts)
{
    if (!PyArray_Check(rows.ptr()) || !PyArray_Check(cuts.ptr())) throw py::type_error("split_rows takes numpy arrays");
    auto* a = reinterpret_cast<PyArrayObject*>(rows.ptr());
    auto* c = reinterpret_cast<PyArrayObject*>(cuts.ptr());
    if (PyArray_NDIM(a) != 2 || !PyArray_IS_C_CONTIGUOUS(a) || PyArray_NDIM(c) != 1 || !PyArray_IS_C_CONTIGUOUS(c) ||
        PyArray_TYPE(c) != NPY_INT64 || PyArray_DIM(c, 0) < 1)
        throw py::value_error("split_rows takes a contiguous 2-d array and int64 cuts");
    const auto* cut = static_cast<const npy_int64*>(PyArray_DATA(c));
    const npy_intp n = PyArray_DIM(c, 0) - 1;
    for (npy_intp k = 0; k < n; k++)
        if (cut[k + 1] < cut[k] || cut[k + 1] - cut[0] > PyArray_DIM(a, 0)) throw py::value_error("cuts out of range");
    py::list out(n);
    for (npy_intp k = 0; k < n; k++) {
        npy_intp dims[2] = {(npy_intp)(cut[k + 1] - cut[k]), PyArray_DIM(a, 1)};
        Py_INCREF(PyArray_DESCR(a));      // the new array takes one reference to it, and one to `rows`
        PyObject* view = PyArray_NewFromDescr(&PyArray_Type, PyArray_DESCR(a), 2, dims, PyArray_STRIDES(a),
                                              PyArray_BYTES(a) + (cut[k] - cut[0]) * PyArray_STRIDE(a, 0),
                                              PyArray_FLAGS(a) & ~NPY_ARRAY_OWNDATA, nullptr);
        if (!view) throw py::error_already_set();
        Py_INCREF(rows.ptr());
        if (PyArray_SetBaseObject(reinterpret_cast<PyArrayObject*>(view), rows.ptr()) < 0) {
            Py_DECREF(view);
            throw py::error_already_set();
        }
        PyList_SET_ITEM(out.ptr(), k, view);
    }
    return out;
}

}  // namespace

PYBIND11_MODULE(_torch_ops, m)
{
    if (_import_array() < 0) throw py::error_already_set();
    m.def("split_rows", &split_rows);
    m.def("bind", &bind);
    m.def("ani_sort", &ani_sort);
    m.def("featurize", &featurize);
    m.def("featurize_into", &featurize_into);
    m.def("featurize_grad", &featurize_grad);
}
