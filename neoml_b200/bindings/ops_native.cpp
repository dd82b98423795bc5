// The host side of the calls in neoml_b200/ops.py that a network issues by the dozen, in native code: argument checks, the
// result and work-space tensors, and the C ABI call.  A layer's kernels take a few microseconds at small batches; the
// same steps in Python (two torch.empty, a ctypes structure or two, fifteen converted arguments) took 15-20 us a call,
// here 5-7.
//
// Every function takes positional arguments and returns the result tensor; an int is the C ABI's error code; None means
// that an argument is not what this path takes (not a plain contiguous fp32 CUDA tensor, a size that does not fit): the
// caller then runs its own code, which raises or handles it.  Nothing is kept between calls.
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/python_arg_parser.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/cuda/CUDAStream.h>
#include "../../include/neoml_b200.h"

#include <exception>

namespace {

struct NotHere {}; // "run the Python code"

const at::Tensor& tensor(PyObject* o)
{
	if(!THPVariable_CheckExact(o)) throw NotHere();
	const at::Tensor& t = THPVariable_Unpack(o);
	if(!t.has_storage() || !t.is_cuda() || !t.is_contiguous()) throw NotHere();
	return t;
}

const float* data(PyObject* o) // None: null
{
	return o == Py_None ? nullptr : static_cast<const float*>(tensor(o).data_ptr());
}

const at::Tensor& fp32(PyObject* o)
{
	const at::Tensor& t = tensor(o);
	if(t.scalar_type() != at::kFloat) throw NotHere();
	return t;
}

int integer(PyObject* o)
{
	if(!PyLong_Check(o)) throw NotHere();
	int overflow = 0;
	const long v = PyLong_AsLongAndOverflow(o, &overflow);
	if(overflow != 0 || v < INT32_MIN || v > INT32_MAX) throw NotHere();
	return static_cast<int>(v);
}

int size_of(const at::Tensor& t, int dim)
{
	const int64_t v = t.size(dim);
	if(v > INT32_MAX) throw NotHere();
	return static_cast<int>(v);
}

float number(PyObject* o)
{
	if(PyFloat_CheckExact(o)) return static_cast<float>(PyFloat_AS_DOUBLE(o));
	return static_cast<float>(integer(o));
}

bool truth(PyObject* o)
{
	const int v = PyObject_IsTrue(o);
	if(v < 0) { PyErr_Clear(); throw NotHere(); }
	return v != 0;
}

at::Tensor floats_like(const at::Tensor& like, at::IntArrayRef sizes)
{
	return at::empty(sizes, at::TensorOptions().dtype(at::kFloat).device(like.device()));
}

void* stream()
{
	return c10::cuda::getCurrentCUDAStream().stream();
}

template<typename F>
int without_gil(F&& f)
{
	int rc;
	Py_BEGIN_ALLOW_THREADS
	rc = f();
	Py_END_ALLOW_THREADS
	return rc;
}

PyObject* answer(int rc, const at::Tensor& result)
{
	return rc != NB200_OK ? PyLong_FromLong(rc) : THPVariable_Wrap(result);
}

template<typename F>
PyObject* guarded(Py_ssize_t n, Py_ssize_t expected, F&& f)
{
	if(n != expected) {
		PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", expected, n);
		return nullptr;
	}
	// a mode that wants to see torch.empty and the like sees them in the Python code
	if(at::impl::torch_function_mode_enabled()) Py_RETURN_NONE;
	try {
		return f();
	} catch(const NotHere&) {
		Py_RETURN_NONE;
	} catch(const c10::OutOfMemoryError&) {
		Py_RETURN_NONE; // the Python code does without the work space, or raises torch's own error
	} catch(const std::exception& e) {
		PyErr_SetString(PyExc_RuntimeError, e.what());
		return nullptr;
	}
}

nb200_epilogue epilogue(PyObject* bias, PyObject* residual, int ldResidual, PyObject* act, PyObject* actParam, bool accumulate)
{
	nb200_epilogue e = {};
	e.bias = data(bias);
	e.residual = data(residual);
	e.ld_residual = ldResidual;
	e.act = integer(act);
	e.act_param = number(actParam);
	e.accumulate = accumulate ? 1 : 0;
	return e;
}

int out_size(int size, int filter, int pad, int stride, int dilation)
{
	if(stride <= 0) throw NotHere();
	const int span = size - (filter - 1) * dilation - 1 + 2 * pad;
	if(span < 0) throw NotHere();
	return 1 + span / stride;
}

// source, filter, free_term, result, pad_h, pad_w, stride_h, stride_w, dil_h, dil_w, residual, act, act_param, precision, use_scratch
PyObject* blob_convolution(PyObject*, PyObject* const* a, Py_ssize_t count)
{
	return guarded(count, 15, [&]() -> PyObject* {
		const at::Tensor &x = fp32(a[0]), &f = fp32(a[1]);
		if(x.dim() != 4 || f.dim() != 4 || f.size(3) != x.size(3)) throw NotHere();
		nb200_conv_desc d = {};
		d.batch = size_of(x, 0); d.h = size_of(x, 1); d.w = size_of(x, 2); d.c = size_of(x, 3);
		d.k = size_of(f, 0); d.r = size_of(f, 1); d.s = size_of(f, 2);
		d.pad_h = integer(a[4]); d.pad_w = integer(a[5]); d.stride_h = integer(a[6]); d.stride_w = integer(a[7]);
		d.dil_h = integer(a[8]); d.dil_w = integer(a[9]);
		d.ho = out_size(d.h, d.r, d.pad_h, d.stride_h, d.dil_h);
		d.wo = out_size(d.w, d.s, d.pad_w, d.stride_w, d.dil_w);
		const nb200_epilogue e = epilogue(a[2], a[10], d.k, a[11], a[12], false);
		const int precision = integer(a[13]);
		at::Tensor y = a[3] == Py_None ? floats_like(x, { d.batch, d.ho, d.wo, d.k }) : tensor(a[3]);
		const size_t need = truth(a[14]) ? nb200_blob_convolution_scratch_floats(&d) : 0;
		at::Tensor scratch;
		if(need > 0) scratch = floats_like(x, { static_cast<int64_t>(need) });
		void* const s = stream();
		const float *xp = static_cast<const float*>(x.data_ptr()), *fp = static_cast<const float*>(f.data_ptr());
		float *yp = static_cast<float*>(y.data_ptr()), *sp = need > 0 ? static_cast<float*>(scratch.data_ptr()) : nullptr;
		return answer(without_gil([&] { return nb200_blob_convolution(s, &d, xp, fp, yp, sp, &e, precision); }), y);
	});
}

// first, second, result, m, k, n, lda, ldb, ldc, free_term, residual, act, act_param, accumulate, precision, use_scratch
PyObject* multiply_by_transposed(PyObject*, PyObject* const* a, Py_ssize_t count)
{
	return guarded(count, 16, [&]() -> PyObject* {
		const at::Tensor &first = fp32(a[0]), &second = fp32(a[1]);
		const int m = integer(a[3]), k = integer(a[4]), n = integer(a[5]), lda = integer(a[6]), ldb = integer(a[7]), ldc = integer(a[8]);
		if(m < 0 || ldc < 0) throw NotHere();
		const nb200_epilogue e = epilogue(a[9], a[10], ldc, a[11], a[12], truth(a[13]));
		const int precision = integer(a[14]);
		at::Tensor result = a[2] == Py_None ? floats_like(first, { m, ldc }) : tensor(a[2]);
		const size_t need = truth(a[15]) ? nb200_matrix_product_scratch_floats(1, m, n, k, ldb) : 0;
		at::Tensor scratch;
		if(need > 0) scratch = floats_like(first, { static_cast<int64_t>(need) });
		void* const s = stream();
		const float *ap = static_cast<const float*>(first.data_ptr()), *bp = static_cast<const float*>(second.data_ptr());
		float *cp = static_cast<float*>(result.data_ptr()), *sp = need > 0 ? static_cast<float*>(scratch.data_ptr()) : nullptr;
		return answer(without_gil([&] {
			return need > 0 ? nb200_multiply_matrix_by_transposed_matrix_with_scratch(s, 1, ap, m, k, lda, bp, n, ldb, cp, ldc, sp, &e, precision)
				: nb200_multiply_matrix_by_transposed_matrix(s, ap, m, k, lda, bp, n, ldb, cp, ldc, &e, precision);
		}), result);
	});
}

int batch_product(void* s, int batch, const float* a, int m, int k, const float* b, int n, float* c, float* scratch, int precision)
{
	return scratch != nullptr
		? nb200_multiply_matrix_by_transposed_matrix_with_scratch(s, batch, a, m, k, k, b, n, k, c, n, scratch, nullptr, precision)
		: nb200_batch_multiply_matrix_by_transposed_matrix(s, batch, a, m, k, b, n, c, nullptr, precision);
}

// first [b, m, k], second [b, n, k], result, precision, use_scratch
PyObject* batch_multiply_by_transposed(PyObject*, PyObject* const* a, Py_ssize_t count)
{
	return guarded(count, 5, [&]() -> PyObject* {
		const at::Tensor &first = fp32(a[0]), &second = fp32(a[1]);
		if(first.dim() != 3 || second.dim() != 3) throw NotHere();
		const int b = size_of(first, 0), m = size_of(first, 1), k = size_of(first, 2), n = size_of(second, 1);
		const int precision = integer(a[3]);
		at::Tensor result = a[2] == Py_None ? floats_like(first, { b, m, n }) : tensor(a[2]);
		const size_t need = truth(a[4]) ? nb200_matrix_product_scratch_floats(b, m, n, k, k) : 0;
		at::Tensor scratch;
		if(need > 0) scratch = floats_like(first, { static_cast<int64_t>(need) });
		void* const s = stream();
		const float *ap = static_cast<const float*>(first.data_ptr()), *bp = static_cast<const float*>(second.data_ptr());
		float *cp = static_cast<float*>(result.data_ptr()), *sp = need > 0 ? static_cast<float*>(scratch.data_ptr()) : nullptr;
		return answer(without_gil([&] { return batch_product(s, b, ap, m, k, bp, n, cp, sp, precision); }), result);
	});
}

// first [b, m, k], second [b, k, n], result, precision: with work space, k and n at least four (the second operand is
// transposed once)
PyObject* multiply_by_matrix(PyObject*, PyObject* const* a, Py_ssize_t count)
{
	return guarded(count, 4, [&]() -> PyObject* {
		const at::Tensor &first = fp32(a[0]), &second = fp32(a[1]);
		if(first.dim() != 3 || second.dim() != 3) throw NotHere();
		const int b = size_of(first, 0), m = size_of(first, 1), k = size_of(first, 2), n = size_of(second, 2);
		if(k < 4 || n < 4) throw NotHere();
		const int precision = integer(a[3]);
		at::Tensor result = a[2] == Py_None ? floats_like(first, { b, m, n }) : tensor(a[2]);
		const size_t need = nb200_matrix_product_scratch_floats(b, m, n, k, k);
		const int64_t across = (static_cast<int64_t>(b) * n * k + 3) / 4 * 4;
		// one block: the transposed operand, then the product's own room
		at::Tensor room = floats_like(first, { across + static_cast<int64_t>(need) });
		void* const s = stream();
		const float *ap = static_cast<const float*>(first.data_ptr()), *bp = static_cast<const float*>(second.data_ptr());
		float *cp = static_cast<float*>(result.data_ptr()), *tp = static_cast<float*>(room.data_ptr());
		return answer(without_gil([&] {
			const int rc = nb200_transpose_matrix(s, b, bp, k, 1, n, 1, tp);
			return rc != NB200_OK ? rc : batch_product(s, b, ap, m, k, tp, n, cp, need > 0 ? tp + across : nullptr, precision);
		}), result);
	});
}

// batch, first, height, medium, width, channels, result
PyObject* transpose(PyObject*, PyObject* const* a, Py_ssize_t count)
{
	return guarded(count, 7, [&]() -> PyObject* {
		const int batch = integer(a[0]), h = integer(a[2]), m = integer(a[3]), w = integer(a[4]), c = integer(a[5]);
		const at::Tensor& first = fp32(a[1]);
		at::Tensor result = a[6] == Py_None ? floats_like(first, first.sizes()) : tensor(a[6]);
		void* const s = stream();
		const float* ap = static_cast<const float*>(first.data_ptr());
		float* rp = static_cast<float*>(result.data_ptr());
		return answer(without_gil([&] { return nb200_transpose_matrix(s, batch, ap, h, m, w, c, rp); }), result);
	});
}

// op code, first, second, scalar, value, result, count (None: the result's size); first or result given
PyObject* vector_op(PyObject*, PyObject* const* a, Py_ssize_t count)
{
	return guarded(count, 7, [&]() -> PyObject* {
		const int op = integer(a[0]);
		const float *first = data(a[1]), *second = data(a[2]), *scalar = data(a[3]);
		const float value = number(a[4]);
		if(a[5] == Py_None && a[1] == Py_None) throw NotHere();
		at::Tensor result = a[5] == Py_None ? floats_like(fp32(a[1]), tensor(a[1]).sizes()) : tensor(a[5]);
		const int64_t n = a[6] == Py_None ? result.numel() : integer(a[6]);
		if(n > INT32_MAX) throw NotHere();
		void* const s = stream();
		float* rp = static_cast<float*>(result.data_ptr());
		return answer(without_gil([&] { return nb200_vector_op(s, op, first, second, scalar, value, rp, static_cast<int>(n)); }), result);
	});
}

PyMethodDef methods[] = {
#define FAST(name) { #name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr }
	FAST(blob_convolution), FAST(multiply_by_transposed), FAST(batch_multiply_by_transposed), FAST(multiply_by_matrix),
	FAST(transpose), FAST(vector_op),
#undef FAST
	{ nullptr, nullptr, 0, nullptr }
};

PyModuleDef module = { PyModuleDef_HEAD_INIT, "_ops_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr };

} // namespace

PyMODINIT_FUNC PyInit__ops_native()
{
	return PyModule_Create(&module);
}
