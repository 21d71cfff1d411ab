// The operators of cnet_b200/ops.py that small calls spend their time in, as a CPython module: results are made by
// at::empty and the C ABI is called here.  Through ctypes and torch's Python functions an operator's call cost 6 us beside
// its launch (two results 3.2, the foreign call, attributes and checks); at 16 x 100 a whole loss, three operators, took
// 30 us on the host and 5 on the device.
//
// A complex tensor is a pair of planes.  Planes are torch tensors or anything with shape and data_ptr(); they are read as
// contiguous float32, as through the C ABI itself.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>

#include "../../include/cnet_b200.h"

namespace {

PyObject* g_error = nullptr;                     // cnet_b200.lib.CnetError

// a Python error is set
struct Raised {};

// Nothing (None) is the null pointer, which the C ABI refuses where it needs a plane.
float* address(PyObject* o) {
	if (o == Py_None) return nullptr;
	if (THPVariable_Check(o)) return static_cast<float*>(THPVariable_Unpack(o).data_ptr());
	PyObject* v = PyObject_CallMethod(o, "data_ptr", nullptr);
	if (!v) throw Raised();
	void* p = PyLong_AsVoidPtr(v);
	Py_DECREF(v);
	if (PyErr_Occurred()) throw Raised();
	return static_cast<float*>(p);
}

void shape2(PyObject* o, int64_t* rows, int64_t* cols) {
	if (THPVariable_Check(o)) {
		const at::Tensor& t = THPVariable_Unpack(o);
		if (t.dim() != 2) {
			PyErr_Format(PyExc_ValueError, "a plane of %lld dimensions (expected 2)", (long long) t.dim());
			throw Raised();
		}
		*rows = t.size(0); *cols = t.size(1);
		return;
	}
	PyObject* s = PyObject_GetAttrString(o, "shape");
	if (!s) throw Raised();
	PyObject* two = PySequence_Tuple(s);
	Py_DECREF(s);
	if (!two) throw Raised();
	const bool ok = PyTuple_GET_SIZE(two) == 2;
	if (ok) { *rows = PyLong_AsLongLong(PyTuple_GET_ITEM(two, 0)); *cols = PyLong_AsLongLong(PyTuple_GET_ITEM(two, 1)); }
	Py_DECREF(two);
	if (!ok) PyErr_SetString(PyExc_ValueError, "a plane has two dimensions");
	if (PyErr_Occurred()) throw Raised();
}

// One extent of a plane that may have more dimensions than two: of a weight [out, 28, 28] only what the product cannot take
// from the other operand is asked for.
int64_t extent(PyObject* o, int axis) {
	if (THPVariable_Check(o)) {
		const at::Tensor& t = THPVariable_Unpack(o);
		if (t.dim() <= axis) {
			PyErr_SetString(PyExc_IndexError, "a plane of too few dimensions");
			throw Raised();
		}
		return t.size(axis);
	}
	PyObject* s = PyObject_GetAttrString(o, "shape");
	PyObject* v = s ? PySequence_GetItem(s, axis) : nullptr;
	Py_XDECREF(s);
	if (!v) throw Raised();
	const int64_t n = PyLong_AsLongLong(v);
	Py_DECREF(v);
	if (PyErr_Occurred()) throw Raised();
	return n;
}

// The two planes of a pair, as references of their own.  A pair is whatever o[0] and o[1] work for in Python: a tensor of two
// planes is no sequence to C.
struct Pair {
	PyObject *re = nullptr, *im = nullptr;
	explicit Pair(PyObject* o) {
		re = item(o, 0);
		im = re ? item(o, 1) : nullptr;
		if (!im) { Py_XDECREF(re); throw Raised(); }
	}
	static PyObject* item(PyObject* o, Py_ssize_t k) {
		if (PyTuple_Check(o) || PyList_Check(o)) return PySequence_GetItem(o, k);
		PyObject* key = PyLong_FromSsize_t(k);
		PyObject* v = key ? PyObject_GetItem(o, key) : nullptr;
		Py_XDECREF(key);
		return v;
	}
	Pair(const Pair&) = delete;
	~Pair() { Py_DECREF(re); Py_DECREF(im); }
	float* r() const { return address(re); }
	float* i() const { return address(im); }
};

at::Device device_of(PyObject* o) { return THPVariable_Check(o) ? THPVariable_Unpack(o).device() : at::Device(at::kCUDA); }

at::Tensor fresh(at::IntArrayRef sizes, at::Device device) { return at::empty(sizes, at::TensorOptions().dtype(at::kFloat).device(device)); }

// takes both references
PyObject* two(PyObject* a, PyObject* b) {
	PyObject* t = a && b ? PyTuple_New(2) : nullptr;
	if (!t) { Py_XDECREF(a); Py_XDECREF(b); throw Raised(); }
	PyTuple_SET_ITEM(t, 0, a);
	PyTuple_SET_ITEM(t, 1, b);
	return t;
}

// a result that is passed in, or a new pair
struct Result {
	at::Tensor re, im;
	PyObject* given = nullptr;
	float *r = nullptr, *i = nullptr;
	Result(PyObject* out, int64_t rows, int64_t cols, at::Device device) {
		if (out && out != Py_None) {
			given = out;
			const Pair p(out);
			r = p.r(); i = p.i();
			return;
		}
		re = fresh({rows, cols}, device); im = fresh({rows, cols}, device);
		r = static_cast<float*>(re.data_ptr()); i = static_cast<float*>(im.data_ptr());
	}
	PyObject* py() {
		if (given) { Py_INCREF(given); return given; }
		PyObject* a = THPVariable_Wrap(std::move(re));
		return two(a, THPVariable_Wrap(std::move(im)));
	}
};

cnb_ctx* context(PyObject* o) {
	void* p = o == Py_None ? nullptr : PyLong_AsVoidPtr(o);
	if (!p && PyErr_Occurred()) throw Raised();
	return static_cast<cnb_ctx*>(p);
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// Other threads may run Python meanwhile; the interpreter is this thread's again however that ends, also by an exception.
struct Unlocked {
	PyThreadState* state = PyEval_SaveThread();
	~Unlocked() { PyEval_RestoreThread(state); }
};

template <class F> void call(const char* what, F f) {
	const int rc = [&] { const Unlocked unlocked; return f(); }();
	if (rc < 0) {
		PyErr_Format(g_error ? g_error : PyExc_RuntimeError, "%s failed (%d): %s", what, rc, cnb_last_error());
		throw Raised();
	}
}

// f() with C++ errors turned into Python's
template <class F> PyObject* guarded(Py_ssize_t n, Py_ssize_t want, F f) {
	HANDLE_TH_ERRORS
	if (n != want) { PyErr_Format(PyExc_TypeError, "%zd arguments (expected %zd)", n, want); return nullptr; }
	try { return f(); } catch (const Raised&) { return nullptr; }
	END_HANDLE_TH_ERRORS
}

// (context, x, w, res or None) -> y
PyObject* linear_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
	return guarded(n, 4, [&]() -> PyObject* {
		cnb_ctx* ctx = context(a[0]);
		const Pair x(a[1]), w(a[2]);
		int64_t B, in;
		shape2(x.re, &B, &in);
		const int64_t out = extent(w.re, 0);
		float *rr = nullptr, *ri = nullptr;
		const int has = PyObject_IsTrue(a[3]);
		if (has < 0) throw Raised();
		if (has) { const Pair res(a[3]); rr = res.r(); ri = res.i(); }
		Result y(nullptr, B, out, at::Device(at::kCUDA));
		const float *xr = x.r(), *xi = x.i(), *wr = w.r(), *wi = w.i();
		void* st = stream();
		call("linear_fwd", [&] { return cnb_linear_fwd(ctx, xr, xi, wr, wi, rr, ri, y.r, y.i, (int) B, (int) in, (int) out, st); });
		return y.py();
	});
}

// (context, g, w, out or None) -> dx
PyObject* linear_bwd_x(PyObject*, PyObject* const* a, Py_ssize_t n) {
	return guarded(n, 4, [&]() -> PyObject* {
		cnb_ctx* ctx = context(a[0]);
		const Pair g(a[1]), w(a[2]);
		int64_t B, out;
		shape2(g.re, &B, &out);
		const int64_t in = extent(w.re, 1);
		Result dx(a[3], B, in, at::Device(at::kCUDA));
		const float *gr = g.r(), *gi = g.i(), *wr = w.r(), *wi = w.i();
		void* st = stream();
		call("linear_bwd_x", [&] { return cnb_linear_bwd_x(ctx, gr, gi, wr, wi, dx.r, dx.i, (int) B, (int) in, (int) out, dx.given ? 1 : 0, st); });
		return dx.py();
	});
}

// (context, g, x, out or None) -> dw
PyObject* linear_bwd_w(PyObject*, PyObject* const* a, Py_ssize_t n) {
	return guarded(n, 4, [&]() -> PyObject* {
		cnb_ctx* ctx = context(a[0]);
		const Pair g(a[1]), x(a[2]);
		int64_t B, out;
		shape2(g.re, &B, &out);
		const int64_t in = extent(x.re, 1);
		Result dw(a[3], out, in, at::Device(at::kCUDA));
		const float *gr = g.r(), *gi = g.i(), *xr = x.r(), *xi = x.i();
		void* st = stream();
		call("linear_bwd_w", [&] { return cnb_linear_bwd_w(ctx, gr, gi, xr, xi, dw.r, dw.i, (int) B, (int) in, (int) out, dw.given ? 1 : 0, st); });
		return dw.py();
	});
}

// (context, x) -> y
PyObject* dft_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
	return guarded(n, 2, [&]() -> PyObject* {
		cnb_ctx* ctx = context(a[0]);
		const Pair x(a[1]);
		int64_t B, N;
		shape2(x.re, &B, &N);
		Result y(nullptr, B, N, device_of(x.re));
		const float *xr = x.r(), *xi = x.i();
		void* st = stream();
		call("dft_fwd", [&] { return cnb_dft_fwd(ctx, xr, xi, y.r, y.i, (int) B, (int) N, st); });
		return y.py();
	});
}

// (context, g, out or None) -> dx
PyObject* dft_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
	return guarded(n, 3, [&]() -> PyObject* {
		cnb_ctx* ctx = context(a[0]);
		const Pair g(a[1]);
		int64_t B, N;
		shape2(g.re, &B, &N);
		Result dx(a[2], B, N, device_of(g.re));
		const float *gr = g.r(), *gi = g.i();
		void* st = stream();
		call("dft_bwd", [&] { return cnb_dft_bwd(ctx, gr, gi, dx.r, dx.i, (int) B, (int) N, dx.given ? 1 : 0, st); });
		return dx.py();
	});
}

// (context, z) -> y, inverse norms
PyObject* softmax_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
	return guarded(n, 2, [&]() -> PyObject* {
		cnb_ctx* ctx = context(a[0]);
		const Pair z(a[1]);
		int64_t B, N;
		shape2(z.re, &B, &N);
		Result y(nullptr, B, N, device_of(z.re));
		at::Tensor inv = fresh({B}, at::Device(at::kCUDA));
		const float *zr = z.r(), *zi = z.i();
		float* pi = static_cast<float*>(inv.data_ptr());
		void* st = stream();
		call("softmax_fwd", [&] { return cnb_softmax_fwd(ctx, zr, zi, y.r, y.i, pi, (int) B, (int) N, st); });
		PyObject* first = y.py();
		return two(first, THPVariable_Wrap(std::move(inv)));
	});
}

// (context, g, z, inverse norms) -> dz
PyObject* softmax_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
	return guarded(n, 4, [&]() -> PyObject* {
		cnb_ctx* ctx = context(a[0]);
		const Pair g(a[1]), z(a[2]);
		int64_t B, N;
		shape2(z.re, &B, &N);
		Result d(nullptr, B, N, device_of(z.re));
		const float *gr = g.r(), *gi = g.i(), *zr = z.r(), *zi = z.i(), *inv = address(a[3]);
		void* st = stream();
		call("softmax_bwd", [&] { return cnb_softmax_bwd(ctx, gr, gi, zr, zi, inv, d.r, d.i, (int) B, (int) N, 0, st); });
		return d.py();
	});
}

// (context, z, labels, backward) -> loss, dz (a pair, of None without backward)
PyObject* crossent(PyObject*, PyObject* const* a, Py_ssize_t n) {
	return guarded(n, 4, [&]() -> PyObject* {
		cnb_ctx* ctx = context(a[0]);
		const Pair z(a[1]);
		int64_t B, M;
		shape2(z.re, &B, &M);
		const int backward = PyObject_IsTrue(a[3]);
		if (backward < 0) throw Raised();
		at::Tensor loss = fresh({B}, at::Device(at::kCUDA));
		float* pl = static_cast<float*>(loss.data_ptr());
		const float *zr = z.r(), *zi = z.i();
		const int32_t* labels = reinterpret_cast<const int32_t*>(address(a[2]));
		void* st = stream();
		PyObject* second;
		if (backward) {
			Result d(nullptr, B, M, device_of(z.re));
			call("crossent", [&] { return cnb_crossent_fwd_bwd(ctx, zr, zi, labels, pl, d.r, d.i, (int) B, (int) M, st); });
			second = d.py();
		} else {
			call("crossent", [&] { return cnb_crossent_fwd_bwd(ctx, zr, zi, labels, pl, nullptr, nullptr, (int) B, (int) M, st); });
			second = PyTuple_Pack(2, Py_None, Py_None);
		}
		return two(THPVariable_Wrap(std::move(loss)), second);
	});
}

// the class of errors
PyObject* set_error_class(PyObject*, PyObject* cls) {
	Py_INCREF(cls);
	Py_XSETREF(g_error, cls);
	Py_RETURN_NONE;
}

#define CNET_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
	CNET_FAST(linear_fwd), CNET_FAST(linear_bwd_x), CNET_FAST(linear_bwd_w), CNET_FAST(dft_fwd), CNET_FAST(dft_bwd),
	CNET_FAST(softmax_fwd), CNET_FAST(softmax_bwd), CNET_FAST(crossent),
	{"set_error_class", set_error_class, METH_O, nullptr},
	{nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "ops_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

#ifndef CNET_BUILT_FOR
#define CNET_BUILT_FOR ""
#endif

PyMODINIT_FUNC PyInit_ops_native() {
	PyObject* m = PyModule_Create(&module);
	if (m && PyModule_AddStringConstant(m, "built_for", CNET_BUILT_FOR) < 0) { Py_DECREF(m); return nullptr; }
	return m;
}
