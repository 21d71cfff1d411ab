// A call of the native operators' kind that ends by a C++ exception.
#include "../../cnet_b200/host/ops_native.cpp"

#include <new>

static PyObject* throwing(PyObject*, PyObject*) {
	return guarded(0, 0, []() -> PyObject* {
		call("throwing", []() -> int { throw std::bad_alloc(); });
		return nullptr;
	});
}

static PyMethodDef probe_methods[] = {{"throwing", throwing, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
static PyModuleDef probe = {PyModuleDef_HEAD_INIT, "ops_throw_probe", nullptr, -1, probe_methods, nullptr, nullptr, nullptr, nullptr};
PyMODINIT_FUNC PyInit_ops_throw_probe() { return PyModule_Create(&probe); }
