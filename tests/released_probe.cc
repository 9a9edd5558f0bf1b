// released_probe.cc - an extension module for test_native_calls.py: calls made through csrc/torch/released.h.
#include "../csrc/torch/released.h"

#include <new>

namespace {

// whether the interpreter lock was free inside a call, whether it is held again behind it
PyObject *Returns(PyObject *, PyObject *)
{
    const int inside = hcomm_torch::Released([] { return PyGILState_Check(); });
    return Py_BuildValue("(ii)", inside, PyGILState_Check());
}
// whether the lock is held where an exception that came out of such a call is caught
PyObject *Throws(PyObject *, PyObject *)
{
    int held = -1;
    try {
        hcomm_torch::Released([]() -> int { throw std::bad_alloc(); });
    } catch (const std::bad_alloc &) {
        held = PyGILState_Check();
    }
    if (held != 1) PyGILState_Ensure();     // so that the test can say so
    return PyLong_FromLong(held);
}

PyMethodDef kMethods[] = {{"returns", Returns, METH_NOARGS, nullptr}, {"throws", Throws, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "released_probe", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_released_probe() { return PyModule_Create(&kModule); }
