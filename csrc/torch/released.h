// released.h - a call made without the interpreter lock, which is held again however the call ends: what catches a C++ exception
// from it (a failed allocation, say) makes a Python error of it.
#pragma once
#include <Python.h>

namespace hcomm_torch {

template <typename Call> int Released(Call call)
{
    struct Unlocked {
        PyThreadState *save = PyEval_SaveThread();
        ~Unlocked() { PyEval_RestoreThread(save); }
    } unlocked;
    return call();
}

}  // namespace hcomm_torch
