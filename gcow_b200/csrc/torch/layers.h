// Training-layer functions of the extension module (layers.cpp).
#pragma once
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>

namespace gcow_ext {

// The device word that the tensor-core kernels set when they abandon a wait: one int32 per device, made on first use.
at::Tensor error_word(int device);

extern PyMethodDef layer_methods[];

}  // namespace gcow_ext
