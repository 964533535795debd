// Training-layer functions of the extension module (layers.cpp).
#pragma once
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>

namespace gcow_ext {

// The device word that the tensor-core kernels set when they abandon a wait: one int32 per device, made on first use.
at::Tensor error_word(int device);

// Refuses a tensor that names a device without memory there (a FakeTensor): a kernel would get a null address.
inline const at::Tensor& in_memory(const at::Tensor& t) {
  TORCH_CHECK(!t.defined() || t.storage().device_type() == t.device().type(), "expected a tensor in the memory of ", t.device(),
              ", got one without (a FakeTensor?)");
  return t;
}

extern PyMethodDef layer_methods[];

}  // namespace gcow_ext
