// Shared parts of the PyTorch binding (liblact_b200_torch.so): the registered operators' host side.  Everything here
// allocates through PyTorch, validates, and enqueues through the C ABI of liblact_b200.so; no kernel lives here.
#pragma once
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/autograd_not_implemented_fallback.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

#include <optional>
#include <vector>

#include "../../../include/lact_b200.h"

namespace lact_torch {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

enum Step : int64_t { kApply = LACT_STEP_APPLY, kUpdate = LACT_STEP_UPDATE };

// Throws the Python package's LactError, from forwards and backwards alike (status.cpp).
[[noreturn]] void fail(const std::string& message);

// Return code of the C ABI -> exception (ValueError for arguments, LactError for the device).
inline void check(int rc, const char* what) {
  if (rc == LACT_OK) return;
  const char* msg = lact_error_string(rc);
  TORCH_CHECK_VALUE(!(rc == LACT_ERR_NULL || rc == LACT_ERR_SHAPE || rc == LACT_ERR_DTYPE || rc == LACT_ERR_CONFIG ||
                      rc == LACT_ERR_STEPS),
                    what, ": ", msg, " (code ", rc, ")");
  fail(c10::str("lact_b200: ", what, ": ", msg, " (code ", rc, ")"));
}

inline int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kFloat) return LACT_F32;
  TORCH_CHECK_TYPE(t.scalar_type() == at::kBFloat16, "unsupported dtype: expected float32 or bfloat16");
  return LACT_BF16;
}

inline void* ptr(const Tensor& t) { return t.data_ptr(); }
inline void* ptr(const OptTensor& t) { return t.has_value() && t->defined() ? t->data_ptr() : nullptr; }
inline bool given(const OptTensor& t) { return t.has_value() && t->defined(); }
inline Tensor value(const OptTensor& t) { return given(t) ? *t : Tensor(); }
inline OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); }

inline void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

inline Tensor empty(at::IntArrayRef shape, at::ScalarType dt, const Tensor& like) {
  return at::empty(shape, like.options().dtype(dt).requires_grad(false));
}
inline Tensor bytes(size_t n, const Tensor& like) {
  return empty({static_cast<int64_t>(n < 256 ? 256 : n)}, at::kByte, like);
}

// Device status word of the calls on (device of `like`, current stream): cleared once, shared by consecutive calls.  A
// call that is being captured gets a word of its own, which the graph clears at every replay: keep the object for as long
// as kernels that use the word are enqueued.  Throws if a call has recorded a failure since the last look (see status.cpp);
// costs one read of host memory and a query of the stream.
struct StatusWord {
  Tensor own;  // defined inside a capture
  int32_t* word;
  operator int32_t*() const { return word; }
};
StatusWord status_word(const Tensor& like);
void poll_status(const Tensor& like);
// End of a backward: with LACT_B200_SYNC_CHECK=1 (and no capture) waits for the stream and reports what it has left (forwards
// are waited for in Python).
void settle(const Tensor& like);

// A [batch, rows, cols] bf16 activation whose last axis is contiguous and whose strides and base keep 16-byte alignment
// (views of fused projections pass through); anything else is copied.
inline Tensor aligned(const Tensor& t, int64_t elems = 8) {
  if (t.stride(-1) != 1 || t.stride(1) % elems || t.stride(0) % elems || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 ||
      t.stride(1) < t.size(-1))
    return t.contiguous();
  return t;
}

}  // namespace lact_torch
