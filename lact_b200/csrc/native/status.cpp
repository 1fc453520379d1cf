// Device status without copies: every kernel that gives up leaves its code in a word of mapped host memory
// (lact_status_host_word).  An operator reads that word before it enqueues (one load); a non-zero word is reported as an
// exception and cleared together with the device-side words.  (A 4-byte device-to-host copy, an event and a memset per
// call cost about 5 us of stream time and 12 us of host time.)
#include <Python.h>

#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <torch/csrc/Exceptions.h>

#include <atomic>
#include <cstdlib>
#include <mutex>
#include <string_view>
#include <unordered_map>

#include "common.h"

namespace lact_torch {
namespace {

std::atomic<PyObject*> g_error_type{nullptr};  // lact_b200.LactError, kept alive by its module

// PyTorch turns exceptions of this kind into Python ones of their type, also those that leave an autograd node.
struct Failure : torch::PyTorchError {
  using torch::PyTorchError::PyTorchError;
  PyObject* python_type() override {
    PyObject* t = g_error_type.load();
    return t != nullptr ? t : PyExc_RuntimeError;
  }
};

constexpr int kMaxDevices = 64;
std::atomic<int32_t*> g_host[kMaxDevices];
std::atomic<uint64_t> g_epoch{1};  // raised when a failure is reported: device words of older epochs are cleared before use

struct Word {
  Tensor buf;
  uint64_t epoch = 0;
};
std::mutex g_mu;
// 256 bytes per (device, stream) in use; never destroyed (the CUDA context may be gone before static destructors run)
std::unordered_map<uint64_t, Word>& g_words = *new std::unordered_map<uint64_t, Word>();

volatile int32_t* host_word(int dev) {
  int32_t* w = g_host[dev].load(std::memory_order_acquire);
  if (w == nullptr) {
    check(lact_status_host_word(&w), "lact_status_host_word");
    g_host[dev].store(w, std::memory_order_release);
  }
  return w;
}

}  // namespace

void fail(const std::string& message) { throw Failure(message); }

void poll_status(const Tensor& like) {
  const int dev = like.device().index();
  TORCH_CHECK(dev >= 0 && dev < kMaxDevices, "unsupported device index");
  volatile int32_t* w = host_word(dev);
  const int32_t st = *w;
  if (st == 0) return;
  *w = 0;
  g_epoch.fetch_add(1);
  fail(c10::str("lact_b200: device status: ", lact_error_string(st), " (code ", st, ")"));
}

static bool capturing() { return c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None; }

void settle(const Tensor& like) {
  static const bool on = [] {
    const char* v = std::getenv("LACT_B200_SYNC_CHECK");
    return v != nullptr && std::string_view(v) == "1";
  }();
  if (!on || capturing()) return;
  c10::cuda::getCurrentCUDAStream(like.device().index()).synchronize();
  poll_status(like);
}

StatusWord status_word(const Tensor& like) {
  poll_status(like);
  if (capturing()) {
    // The stream's shared word would be cleared (or not) by whatever runs between the replays, and if its clearing fell
    // into this capture it would only be recorded.
    Tensor own = empty({64}, at::kInt, like).zero_();
    return {own, own.data_ptr<int32_t>()};
  }
  const int dev = like.device().index();
  const auto stream = c10::cuda::getCurrentCUDAStream(dev);
  const uint64_t key = (static_cast<uint64_t>(dev) << 56) ^ static_cast<uint64_t>(reinterpret_cast<uintptr_t>(stream.stream()));
  const uint64_t epoch = g_epoch.load();
  std::lock_guard<std::mutex> lock(g_mu);
  Word& w = g_words[key];
  if (!w.buf.defined()) w.buf = empty({64}, at::kInt, like);
  if (w.epoch != epoch) {
    w.buf.zero_();
    w.epoch = epoch;
  }
  return {Tensor(), w.buf.data_ptr<int32_t>()};
}

}  // namespace lact_torch

// Status recorded on `device` so far (0: none), cleared by the read; what the Python side calls after a synchronisation.
extern "C" int lact_torch_take_status(int device) {
  if (device < 0 || device >= lact_torch::kMaxDevices) return 0;
  int32_t* w = lact_torch::g_host[device].load(std::memory_order_acquire);
  if (w == nullptr) return 0;
  const int32_t st = *reinterpret_cast<volatile int32_t*>(w);
  if (st != 0) {
    *reinterpret_cast<volatile int32_t*>(w) = 0;
    lact_torch::g_epoch.fetch_add(1);
  }
  return st;
}

// Makes the word failures on `device` are reported in, if no operator has yet: called before kernels are launched past the
// operators.  Returns the C ABI's code.
extern "C" int lact_torch_prepare_status(int device) {
  if (device < 0 || device >= lact_torch::kMaxDevices) return LACT_ERR_DEVICE;
  if (lact_torch::g_host[device].load(std::memory_order_acquire) != nullptr) return LACT_OK;
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
  int32_t* w = nullptr;
  const int rc = lact_status_host_word(&w);
  if (rc == LACT_OK) lact_torch::g_host[device].store(w, std::memory_order_release);
  return rc;
}

// The PyTorch this library was compiled against (LACT_TORCH_BUILD, from build.py, which looks for it in the file).
extern "C" const char lact_torch_build[] = LACT_TORCH_BUILD;

// The class of `fail`'s exceptions.
extern "C" void lact_torch_set_error_type(PyObject* type) { lact_torch::g_error_type.store(type); }
