// Per-thread device context of the engine: mode, device ordinal, the stream
// all of this thread's kernels and copies run on, and the status word that
// kernels with bounded waits report into.
//
// mini-caffe keeps mode and cuBLAS handle in a thread-local `Caffe` singleton
// (src/common.hpp:76-117, src/common.cpp:7-10); this is the counterpart.  A
// thread that never calls SetMode runs on GPU 0.
#ifndef MCB200_CONTEXT_H_
#define MCB200_CONTEXT_H_

#include <cuda_runtime.h>

#include <exception>

#include "caffe/base.hpp"

#define CUDA_CHECK(expr)                                                            \
  do {                                                                              \
    cudaError_t cuda_check_err_ = (expr);                                           \
    CHECK_EQ(static_cast<int>(cuda_check_err_), static_cast<int>(cudaSuccess))      \
        << " " << cudaGetErrorString(cuda_check_err_);                              \
  } while (0)

// Kernel-level entry points return 0, a negative argument error, or a cudaError_t.
#define KERNEL_CHECK(expr)                                                          \
  do {                                                                              \
    int kernel_check_rc_ = (expr);                                                  \
    CHECK_EQ(kernel_check_rc_, 0) << " kernel launcher failed: " #expr              \
        << (kernel_check_rc_ > 0 ? cudaGetErrorString(static_cast<cudaError_t>(kernel_check_rc_)) : ""); \
  } while (0)

namespace caffe {

class Context {
 public:
  static Context& Get();  // of the calling thread

  DeviceMode mode() const { return mode_; }
  int device() const { return device_; }
  void Set(DeviceMode mode, int device);

  // Binds the thread to its device and creates the stream on first use.
  // Throws caffe::Error in CPU mode or without a usable device.
  void Activate();
  cudaStream_t stream() { Activate(); return stream_; }
  void* stream_ptr() { return static_cast<void*>(stream()); }
  // The stream if this thread has one already, else NULL (never creates one, never throws).
  void* stream_if_active() const { return active_ ? static_cast<void*>(stream_) : nullptr; }
  // Word that kernels raise on a timed-out wait; checked by Net::Forward.  It lies in pinned host
  // memory that the device writes through its mapped address: kernels touch it only when something
  // went wrong, and a pass does not pay a device-to-host copy to learn that nothing did.
  int* status_word() { Activate(); return status_dev_; }
  // Copies of new input that run beside the kernels, on a second stream.  CopiesBegin: copies queued
  // from here on start after the work queued so far (which may still use their destinations), and
  // the stream to queue them on is returned.  CopiesArrived: work queued on stream() from here on
  // starts after the copies queued so far.
  cudaStream_t CopiesBegin();
  void CopiesArrived();
  // The forward passes under way on this thread's device, in all threads of the process (see PassInFlight).
  int passes_in_flight() const;
  // Blocks until the stream is idle and throws if a kernel raised the status word.
  void SyncAndCheck();
  void Sync();

  ~Context();

 private:
  Context() : mode_(GPU), device_(0), active_(false), stream_(nullptr), copy_stream_(nullptr), event_(nullptr),
              status_dev_(nullptr), status_host_(nullptr) {}
  DeviceMode mode_;
  int device_;
  bool active_;
  cudaStream_t stream_, copy_stream_;
  cudaEvent_t event_;      // one event serves every hand-over: a wait refers to the record before it
  int* status_dev_;
  int* status_host_;
  void Release();
};

// A forward pass, from its first launch to its wait.  Input in parts hides the copy behind kernels on a GPU that would
// otherwise idle, at the price of a launch per part and layer.  With other nets' passes in flight there is no idle time
// to fill, and input is copied whole: three threads with a net each made 32 600 images/s in parts and 34 700 whole of
// ResNet-50 at batch 64, 75 100 and 89 500 of MobileNet-v1, 55 700 and 60 900 of DetectionOutput at 32; one thread
// 28 250 and 24 400 of ResNet-50.  (The results are the same bits either way.)
class PassInFlight {
 public:
  explicit PassInFlight(int device);
  ~PassInFlight();
  PassInFlight(const PassInFlight&) = delete;
  PassInFlight& operator=(const PassInFlight&) = delete;

 private:
  const int device_;
};

// For a scope that queues work on blobs' host memory itself.  A blob whose host copy is the only current one is
// released without a wait, so when an exception leaves the scope that work ends before it does.
class DrainOnError {
 public:
  explicit DrainOnError(Context& ctx) : ctx_(ctx), before_(std::uncaught_exceptions()) {}
  ~DrainOnError() {
    if (std::uncaught_exceptions() == before_) return;
    try { ctx_.Sync(); } catch (...) {}
  }
  DrainOnError(const DrainOnError&) = delete;
  DrainOnError& operator=(const DrainOnError&) = delete;

 private:
  Context& ctx_;
  const int before_;
};

// Number of usable CUDA devices (0 without a driver); cached.
int DeviceCount();

}  // namespace caffe

#endif  // MCB200_CONTEXT_H_
