// Independent units of a call spread over a few host threads, each with a CUDA
// stream and buffers of its own.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <condition_variable>
#include <exception>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "qg_internal.h"

namespace qg {

// Non-blocking stream of a lane.
struct LaneStream {
  cudaStream_t s = nullptr;
  int create() {
    QG_CUDA_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    return QPMS_SUCCESS;
  }
  ~LaneStream() {
    if (s) cudaStreamDestroy(s);
  }
};

// Device memory that the lanes beyond the first of all calls in flight were
// granted, per device.  A call's first lane needs no grant: it is what the call
// takes without lanes.
class LaneMemory {
 public:
  static LaneMemory &of(int dev) {
    static LaneMemory m[kDevices];
    return m[dev < 0 || dev >= kDevices ? 0 : dev];
  }
  // At most `most` lanes, and no more than fit half the free memory at `bytes`
  // each beside what other calls were granted; one while a call waits for memory.
  int grant(int most, size_t bytes) {
    std::lock_guard<std::mutex> g(mu_);
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
      cudaGetLastError();
      return 1;
    }
    fr /= 2;
    if (waiting_ || granted_ >= fr) return 1;
    bytes = std::max<size_t>(bytes, 1);
    const int n = (int)std::max<size_t>(1, std::min<size_t>((size_t)most, (fr - granted_) / bytes));
    granted_ += (n - 1) * bytes;
    return n;
  }
  void release(size_t bytes) {
    std::lock_guard<std::mutex> g(mu_);
    granted_ -= bytes;
    if (!granted_) cv_.notify_all();
  }
  // Waits until no lane beyond a call's first is in flight (the caller's own are
  // released); none is granted meanwhile.  False if there was none.
  bool wait_for_none() {
    std::unique_lock<std::mutex> l(mu_);
    if (!granted_) return false;
    ++waiting_;
    cv_.wait(l, [&] { return !granted_; });
    --waiting_;
    return true;
  }

 private:
  static constexpr int kDevices = 64;
  std::mutex mu_;
  std::condition_variable cv_;
  size_t granted_ = 0;
  int waiting_ = 0;
};

// The lanes of one call and the memory granted for those beyond the first.
class LaneGrant {
 public:
  LaneGrant(int most, size_t bytes) {
    if (most <= 1 || cudaGetDevice(&dev_) != cudaSuccess) return;
    lanes_ = LaneMemory::of(dev_).grant(most, bytes);
    held_ = (lanes_ - 1) * std::max<size_t>(bytes, 1);
  }
  ~LaneGrant() { release(); }
  LaneGrant(const LaneGrant &) = delete;
  LaneGrant &operator=(const LaneGrant &) = delete;
  int lanes() const { return lanes_; }
  void release() {
    if (held_) LaneMemory::of(dev_).release(held_);
    held_ = 0;
  }

 private:
  int dev_ = 0, lanes_ = 1;
  size_t held_ = 0;
};

// Runs body(0) .. body(lanes - 1), lane 0 on the calling thread, the others on
// threads with the same current device; returns after all have ended, with the
// first failing lane's code and message.  A lane whose thread cannot be started
// runs after lane 0.  A lane that found no device memory is run again, on the
// calling thread, once the others have given theirs back and no other call has
// lanes beyond its first: from then on the call needs no more than on one lane.
// So body(i) frees what it allocates, or finds it again, and may start over.
template <class F>
int run_lanes(LaneGrant &grant, F body) {
  const int lanes = grant.lanes();
  int dev = 0;
  QG_CUDA_TRY(cudaGetDevice(&dev));
  std::vector<int> rc(lanes, QPMS_SUCCESS);
  std::vector<char> memory(lanes, 0);
  std::vector<std::string> msg(lanes);
  auto run = [&](int i) {
    rc[i] = body(i);
    if (rc[i]) {
      msg[i] = qpms_gpu_last_error();
      memory[i] = cudaPeekAtLastError() == cudaErrorMemoryAllocation;
    }
  };
  auto lane = [&](int i) {
    try {
      run(i);
    } catch (const std::exception &ex) {
      rc[i] = QPMS_ENOMEM;
      msg[i] = ex.what();
    }
  };
  if (lanes == 1) {
    run(0);
  } else {
    std::vector<std::thread> th;
    int started = 1;
    try {
      th.reserve(lanes - 1);
      for (; started < lanes; ++started)
        th.emplace_back([&, i = started] {
          if (cudaSetDevice(dev) != cudaSuccess) {
            rc[i] = QPMS_ERROR;
            msg[i] = "cudaSetDevice failed";
            return;
          }
          lane(i);
        });
    } catch (const std::exception &) {
    }
    lane(0);
    for (int i = started; i < lanes; ++i) lane(i);
    for (auto &t : th) t.join();
  }
  if (std::find(memory.begin(), memory.end(), 1) != memory.end()) {
    grant.release();
    const bool waited = LaneMemory::of(dev).wait_for_none();
    if (lanes > 1 || waited)
      for (int i = 0; i < lanes; ++i)
        if (memory[i]) {
          cudaGetLastError();  // the failed allocation's, on this thread
          if (lanes > 1)
            lane(i);
          else
            run(i);
        }
  }
  for (int i = 0; i < lanes; ++i)
    if (rc[i]) {
      set_error("%s", msg[i].c_str());
      return rc[i];
    }
  return QPMS_SUCCESS;
}

}  // namespace qg
