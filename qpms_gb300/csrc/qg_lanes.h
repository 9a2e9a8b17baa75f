// Independent units of a call spread over a few host threads, each with a CUDA
// stream and buffers of its own.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <exception>
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

// Runs body(0) .. body(lanes - 1), lane 0 on the calling thread, the others on
// threads with the same current device; returns after all have ended, with the
// first failing lane's code and message.  A lane whose thread cannot be started
// runs after lane 0.
template <class F>
int run_lanes(int lanes, F body) {
  if (lanes <= 1) return body(0);
  int dev = 0;
  QG_CUDA_TRY(cudaGetDevice(&dev));
  std::vector<int> rc(lanes, QPMS_SUCCESS);
  std::vector<std::string> msg(lanes);
  auto lane = [&](int i) {
    try {
      rc[i] = body(i);
      if (rc[i]) msg[i] = qpms_gpu_last_error();
    } catch (const std::exception &ex) {
      rc[i] = QPMS_ENOMEM;
      msg[i] = ex.what();
    }
  };
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
  for (int i = 0; i < lanes; ++i)
    if (rc[i]) {
      set_error("%s", msg[i].c_str());
      return rc[i];
    }
  return QPMS_SUCCESS;
}

// At most `lanes`, and no more than fit half the free device memory at
// `bytes` each.
inline int lanes_that_fit(int lanes, size_t bytes) {
  if (lanes <= 1) return 1;
  size_t fr = 0, tot = 0;
  if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return (int)std::max<size_t>(1, std::min<size_t>((size_t)lanes, fr / 2 / std::max<size_t>(bytes, 1)));
}

}  // namespace qg
