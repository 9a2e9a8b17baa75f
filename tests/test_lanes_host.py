"""The lanes of a call (qg_lanes.h) on the CPU, against a fake of the few CUDA calls they make: errors of any lane
reach the caller after all lanes have ended, the memory granted to lanes stays within half of what is free over all
calls, a lane that finds no memory starts over on the calling thread, and a call whose only lane finds none waits for
the lanes of the others."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

SOURCE = r"""
#include "qg_lanes.h"
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <atomic>
#include <chrono>
#include <mutex>
#include <stdexcept>

// ---- fake device: `total` bytes, a thread-local last error ----
static std::mutex mu;
static size_t total = 1000, used = 0;
static thread_local cudaError_t last = cudaSuccess;
static thread_local char message[256];
static cudaError_t fail(cudaError_t e) { return last = e; }
extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  std::lock_guard<std::mutex> g(mu);
  *f = total - used;
  *t = total;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError(void) { return last; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
const char *qpms_gpu_last_error(void) { return message; }
}
namespace qg {
void set_error(const char *fmt, ...) {
  va_list a;
  va_start(a, fmt);
  vsnprintf(message, sizeof message, fmt, a);
  va_end(a);
}
}  // namespace qg

struct Mem {  // an allocation of the fake device
  size_t n = 0;
  bool get(size_t bytes) {
    std::lock_guard<std::mutex> g(mu);
    if (used + bytes > total) {
      fail(cudaErrorMemoryAllocation);
      qg::set_error("out of memory");
      return false;
    }
    used += bytes;
    n = bytes;
    return true;
  }
  ~Mem() {
    std::lock_guard<std::mutex> g(mu);
    used -= n;
  }
};
static void nap(int ms) { std::this_thread::sleep_for(std::chrono::milliseconds(ms)); }
static void expect(bool ok, const char *what) {
  if (ok) return;
  fprintf(stderr, "failed: %s\n", what);
  exit(1);
}

// lanes of `mask` fail (code 10 + lane), those of `thrown` throw
static void errors(int lanes, unsigned mask, unsigned thrown) {
  qg::LaneGrant grant(lanes, 1);
  expect(grant.lanes() == lanes, "lanes");
  std::atomic<int> ended{0};
  const int rc = qg::run_lanes(grant, [&](int i) -> int {
    if (i) nap(20);
    ++ended;
    if (thrown >> i & 1) throw std::runtime_error("thrown");
    if (mask >> i & 1) {
      qg::set_error("lane %d", i);
      return 10 + i;
    }
    return QPMS_SUCCESS;
  });
  expect(ended == lanes, "every lane ends, once");
  int first = -1;
  for (int i = lanes - 1; i >= 0; --i)
    if ((mask | thrown) >> i & 1) first = i;
  if (first < 0) {
    expect(rc == QPMS_SUCCESS, "success");
  } else if (thrown >> first & 1) {
    expect(rc == QPMS_ENOMEM && !strcmp(message, "thrown"), "an exception's code and message");
  } else {
    char m[16];
    snprintf(m, sizeof m, "lane %d", first);
    expect(rc == 10 + first && !strcmp(message, m), "the first failing lane's code and message");
  }
}

// grants of calls in flight stay within half of the free memory
static void grants() {
  qg::LaneGrant a(4, 100);
  expect(a.lanes() == 4, "500 bytes: four lanes of 100");
  qg::LaneGrant b(4, 100);  // nothing allocated yet: 1000 still look free
  expect(b.lanes() == 2, "300 of 500 are granted: two lanes");
  qg::LaneGrant c(4, 100);
  expect(c.lanes() == 1, "400 of 500 are granted: one lane");
  a.release();
  qg::LaneGrant d(4, 100);
  expect(d.lanes() == 4, "released memory is granted again");
  expect(qg::LaneGrant(2, 600).lanes() == 1, "one lane where two do not fit");
  expect(qg::LaneGrant(1, 1).lanes() == 1, "one lane");
}

// what another program took after the grant: the lanes that find none start over
static void retreat(size_t other) {
  qg::LaneGrant grant(4, 100);
  expect(grant.lanes() == 4, "four lanes");
  Mem taken;
  expect(taken.get(other), "the other program's memory");
  std::atomic<int> runs{0}, waiting{4};
  std::vector<int> done(4, 0);
  const int rc = qg::run_lanes(grant, [&](int i) -> int {
    ++runs;
    Mem m;
    const bool ok = m.get(100);
    for (--waiting; waiting > 0;) nap(1);  // the first four runs hold their memory at the same time
    if (!ok) return QPMS_ERROR;
    ++done[i];
    return QPMS_SUCCESS;
  });
  expect(rc == (other > 900 ? QPMS_ERROR : QPMS_SUCCESS), "result");
  for (int i = 0; i < 4; ++i) expect(done[i] == (other > 900 ? 0 : 1), "every lane done, once");
  expect(runs == 4 + (other > 900 ? 4 : 4 - (int)((1000 - other) / 100)), "only the lanes without memory start over");
}

// a call on one lane waits for the lanes of another call
static void wait_for_others() {
  total = 400;
  std::atomic<int> stage{0};
  std::thread other([&] {
    qg::LaneGrant grant(2, 100);
    expect(grant.lanes() == 2, "two lanes");
    const int rc = qg::run_lanes(grant, [&](int) -> int {
      Mem m;
      if (!m.get(150)) return QPMS_ERROR;
      ++stage;
      nap(200);
      return QPMS_SUCCESS;
    });
    expect(rc == QPMS_SUCCESS, "the other call");
  });
  while (stage < 2) nap(1);
  qg::LaneGrant grant(1, 300);
  int runs = 0;
  const int rc = qg::run_lanes(grant, [&](int) -> int {
    ++runs;
    Mem m;
    return m.get(300) ? QPMS_SUCCESS : QPMS_ERROR;
  });
  expect(rc == QPMS_SUCCESS && runs == 2, "the call starts over once the others' lanes have ended");
  other.join();
  runs = 0;
  expect(qg::run_lanes(grant, [&](int) -> int {
    ++runs;
    Mem m;
    return m.get(500) ? QPMS_SUCCESS : QPMS_ERROR;
  }) == QPMS_ERROR && runs == 1, "no other lanes: the failure stands");
}

// many calls at once on little memory: all end, none fails
static void many() {
  total = 1000;
  std::atomic<int> bad{0};
  std::vector<std::thread> th;
  for (int t = 0; t < 6; ++t)
    th.emplace_back([&] {
      for (int r = 0; r < 20; ++r) {
        qg::LaneGrant grant(4, 100);
        bad += qg::run_lanes(grant, [&](int) -> int {
          Mem m;
          if (!m.get(150)) return QPMS_ERROR;
          nap(1);
          return QPMS_SUCCESS;
        }) != QPMS_SUCCESS;
      }
    });
  for (auto &t : th) t.join();
  expect(bad == 0, "six calls of 150 bytes on 1000 succeed");
}

int main(int argc, char **argv) {
  const char *what = argv[1];
  if (!strcmp(what, "errors")) errors(atoi(argv[2]), atoi(argv[3]), atoi(argv[4]));
  if (!strcmp(what, "grants")) grants();
  if (!strcmp(what, "retreat")) retreat(atoi(argv[2]));
  if (!strcmp(what, "wait")) wait_for_others();
  if (!strcmp(what, "many")) many();
  expect(used == 0, "all memory is given back");
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("no g++ or CUDA headers")
    d = tmp_path_factory.mktemp("lanes")
    src, exe = str(d / "lanes.cpp"), str(d / "lanes")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-pthread", "-I", CUDA,
                    "-I", os.path.join(ROOT, "qpms_gb300", "csrc"), src, "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("args", [
    ["errors", 1, 0, 0], ["errors", 1, 1, 0], ["errors", 4, 0, 0], ["errors", 4, 1, 0], ["errors", 4, 8, 0],
    ["errors", 4, 14, 0], ["errors", 4, 15, 0], ["errors", 3, 0, 1], ["errors", 3, 4, 2], ["errors", 3, 2, 4],
    ["grants"], ["retreat", 600], ["retreat", 700], ["retreat", 900], ["retreat", 950], ["wait"], ["many"]],
    ids=lambda a: "-".join(map(str, a)))
def test_lanes(program, args):
    r = subprocess.run([program, *map(str, args)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
