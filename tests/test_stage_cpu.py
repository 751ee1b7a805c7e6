"""Staged copies of host-pointer calls against a stand-in for the CUDA runtime (compiled here, no GPU):
when the worker threads run."""
import pathlib
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "pseudoctimaging_b200" / "csrc"
CUDA = pathlib.Path("/usr/local/cuda/include")

# The stand-in's device memory is host memory. Its one stream is busy until `busy_until`: copies are
# made at once, but events and the stream are done only then.
RUNTIME = r"""
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <time.h>
#include <atomic>
#include <chrono>
#include <thread>
#include <vector>
#include "pct_stage.h"

using Clock = std::chrono::steady_clock;
static Clock::time_point busy_until = Clock::now();
static std::atomic<long> early_queries{0}, registered{0};
static std::atomic<int> register_ms{0};
static std::thread::id caller;
static std::atomic<bool> registered_by_caller{false};
static bool busy() { return Clock::now() < busy_until; }

extern "C" {
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
  memset(a, 0, sizeof(*a));
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaHostRegister(void *, size_t, unsigned) {
  if (std::this_thread::get_id() == caller) registered_by_caller = true;
  std::this_thread::sleep_for(std::chrono::milliseconds(register_ms.load()));
  ++registered;
  return cudaSuccess;
}
cudaError_t cudaHostUnregister(void *) { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  *e = (cudaEvent_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  free((void *)e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) {
  if (!busy()) return cudaSuccess;
  ++early_queries;
  return cudaErrorNotReady;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) {
  std::this_thread::sleep_until(busy_until);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  std::this_thread::sleep_until(busy_until);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
}

static double ms(Clock::time_point t) {
  return std::chrono::duration<double, std::milli>(Clock::now() - t).count();
}
static double cpu_ms() {
  timespec t;
  clock_gettime(CLOCK_PROCESS_CPUTIME_ID, &t);
  return 1e3 * t.tv_sec + 1e-6 * t.tv_nsec;
}
static std::vector<char> data(size_t n, int seed) {
  std::vector<char> v(n);
  for (size_t i = 0; i < n; i += 61) v[i] = (char)(i / 61 + seed);
  return v;
}
// One upload of v; whether it was staged.
static bool upload(pct::HostStager &st, const std::vector<char> &v) {
  std::vector<char> dev(v.size());
  if (!BEGIN(st, v)) return false;
  if (st.copy(dev.data(), v.data(), v.size(), nullptr) != cudaSuccess) exit(2);
  st.end();
  if (dev != v) exit(3);
  return true;
}
"""

BEGIN = "#define BEGIN(st, v) (st).begin(0, {{(v).data(), (v).size()}}, nullptr)\n#define END(st) (st).pin_ahead()\n"


def run(tmp_path, main):
    if not CUDA.exists() or not shutil.which("g++"):
        pytest.skip("no CUDA headers or compiler")
    src = tmp_path / "t.cpp"
    src.write_text(BEGIN + RUNTIME + main)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{CUDA}", f"-I{CSRC}", str(src),
                    str(CSRC / "pct_stage.cpp"), "-o", str(exe), "-lpthread"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, (out.returncode, out.stdout, out.stderr)
    return [float(x) for x in out.stdout.split()]


def test_nobody_polls_before_the_data_is_there(tmp_path):
    """Downloads and uploads behind 300 ms of other work on the stream: no event is asked for, and the
    threads sleep, until it is done."""
    queries, cpu, ok = run(tmp_path, r"""
int main() {
  caller = std::this_thread::get_id();
  pct::HostStager st;
  const std::vector<char> big = data(64u << 20, 1), v = data((20u << 20) + 4, 2);
  if (!upload(st, big)) return 4;
  std::vector<char> out(v.size());
  early_queries = 0;
  double c = cpu_ms();
  busy_until = Clock::now() + std::chrono::milliseconds(300);
  if (st.download(0, out.data(), v.data(), v.size(), nullptr) != cudaSuccess) return 5;
  busy_until = Clock::now() + std::chrono::milliseconds(300);
  if (!upload(st, v)) return 6;
  c = cpu_ms() - c;
  printf("%ld %.1f %d\n", early_queries.load(), c, out == v);
}""")
    assert ok == 1 and queries == 0
    assert cpu < 250, f"{cpu} ms of CPU time for 600 ms of waiting"


def test_no_small_call_pays_for_pinning(tmp_path):
    """Pinning takes 400 ms here. Calls of 25 MB never wait for it, whether they cross the line after which
    slots are worth having or come while they are pinned; once they are, calls use them. A call that
    is worth slots by itself pins them at once."""
    slowest, by_caller, staged, again, handed, at_once, leftover = run(tmp_path, r"""
int main() {
  caller = std::this_thread::get_id();
  register_ms = 400;
  const std::vector<char> v = data(25u << 20, 1), big = data(62u << 20, 2);
  double slowest = 0;
  int staged = 0, again = 0, handed = 0, at_once = 0;
  {
    pct::HostStager st;
    for (int k = 0; k < 6; ++k) {
      const auto t = Clock::now();
      if (BEGIN(st, v)) return 4;  // not pinned yet: copied directly
      END(st);
      if (ms(t) > slowest) slowest = ms(t);
    }
    for (int k = 0; k < 100 && !registered; ++k) std::this_thread::sleep_for(std::chrono::milliseconds(20));
    std::this_thread::sleep_for(std::chrono::milliseconds(50));
    staged = upload(st, v);
    again = upload(st, v);
    pct::HostStager other;
    {
      pct::HostStager closing;
      for (int k = 0; k < 3; ++k) {
        BEGIN(closing, v);
        END(closing);
      }
    }  // closed while it pins: the slots pass on
    handed = upload(other, v);
  }
  const bool small_by_caller = registered_by_caller;
  pct::HostStager st;
  at_once = upload(st, big);
  printf("%.1f %d %d %d %d %d %ld\n", slowest, small_by_caller, staged, again, handed, at_once,
         registered.load());
}""")
    assert slowest < 200 and by_caller == 0
    assert staged == again == handed == at_once == 1
    assert leftover == 3  # one per stager that asked for slots and found none
