"""Host copies of the drop-ins (staging.cu) against a stand-in for the CUDA runtime
whose copies run only when an event or the stream is waited for (no GPU needed): after a
copy that failed none is left under way, since the next call refills the pinned slots,
and copies towards the host are done on return."""
import os
import subprocess

import pytest

from vtkmakecompare_b200 import build as B

FAKE = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <vector>
#include "common.cuh"
static std::mutex mu;
static std::vector<std::function<void()>> fifo;
static size_t done = 0;
static long calls = 0, fail_at = -1;
static std::map<cudaEvent_t, size_t> at;
static void run_to(size_t n) { for (; done < n; ++done) fifo[done](); }
static cudaError_t queue(std::function<void()> f) {
  std::lock_guard<std::mutex> lk(mu);
  if (calls++ == fail_at) return cudaErrorInvalidValue;
  fifo.push_back(f);
  return cudaSuccess;
}
extern "C" {
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return queue([=]() { memcpy(d, s, n); });
}
cudaError_t cudaMemcpy3DAsync(const cudaMemcpy3DParms* p, cudaStream_t) {
  const cudaMemcpy3DParms q = *p;
  return queue([=]() {
    for (size_t k = 0; k < q.extent.depth; ++k)
      for (size_t j = 0; j < q.extent.height; ++j) {
        const size_t o = q.srcPos.x + q.srcPtr.pitch * ((q.srcPos.y + j) + q.srcPtr.ysize * k);
        memcpy((char*)q.dstPtr.ptr + o, (char*)q.srcPtr.ptr + o, q.extent.width);
      }
  });
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = (cudaEvent_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  std::lock_guard<std::mutex> lk(mu);
  at[e] = fifo.size();
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::lock_guard<std::mutex> lk(mu);
  run_to(at[e]);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  std::lock_guard<std::mutex> lk(mu);
  run_to(fifo.size());
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
}
namespace nse { bool cuda_ok(cudaError_t, const char*) { return false; } }
// arguments: to_device, the copy that fails (-1: none), doubles per array
int main(int, char** argv) {
  const bool up = atoi(argv[1]);
  fail_at = atol(argv[2]);
  const size_t n = atol(argv[3]), row = 16;
  std::vector<double> host(2 * n), dev(2 * n);
  for (size_t i = 0; i < 2 * n; ++i) { host[i] = 1.0 + i; dev[i] = -1.0 - i; }
  const std::vector<double> h0 = host, d0 = dev;
  // a whole array, and rows 1 and 2 of four with entries 3 .. 12 of 16
  const nse::HostCopy list[2] = {
      {host.data(), dev.data(), n * 8, n * 8, 0, n * 8, 1, 0, 0},
      {host.data() + n, dev.data() + n, n * 8, row * 8, 3 * 8, 10 * 8, 4, 1, 2}};
  const bool ok = nse::host_copies(list, 2, up, nullptr);
  // (an upload that succeeds may still be queued: its call waits at its end)
  const bool idle = (up && ok) || done == fifo.size();
  bool right = true;
  for (int rep = 0; rep < 2; ++rep) {  // then a call without a failure
    if (rep) { fail_at = -1; host = h0; dev = d0; right = nse::host_copies(list, 2, up, nullptr); }
    if (rep == 0 && !ok) continue;
    if (up) cudaStreamSynchronize(nullptr);
    right = right && done == fifo.size();
    for (size_t i = 0; i < 2 * n; ++i) {
      const size_t e = i % n, r = e / row % 4;
      const bool in = i < n || (r >= 1 && r <= 2 && e % row >= 3 && e % row < 13);
      right = right && (up ? dev[i] == h0[i] : host[i] == (in ? d0[i] : h0[i]));
    }
  }
  printf("%d %d %d\n", ok, idle, right);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("staging")
    src, exe = d / "fake.cpp", d / "staging"
    src.write_text(FAKE)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(B.nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + inc, "-I" + B.CSRC, "-x", "c++",
                    os.path.join(B.CSRC, "staging.cu"), str(src), "-o", str(exe)], check=True)
    return str(exe)


# 2 x 80 KB go as plain copies, 2 x 8 MB in 32 chunks through the slots
@pytest.mark.parametrize("up", [0, 1])
@pytest.mark.parametrize("n,fail", [(64 * 160, -1), (64 * 160, 1), (1 << 20, -1), (1 << 20, 0),
                                    (1 << 20, 5), (1 << 20, 20), (1 << 20, 31)])
def test_no_copy_is_left_under_way(program, up, n, fail):
    r = subprocess.run([program, str(up), str(fail), str(n)], capture_output=True, text=True,
                       timeout=60, check=True)
    assert r.stdout.split() == [str(int(fail < 0)), "1", "1"]
