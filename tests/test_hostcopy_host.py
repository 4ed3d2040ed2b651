"""Copies of large pageable host arrays (vls_hostcopy.h) against a runtime that
does nothing before it must: queued copies run when their event or stream is
waited for, so a chunk that is filled again or emptied too early gives wrong
bytes.  Element by element, around the chunks' borders, from several threads,
where no memory can be page-locked, and with a single thread."""

import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SRC = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <map>
#include <mutex>
#include <set>
#include <thread>
#include <vector>
#include "vls_hostcopy.h"

// ------------------------------------------------------------ fake runtime
struct Stream {
  std::vector<std::function<void()>> ops;
  size_t done = 0;
};
struct Event {
  Stream *s = nullptr;
  size_t upto = 0;
};
static std::mutex mu;
static std::set<void *> locked;  // live page-locked blocks
static std::atomic<int> allocs_left{1 << 30}, staged{0};
static cudaError_t last = cudaSuccess;
static void run(Stream *s, size_t upto) {
  for (; s->done < upto; ++s->done) s->ops[s->done]();
}
extern "C" {
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
  std::lock_guard<std::mutex> lk(mu);
  if (allocs_left-- <= 0) return last = cudaErrorMemoryAllocation;
  *p = std::malloc(n);
  locked.insert(*p);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
  std::lock_guard<std::mutex> lk(mu);
  if (!locked.erase(p)) return last = cudaErrorInvalidValue;
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
  *a = cudaPointerAttributes();
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  if (n == vls::ChunkPool::CHUNK) ++staged;
  ((Stream *)st)->ops.push_back([=] { std::memcpy(d, s, n); });
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  *e = (cudaEvent_t) new Event;
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete (Event *)e;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
  ((Event *)e)->s = (Stream *)st;
  ((Event *)e)->upto = ((Stream *)st)->ops.size();
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  run(((Event *)e)->s, ((Event *)e)->upto);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
  run((Stream *)st, ((Stream *)st)->ops.size());
  return cudaSuccess;
}
}
// ------------------------------------------------------------------- cases
static int bad = 0;
static void roundtrip(size_t bytes, size_t off, unsigned seed) {
  Stream st;
  std::vector<unsigned char> host(bytes + off), dev(bytes, 0), back(bytes + off, 0xEE);
  for (size_t i = 0; i < host.size(); ++i) host[i] = (unsigned char)((i * 2654435761u + seed) >> 9);
  vls::HostCopy c;
  if (c.upload(dev.data(), host.data() + off, bytes, (cudaStream_t)&st) != cudaSuccess) ++bad;
  cudaStreamSynchronize((cudaStream_t)&st);
  if (std::memcmp(dev.data(), host.data() + off, bytes)) ++bad;
  if (c.download(back.data() + off, dev.data(), bytes, (cudaStream_t)&st) != cudaSuccess) ++bad;
  cudaStreamSynchronize((cudaStream_t)&st);
  if (std::memcmp(back.data() + off, host.data() + off, bytes)) ++bad;
  for (size_t i = 0; i < off; ++i) bad += back[i] != 0xEE;
  c.release();
}
int main(int argc, char **argv) {
  const size_t M = vls::HostCopy::MIN_BYTES, C = vls::ChunkPool::CHUNK;
  if (std::atoi(argv[1]) == 0) {
    for (size_t n : {M - 8, M, M + 1, M + C - 1, M + C, M + C + 8, 2 * M + 12345, 9 * C + 7})
      for (size_t off : {0, 8, 4093}) roundtrip(n, off, (unsigned)(n + off));
    if (!staged) ++bad;
  } else if (std::atoi(argv[1]) == 1) {
    std::vector<std::thread> t;
    for (unsigned k = 0; k < 5; ++k)
      t.emplace_back([=] { for (unsigned i = 0; i < 3; ++i) roundtrip(M + k * C + 8 * i, 8 * k, 31 * k + i); });
    for (std::thread &x : t) x.join();
  } else if (std::atoi(argv[1]) == 2) {
    // no page-locked memory at all, then one block (half a pair), then enough
    for (int left : {0, 1, 1 << 20}) {
      allocs_left = left;
      roundtrip(M + 3 * C + 8, 8, (unsigned)left);
      if (cudaGetLastError() != cudaSuccess) ++bad;
    }
  }
  if (std::atoi(argv[1]) == 3) {
    // one thread: no chunks
    staged = 0;
    allocs_left = 0;
    roundtrip(M + 3 * C + 8, 8, 5);
    if (staged || allocs_left != 0) ++bad;
  }
  if (!locked.empty()) ++bad;  // the last object gave the chunks back
  std::printf("%d\n", bad);
  return bad != 0;
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if not shutil.which("g++") or not os.path.exists(CUDA + "/include/cuda_runtime.h"):
        pytest.skip("no g++ or no CUDA headers")
    d = tmp_path_factory.mktemp("hostcopy")
    (d / "t.cpp").write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fopenmp", "-pthread",
                           "-I" + CUDA + "/include",
                           "-I" + os.path.join(REPO, "vlasolve_b200", "csrc"),
                           str(d / "t.cpp"), "-o", str(d / "t")])
    return str(d / "t")


CASES = ["borders", "threads", "no_locked_memory", "one_thread"]


@pytest.mark.parametrize("case", CASES)
def test_copies(exe, case):
    env = dict(os.environ, OMP_NUM_THREADS="1" if case == "one_thread" else "4")
    r = subprocess.run([exe, str(CASES.index(case))], capture_output=True, text=True, timeout=300,
                       env=env)
    assert r.returncode == 0, r.stdout + r.stderr
