"""chain_launch (launches set up while the previous kernel runs): its arguments
must fit the kernel's parameters without a cast, and a refused launch leaves no
error for the next unrelated call (the runtime refuses a block of more threads
than a block can have)."""

import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <type_traits>
#include "vls_async.cuh"
using namespace vls;
__global__ void kern(const float *a, double *b, int64_t n, float x) {
  chain_begin();
  if (n < 0) b[0] = a[0] + x;
}
template <class... A>
auto fits(int, const A &...a)
    -> decltype(chain_launch(kern, dim3(1), dim3(1), size_t(0), cudaStream_t(0), a...),
                std::true_type());
template <class... A>
std::false_type fits(long, const A &...);
using F = float *;
using D = double *;
static_assert(decltype(fits(0, (const float *)0, D(), 1, 1.f))::value, "as declared");
static_assert(decltype(fits(0, F(), D(), int64_t(1), 1))::value, "implicit conversions");
static_assert(decltype(fits(0, nullptr, nullptr, 1, 1))::value, "null pointers");
static_assert(!decltype(fits(0, D(), D(), 1, 1.f))::value, "another type's pointer");
static_assert(!decltype(fits(0, F(), (const double *)0, 1, 1.f))::value, "const dropped");
static_assert(!decltype(fits(0, D(), F(), 1, 1.f))::value, "swapped");
static_assert(!decltype(fits(0, F(), 1, D(), 1.f))::value, "a number for a pointer");
int main() {
  const cudaError_t e = chain_launch(kern, dim3(1), dim3(4096), 0, 0, nullptr, nullptr, 1, 1.f);
  const cudaError_t left = cudaGetLastError();
  std::printf("%s, left: %s\n", cudaGetErrorName(e), cudaGetErrorName(left));
  return e != cudaSuccess && left == cudaSuccess ? 0 : 1;
}
"""


def _compile(tmp_path, *opts):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if not shutil.which(nvcc):
        pytest.skip("no nvcc")
    src, out = tmp_path / "t.cu", str(tmp_path / "t")
    src.write_text(SRC)
    subprocess.check_call([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                           "-I" + os.path.join(REPO, "vlasolve_b200", "csrc"), str(src), "-o", out,
                           *opts])
    return out


def test_arguments_are_checked(tmp_path):
    _compile(tmp_path, "-c")


@pytest.mark.gpu
def test_refused_launch_leaves_no_error(tmp_path):
    r = subprocess.run([_compile(tmp_path)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
