"""A kernel launch that the runtime refuses is reported by the helper that issues it
(csrc/launch.cuh), whatever is queried between it and the end of the call, and leaves no error
behind.  A block of 2048 threads is refused on the host; without a GPU every launch is."""

import subprocess

import pytest

from materialite_b200.csrc import build

PROGRAM = r"""
#include <cstdio>
#include "launch.cuh"
static std::string last;
int ssfft_internal_fail(int code, const std::string &msg) { last = msg; return code; }
__global__ void nothing(int) {}
template <int> __global__ void other(int) {}
static int passes() {  // as a projection: a refused pass, then a query for the next one
  CKR(launch_kernel(PDL, nothing, 1, 2048, 0, 0, 1));
  resident_blocks(other<1>, 32, 0, 0);
  return 0;
}
static int clustered() {
  CKR(launch_clustered(nothing, 2, 2048, 0, 1, 0, 0, 1));
  return 0;
}
int main() {
  const int a = passes();
  const bool named = last.find("kernel launch") == 0;
  const int b = clustered();
  std::printf("%d %d %d %d\n", a, (int)named, b, (int)cudaGetLastError());
}
"""


def refused(tmp_path, pdl):
    src, exe = tmp_path / "launch.cu", tmp_path / "launch"
    src.write_text(PROGRAM)
    try:
        subprocess.run([build.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                        f"-DPDL={pdl}", "-I", build.HERE, "-o", str(exe), str(src)], check=True)
    except FileNotFoundError:
        pytest.skip("no nvcc")
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()


# SSFFT_E_CUDA from both helpers, the launch named in the message
@pytest.mark.parametrize("pdl", ["false", "true"])
def test_refused_launch_is_returned(tmp_path, pdl):
    assert refused(tmp_path, pdl)[:3] == ["-2", "1", "-2"]


@pytest.mark.gpu
def test_refused_launch_leaves_no_error(tmp_path):
    assert refused(tmp_path, "true") == ["-2", "1", "-2", "0"]
