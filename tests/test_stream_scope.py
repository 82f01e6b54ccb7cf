"""Host code of the launches, compiled here; no CUDA call is made.  A launch that fails while
the operator's independent launches run on branches leaves the state as it was: the library
stream and the branch switch come back with the exception.  The parts of the near lists
follow from the number of items and the device's SMs alone, whichever entry point ran first."""
import subprocess

from erosion_b200 import build

SCOPE = r"""
#include "state.h"
#include <cstdio>
using namespace eb;
int main() {
  State s;
  const cudaStream_t lib = (cudaStream_t)0x10, branch = (cudaStream_t)0x20;
  s.st = lib;
  cudaStream_t seen = nullptr;
  on_stream(s, branch, [&] { seen = s.st; });
  if (seen != branch || s.st != lib) return 1;
  for (int depth = 0; depth < 2; ++depth) {
    try {
      const Scoped<bool> forked(s.forked, true);
      on_stream(s, branch, [&] {
        if (!s.forked) std::abort();
        if (depth) on_stream(s, (cudaStream_t)0x30, [] { throw Error(EROSION_CUDA_ERROR, "inner launch"); });
        throw Error(EROSION_CUDA_ERROR, "launch");
      });
      return 2;
    } catch (const Error&) {
    }
    if (s.st != lib || s.forked) return 3;
  }
  std::puts("ok");
  return 0;
}
"""


PARTS = r"""
#include "state.h"
#include <cstdio>
int main() {
  for (int sms : {74, 132, 148})
    for (int items : {1, 72, 464, 592, 593, 5000}) std::printf("%d ", eb::near_parts(items, sms));
  return 0;
}
"""


def run(tmp_path, source):
    src, exe = tmp_path / "host.cu", tmp_path / "host"
    src.write_text(source)
    subprocess.run([build.nvcc_path(), *build.COMPILE_FLAGS, "-I", build.INCLUDE, "-I", build.CSRC, "-o", str(exe),
                    str(src)], check=True, capture_output=True, text=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout


def test_a_throw_restores_the_library_stream(tmp_path):
    assert run(tmp_path, SCOPE) == "ok\n"


def test_near_parts_follow_the_device(tmp_path):
    want = [max(1, min(8, -(-4 * sms // items))) for sms in (74, 132, 148) for items in (1, 72, 464, 592, 593, 5000)]
    assert run(tmp_path, PARTS).split() == [str(v) for v in want]
