"""A launch that fails while the operator's independent launches run on branches leaves the
state as it was: the library stream and the branch switch come back with the exception.
Host code alone, compiled here: no CUDA call is made."""
import subprocess

from erosion_b200 import build

SOURCE = r"""
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


def test_a_throw_restores_the_library_stream(tmp_path):
    src, exe = tmp_path / "scope.cu", tmp_path / "scope"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc_path(), *build.COMPILE_FLAGS, "-I", build.INCLUDE, "-I", build.CSRC, "-o", str(exe),
                    str(src)], check=True, capture_output=True, text=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout == "ok\n"
