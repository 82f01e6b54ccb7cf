"""Host code of the launches, compiled here; no CUDA call is made.  A launch that fails while
the operator's independent launches run on branches leaves the state as it was: the library
stream and the branch switch come back with the exception.  The parts of the near lists
follow from the number of items and the device's SMs alone, whichever entry point ran first.
A host thread that the system refuses does not end the process: the others run its jobs."""
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

POOL = r"""
#include "pool.h"
#include <cstdio>
#include <mutex>
#include <numeric>
#include <sys/resource.h>
#include <unistd.h>
int main() {
  std::vector<int> order(200), done;
  std::iota(order.begin(), order.end(), 0);
  long pages = 0;   // address space for a few thread stacks more, not for sixteen
  if (FILE* f = std::fopen("/proc/self/statm", "r")) {
    if (std::fscanf(f, "%ld", &pages) != 1) return 1;
    std::fclose(f);
  }
  rlimit stack;
  getrlimit(RLIMIT_STACK, &stack);
  const rlim_t each = stack.rlim_cur == RLIM_INFINITY ? (rlim_t)2 << 20 : stack.rlim_cur;
  const rlim_t bytes = (rlim_t)pages * sysconf(_SC_PAGESIZE) + 3 * each;
  const rlimit lim{bytes, bytes};
  if (setrlimit(RLIMIT_AS, &lim)) return 2;
  std::mutex mu;
  int entered = 0;
  eb::on_pool(16, order, [&] { std::lock_guard<std::mutex> lk(mu); ++entered; },
              [&](int i) { std::lock_guard<std::mutex> lk(mu); done.push_back(i); usleep(2000); });
  std::sort(done.begin(), done.end());
  std::printf("%d %d\n", done == order, entered > 0 && entered < 16);
  try {
    eb::on_pool(4, order, [] {}, [](int i) { if (i == 7) throw std::runtime_error("seven"); });
  } catch (const std::runtime_error& e) {
    std::puts(e.what());
  }
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


def test_a_refused_thread_is_done_without(tmp_path):
    assert run(tmp_path, POOL) == "1 1\nseven\n"
