"""csrc/fault_ahead.h on the CPU when the host has no memory for another thread: no exception
leaves a C entry, and no thread that runs already is abandoned."""
import subprocess

from test_fault_ahead import CSRC, FAKE


THROWS = r"""
#include "fault_ahead.h"
#include <assert.h>
#include <stdlib.h>
#include <new>
int g_type = cudaMemoryTypeUnregistered;
static int g_left = -1;  // allocations until the next one fails
void *operator new(size_t n) {
  if (g_left == 0) throw std::bad_alloc();
  if (g_left > 0) --g_left;
  return malloc(n);
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }
int main() {
  const size_t n = 16u << 20;
  char *p = (char *)mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  for (int k = 0; k < 5; ++k) {
    g_left = k;
    { tg::FaultAhead f(p, n); }  // must neither throw nor end the process
    g_left = -1;
  }
  return 0;
}
"""


def test_no_memory_for_a_thread_leaves_the_pages_to_the_copy(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "main.cpp").write_text(THROWS)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-UNDEBUG", f"-I{tmp_path}", f"-I{CSRC}", str(tmp_path / "main.cpp"),
                    "-o", str(exe), "-lpthread"], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)
