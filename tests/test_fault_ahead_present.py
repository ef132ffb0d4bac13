"""csrc/fault_ahead.h on the CPU: a buffer whose pages are there starts no thread (a download
into memory that an earlier one filled has nothing to wait for)."""
import subprocess

from test_fault_ahead import CSRC, FAKE

MAIN = r"""
#include "fault_ahead.h"
#include <assert.h>
#include <stdlib.h>
#include <string.h>
#include <new>
int g_type = cudaMemoryTypeUnregistered;
static int g_news = 0;  // a thread's start allocates its state
void *operator new(size_t n) { ++g_news; return malloc(n); }
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }
static int threads(char *p, size_t n) {
  const int before = g_news;
  { tg::FaultAhead f(p, n); }
  return g_news - before;
}
int main() {
  const size_t n = 21u << 20;
  for (size_t off : {size_t(0), size_t(64)}) {
    char *p = (char *)mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    assert(threads(p + off, n - off) > 0);   // fresh
    memset(p, 1, n);
    assert(threads(p + off, n - off) == 0);  // filled
    for (size_t cut : {size_t(0), n / 2, n - (4u << 20)}) {
      memset(p, 1, n);
      madvise(p + cut, 4u << 20, MADV_DONTNEED);
      assert(threads(p + off, n - off) > 0);  // a part is gone
    }
    munmap(p, n);
  }
  return 0;
}
"""


def test_pages_that_are_there_start_no_thread(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-UNDEBUG", f"-I{tmp_path}", f"-I{CSRC}", str(tmp_path / "main.cpp"),
                    "-o", str(exe), "-lpthread"], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)
