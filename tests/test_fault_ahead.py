"""csrc/fault_ahead.h on the CPU, with a stand-in for the pointer query: the
contents of a buffer stay, its pages are there afterwards, and ranges that end
off a page, short ranges and read-only or unmapped memory are left to the copy."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(__file__), "..", "imod-rs_b200", "csrc")

FAKE = """
#pragma once
typedef int cudaError_t;
enum { cudaSuccess = 0, cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
struct cudaPointerAttributes { int type; };
extern int g_type;
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) { a->type = g_type; return 0; }
inline cudaError_t cudaGetLastError() { return 0; }
"""

MAIN = r"""
#include "fault_ahead.h"
#include <assert.h>
#include <string.h>
#include <vector>
int g_type = cudaMemoryTypeUnregistered;
static size_t resident(char *p, size_t n) {
  std::vector<unsigned char> v((n + 4095) / 4096);
  assert(mincore(p, n, v.data()) == 0);
  size_t c = 0;
  for (unsigned char x : v) c += x & 1;
  return c;
}
static char *map(size_t n, int prot) {
  return (char *)mmap(nullptr, n, prot, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
}
int main() {
  const size_t n = 37u << 20;
  for (size_t off : {size_t(0), size_t(64), size_t(4095)}) {
    char *p = map(n, PROT_READ | PROT_WRITE);
    p[off] = 7;
    p[n / 2] = 8;
    { tg::FaultAhead f(p + off, n - off - 100); }
    assert(p[off] == 7 && p[n / 2] == 8 && p[n / 2 + 1] == 0);
    if (madvise(map(4096, PROT_READ | PROT_WRITE), 4096, MADV_POPULATE_WRITE) == 0) assert(resident(p, n) >= n / 4096 - 2);
    munmap(p, n);
  }
  char *p = map(n, PROT_READ | PROT_WRITE);
  { tg::FaultAhead f(p, 1u << 20); }
  { tg::FaultAhead f(nullptr, n); }
  g_type = cudaMemoryTypeHost;
  { tg::FaultAhead f(p, n); }
  assert(resident(p, n) == 0);
  g_type = cudaMemoryTypeUnregistered;
  { tg::FaultAhead f(map(n, PROT_READ), n); }   // read-only
  munmap(p + (8 << 20), 8 << 20);
  { tg::FaultAhead f(p, n); }                   // a hole
  return 0;
}
"""


def test_fault_ahead(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-UNDEBUG", f"-I{tmp_path}", f"-I{CSRC}", str(tmp_path / "main.cpp"),
                    "-o", str(exe), "-lpthread"], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)
