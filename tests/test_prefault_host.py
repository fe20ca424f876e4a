"""Host build of the pages of result arrays (csrc/prefault.cu), on CPU: which sizes get
their pages in the background."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
SRC = r'''
#include <sys/mman.h>
#include <unistd.h>
#include <cstdio>
#include <cstdlib>
#include "common.cuh"
// megabytes of a fresh mapping of argv[1] MB that are resident after a HostPrefault
int main(int, char** argv) {
  const size_t n = (size_t)std::atoll(argv[1]) << 20, page = sysconf(_SC_PAGESIZE);
  void* p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (p == MAP_FAILED) return 1;
  {
    pgb::HostPrefault pages(p, n);
    pages.join();
  }
  std::vector<unsigned char> in(n / page);
  if (mincore(p, n, in.data()) != 0) return 1;
  size_t have = 0;
  for (unsigned char c : in) have += c & 1;
  printf("%zu\n", have * page >> 20);
  return 0;
}
'''


def compile_host(tmp_path, source, name, plain=None):
    """source: a .cu file; plain: a C++ file beside it"""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not found")
    csrc = ROOT / "pyrpa_gb300" / "csrc"
    (tmp_path / f"{name}.cu").write_text(source)
    exe = tmp_path / name
    files = [tmp_path / f"{name}.cu", csrc / "prefault.cu"]
    if plain:
        files.append(tmp_path / f"{name}_plain.cpp")
        files[-1].write_text(plain)
    subprocess.run([nvcc, "-std=c++17", "-O2", "-I", str(csrc), *map(str, files), "-o", str(exe)], check=True,
                   capture_output=True, text=True)
    return exe


def test_sizes_that_get_their_pages(tmp_path):
    exe = compile_host(tmp_path, SRC, "pages")
    have = {mb: int(subprocess.run([str(exe), str(mb)], check=True, capture_output=True, text=True).stdout)
            for mb in (16, 64, 1024 + 64)}
    assert have[16] == 0
    if have[64] == 0:
        pytest.skip("no MADV_POPULATE_WRITE in this kernel")
    assert have[64] == 64
    assert have[1024 + 64] == 0


ALLOC = r'''
#include <cstdlib>
#include <new>
thread_local int left = -1;  // allocations of the calling thread until one fails; -1: none fails
void* operator new(size_t n) {
  if (left >= 0 && left-- == 0) throw std::bad_alloc();
  void* p = std::malloc(n);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
'''
NO_MEMORY = r'''
#include <sys/mman.h>
#include <cstdio>
#include "common.cuh"
extern thread_local int left;
int main() {
  const size_t n = 256u << 20;
  void* p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (p == MAP_FAILED) return 1;
  for (int k = 0; k < 16; ++k) {
    left = k;
    pgb::HostPrefault pages(p, n);
    left = -1;
    pages.join();
  }
  std::puts("done");
  return 0;
}
'''


def test_failed_allocations_leave_the_pages_to_the_copy(tmp_path):
    """Every allocation of the constructor fails once, also after threads have started."""
    exe = compile_host(tmp_path, NO_MEMORY, "no_memory", ALLOC)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "done\n", r.stderr
