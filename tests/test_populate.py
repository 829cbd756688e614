"""The helper that populates the pages of host outputs (csrc/vti_populate.h), compiled
for the host with a stand-in for the pointer query: what an array holds stays, and
no exception leaves it when there is no memory for its threads."""
import subprocess

from conftest import ROOT

SRC = r"""
#include <cstdlib>
#include <cstring>
#include <new>
static bool refuse = false;
void* operator new(std::size_t n) {
  void* p = refuse ? nullptr : std::malloc(n);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
#include "vti_populate.h"
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
int main() {
  const size_t n = (size_t)24 << 20;
  unsigned char* p = static_cast<unsigned char*>(std::calloc(n, 1));
  for (size_t i = 0; i < n; i += 4097) p[i] = (unsigned char)i;
  for (int round = 0; round < 2; ++round) {
    refuse = round == 1;
    vti::Populate pages;
    pages.start(p + 3, n - 5);
    pages.join();
    refuse = false;
  }
  for (size_t i = 0; i < n; ++i)
    if (p[i] != (i % 4097 == 0 ? (unsigned char)i : 0)) return 2;
  return 0;
}
"""


def test_contents_stay_and_nothing_is_thrown(tmp_path):
    (tmp_path / "use.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'thesis-source-code_b200' / 'csrc'}",
                    "-I/usr/local/cuda/include", str(tmp_path / "use.cpp"), "-o",
                    str(tmp_path / "use"), "-lpthread"], check=True)
    assert subprocess.run([str(tmp_path / "use")]).returncode == 0
