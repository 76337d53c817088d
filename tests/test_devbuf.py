"""A device buffer whose allocation was refused is empty and of size 0: code that
keeps a workspace while it is large enough must not take a refused one for it.
A C++ program over the library's own header, with a size that no device has."""
import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include <string>
#include "nmg_internal.h"
int main() {
  nmg::DevBuf<double> b;
  const bool refused = b.alloc((size_t)1 << 57) != cudaSuccess;
  std::printf("%d %d %zu\n", (int)refused, (int)(b.p == nullptr), b.n);
  const bool empty = b.alloc(0) == cudaSuccess;
  std::printf("%d %d %zu\n", (int)empty, (int)(b.p == nullptr), b.n);
  return 0;
}
"""


def test_refused_allocation(tmp_path):
    from nmag import _build
    src, exe = tmp_path / "devbuf.cu", tmp_path / "devbuf"
    src.write_text(PROGRAM)
    subprocess.run([_build.nvcc()] + _build.ARCH + ["-std=c++17", "-I", os.path.join(ROOT, "nmag-src_gb300", "csrc"),
                                                    "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split("\n")[:2] == ["1 1 0", "1 1 0"]
