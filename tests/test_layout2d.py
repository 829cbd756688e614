"""The cut of a 2D grid into tiles (csrc/vti_tile2d.h), compiled for the host:
every index of a layout that is used fits its type."""
import subprocess

import pytest

from conftest import ROOT

PKG = ROOT / "thesis-source-code_b200"
SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "vti_tile2d.h"
int main(int argc, char** argv) {
  for (int i = 1; i + 3 < argc; i += 4) {
    const auto L = vti::tile2d::make_layout(148, atoi(argv[i]), atoi(argv[i + 1]),
                                            atoi(argv[i + 2]), atoi(argv[i + 3]));
    printf("%d %d %d %d %d %zu\n", L.T, L.tile, L.ntx, L.ntz, L.W, L.n);
  }
}
"""


@pytest.fixture(scope="module")
def layouts(tmp_path_factory):
    d = tmp_path_factory.mktemp("layout")
    (d / "layout.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{PKG / 'csrc'}", f"-I{ROOT / 'include'}",
                    "-I/usr/local/cuda/include", str(d / "layout.cpp"), "-o", str(d / "layout"),
                    "-L/usr/local/cuda/lib64", "-lcudart"], check=True)

    def run(*grids):  # (nnx, nnz, shots, backward) -> (T, tile, ntx, ntz, W, n)
        args = [str(int(v)) for g in grids for v in g]
        out = subprocess.run([str(d / "layout"), *args], check=True, capture_output=True,
                             text=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]
    return run


def test_indices_of_thin_long_grids_fit_their_types(layouts):
    grids = [(9, 2 ** 30 // 9), (2 ** 30 // 9, 9), (40, 2 ** 30 // 40), (2 ** 30 // 40, 40),
             (9, 2 ** 24), (2 ** 24, 9), (2 ** 15, 2 ** 15), (9, 2 ** 21), (9, 9), (461, 261)]
    cases = [(a, b, 1, back) for a, b in grids for back in (0, 1)]
    taken = 0
    for (nnx, nnz, _, back), (T, tile, ntx, ntz, W, n) in zip(cases, layouts(*cases)):
        if not T:
            assert 64 * max(nnx, nnz) >= 2 ** 31 or nnz / 48 > 65535  # nothing small is left out
            continue
        taken += 1
        assert T >= (3 if back else 2) and n < 2 ** 31 and ntz <= 65535
        off = 4 * T - 4
        assert (nnx - 1 + off) < W and (nnx - 1 + off) + (nnz - 1 + off) * W < n
        assert (ntx - 1) * tile + 64 <= W and ((ntz - 1) * tile + 64) * W <= n
    assert 6 <= taken < len(cases)
