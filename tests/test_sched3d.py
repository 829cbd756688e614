"""The cut of a 3D launch into segments (csrc/vti_sched.h), compiled for the host."""
import itertools
import subprocess

import pytest

from conftest import ROOT

PKG = ROOT / "thesis-source-code_b200"
SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "vti_sched.h"
int main(int argc, char** argv) {
  for (int i = 1; i + 5 < argc; i += 6) {
    vti::Dims3 d{};
    d.nx = atoi(argv[i]);
    d.ny = atoi(argv[i + 1]);
    d.nz = atoi(argv[i + 2]);
    const auto s = vti::plan_sched(148, d, atoi(argv[i + 3]), atoi(argv[i + 4]), atoll(argv[i + 5]));
    printf("%d %d %d %d %lld\n", s.seg, s.items, s.grid, s.gx * s.gy, vti::sched_columns(d));
  }
}
"""


@pytest.fixture(scope="module")
def scheds(tmp_path_factory):
    d = tmp_path_factory.mktemp("sched")
    (d / "sched.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{PKG / 'csrc'}", f"-I{ROOT / 'include'}",
                    "-I/usr/local/cuda/include", str(d / "sched.cpp"), "-o", str(d / "sched"),
                    "-L/usr/local/cuda/lib64", "-lcudart"], check=True)

    def run(cases):  # (nx, ny, nz, CTAs per SM, copies, launch planes) -> (seg, items, grid, cols)
        args = [str(int(v)) for c in cases for v in c]
        out = subprocess.run([str(d / "sched"), *args], check=True, capture_output=True,
                             text=True).stdout
        rows = [tuple(map(int, line.split())) for line in out.splitlines()]
        assert all(r[3] == r[4] for r in rows)
        return [r[:4] for r in rows]
    return run


SIZES = [9, 40, 41, 64, 97, 110, 160, 250, 400]
DEPTHS = [1, 3, 7, 20, 21, 64, 83, 100, 150]


def test_items_cover_the_volume(scheds):
    cases = [(nx, ny, nz, c, k, 0) for nx, ny in itertools.product(SIZES, SIZES) for nz in DEPTHS
             for c in (2, 3) for k in (1, 2)]
    for (nx, ny, nz, ctas, copies, _), (seg, items, grid, cols) in zip(cases, scheds(cases)):
        assert 1 <= seg <= nz and items == cols * -(-nz // seg)
        assert 32 * (-(-(nx - 4) // 32)) >= nx - 4
        assert grid == min(items * copies, 148 * ctas)
        if seg < min(8, nz):  # short segments only while every item is resident
            assert seg >= 4 and items * copies <= 148 * ctas


def test_shared_launch_counts_every_volume(scheds):
    """Volumes that share a launch: short segments only where all items of the launch
    are resident at once; a volume that shares with nothing is cut as alone."""
    jobs = [(nx, ny) for nx in (48, 64, 80, 96) for ny in (48, 64, 80, 96)]
    for nz in (20, 64, 80, 100):
        for ctas in (2, 3):
            alone = scheds([(nx, ny, nz, ctas, 1, 0) for nx, ny in jobs])
            assert alone == scheds([(nx, ny, nz, ctas, 1, a[3] * nz)
                                    for (nx, ny), a in zip(jobs, alone)])
            for n in (2, 4, 16):
                planes = sum(a[3] for a in alone[:n]) * nz
                got = scheds([(nx, ny, nz, ctas, 1, planes) for nx, ny in jobs[:n]])
                total = sum(g[1] for g in got)
                assert len({g[0] for g in got}) == 1  # one depth, one segment length
                if got[0][0] < 8:
                    assert total <= 148 * ctas


def test_segments_of_the_march_test(scheds):
    """The grids that the GPU test of the march is written for have the segments it
    names: off the 4-plane blocks, and the whole depth."""
    from test_gpu_march import GRIDS
    for per_sm, col in ((3, 4), (2, 5)):
        got = scheds([(g[0], g[1], g[2], per_sm, 1, 0) for g in GRIDS])
        assert [s[0] for s in got] == [g[col] for g in GRIDS]
