"""The 3D step kernels walk the volume down z on even levels and up z on odd
ones. Depths whose last 4-plane sponge block is partial, segments that start
and end off a block boundary, and a volume of a single segment, against the
FP64 oracle (the reference's FP32 trace tolerance 1e-5, gradients 1e-4)."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_l2

import vtib200 as V
import vtib200.synth as S

pytestmark = pytest.mark.gpu


# nx, ny, nz, npad, planes per segment of the forward and of the backward step on 148
# SMs (tests/test_sched3d.py computes them)
GRIDS = [(40, 36, 24, 6, 4, 4), (41, 25, 21, 5, 4, 4), (33, 37, 26, 7, 4, 4), (70, 26, 35, 9, 4, 4),
         (250, 250, 21, 5, 7, 11), (250, 250, 26, 6, 9, 13), (330, 360, 21, 5, 21, 21)]


@pytest.mark.parametrize("nx,ny,nz,npad", [g[:4] for g in GRIDS])
def test_alternating_march_matches_oracle(ctx, nx, ny, nz, npad):
    s = S.small3d(nx=nx, ny=ny, nz=nz, nt=131, npad=npad, rate=2.8e-3)
    t = S.small3d(nx=nx, ny=ny, nz=nz, nt=131, npad=npad, rate=2.8e-3, seed=11)
    g, n = s.geom(), s.nxyz
    padb, randb = S.boundaries3d(s)
    ct = t.cij()
    ct = [ct[k * n:(k + 1) * n] for k in range(3)]
    d = V.modelDataCij3d_f(ctx, g, s.souloc, [0], s.recloc, s.wavelet, *ct)
    od = O.model_data3d(g, *ct, s.wavelet, s.souloc, [0], s.recloc)
    assert np.abs(od).max() > 0
    assert rel_l2(d, od) < 1e-5
    fg, mis = V.objFuncGradientCij3d_f(ctx, g, s.souloc, [0], s.recloc, s.wavelet, s.cij(), padb,
                                       randb, od)
    o, mod = O.gradient3d(g, s.cij(), padb, randb, s.wavelet, s.souloc, [0], s.recloc, od,
                          want_modeled=True)
    # the residual r carries the trace error magnified by |d| / |r|: |dJ|/J is
    # twice that to first order, and the gradient, linear in r, gains it once
    res_tol = 1e-5 * np.linalg.norm(od) / np.linalg.norm(mod - od)
    assert abs(mis - o[0]) / o[0] < 2 * res_tol
    for k in range(3):
        a, b = fg[1 + k * n:1 + (k + 1) * n], o[1 + k * n:1 + (k + 1) * n]
        assert rel_l2(a, b) < 1e-4 + res_tol, k
