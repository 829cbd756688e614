"""2D propagation several levels per launch against the per-level kernels
(Context.set_2d_resident(False)): the tiles split the grid and the levels, not
the arithmetic, so traces are equal bit for bit; gradients and images within
the FP32 rounding of their sums (1e-5), and against the FP64 oracle elsewhere."""
import numpy as np
import pytest

from conftest import rel_l2

import vtib200 as V
import vtib200.synth as S

pytestmark = pytest.mark.gpu


def both(ctx, call):
    out = []
    for on in (False, True):
        ctx.set_2d_resident(on)
        try:
            out.append(call())
        finally:
            ctx.set_2d_resident(True)
    return out


def shots(s, pos, per, depth):
    """Sources at `pos`, each recorded by its own `per` cells at `depth`."""
    s.sloc = np.array([[x, s.npad + 2, per, k * per] for k, x in enumerate(pos)], np.int32)
    s.rloc = np.array([[4 + (7 * k + 3 * i) % (s.nx + 2 * s.npad - 8), depth + i % 3]
                       for k in range(len(pos)) for i in range(per)], np.int32)
    return s


# grids of one tile and just over, ragged tiles, a grid wider than one cluster;
# records whose levels are not a multiple of the levels of a launch
@pytest.mark.parametrize("nx,nz,pad,nt,rate", [(20, 20, 10, 30, 1e-3), (21, 21, 10, 31, 2e-3),
                                               (57, 30, 12, 65, 3e-3), (40, 90, 9, 130, 2e-3),
                                               (1030, 25, 10, 72, 2e-3)])
def test_tiled_traces_equal_per_level_traces(ctx, nx, nz, pad, nt, rate):
    s = S.survey2d(nx=nx, nz=nz, nt=nt, npad=pad, rate=rate)
    s = shots(s, [pad + 3, 4, nx + 2 * pad - 5], min(nx // 3, 40), pad + 1)
    a, b = both(ctx, lambda: V.synthetic_f(ctx, s.geom(), s.c11, s.c13, s.c33, s.wavelet, s.sloc,
                                           s.rloc, s.taper))
    assert np.abs(a).max() > 0
    assert np.array_equal(a, b)


@pytest.mark.parametrize("nx,nz,pad,nt,rate,ns", [(20, 20, 10, 31, 2e-3, 1), (57, 30, 12, 64, 3e-3, 2),
                                                  (40, 90, 9, 133, 2e-3, 1),
                                                  (101, 61, 15, 202, 4e-3, 2)])
def test_tiled_gradient_and_migration_match_per_level(ctx, nx, nz, pad, nt, rate, ns):
    s = S.survey2d(nx=nx, nz=nz, nt=nt, npad=pad, rate=rate)
    s = shots(s, [pad + nx // 2, pad + 4][:ns], nx // 3, pad + 1)
    g = s.geom()
    data = V.synthetic_f(ctx, g, 0.95 * s.c11, 0.96 * s.c13, 0.97 * s.c33, s.wavelet, s.sloc, s.rloc,
                         s.taper)
    a, b = both(ctx, lambda: V.objFuncGradient_f(ctx, g, data, s.c11, s.c13, s.c33, s.wavelet,
                                                 s.sloc, s.rloc, s.taper))
    assert a[3] > 0 and a[3] == b[3]
    for x, y in zip(a[:3], b[:3]):
        assert np.abs(x).max() > 0
        assert rel_l2(y, x) < 1e-5
    a, b = both(ctx, lambda: V.rtm_f(ctx, g, data, s.c11, s.c13, s.c33, s.wavelet, s.sloc, s.rloc,
                                     s.taper))
    assert np.abs(a).max() > 0
    assert rel_l2(b, a) < 1e-5
