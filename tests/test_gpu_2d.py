"""GPU parity tests of the 2D forward path (synthetic_f / modeling_f)."""
import numpy as np
import pytest

import cases as K
import oracle as O
from conftest import load_golden, rel_l2

import vtib200 as V
import vtib200.synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", K.CASES2D)
def test_synthetic_matches_oracle_and_reference(ctx, name):
    s = K.case2d(name)["s"]
    g = s.geom()
    d = V.synthetic_f(ctx, g, s.c11, s.c13, s.c33, s.wavelet, s.sloc, s.rloc, s.taper)
    o = O.forward2d(g, s.c11, s.c13, s.c33, s.wavelet, s.sloc, s.rloc, s.taper)
    assert np.abs(o).max() > 0
    assert rel_l2(d, o) < 1e-5
    assert rel_l2(d.reshape(-1), load_golden(name)["data"]) < 1e-5


# Whole-wavefield snapshots carry more FP32 rounding than traces: the
# reference's own snapshots of this case are 9.3e-6 from the FP64 oracle
# (1.9e-5 at the last one), so two FP32 implementations may differ by 2x that.
SNAP_TOL = 3e-5


@pytest.mark.parametrize("name", K.CASES2D)
def test_modeling_matches_oracle_and_reference(ctx, name):
    s = K.case2d(name)["s"]
    g = s.geom()
    sxz = int(s.sloc[0] + s.sloc[1] * (s.nx + 2 * s.npad))
    w = V.modeling_f(ctx, g, s.c11, s.c13, s.c33, s.wavelet, sxz, s.taper)
    o = O.forward2d(g, s.c11, s.c13, s.c33, s.wavelet, None, None, s.taper, mode=1, slocxz=sxz)
    assert rel_l2(w[: o.shape[0]], o) < SNAP_TOL
    gold = load_golden(name)
    assert np.abs(gold["snaps"]).max() > 0
    assert rel_l2(w[gold["snap_rows"]], gold["snaps"]) < SNAP_TOL


@pytest.mark.parametrize("name", K.CASES2D)
def test_gradient_matches_oracle_and_reference(ctx, name):
    c = K.case2d(name)
    s = c["s"]
    g = s.geom()
    n = (s.nx + 2 * s.npad) * (s.nz + 2 * s.npad)
    gold = load_golden(name)
    g11, g13, g33, mis = V.objFuncGradient_f(ctx, g, gold["dobs"], s.c11, s.c13, s.c33, s.wavelet,
                                             s.sloc, s.rloc, s.taper)
    o = O.gradient2d(g, s.c11, s.c13, s.c33, s.wavelet, s.sloc, s.rloc, s.taper,
                     data=gold["dobs"])
    ref = gold["grad"]
    assert abs(mis - o[3]) / o[3] < 1e-5
    assert abs(mis - ref[3 * n]) / ref[3 * n] < 1e-5
    for k, a in enumerate((g11, g13, g33)):
        assert rel_l2(a, o[k]) < 1e-4, k
        assert rel_l2(a, ref[k * n:(k + 1) * n]) < 1e-4, k


@pytest.mark.parametrize("name", K.CASES2D)
def test_gn_hessian_matches_oracle_and_reference(ctx, name):
    c = K.case2d(name)
    s = c["s"]
    g = s.geom()
    n = (s.nx + 2 * s.npad) * (s.nz + 2 * s.npad)
    dc = (c["dc"]["c11"], c["dc"]["c13"], c["dc"]["c33"])
    h = V.GNhessian_f(ctx, g, s.c11, s.c13, s.c33, *dc, s.wavelet, s.sloc, s.rloc, s.taper)
    o = O.gradient2d(g, s.c11, s.c13, s.c33, s.wavelet, s.sloc, s.rloc, s.taper, dc=dc)
    ref = load_golden(name)["gnhess"]
    for k in range(3):
        assert rel_l2(h[k], o[k]) < 1e-4, k
        assert rel_l2(h[k], ref[k * n:(k + 1) * n]) < 1e-4, k
    # linear in the perturbation
    h2 = V.GNhessian_f(ctx, g, s.c11, s.c13, s.c33, *(2 * x for x in dc), s.wavelet, s.sloc,
                       s.rloc, s.taper)
    for k in range(3):
        assert rel_l2(h2[k], 2 * h[k]) < 1e-5


def test_synthetic_config_size(ctx):
    """The 2D benchmark grid (201 x 401 + 30-cell pad, 2000 steps), one shot."""
    s = S.survey2d()
    g = s.geom()
    d = V.synthetic_f(ctx, g, s.c11, s.c13, s.c33, s.wavelet, s.sloc, s.rloc, s.taper)
    o = O.forward2d(g, s.c11, s.c13, s.c33, s.wavelet, s.sloc, s.rloc, s.taper)
    assert rel_l2(d, o) < 1e-5


@pytest.mark.parametrize("kw", [
    dict(),  # the benchmark grid, 461 x 261: one shot runs in tiles
    dict(nx=97, nz=37, nt=240, npad=9, d=10.0, dt=1e-3, rate=1e-3, freq=20.0, src_x=480.0,
         src_z=120.0, rec_z=0.0, ns=3),  # shots on receivers of their own in a cluster each
    # (ragged rows, every step sampled, source in exchanged rows), on shared ones in tiles
    dict(nx=1100, nz=24, nt=120, npad=8, d=10.0, dt=1e-3, rate=2e-3, freq=15.0, src_x=5000.0,
         src_z=100.0, rec_z=20.0),  # wider than one cluster: tiles
])
def test_resident_traces_equal_per_step_traces(ctx, kw):
    """The shared-memory resident launch (one cluster per shot), the tiles and
    the per-step launches compute every point with the same operations: the
    traces are bitwise equal."""
    s = S.survey2d(**kw)
    g = s.geom()
    args = (ctx, g, s.c11, s.c13, s.c33, s.wavelet, s.sloc, s.rloc, s.taper)
    if kw.get("ns", 1) > 1:
        # the survey's shots all record every receiver (a later shot
        # overwrites); also run disjoint receiver blocks (all shots in one
        # launch, one cluster each)
        sl = s.sloc.reshape(-1, 4).copy()
        nrb = (s.rloc.size // 2) // len(sl)
        sl[:, 2] = nrb
        sl[:, 3] = np.arange(len(sl)) * nrb
        args2 = (ctx, g, s.c11, s.c13, s.c33, s.wavelet, sl.reshape(-1), s.rloc, s.taper)
        before = ctx.launches
        res2 = V.synthetic_f(*args2)
        assert ctx.launches - before == 1
        ctx.set_2d_resident(False)
        try:
            step2 = V.synthetic_f(*args2)
        finally:
            ctx.set_2d_resident(True)
        assert np.abs(step2).max() > 0
        np.testing.assert_array_equal(res2, step2)
    res = V.synthetic_f(*args)
    ctx.set_2d_resident(False)
    try:
        step = V.synthetic_f(*args)
    finally:
        ctx.set_2d_resident(True)
    assert np.abs(step).max() > 0
    np.testing.assert_array_equal(res, step)


@pytest.mark.parametrize("nx,nz,ns", [(97, 37, 1), (97, 37, 3), (401, 201, 1)])
def test_receivers_outside_the_grid_are_refused_whatever_the_path(ctx, nx, nz, ns):
    """Grids that fit one cluster: a receiver outside the grid is refused even if no
    shot records it, whether the cluster or the tiles would run the call."""
    s = S.survey2d(nx=nx, nz=nz, nt=60, npad=10, ns=ns)
    rloc = np.concatenate([s.rloc, np.array([nx + 20, 5], np.int32)])  # first column outside
    args = (ctx, s.geom(), s.c11, s.c13, s.c33, s.wavelet, s.sloc)
    with pytest.raises(V.VtiError, match="outside the grid"):
        V.synthetic_f(*args, rloc, s.taper)
    ctx.set_2d_resident(False)
    try:  # the per-level path reads only the receivers of the shots
        V.synthetic_f(*args, rloc, s.taper)
    finally:
        ctx.set_2d_resident(True)


@pytest.mark.parametrize("nx,nz,nt,ns,cluster", [
    (41, 31, 200, 1, True),     # 101 x 91: a cluster's level is shorter
    (201, 101, 10, 1, True),    # 261 x 161, a short record: the tiles' preparation costs more
    (201, 101, 1000, 1, False),
    (201, 101, 500, 4, True),   # four shots fill the GPU either way
    (401, 201, 500, 14, True),  # 461 x 261, 16 CTAs of 16 rows, more shots than clusters
    (401, 201, 500, 2, False)])
def test_cluster_or_tiles_by_cost(ctx, nx, nz, nt, ns, cluster):
    """Shots on receivers of their own run where they take less time: one launch with
    a cluster per shot, or tiles; the traces are those of the per-step path."""
    s = S.survey2d(nx=nx, nz=nz, nt=nt, ns=ns)
    sl = s.sloc.reshape(-1, 4)
    sl[:, 2] = nx // ns
    sl[:, 3] = np.arange(ns) * (nx // ns)
    args = (ctx, s.geom(), s.c11, s.c13, s.c33, s.wavelet, s.sloc, s.rloc, s.taper)
    before = ctx.launches
    res = V.synthetic_f(*args)
    assert (ctx.launches - before == 1) == cluster
    ctx.set_2d_resident(False)
    try:
        step = V.synthetic_f(*args)
    finally:
        ctx.set_2d_resident(True)
    assert nt < 100 or np.abs(step).max() > 0
    np.testing.assert_array_equal(res, step)


@pytest.mark.parametrize("shared", [False, True])
def test_cluster_takes_what_the_tiles_refuse(ctx, shared):
    """Two receivers of a shot on one cell: every shot runs in a cluster, all of them
    in one launch or, where they share receivers, one launch after another."""
    s = S.survey2d(nx=97, nz=37, nt=240, npad=9, rate=1e-3, ns=3)
    sl, rl = s.sloc.reshape(-1, 4), s.rloc.reshape(-1, 2)
    if not shared:
        sl[:, 2], sl[:, 3] = 32, np.arange(3) * 32
    rl[1::32] = rl[0::32][: len(rl[1::32])]
    args = (ctx, s.geom(), s.c11, s.c13, s.c33, s.wavelet, s.sloc, s.rloc, s.taper)
    before = ctx.launches
    res = V.synthetic_f(*args)
    assert ctx.launches - before == (3 if shared else 1)
    ctx.set_2d_resident(False)
    try:
        step = V.synthetic_f(*args)
    finally:
        ctx.set_2d_resident(True)
    assert np.abs(step).max() > 0
    np.testing.assert_array_equal(res, step)
