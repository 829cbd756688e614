"""2D propagation several levels per launch against the per-level kernels
(Context.set_2d_resident(False)): the tiles split the grid and the levels, not
the arithmetic, so traces, gradients and images are equal bit for bit. (Images of
traces with values below 1e-31 are not: the per-level path's atomics flush
subnormal contributions.) Every case says how many levels its launches take, and
the number of launches confirms it."""
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


def step_launches(ctx, call):
    """Launches of the 2D step kernels that a call makes."""
    ctx.set_timing(True)
    try:
        call()
        return ctx.kernel_time("step2d")[1]
    finally:
        ctx.set_timing(False)


def shots(s, pos, per, depth, step=None):
    """Sources at `pos`, each recorded by `per` cells from row `depth` on, `step` of
    them (all by default) not recorded by the shot before."""
    n = s.nx + 2 * s.npad - 8
    step = per if step is None else step
    m = next(k for k in (7, 11, 13, 17) if n % k)  # 7th cell by 7th cell, row after row
    s.sloc = np.array([[x, s.npad + 2, per, k * step] for k, x in enumerate(pos)], np.int32)
    s.rloc = np.array([[4 + m * j % n, depth + j // n]
                       for j in range(per + (len(pos) - 1) * step)], np.int32)
    return s


# levels per launch T and grids of: one tile exactly and one cell more (tiles of 24
# cells a side), ragged tiles in both directions, a row of tiles wider than a cluster,
# one wave of 32-cell tiles, two of 40 and four of 48; records whose levels are not a
# multiple of T, and every level sampled with a receiver on the source
@pytest.mark.parametrize("nx,nz,pad,nt,rate,ns,T", [
    (12, 12, 10, 60, 1e-3, 3, 5), (13, 13, 10, 61, 2e-3, 3, 5), (57, 30, 12, 65, 3e-3, 3, 5),
    (40, 90, 9, 130, 2e-3, 3, 5), (1030, 25, 10, 72, 2e-3, 3, 3), (401, 201, 30, 65, 2e-3, 1, 4),
    (401, 201, 30, 80, 1e-3, 2, 2), (801, 401, 30, 63, 2e-3, 1, 3), (801, 401, 30, 64, 4e-3, 3, 2)])
def test_tiled_traces_equal_per_level_traces(ctx, nx, nz, pad, nt, rate, ns, T):
    s = S.survey2d(nx=nx, nz=nz, nt=nt, npad=pad, rate=rate)
    per = min(nx // 3, 40)
    # shots on shared receivers: with receivers of their own small grids run in clusters
    s = shots(s, [pad + 3, 4, nx + 2 * pad - 5][:ns], per, pad + 2, max(1, per // 2))
    call = lambda: V.synthetic_f(ctx, s.geom(), s.c11, s.c13, s.c33, s.wavelet,  # noqa: E731
                                 s.sloc, s.rloc, s.taper)
    a, b = both(ctx, call)
    assert np.abs(a).max() > 0
    assert np.array_equal(a, b)
    assert step_launches(ctx, call) == -(-(nt - 2) // T)


@pytest.mark.parametrize("nx,nz,pad,nt,rate,ns,T", [
    (20, 20, 10, 31, 2e-3, 1, 5), (57, 30, 12, 64, 3e-3, 2, 5), (40, 90, 9, 133, 2e-3, 1, 5),
    (101, 61, 15, 202, 4e-3, 2, 5), (401, 201, 30, 65, 2e-3, 2, 4), (801, 401, 30, 63, 3e-3, 1, 3),
    (801, 401, 30, 31, 1e-3, 1, 3)])
def test_tiled_gradient_and_migration_equal_per_level(ctx, nx, nz, pad, nt, rate, ns, T):
    s = S.survey2d(nx=nx, nz=nz, nt=nt, npad=pad, rate=rate)
    s = shots(s, [pad + nx // 2, pad + 4][:ns], nx // 3, pad + 1)
    g = s.geom()
    per = int(rate / s.dt + 0.5)
    data = np.random.default_rng(nt).standard_normal(
        ((nt - 1) // per + 1, s.rloc.shape[0])).astype(np.float32)
    call = lambda: V.objFuncGradient_f(ctx, g, data, s.c11, s.c13, s.c33, s.wavelet,  # noqa: E731
                                       s.sloc, s.rloc, s.taper)
    a, b = both(ctx, call)
    assert a[3] > 0 and a[3] == b[3]
    for x, y in zip(a[:3], b[:3]):
        assert np.abs(x).max() > 0
        assert np.array_equal(x, y)
    sweep = -(-(nt - 2) // T)
    assert step_launches(ctx, call) == ns * (2 * sweep + 1)  # and the last level's checkpoint
    call = lambda: V.rtm_f(ctx, g, data, s.c11, s.c13, s.c33, s.wavelet, s.sloc,  # noqa: E731
                           s.rloc, s.taper)
    a, b = both(ctx, call)
    assert np.abs(a).max() > 0
    assert np.array_equal(a, b)
    assert step_launches(ctx, call) == ns * 2 * sweep


@pytest.mark.parametrize("kind,room", [("synthetic", 60), ("gradient", 180), ("migration", 100)])
def test_calls_run_where_the_tiles_have_no_room(kind, room):
    """The tiles' padded arrays (131 x 91 cells in 192 x 136) need about twice the
    memory of the other paths: with `room` MB free the tiles do not fit and the
    call runs all the same. Levels kept: 250 MB padded, 114 MB not (gradient), 125 and
    57 MB (migration); 100 shots side by side 94 MB, one after another 2 MB."""
    import torch
    synth = kind == "synthetic"
    s = S.survey2d(nx=111, nz=71, nt=41 if synth else 1201, npad=10, rate=1e-3, ns=100 if synth else 1)
    a = (s.c11, s.c13, s.c33, s.wavelet, s.sloc, s.rloc, s.taper)
    small = V.Context(0)
    try:
        g = s.geom()
        data = np.random.default_rng(3).standard_normal(s.nt * (s.rloc.size // 2)).astype(np.float32)
        call = {"synthetic": lambda c: [V.synthetic_f(c, g, *a)],
                "gradient": lambda c: V.objFuncGradient_f(c, g, data, *a),
                "migration": lambda c: [V.rtm_f(c, g, data, *a)]}[kind]
        warm = V.Context(0)  # loads every kernel while there is room
        try:
            tiled = call(warm)
            warm.set_2d_resident(False)
            ref = call(warm)
        finally:
            warm.close()
        torch.cuda.empty_cache()
        torch.cuda.synchronize()
        hold = torch.empty(torch.cuda.mem_get_info()[0] - (room << 20), dtype=torch.uint8, device="cuda")
        try:
            out = call(small)
        finally:
            del hold
            torch.cuda.empty_cache()
        for x, y, t in zip(out, ref, tiled):
            assert np.abs(x).max() > 0
            assert rel_l2(x, y) < 1e-5 and rel_l2(t, y) < 1e-5
    finally:
        small.close()


def test_many_shots_on_shared_receivers(ctx):
    """1000 shots, each on 200 receivers of which the next shots record most again
    (the last one to record a receiver stands): several chunks of shots, traces equal
    to one shot after another, and device memory of a chunk, not of the 320 MB of all
    shots' traces beside it."""
    import torch
    s = S.survey2d(nx=220, nz=60, nt=400, npad=10, rate=1e-3)
    ns, nri = 1000, 200
    s.rloc = np.array([[10 + (7 * k) % 220, 11 + k // 220] for k in range(1100)], np.int32).reshape(-1)
    s.sloc = np.array([[14 + (5 * k) % 210, 12, nri, (37 * k) % 900] for k in range(ns)],
                      np.int32).reshape(-1)
    a = (s.geom(), s.c11, s.c13, s.c33, s.wavelet, s.sloc, s.rloc, s.taper)
    own = V.Context(0)
    try:
        V.synthetic_f(own, a[0], *a[1:5], s.sloc[:4], s.rloc, s.taper)  # loads the kernels
        before = torch.cuda.mem_get_info()[0]
        out = V.synthetic_f(own, *a)
        assert before - torch.cuda.mem_get_info()[0] < 300 << 20
    finally:
        own.close()
    ctx.set_2d_resident(False)
    try:
        ref = V.synthetic_f(ctx, *a)
    finally:
        ctx.set_2d_resident(True)
    assert np.abs(ref).max() > 0
    assert np.array_equal(out, ref)


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("nx,nz", [(57, 30), (60, 60)])
def test_nonfinite_samples_spread_as_per_level(ctx, value, nx, nz):
    """A NaN or infinite observed sample makes the same cells of gradient and image
    NaN as one launch per level does; the frame that no step updates stays zero."""
    s = S.survey2d(nx=nx, nz=nz, nt=62, npad=12, rate=2e-3)
    s = shots(s, [12 + nx // 2], nx // 3, nz + 14)  # receivers near the far side
    data = np.random.default_rng(2).standard_normal((31, nx // 3)).astype(np.float32)
    data[20, 5] = value
    nnx, nnz = nx + 24, nz + 24
    for call in (lambda: V.objFuncGradient_f(ctx, s.geom(), data, s.c11, s.c13, s.c33, s.wavelet,
                                             s.sloc, s.rloc, s.taper)[:3],
                 lambda: [V.rtm_f(ctx, s.geom(), data, s.c11, s.c13, s.c33, s.wavelet, s.sloc,
                                  s.rloc, s.taper)]):
        for x, y in zip(*both(ctx, call)):
            x, y = x.reshape(nnz, nnx), y.reshape(nnz, nnx)
            assert np.isnan(x).any() and np.isfinite(x).any()
            assert np.array_equal(np.isnan(x), np.isnan(y)) and np.array_equal(np.isinf(x), np.isinf(y))
            frame = np.ones((nnz, nnx), bool)
            frame[4:-4, 4:-4] = False
            assert not y[frame].any()


def test_calls_of_two_threads_on_one_context(ctx):
    """Gradients and migrations that two threads run on one context at the same time:
    only one of them has the context's scratch, the results are those of calls alone."""
    import threading
    rng = np.random.default_rng(6)
    calls = []
    for nx, nz, pad, nt in ((57, 30, 12, 301), (201, 101, 20, 201)):
        s = shots(S.survey2d(nx=nx, nz=nz, nt=nt, npad=pad, rate=2e-3), [pad + nx // 2], nx // 3,
                  pad + 1)
        data = rng.standard_normal(((nt - 1) // 2 + 1, nx // 3)).astype(np.float32)
        a = (s.c11, s.c13, s.c33, s.wavelet, s.sloc, s.rloc, s.taper)
        calls.append(lambda s=s, a=a, data=data: [*V.objFuncGradient_f(ctx, s.geom(), data, *a)[:3],
                                                  V.rtm_f(ctx, s.geom(), data, *a)])
    alone = [c() for c in calls]
    got = [[], []]

    def run(k):
        for _ in range(8):
            got[k].append(calls[k]())

    threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert len(got[k]) == 8
        for out in got[k]:
            for x, y in zip(out, alone[k]):
                assert np.abs(y).max() > 0 and np.array_equal(x, y)
