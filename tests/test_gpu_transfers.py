"""Host arrays of pitched volumes (staged, packed and unpacked on the device,
pages populated beforehand) against device arrays of the same calls, and the
offset gathers summed eight levels at a time: equal bit for bit."""
import numpy as np
import pytest

import vtib200 as V
import vtib200.synth as S

pytestmark = pytest.mark.gpu


# below the staging limit; rows of one pitch; several planes; more than one
# 32 MB block, with an output of more than 4 MB
@pytest.mark.parametrize("nx,ny,nz", [(25, 21, 20), (64, 30, 24), (70, 41, 33), (250, 200, 190)])
def test_host_and_device_arrays_agree(ctx, nx, ny, nz):
    import torch
    s = S.small3d(nx=nx, ny=ny, nz=nz, nt=12, npad=5, rate=2.1e-3)
    n = s.nxyz
    c = s.cij().reshape(3, n)
    dobs = np.zeros(V.nnt3d(s.geom()) * (s.recloc.size // 4), dtype=np.float32)
    res = []
    for mem in (V.MEM_HOST, V.MEM_DEVICE):
        plan = V.Plan3d(ctx, s.geom(), V.OPT_FULL_STEPS)
        plan.set_wavelet(s.wavelet)
        plan.set_receivers(s.recloc)
        if mem == V.MEM_HOST:
            plan.set_model(*c)
            out = np.full(2 + 3 * n, np.nan, dtype=np.float32)[1:]  # not page aligned
            plan.gradient(s.souloc, [0], dobs, V.MEM_HOST, out, V.MEM_HOST)
            fresh = plan.gradient(s.souloc, [0], dobs)[0]
            assert np.array_equal(out, fresh)
        else:
            dc = [torch.tensor(k, device="cuda") for k in c]
            dd, fg = torch.tensor(dobs, device="cuda"), torch.zeros(1 + 3 * n, device="cuda")
            torch.cuda.synchronize()
            plan.set_model(*[k.data_ptr() for k in dc], mem=V.MEM_DEVICE)
            plan.gradient(s.souloc, [0], dd.data_ptr(), V.MEM_DEVICE, fg.data_ptr(), V.MEM_DEVICE)
            out = fg.cpu().numpy()
        res.append(out)
        plan.close()
    assert np.abs(res[0][1:]).max() > 0
    assert np.array_equal(res[0], res[1])


# 6 to 16 backward levels: fewer than, exactly and just over the eight summed at
# a time; lag ranges that are not a multiple of four; odd row lengths
@pytest.mark.parametrize("nt,nx", [(8, 40), (10, 41), (11, 47), (18, 38)])
def test_gathers_do_not_depend_on_the_lag_range(ctx, nt, nx):
    s = S.small3d(nx=nx, ny=24, nz=22, nt=nt, npad=5, rate=2.1e-3)
    plan = V.Plan3d(ctx, s.geom(), V.OPT_FULL_STEPS)
    plan.set_model(*s.cij().reshape(3, s.nxyz))
    plan.set_wavelet(s.wavelet)
    plan.set_receivers(s.recloc)
    data = np.random.default_rng(1).standard_normal(
        V.nnt3d(s.geom()) * (s.recloc.size // 4)).astype(np.float32)
    im = plan.rtm(s.souloc, [0], data).reshape(22, 24, nx)
    ref = plan.odcig(s.souloc, [0], data, 13).reshape(27, 22, 24, nx)
    assert np.abs(ref).max() > 0
    for nlag in (0, 1, 3, 4, 6):
        g = plan.odcig(s.souloc, [0], data, nlag).reshape(2 * nlag + 1, 22, 24, nx)
        assert np.array_equal(g[:, :, :, 13:nx - 13], ref[13 - nlag:14 + nlag, :, :, 13:nx - 13])
        lo = max(4, nlag)
        assert np.array_equal(g[nlag][:, :, lo:nx - lo], im[:, :, lo:nx - lo])
        assert not g[:, :, :, :lo].any() and not g[:, :, :, nx - lo:].any()
    plan.close()


@pytest.mark.parametrize("nt", [5, 40])
def test_product_with_blocks_longer_than_the_record(ctx, nt):
    """Checkpoint blocks longer than the record hold only its levels: one block
    either way, the same sums."""
    s = S.small3d(nx=40, ny=36, nz=32, nt=nt, npad=8, rate=2.1e-3)
    n = s.nxyz
    c = s.cij()
    dc = (0.02 * c).astype(np.float32)
    dobs = np.zeros(V.nnt3d(s.geom()) * (s.recloc.size // 4), dtype=np.float32)
    out = [V.gnhv_exact(ctx, s.geom(), *c.reshape(3, n), s.wavelet, s.souloc, s.recloc, dc=dc,
                        dobs=dobs, checkpoint_every=k) for k in (nt, 64, 500)]
    assert nt == 5 or np.abs(out[0]["hv"]).max() > 0  # nothing has reached a receiver by then
    for o in out[1:]:
        for k in ("hv", "grad", "traces", "born"):
            assert np.array_equal(o[k], out[0][k]), k


def test_transfers_of_two_threads_on_one_context(ctx):
    """Two threads set models and fetch gradients of their own plans on one context:
    the staging block carries one piece at a time."""
    import threading
    plans, models = [], []
    for k, (nx, ny, nz) in enumerate(((70, 121, 93), (90, 110, 105))):
        s = S.small3d(nx=nx, ny=ny, nz=nz, nt=12, npad=5, rate=2.1e-3, seed=3 + k)
        p = V.Plan3d(ctx, s.geom(), V.OPT_FULL_STEPS)
        p.set_wavelet(s.wavelet)
        p.set_receivers(s.recloc)
        dobs = np.random.default_rng(k).standard_normal(
            V.nnt3d(s.geom()) * (s.recloc.size // 4)).astype(np.float32)
        plans.append(p)
        models.append((s.cij().reshape(3, s.nxyz), s.souloc, dobs))

    def call(k):
        c, sou, dobs = models[k]
        plans[k].set_model(*c)
        return plans[k].gradient(sou, [0], dobs)[0]

    alone = [call(0), call(1)]
    got = [[], []]
    threads = [threading.Thread(target=lambda k=k: got[k].extend(call(k) for _ in range(40)))
               for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for p in plans:
        p.close()
    for k in range(2):
        assert len(got[k]) == 40 and np.abs(alone[k][1:]).max() > 0
        for g in got[k]:
            assert np.array_equal(g, alone[k])
