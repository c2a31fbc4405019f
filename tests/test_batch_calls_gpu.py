"""Admission to a batch and to the serving loop: what a member is charged, and what
is left when an admission fails."""
import pytest

import fdtd_2d_gb300 as F

pytestmark = pytest.mark.gpu

SWITCHES = ("FDTD2D_KERNEL", "FDTD2D_TMA", "FDTD2D_TMAT", "FDTD2D_TB", "FDTD2D_PERSIST", "FDTD2D_TILE", "FDTD2D_RESIDENT",
            "FDTD2D_BATCH_SOLO_CELLS")


@pytest.fixture(autouse=True)
def _no_switches(monkeypatch):
    for v in SWITCHES:
        monkeypatch.delenv(v, raising=False)


def _shot(nx, ny, **kw):
    return F.Problem.from_spec(nx=nx, ny=ny, npml=12, n_steps=24, src_i=nx // 2, src_j=ny // 2, det_i=nx // 2 + 3, det_j=ny // 2, **kw)


@pytest.mark.parametrize("nx,ny,store", [(300, 200, F.STORE_F16), (300, 200, F.STORE_BF16), (1500, 1450, F.STORE_F32)])
def test_solo_member_needs_what_it_holds(gpu, monkeypatch, nx, ny, store):
    """A solo member is admitted under a budget of its device bytes; where a variable
    selects the paths with two more field buffers, their room is asked for too."""
    p = _shot(nx, ny, storage=store, field_max=16.0)
    with F.Batch(gpu, budget_bytes=p.device_bytes()) as b:
        i = b.add(p)
        assert i is not None and b.free_bytes() == 0
        assert b.shot(i).kernel_name().startswith("step_tmat_kernel<tile,")   # its own kernels: a solo member
        b.run(24)
        b.synchronize()
        assert b.finished(i)
    with F.Server(gpu, budget_bytes=p.device_bytes()) as srv:
        srv.submit(p, 5)
        got = None
        while got is None:
            srv.step()
            got = srv.pop()
        assert got["tag"] == 5
    monkeypatch.setenv("FDTD2D_TILE", "0")
    with F.Batch(gpu, budget_bytes=p.device_bytes()) as b:
        if store != F.STORE_F32:
            assert b.add(p) is None
        else:
            assert b.shot(b.add(p)).kernel_name() == ""   # on the batch's kernel instead
    if store != F.STORE_F32:
        with F.Server(gpu, budget_bytes=p.device_bytes()) as srv:
            with pytest.raises(F.FdtdError) as e:
                srv.submit(p, 6)
            assert e.value.status == F.ERR_BUDGET


def test_add_that_fails_leaves_no_member(gpu, monkeypatch):
    """Every allocation of an add fails in turn (its tile list the last of them): out
    of memory, nothing charged, no member left that later passes would step; the
    members before and after it give a single shot's results."""
    import numpy as np

    probs = [_shot(300, 200), _shot(260, 220)]
    alone = []
    for p in probs:
        with F.Shot(p, gpu) as shot:
            shot.run(1, 24)
            alone.append((shot.traces()["det_ez"], shot.dft()))
    failed = 0
    with F.Batch(gpu) as b:
        first = b.add(probs[0])
        b.run(3)
        free = b.free_bytes()
        for k in range(1, 200):
            monkeypatch.setenv("FDTD2D_TEST_FAIL_ALLOC", str(k))
            try:
                i = b.add(probs[1])
            except F.FdtdError as e:
                assert e.status == F.ERR_NOMEM, (k, e)
                assert b.free_bytes() == free, k
                failed = k
                continue
            b.remove(i)
            break
        monkeypatch.delenv("FDTD2D_TEST_FAIL_ALLOC")
        assert failed == k - 1 >= 8
        second = b.add(probs[1])
        assert second == first + 1          # the slot of the failed ones
        b.run(24)
        b.synchronize()
        for i, (tr, dft) in zip((first, second), alone):
            assert b.finished(i)
            assert np.array_equal(b.shot(i).traces()["det_ez"], tr) and np.array_equal(b.shot(i).dft(), dft)


def test_batch_of_lossy_and_lossless_shots(gpu):
    """Members of lossy and lossless media and of different lengths, one with
    denominators that vary everywhere, so that the passes' kernel changes as members end
    and join: a single shot's bits."""
    import numpy as np

    probs = []
    for k, (nx, ny, n, ca) in enumerate([(300, 200, 37, 1.0), (410, 260, 22, 0.998), (260, 333, 50, 1.0), (390, 180, 64, 0.999)]):
        p = F.Problem.from_spec(nx=nx, ny=ny, npml=8 + k, n_steps=n, profile=1, x_lo=nx // 2, x_hi=nx - 8, ne_peak=2e19,
                                src_i=nx // 2, src_j=ny // 2, det_i=nx // 2 + 3, det_j=ny // 2)
        p.setup.ca = p.setup.da = ca
        if k == 2:
            a = np.ctypeslib.as_array(p.setup.den_ey, (ny - 1,))
            a *= np.random.default_rng(3).uniform(0.8, 1.0, ny - 1).astype(np.float32)
        probs.append(p)
    fields = ("ez", "hx", "hy", "jz")

    def outputs(shot):
        return [shot.traces()["det_ez"], shot.dft()] + [shot.read_field(f) for f in fields]

    alone = []
    for p in probs:
        with F.Shot(p, gpu) as shot:
            shot.run(1, p.n_steps)
            alone.append(outputs(shot))
    with F.Batch(gpu) as b:
        ids = [b.add(p) for p in probs[:3]]
        b.run(13)
        ids.append(b.add(probs[3]))
        for k in (1, 6, 10, 3, 44):
            b.run(k)
        b.synchronize()
        for i, ref in zip(ids, alone):
            assert b.finished(i)
            for x, y in zip(outputs(b.shot(i)), ref):
                assert np.array_equal(x, y)
