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
