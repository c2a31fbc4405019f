"""Calls around the register-tile and on-chip kernels that a program makes in
other ways than one shot in one thread with long run calls."""
import threading

import numpy as np
import pytest

import fdtd_2d_gb300 as F

pytestmark = pytest.mark.gpu

SWITCHES = ("FDTD2D_KERNEL", "FDTD2D_TMA", "FDTD2D_TMAT", "FDTD2D_TB", "FDTD2D_PERSIST", "FDTD2D_TILE", "FDTD2D_RESIDENT")


@pytest.fixture(autouse=True)
def _no_switches(monkeypatch):
    for v in SWITCHES:
        monkeypatch.delenv(v, raising=False)


def _point_shot(nx, ny, P, n_steps, **kw):
    return F.Problem.from_spec(nx=nx, ny=ny, npml=P, n_steps=n_steps, src_i=nx // 2, src_j=ny // 2, det_i=nx // 2 + 3,
                               det_j=ny // 2 + 1, **kw)


def _in_threads(*calls):
    """The calls' results, each from its own thread; an exception in one is raised here."""
    out, start = [None] * len(calls), threading.Barrier(len(calls))

    def go(k):
        start.wait()
        try:
            out[k] = calls[k]()
        except Exception as e:  # noqa: BLE001
            out[k] = e

    threads = [threading.Thread(target=go, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for r in out:
        if isinstance(r, Exception):
            raise r
    return out


def test_shots_in_two_threads(gpu):
    """Two shots whose tiles take different amounts of shared memory (CPMLs of 3
    and 120 cells), stepped by a thread each, a step a call: every call launches,
    the results are those of one thread."""
    n = 4000
    probs = [_point_shot(400, 400, P, n) for P in (3, 120)]

    def stepped(p):
        with F.Shot(p, gpu) as shot:
            for k in range(1, n + 1):
                shot.run(k, k)
            shot.synchronize()
            return [shot.read_field("ez"), shot.traces()["det_ez"], shot.dft()]

    alone = [stepped(p) for p in probs]
    for a, b in zip(alone, _in_threads(*[lambda p=p: stepped(p) for p in probs])):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)


def test_batches_in_two_threads(gpu):
    """The same with a batch in each thread."""
    n = 4000
    probs = [_point_shot(400, 400, P, n) for P in (3, 120)]

    def stepped(p):
        with F.Batch(gpu) as b:
            k = b.add(p)
            for _ in range(n):
                b.run(1)
            b.synchronize()
            return [b.shot(k).traces()["det_ez"], b.shot(k).dft()]

    alone = [stepped(p) for p in probs]
    for a, b in zip(alone, _in_threads(*[lambda p=p: stepped(p) for p in probs])):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
