"""Calls around the register-tile and on-chip kernels that a program makes in
other ways than one shot in one thread with long run calls."""
import threading

import numpy as np
import pytest

import fdtd_2d_gb300 as F
from helpers import FIELDS, PSI_FIELDS, load_state, random_state

pytestmark = pytest.mark.gpu

SWITCHES = ("FDTD2D_KERNEL", "FDTD2D_TMA", "FDTD2D_TMAT", "FDTD2D_TB", "FDTD2D_PERSIST", "FDTD2D_TILE", "FDTD2D_RESIDENT",
            "FDTD2D_ONE_STEP")


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


@pytest.mark.parametrize("nx,ny,P,store,ca", [
    (800, 90, 3, 0, 1.0), (1283, 333, 17, 0, 0.999), (900, 300, 120, 0, 1.0), (1024, 401, 32, 1, 1.0), (1411, 200, 5, 2, 0.998)])
def test_one_step_calls(gpu, monkeypatch, nx, ny, P, store, ca):
    """Run calls that leave a single step to the form for it, between passes of
    two to four steps after which the buffers have or have not traded places: the
    one-row kernel's bits in every field, psi array, trace and DFT sum."""
    chunks = (1, 4, 1, 1, 2, 1, 5, 3, 1, 9, 1)
    n = sum(chunks)
    prob = F.Problem.from_spec(nx=nx, ny=ny, npml=P, n_steps=n, profile=1, x_lo=nx // 3, x_hi=nx - 3, ne_peak=2e19, nu=3e9,
                               n_elem=6, src_i=nx // 2 - 300, src_j=ny // 2, src_di=97, src_dj=1, n_det=9, det_i=P + 4,
                               det_j=ny // 2 - 3, det_di=(nx - 2 * P) // 10, det_dj=1, storage=store, field_max=16.0)
    prob.setup.ca = prob.setup.da = ca
    st = random_state(None, nx, ny, P, np.random.default_rng(nx))

    def stepped(parts):
        with F.Shot(prob, gpu) as shot:
            load_state([shot], st)
            first = 1
            for c in parts:
                shot.run(first, first + c - 1)
                first += c
            out = {w: shot.read_field(w) for w in FIELDS + PSI_FIELDS}
            out["det"], out["dft"] = shot.traces()["det_ez"], shot.dft()
            shot.synchronize()
            return shot.kernel_name(), shot.launches(), out

    monkeypatch.setenv("FDTD2D_TILE", "7")
    monkeypatch.setenv("FDTD2D_ONE_STEP", "0")
    name, tiles, _ = stepped(chunks)
    monkeypatch.setenv("FDTD2D_ONE_STEP", "1")
    name, launches, got = stepped(chunks)
    assert name == "step_tmat_kernel<tile,7>", name
    assert launches == tiles + 8   # a second launch for each single step
    for v in ("FDTD2D_TILE", "FDTD2D_ONE_STEP"):
        monkeypatch.delenv(v)
    monkeypatch.setenv("FDTD2D_TMAT", "0")
    monkeypatch.setenv("FDTD2D_TMA", "4,3")
    monkeypatch.setenv("FDTD2D_PERSIST", "0")
    name, _, ref = stepped((n,))
    assert name == "step_tma_kernel<4,3>", name
    for k in ref:
        assert np.array_equal(ref[k], got[k]), k


@pytest.mark.parametrize("nx,ny", [(64, 40), (700, 300), (3100, 3000)])
def test_read_into_kept_new_and_odd_buffers(gpu, nx, ny):
    """A field read into new pages, pages that are there, some of each, and a buffer
    that starts inside a page: the same values, nothing outside the buffer touched."""
    import mmap

    prob = _point_shot(nx, ny, 8, 8)
    a = np.random.default_rng(nx).standard_normal((ny, nx)).astype(np.float32)
    n = a.nbytes
    with F.Shot(prob, gpu) as shot:
        shot.write_field("ez", a)
        assert np.array_equal(shot.read_field("ez"), a)
        for at in (0, 4, 4096 - 8, 70004):
            mem = mmap.mmap(-1, n + (1 << 18))
            buf = np.frombuffer(mem, np.uint8)
            got = buf[at:at + n].view(np.float32)
            for fill in (0, 3, 7):   # new pages, then present ones; at last every second MB of a new map
                if fill == 7:
                    del got, buf
                    mem = mmap.mmap(-1, n + (1 << 18))
                    buf = np.frombuffer(mem, np.uint8)
                    got = buf[at:at + n].view(np.float32)
                    for m in range(0, n, 2 << 20):
                        buf[at + m:at + min(m + (1 << 20), n)] = 7
                elif fill:
                    buf[:] = fill
                rc = F._lib().fdtd2d_read_field(shot._h, F.FIELD_EZ, got.ctypes.data_as(F._fp))
                assert rc == F.OK
                assert np.array_equal(got, a.ravel())
                out = 0 if fill == 7 else fill
                assert (buf[:at] == out).all() and (buf[at + n:] == out).all()
            del got, buf


def _tracker_shot(n_steps, lines):
    """A 500 x 300 shot with so many tracker lines, its scan columns beside its maximum columns."""
    prob = _point_shot(500, 300, 10, n_steps)
    s = prob.setup
    scan = np.arange(100, 100 + 7 * lines, 7, dtype=np.int32)
    most = scan + np.int32(3)
    prob.keep = (scan, most)
    s.n_rc, s.rc_level, s.rc_j_cut, s.rc_edge0 = lines, 0.07, 40, 1e-3
    if lines:
        s.rc_scan_i, s.rc_max_i = (a.ctypes.data_as(type(s.rc_scan_i)) for a in (scan, most))
    return prob


@pytest.mark.parametrize("n_steps", [10, 400])
def test_tracker_memory_is_counted(gpu, n_steps):
    """device_bytes counts the columns a tracker shot keeps, which are no more than
    its steps need."""
    from test_failure_gpu import _pool_used_bytes

    held, said = [], []
    for lines in (0, 12):
        prob = _tracker_shot(n_steps, lines)
        base = _pool_used_bytes(gpu)
        if base is None:
            pytest.skip("no CUDA runtime library to ask")
        with F.Shot(prob, gpu) as shot:
            assert shot.kernel_name().startswith("step_persist_kernel<0>/tile<")
            held.append(_pool_used_bytes(gpu) - base)
            said.append(prob.device_bytes())
    history = min(n_steps, 256) * 24 * 320 * 4
    assert history <= held[1] - held[0] <= history + 100_000
    assert 0 <= said[1] - said[0] - (held[1] - held[0]) + 8192 <= 100_000   # (allocations are rounded up to 512 B each)


def test_tracker_allocation_failures(gpu, monkeypatch):
    """Every allocation of a tracker shot fails in turn: out of memory, or the same
    rows on a path that needs less."""
    prob = _tracker_shot(60, 12)
    st = random_state(None, 500, 300, 10, np.random.default_rng(1))

    def stepped():
        with F.Shot(prob, gpu) as shot:
            load_state([shot], st)
            shot.run(1, 60)
            return [shot.rc(), shot.traces()["det_ez"], shot.read_field("ez")], shot.kernel_name()

    ref, name = stepped()
    assert name.startswith("step_persist_kernel<0>/tile<") and ref[0].max() > 0
    names, in_a_row = set(), 0
    for k in range(1, 200):
        monkeypatch.setenv("FDTD2D_TEST_FAIL_ALLOC", str(k))
        try:
            got, name = stepped()
        except F.FdtdError as e:
            assert e.status == F.ERR_NOMEM, (k, e)
            in_a_row = 0
            continue
        for a, b in zip(ref, got):
            assert np.array_equal(a, b), (k, name)
        names.add(name)
        in_a_row = in_a_row + 1 if name.startswith("step_persist_kernel<0>/tile<") else 0
        if in_a_row == 3:
            break
    assert in_a_row == 3
    assert any(not n.startswith("step_persist_kernel<0>/tile<") for n in names), names


def _outputs(gpu, prob, st, chunks):
    with F.Shot(prob, gpu) as shot:
        load_state([shot], st)
        first = 1
        for c in chunks:
            shot.run(first, first + c - 1)
            first += c
        out = {w: shot.read_field(w) for w in FIELDS + PSI_FIELDS}
        out["det"], out["dft"] = shot.traces()["det_ez"], shot.dft()
        if prob.setup.n_rc:
            out["rc"] = shot.rc()
        shot.synchronize()
        return shot.kernel_name(), out


def _same(ref, got):
    for k in ref:
        assert np.array_equal(ref[k], got[k], equal_nan=np.asarray(ref[k]).dtype.kind in "fc"), k


FORMS = [("FDTD2D_TILE", "7"), ("FDTD2D_TILE", "5"), ("FDTD2D_RESIDENT", "2"), ("FDTD2D_RESIDENT", "4"), ("FDTD2D_RESIDENT", "6"),
         ("FDTD2D_RESIDENT", "8")]


@pytest.mark.parametrize("form", FORMS, ids=lambda f: f[0][7:] + f[1])
@pytest.mark.parametrize("nx,ny,P,store,ca", [(700, 300, 9, 0, 1.0), (700, 300, 9, 0, 0.999), (500, 223, 21, 1, 1.0), (390, 180, 4, 2, 0.998)])
def test_denominators_that_vary(gpu, monkeypatch, form, nx, ny, P, store, ca):
    """Curl denominators that vary outside the CPML too: no plain tile, every warp in
    the form with tables, tiles without a strip lane.  The one-row kernel's bits."""
    if form == ("FDTD2D_RESIDENT", "8") and store:
        pytest.skip("16-bit fields take at most 6 rows")
    chunks = (1, 4, 3, 8, 2, 9)
    n = sum(chunks)
    prob = F.Problem.from_spec(nx=nx, ny=ny, npml=P, n_steps=n, profile=1, x_lo=nx // 3, x_hi=nx - 3, ne_peak=2e19, nu=3e9,
                               n_elem=5, src_i=nx // 2 - 6, src_j=ny // 2, src_di=3, src_dj=1, n_det=6, det_i=nx // 2 - 8,
                               det_j=ny // 2 - 2, det_di=2, det_dj=1, storage=store, field_max=16.0)
    s = prob.setup
    s.ca = s.da = ca
    rng = np.random.default_rng(nx)
    for name, m in (("den_ex", nx - 1), ("den_hx", nx - 1), ("den_ey", ny - 1), ("den_hy", ny - 1)):
        a = np.ctypeslib.as_array(getattr(s, name), (m,))
        a *= rng.uniform(0.8, 1.0, m).astype(np.float32)
    st = random_state(None, nx, ny, P, rng)
    monkeypatch.setenv(*form)
    name, got = _outputs(gpu, prob, st, chunks)
    assert name.endswith("%s>" % form[1]) and "tile" in name, name
    monkeypatch.delenv(form[0])
    monkeypatch.setenv("FDTD2D_TMAT", "0")
    monkeypatch.setenv("FDTD2D_TMA", "4,3")
    monkeypatch.setenv("FDTD2D_PERSIST", "0")
    name, ref = _outputs(gpu, prob, st, (n,))
    assert name == "step_tma_kernel<4,3>", name
    _same(ref, got)


@pytest.mark.parametrize("form", FORMS, ids=lambda f: f[0][7:] + f[1])
@pytest.mark.parametrize("store,ca,lines", [(0, 1.0, 0), (0, 0.999, 12), (1, 1.0, 0), (2, 0.999, 0)])
def test_special_values(gpu, monkeypatch, form, store, ca, lines):
    """NaN, infinities, values near both ends of the range and signed zeros in the
    fields and in psi, with the tracker reading some: they spread as in the kernels of
    one step (FP32: the streaming one, which runs the tracker; 16-bit: the one-row one)."""
    if form == ("FDTD2D_RESIDENT", "8") and store:
        pytest.skip("16-bit fields take at most 6 rows")
    chunks = (1, 4, 3, 8, 2, 12)
    n = sum(chunks)
    nx, ny, P = 500, 300, 10
    prob = _tracker_shot(n, lines) if lines else _point_shot(nx, ny, P, n, storage=store, field_max=16.0, profile=1, x_lo=200, x_hi=490,
                                                             ne_peak=2e19)
    prob.setup.ca = prob.setup.da = ca
    rng = np.random.default_rng(7)
    st = random_state(None, nx, ny, P, rng)
    for w in FIELDS + PSI_FIELDS:
        flat = st[w].reshape(-1)
        at = rng.choice(flat.size, 12, replace=False)
        flat[at] = np.array([np.nan, np.inf, -np.inf, 3e38, -3e38, 1e-40, -1e-40, 0.0, -0.0, 1e-38, 6e4, -6e4], np.float32)
    monkeypatch.setenv(*form)
    name, got = _outputs(gpu, prob, st, chunks)
    assert name.endswith("%s>" % form[1]) and "tile" in name, name
    monkeypatch.delenv(form[0])
    monkeypatch.setenv("FDTD2D_PERSIST", "0")
    monkeypatch.setenv("FDTD2D_TMAT", "0")
    monkeypatch.setenv(*(("FDTD2D_KERNEL", "stream") if store == 0 else ("FDTD2D_TMA", "4,3")))
    name, ref = _outputs(gpu, prob, st, (n,))
    assert name == ("step_stream_kernel<0>" if store == 0 else "step_tma_kernel<4,3>"), name
    assert not np.isfinite(ref[F.FIELD_EZ]).all() and np.isfinite(ref[F.FIELD_EZ]).any()
    if lines:
        assert ref["rc"].max() > 0
    _same(ref, got)


def test_production_shot_on_tiles(gpu, monkeypatch):
    """The 8192^2 production shot from a random state on the path it takes by default
    (register tiles, a single step on the tensor kernel among them): the bits of the
    two-step path, which the production tests hold against the FP64 oracle."""
    chunks = (9, 1, 12)
    n = sum(chunks)
    prob = F.Problem.from_spec(F.production_spec(n_steps=n))
    st = {}
    rng = np.random.default_rng(5)
    for w in FIELDS + PSI_FIELDS:
        a = rng.standard_normal(F.field_shape(w, prob.nx, prob.ny, prob.setup.npml), dtype=np.float32)
        st[w] = a * np.float32({F.FIELD_HX: 1 / 377.0, F.FIELD_HY: 1 / 377.0}.get(w, 1.0 if w in FIELDS else 1e-3))
    name, got = _outputs(gpu, prob, st, chunks)
    assert name.startswith("step_tmat_kernel<tile,"), name
    monkeypatch.setenv("FDTD2D_TB", "1")
    name, ref = _outputs(gpu, prob, st, (n,))
    assert name.startswith("step_tmat2_kernel<"), name
    _same(ref, got)


@pytest.mark.parametrize("store", [F.STORE_F32, F.STORE_F16, F.STORE_BF16])
@pytest.mark.parametrize("lines,probe", [(12, None), (0, 150), (12, 299)])
def test_tracker_and_probe_of_every_storage(gpu, store, lines, probe):
    """Tracker rows and probe samples against the ones formed from the fields read
    after every step, in each storage type (one probe on the grid's last row)."""
    n = 40
    prob = _tracker_shot(n, lines)
    s = prob.setup
    s.storage, s.field_max = store, 16.0
    if probe is not None:
        s.line_n, s.line_i0, s.line_j, s.line_first, s.line_last = 300, 50, probe, 11, 31
    st = random_state(None, 500, 300, 10, np.random.default_rng(1))
    with F.Shot(prob, gpu) as shot:
        load_state([shot], st)
        for a, b in ((1, 9), (10, 12), (13, n)):
            shot.run(a, b)
        rows = shot.rc() if lines else None
        line = shot.line(11, 31) if probe is not None else None
        ez = shot.read_field("ez")
    want_rows, want_line = [], []
    with F.Shot(prob, gpu) as shot:
        load_state([shot], st)
        edge = np.full(lines, s.rc_edge0, np.float32)
        for k in range(1, n + 1):
            shot.run(k, k)
            e = shot.read_field("ez")
            if 11 <= k <= 31 and probe is not None:
                want_line.append(e[probe, 50:350])
            if lines:
                scan, most = prob.keep
                top = np.maximum(e[0, most], e[s.rc_j_cut:298, most].max(axis=0))
                edge = np.maximum(edge, top * np.float32(s.rc_level))
                hit = ~(np.abs(e[1:298, scan]) < edge)
                want_rows.append(np.where(hit, np.arange(1, 298)[:, None], 0).max(axis=0))
    assert np.array_equal(ez, e)
    if lines:
        assert np.array_equal(rows, np.array(want_rows)) and rows.max() > 0
    if probe is not None:
        assert np.array_equal(line, np.array(want_line)) and np.abs(line).max() > 0


@pytest.mark.parametrize("form", [("FDTD2D_TILE", "7"), ("FDTD2D_TILE", "5"), ("FDTD2D_RESIDENT", "4")], ids=lambda f: f[0][7:] + f[1])
@pytest.mark.parametrize("store", [0, 1, 2])
@pytest.mark.parametrize("kind", ["rows", "block", "cell", "spread", "strips"])
def test_many_points(gpu, monkeypatch, form, store, kind):
    """More points than lanes in a warp's rows: lines of sources and detectors along x, a
    block of detectors, many sources and detectors in one cell (subtracted in their
    order), points all over the grid, points in the CPML; component detectors beside
    them.  The one-row kernel's bits."""
    chunks = (1, 4, 3, 8)
    n, nx, ny, P = sum(chunks), 420, 300, 12
    prob = _point_shot(nx, ny, P, n, storage=store, field_max=16.0, profile=1, x_lo=200, x_hi=400, ne_peak=2e19, n_elem=90)
    s = prob.setup
    rng = np.random.default_rng(9)
    at = {"rows": lambda q: (30 + 4 * q % 360, 150 + q % 2), "block": lambda q: (200 + q % 13, 140 + q // 13),
          "cell": lambda q: (211, 150), "spread": lambda q: (int(rng.integers(1, nx - 1)), int(rng.integers(1, ny - 1))),
          "strips": lambda q: (1 + q % (P + 3), 1 + q // (P + 3))}[kind]

    def points(count):
        a = (type(s.det[0]) * count)()
        for q in range(count):
            a[q].i, a[q].j = at(q)
        return a

    prob.keep = src, det, comp = points(s.n_src), points(230), points(70)
    s.src, s.det, s.comp, s.n_det, s.n_comp = src, det, comp, len(det), len(comp)
    phase = np.ctypeslib.as_array(s.src_phase_deg, (s.n_src,))
    phase += rng.uniform(0, 360, s.n_src)   # sources of different values, so that their order shows
    st = random_state(None, nx, ny, P, rng)

    def stepped(parts):
        name, out = _outputs(gpu, prob, st, parts)
        return name, out

    def all_traces(parts):
        with F.Shot(prob, gpu) as shot:
            load_state([shot], st)
            first = 1
            for c in parts:
                shot.run(first, first + c - 1)
                first += c
            return shot.traces()

    monkeypatch.setenv(*form)
    name, got = stepped(chunks)
    got.update(all_traces(chunks))
    assert "tile" in name, name
    monkeypatch.delenv(form[0])
    monkeypatch.setenv("FDTD2D_TMAT", "0")
    monkeypatch.setenv("FDTD2D_TMA", "4,3")
    monkeypatch.setenv("FDTD2D_PERSIST", "0")
    name, ref = stepped((n,))
    ref.update(all_traces((n,)))
    assert name == "step_tma_kernel<4,3>", name
    _same(ref, got)


def test_varying_denominators_step_by_step(gpu, monkeypatch):
    """A 16-bit shot with varying denominators goes a step at a time where single
    steps have a form of their own; in passes elsewhere.  The same bits."""
    nx, ny, P, n = 1100, 300, 9, 22
    prob = _point_shot(nx, ny, P, n, storage=F.STORE_F16, field_max=16.0)
    a = np.ctypeslib.as_array(prob.setup.den_ey, (ny - 1,))
    a *= np.random.default_rng(3).uniform(0.8, 1.0, ny - 1).astype(np.float32)
    st = random_state(None, nx, ny, P, np.random.default_rng(2))
    monkeypatch.setenv("FDTD2D_TILE", "5")
    out = []
    for one in ("0", "1"):
        monkeypatch.setenv("FDTD2D_ONE_STEP", one)
        out.append(_outputs(gpu, prob, st, (1, 13, 8))[1])
        with F.Shot(prob, gpu) as shot:
            before = shot.launches()
            shot.run(1, 8)
            assert shot.launches() - before == (16 if one == "1" else 2)   # two launches a step, one per pass of four
    _same(*out)


@pytest.mark.parametrize("one", ["0", "1"])
def test_single_steps_of_a_tracker_shot(gpu, monkeypatch, one):
    """Run calls of one step, whose tracker rows and probe samples come from the fields,
    between longer ones, whose history the passes keep; on the tiles and on the form
    for single steps.  The streaming kernel's rows, samples and fields."""
    nx, ny, P, n = 900, 300, 10, 60
    prob = _point_shot(nx, ny, P, n)
    s = prob.setup
    scan = np.arange(100, 100 + 37 * 20, 37, dtype=np.int32)
    prob.keep = scan, scan[::-1].copy()
    s.n_rc, s.rc_level, s.rc_j_cut, s.rc_edge0 = 20, 0.07, 40, 1e-3
    s.rc_scan_i, s.rc_max_i = (a.ctypes.data_as(type(s.rc_scan_i)) for a in prob.keep)
    s.line_n, s.line_i0, s.line_j, s.line_first, s.line_last = 500, 50, 140, 3, 40
    st = random_state(None, nx, ny, P, np.random.default_rng(4))

    def stepped(chunks):
        with F.Shot(prob, gpu) as shot:
            load_state([shot], st)
            first = 1
            for c in chunks:
                shot.run(first, first + c - 1)
                first += c
            out = {w: shot.read_field(w) for w in FIELDS + PSI_FIELDS}
            out["rc"], out["line"], out["det"] = shot.rc(), shot.line(3, 40), shot.traces()["det_ez"]
            return shot.kernel_name(), out

    monkeypatch.setenv("FDTD2D_TILE", "7")
    monkeypatch.setenv("FDTD2D_ONE_STEP", one)
    name, got = stepped((1, 1, 1, 4, 1, 9, 1, 20, 1, 1, 17, 3))
    assert name == "step_tmat_kernel<tile,7>", name
    monkeypatch.delenv("FDTD2D_TILE")
    monkeypatch.setenv("FDTD2D_KERNEL", "stream")
    monkeypatch.setenv("FDTD2D_PERSIST", "0")
    name, ref = stepped((n,))
    assert name == "step_stream_kernel<0>", name
    assert ref["rc"].max() > 0
    _same(ref, got)


@pytest.mark.parametrize("rows", ["7", "5"])
@pytest.mark.parametrize("lines,ca", [(0, 1.0), (0, 0.999), (12, 1.0), (12, 0.998)])
def test_few_points(gpu, monkeypatch, rows, lines, ca):
    """A source, a detector and a component detector every 16 rows, in plain tiles, on
    their borders and in the CPML: the kernel for few points gives the streaming one's
    bits, with the tracker and without."""
    chunks = (1, 4, 3, 8)
    n, nx, ny, P = sum(chunks), 500, 300, 10
    prob = _tracker_shot(n, lines)
    s = prob.setup
    s.ca = s.da = ca
    count = 18

    def points(i0):
        a = (type(s.det[0]) * count)()
        for q in range(count):
            a[q].i, a[q].j = (i0 + 27 * q) % (nx - 2) + 1, 3 + 16 * q
        return a

    src = points(60)
    phase, prob.keep2 = np.random.default_rng(1).uniform(0, 360, count), [src]
    s.src, s.n_src, s.src_phase_deg = src, count, phase.ctypes.data_as(type(s.src_phase_deg))
    s.det, s.n_det = prob.keep2.append(points(60)) or prob.keep2[-1], count
    s.comp, s.n_comp = prob.keep2.append(points(61)) or prob.keep2[-1], count
    st = random_state(None, nx, ny, P, np.random.default_rng(3))

    def stepped(parts):
        with F.Shot(prob, gpu) as shot:
            load_state([shot], st)
            first = 1
            for c in parts:
                shot.run(first, first + c - 1)
                first += c
            out = {w: shot.read_field(w) for w in FIELDS + PSI_FIELDS}
            out.update(shot.traces())
            out["dft"] = shot.dft()
            if lines:
                out["rc"] = shot.rc()
            return shot.kernel_name(), out

    monkeypatch.setenv("FDTD2D_TILE", rows)
    name, got = stepped(chunks)
    assert name == f"step_tmat_kernel<tile,{rows}>", name
    monkeypatch.delenv("FDTD2D_TILE")
    monkeypatch.setenv("FDTD2D_KERNEL", "stream")
    monkeypatch.setenv("FDTD2D_PERSIST", "0")
    name, ref = stepped((n,))
    assert name == "step_stream_kernel<0>", name
    _same(ref, got)


def test_few_points_f16_large(gpu, monkeypatch):
    """The F16 kernel for few points, which the largest grids take: the one-row
    kernel's bits."""
    nx, ny, n = 8000, 5010, 9
    prob = _point_shot(nx, ny, 20, n, storage=F.STORE_F16, field_max=16.0, profile=1, x_lo=nx // 2, x_hi=nx - 20, ne_peak=2e19)
    rng = np.random.default_rng(6)
    st = {w: rng.standard_normal(F.field_shape(w, nx, ny, 20), dtype=np.float32) for w in FIELDS}
    st[F.FIELD_HX] /= np.float32(377)
    st[F.FIELD_HY] /= np.float32(377)
    monkeypatch.setenv("FDTD2D_TILE", "7")
    name, got = _outputs(gpu, prob, st, (4, 2, 3))
    assert name == "step_tmat_kernel<tile,7>", name
    monkeypatch.delenv("FDTD2D_TILE")
    monkeypatch.setenv("FDTD2D_TMAT", "0")
    monkeypatch.setenv("FDTD2D_TMA", "4,3")
    name, ref = _outputs(gpu, prob, st, (n,))
    assert name == "step_tma_kernel<4,3>", name
    _same(ref, got)
