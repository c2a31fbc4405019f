"""The register-tile kernel (several time steps per pass, csrc/step_tile.cu)
against the one-row kernel: the same bits in every field, psi array, trace and
DFT sum.  Grids: no plain tile at all, exactly one, widths and heights around
whole tiles, CPMLs of 2 to 40 cells, no plasma, lossy media; points on tile
edges; run calls of 1 to 32 steps (odd and even, so the buffers trade places)."""
import numpy as np
import pytest

import fdtd_2d_gb300 as F
from helpers import FIELDS, PSI_FIELDS, load_state, random_state

pytestmark = pytest.mark.gpu

CHUNKS = (1, 4, 2, 11, 3, 8, 32)
STEPS = sum(CHUNKS)


def _stepped(gpu, prob, st, chunks):
    with F.Shot(prob, gpu) as shot:
        name = shot.kernel_name()
        load_state([shot], st)
        n = 1
        for c in chunks:
            shot.run(n, n + c - 1)
            n += c
        out = {w: shot.read_field(w) for w in FIELDS + PSI_FIELDS}
        out["det"] = shot.traces()["det_ez"]
        out["dft"] = shot.dft()
        shot.synchronize()
    return name, out


def _one_row(gpu, monkeypatch, prob, st, steps):
    """The one-row kernel's results."""
    for v in ("FDTD2D_TILE", "FDTD2D_RESIDENT"):
        monkeypatch.delenv(v, raising=False)
    monkeypatch.setenv("FDTD2D_TMAT", "0")
    monkeypatch.setenv("FDTD2D_TMA", "4,3")
    monkeypatch.setenv("FDTD2D_PERSIST", "0")
    name, ref = _stepped(gpu, prob, st, (steps,))
    assert name == "step_tma_kernel<4,3>", name
    return ref


@pytest.mark.parametrize("rows", ["7", "5"])
@pytest.mark.parametrize("nx,ny,P,store,profile,ca", [
    (40, 40, 2, 0, 1, 1.0), (120, 25, 3, 0, 1, 1.0), (121, 24, 4, 0, 0, 1.0), (203, 157, 7, 0, 1, 0.999),
    (371, 75, 3, 0, 1, 1.0), (372, 76, 3, 0, 3, 1.0), (1100, 90, 9, 0, 1, 1.0), (500, 400, 40, 0, 1, 1.0),
    (777, 601, 17, 0, 3, 0.998), (640, 330, 24, 1, 1, 1.0), (333, 257, 16, 2, 1, 0.999), (900, 700, 32, 1, 3, 1.0)])
def test_tile_equals_one_row(gpu, monkeypatch, rows, nx, ny, P, store, profile, ca):
    for v in ("FDTD2D_KERNEL", "FDTD2D_TMA", "FDTD2D_TMAT", "FDTD2D_TB", "FDTD2D_PERSIST"):
        monkeypatch.delenv(v, raising=False)
    prob = F.Problem.from_spec(nx=nx, ny=ny, npml=P, n_steps=STEPS, profile=profile, x_lo=nx // 3, x_hi=nx - 3,
                               x_center=nx / 2, width=nx / 8, grf_rms=0.05, grf_corr=8, ne_peak=2e19, nu=3e9, n_elem=5,
                               src_i=nx // 2 - 6, src_j=ny // 2, src_di=3, src_dj=1, n_det=6, det_i=nx // 2 - 8,
                               det_j=ny // 2 - 2, det_di=2, det_dj=1, storage=store, field_max=16.0)
    prob.setup.ca = prob.setup.da = ca
    st = random_state(None, nx, ny, P, np.random.default_rng(nx))
    monkeypatch.setenv("FDTD2D_TILE", rows)
    name, got = _stepped(gpu, prob, st, CHUNKS)
    assert name == f"step_tmat_kernel<tile,{rows}>", name
    ref = _one_row(gpu, monkeypatch, prob, st, STEPS)
    for k in ref:
        assert np.array_equal(ref[k], got[k]), k


@pytest.mark.parametrize("rows", [2, 4, 6, 8])
@pytest.mark.parametrize("nx,ny,P,profile,ca", [
    (10, 9, 2, 1, 1.0), (126, 40, 3, 1, 1.0), (127, 41, 5, 0, 1.0), (252, 33, 4, 1, 0.999), (253, 97, 12, 1, 1.0),
    (203, 157, 7, 1, 1.0), (64, 260, 12, 3, 1.0), (1100, 90, 9, 1, 1.0), (500, 400, 40, 1, 0.998), (777, 601, 17, 3, 1.0)])
def test_resident_equals_one_row(gpu, monkeypatch, rows, nx, ny, P, profile, ca):
    """The whole shot on chip: one band of columns, two, several; strips down to
    a single warp; component detectors; the short run calls on the tile passes."""
    for v in ("FDTD2D_KERNEL", "FDTD2D_TMA", "FDTD2D_TMAT", "FDTD2D_TB", "FDTD2D_PERSIST", "FDTD2D_TILE"):
        monkeypatch.delenv(v, raising=False)
    n = 1 if nx < 40 else 5
    prob = F.Problem.from_spec(nx=nx, ny=ny, npml=P, n_steps=STEPS, profile=profile, x_lo=nx // 3, x_hi=nx - 3,
                               x_center=nx / 2, width=nx / 8, grf_rms=0.05, grf_corr=8, ne_peak=2e19, nu=3e9, n_elem=n,
                               src_i=nx // 2 - 6 if nx > 40 else 4, src_j=ny // 2, src_di=3, src_dj=1, n_det=n,
                               det_i=nx // 2 - 8 if nx > 40 else 5, det_j=ny // 2 - 2, det_di=2, det_dj=1)
    s = prob.setup
    s.ca = s.da = ca
    s.n_comp, s.comp = s.n_det, s.det
    st = random_state(None, nx, ny, P, np.random.default_rng(nx))
    monkeypatch.setenv("FDTD2D_RESIDENT", str(rows))
    name, got = _stepped(gpu, prob, st, CHUNKS)
    assert name == f"step_persist_kernel<0>/tile<{rows}>", name
    ref = _one_row(gpu, monkeypatch, prob, st, STEPS)
    for k in ref:
        assert np.array_equal(ref[k], got[k]), k


def test_resident_default_and_limits(gpu, monkeypatch):
    """A small shot runs on chip by default; one with more points than a warp's
    list holds, with two sources in a cell, or too large, on tile passes."""
    for v in ("FDTD2D_KERNEL", "FDTD2D_TMA", "FDTD2D_TMAT", "FDTD2D_TB", "FDTD2D_PERSIST", "FDTD2D_TILE", "FDTD2D_RESIDENT"):
        monkeypatch.delenv(v, raising=False)
    base = dict(ny=160, npml=10, n_steps=40, src_i=60, src_j=80, det_i=62, det_j=80)

    def name_and_check(**kw):
        prob = F.Problem.from_spec(**{**base, **kw})
        st = random_state(None, prob.nx, prob.ny, prob.setup.npml, np.random.default_rng(3))
        with monkeypatch.context() as m:
            name, got = _stepped(gpu, prob, st, (40,))
            ref = _one_row(gpu, m, prob, st, 40)
        for k in ref:
            assert np.array_equal(ref[k], got[k]), (name, k)
        return name

    assert name_and_check(nx=200).startswith("step_persist_kernel<0>/tile<")
    assert name_and_check(nx=200, n_det=60, det_i=63, det_di=1).startswith("step_tmat_kernel<tile")
    assert name_and_check(nx=200, n_elem=2).startswith("step_tmat_kernel<tile")   # both elements in one cell
    assert name_and_check(nx=1300, ny=1300).startswith("step_tmat_kernel<tile")


def test_resident_wait_runs_out(gpu, monkeypatch):
    """A neighbour's edge that never carries the expected tag: the poll gives up
    after its bound, the run reports it, the next shot runs as usual."""
    for v in ("FDTD2D_KERNEL", "FDTD2D_TMA", "FDTD2D_TMAT", "FDTD2D_TB", "FDTD2D_PERSIST", "FDTD2D_TILE", "FDTD2D_RESIDENT"):
        monkeypatch.delenv(v, raising=False)
    prob = F.Problem.from_spec(nx=256, ny=192, n_steps=200, x_lo=128, x_hi=246, src_i=30, src_j=96, det_i=34, det_j=96)
    monkeypatch.setenv("FDTD2D_WAIT_NS", "1000000")
    monkeypatch.setenv("FDTD2D_TEST_BARRIER_EXTRA", "1")
    with F.Shot(prob, gpu) as shot:
        assert shot.kernel_name().startswith("step_persist_kernel<0>/tile<")
        shot.run(1, 100)
        with pytest.raises(F.FdtdError) as e:
            shot.synchronize()
        assert e.value.status == F.ERR_TIMEOUT
    monkeypatch.delenv("FDTD2D_WAIT_NS")
    monkeypatch.delenv("FDTD2D_TEST_BARRIER_EXTRA")
    with F.Shot(prob, gpu) as shot:
        shot.run(1, 200)
        shot.synchronize()
        assert shot.check_finite()


def test_tile_line_probe_and_components(gpu, monkeypatch):
    """A line-probe window opening and closing inside passes, and component
    detectors: single steps where the probe reads, four at a time elsewhere."""
    nx, ny, P = 400, 301, 11
    prob = F.Problem.from_spec(nx=nx, ny=ny, npml=P, n_steps=50, x_lo=nx // 3, x_hi=nx - 3, src_i=200, src_j=150,
                               det_i=203, det_j=151, n_det=3, det_di=5)
    s = prob.setup
    s.line_n, s.line_i0, s.line_j, s.line_first, s.line_last = 300, 50, 140, 15, 22
    s.n_comp, s.comp = s.n_det, s.det

    def stepped():
        with F.Shot(prob, gpu) as shot:
            shot.run(1, 33)
            shot.run(34, 50)
            return shot.kernel_name(), [shot.line(15, 22)] + list(shot.traces().values()) + [shot.read_field("ez")]

    for v in ("FDTD2D_KERNEL", "FDTD2D_TMA", "FDTD2D_TMAT", "FDTD2D_TB", "FDTD2D_PERSIST"):
        monkeypatch.delenv(v, raising=False)
    monkeypatch.setenv("FDTD2D_TILE", "7")
    name, got = stepped()
    assert name == "step_tmat_kernel<tile,7>"
    monkeypatch.setenv("FDTD2D_TILE", "0")
    monkeypatch.setenv("FDTD2D_KERNEL", "stream")
    monkeypatch.setenv("FDTD2D_PERSIST", "0")
    _, ref = stepped()
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)


def test_tracker_and_probe_recorded(gpu, monkeypatch, tmp_path):
    """The wave-front tracker and the line probe recorded by the tile kernels, on
    chip and in passes (a Settings.ini shot of 500 x 1200 cells with 21 tracker
    lines; run calls shorter and longer than the history): the streaming
    kernel's rows, probe samples, traces and fields."""
    import re
    from pathlib import Path

    ini = (Path(__file__).resolve().parent / "golden" / "sphere_fluc_chirp" / "Settings.ini").read_text()
    for key, val in (("Imax", "250"), ("Jmax", "600"), ("Use_Exp_time", "0"), ("Max_time", "420")):
        ini = re.sub(rf"(?m)^{key}\s*=.*$", f"{key} = {val}", ini)
    path = tmp_path / "Settings.ini"
    path.write_text(ini)
    prob = F.Problem.from_ini(path)
    s = prob.setup
    assert (s.nx, s.ny) == (500, 1200) and s.n_rc > 0
    s.line_n, s.line_i0, s.line_j, s.line_first, s.line_last = 400, 50, 700, 120, 180

    def stepped():
        with F.Shot(prob, gpu) as shot:
            n = 1
            for c in (1, 100, 7, 300, 12):
                shot.run(n, n + c - 1)
                n += c
            out = {w: shot.read_field(w) for w in FIELDS + PSI_FIELDS}
            out.update(shot.traces())
            out["rc"], out["line"] = shot.rc(), shot.line(120, 180)
            return shot.kernel_name(), out

    for v in ("FDTD2D_KERNEL", "FDTD2D_TMA", "FDTD2D_TMAT", "FDTD2D_TB", "FDTD2D_PERSIST", "FDTD2D_TILE", "FDTD2D_RESIDENT"):
        monkeypatch.delenv(v, raising=False)
    name, on_chip = stepped()
    assert name.startswith("step_persist_kernel<0>/tile<"), name
    monkeypatch.setenv("FDTD2D_TILE", "7")
    name, passes = stepped()
    assert name == "step_tmat_kernel<tile,7>", name
    monkeypatch.setenv("FDTD2D_TILE", "0")
    monkeypatch.setenv("FDTD2D_KERNEL", "stream")
    monkeypatch.setenv("FDTD2D_PERSIST", "0")
    name, ref = stepped()
    assert name == "step_stream_kernel<0>", name
    assert ref["rc"].max() > 0
    for k in ref:
        assert np.array_equal(ref[k], on_chip[k]), ("on chip", k)
        assert np.array_equal(ref[k], passes[k]), ("passes", k)


@pytest.mark.parametrize("rows,imax,jmax", [("2", 60, 45), ("4", 190, 101), ("6", 127, 160), ("8", 250, 333), ("", 250, 600)])
def test_resident_material(gpu, monkeypatch, tmp_path, rows, imax, jmax):
    """The material-ID medium on chip: random ids (with the perfect conductor's)
    in the three maps, coefficients by material, update launches that stop short
    of their last cells; run calls of 1 to 40 steps, the short ones on the
    one-step kernels.  The streaming kernel's bits."""
    import ctypes
    import re
    from pathlib import Path

    ini = (Path(__file__).resolve().parent / "golden" / "sphere_fluc_chirp" / "Settings.ini").read_text()
    for key, val in (("Imax", imax), ("Jmax", jmax), ("Use_Exp_time", "0"), ("Max_time", "90")):
        ini = re.sub(rf"(?m)^{key}\s*=.*$", f"{key} = {val}", ini)
    path = tmp_path / "Settings.ini"
    path.write_text(ini)
    prob = F.Problem.from_ini(path)
    s = prob.setup
    nx, ny, P, n = s.nx, s.ny, s.npml, s.n_materials
    assert s.medium == F.MEDIUM_MATERIAL_ID
    rng = np.random.default_rng(nx)
    keep = []

    def put(name, a):
        keep.append(a)
        setattr(s, name, a.ctypes.data_as(type(getattr(s, name))))

    for name in ("id1", "id2", "id3"):
        put(name, rng.integers(0, n, (ny, nx)).astype(np.int32))
    for name in ("mat_ca", "mat_da"):
        put(name, rng.uniform(0.9, 1.0, n).astype(np.float32))
    for name in ("mat_cb", "mat_db"):
        put(name, (np.ctypeslib.as_array(getattr(s, name), (n,)) * rng.uniform(0.5, 1.0, n)).astype(np.float32))
    full = [(nx - 1) * (ny - 1), (nx - 1) * (P - 1), (nx - 1) * (ny - 1), (P - 1) * (ny - 1)]
    full += [(nx - 2) * (ny - 2), (nx - 2) * (ny - 2), (P - 1) * (ny - 2), (nx - 2) * (P - 1)]
    s.cover = (ctypes.c_int64 * 8)(*(int(c * f) for c, f in zip(full, rng.uniform(0.6, 1.0, 8))))
    st = random_state(None, nx, ny, P, rng)

    def stepped():
        with F.Shot(prob, gpu) as shot:
            load_state([shot], st)
            first = 1
            for c in (1, 9, 3, 8, 12, 7, 40):
                shot.run(first, first + c - 1)
                first += c
            out = {w: shot.read_field(w) for w in FIELDS + PSI_FIELDS}
            out.update(shot.traces())
            out["rc"] = shot.rc() if s.n_rc else np.zeros(1)
            return shot.kernel_name(), out

    for v in ("FDTD2D_KERNEL", "FDTD2D_TMA", "FDTD2D_TMAT", "FDTD2D_TB", "FDTD2D_PERSIST", "FDTD2D_TILE", "FDTD2D_RESIDENT"):
        monkeypatch.delenv(v, raising=False)
    if rows:
        monkeypatch.setenv("FDTD2D_RESIDENT", rows)
    name, got = stepped()
    assert name.startswith("step_persist_kernel<1>/tile<" + rows), name
    monkeypatch.setenv("FDTD2D_PERSIST", "0")
    name, ref = stepped()
    assert name == "step_stream_kernel<1>", name
    for k in ref:
        assert np.array_equal(ref[k], got[k]), k


@pytest.mark.parametrize("rows,nx,ny,P,store,profile,ca,comp", [
    ("2", 10, 9, 2, 1, 1, 1.0, True), ("2", 253, 97, 12, 2, 1, 0.999, False), ("2", 126, 40, 3, 1, 0, 1.0, False),
    ("4", 203, 157, 7, 1, 1, 1.0, True), ("4", 500, 400, 40, 2, 3, 0.998, False), ("6", 777, 601, 17, 1, 3, 1.0, False),
    ("6", 127, 41, 5, 2, 1, 1.0, True), ("6", 1100, 90, 9, 1, 1, 1.0, False), ("", 1000, 900, 20, 2, 3, 1.0, True)])
def test_resident_16bit_equals_one_row(gpu, monkeypatch, rows, nx, ny, P, store, profile, ca, comp):
    """The whole shot on chip with 16-bit fields, rounded after every step; Ez
    detectors alone and with component ones."""
    for v in ("FDTD2D_KERNEL", "FDTD2D_TMA", "FDTD2D_TMAT", "FDTD2D_TB", "FDTD2D_PERSIST", "FDTD2D_TILE", "FDTD2D_RESIDENT"):
        monkeypatch.delenv(v, raising=False)
    n = 1 if nx < 40 else 5
    prob = F.Problem.from_spec(nx=nx, ny=ny, npml=P, n_steps=STEPS, profile=profile, x_lo=nx // 3, x_hi=nx - 3,
                               x_center=nx / 2, width=nx / 8, grf_rms=0.05, grf_corr=8, ne_peak=2e19, nu=3e9, n_elem=n,
                               src_i=nx // 2 - 6 if nx > 40 else 4, src_j=ny // 2, src_di=3, src_dj=1, n_det=n,
                               det_i=nx // 2 - 8 if nx > 40 else 5, det_j=ny // 2 - 2, det_di=2, det_dj=1, storage=store,
                               field_max=16.0)
    s = prob.setup
    s.ca = s.da = ca
    if comp:
        s.n_comp, s.comp = s.n_det, s.det

    def stepped(chunks):
        with F.Shot(prob, gpu) as shot:
            load_state([shot], st)
            first = 1
            for c in chunks:
                shot.run(first, first + c - 1)
                first += c
            out = {w: shot.read_field(w) for w in FIELDS + PSI_FIELDS}
            out.update(shot.traces())
            out["dft"] = shot.dft()
            return shot.kernel_name(), out

    st = random_state(None, nx, ny, P, np.random.default_rng(nx))
    if rows:
        monkeypatch.setenv("FDTD2D_RESIDENT", rows)
    name, got = stepped(CHUNKS)
    assert name.startswith("step_persist_kernel<0>/tile<" + rows), name
    monkeypatch.delenv("FDTD2D_RESIDENT", raising=False)
    monkeypatch.setenv("FDTD2D_TMAT", "0")
    monkeypatch.setenv("FDTD2D_TMA", "4,3")
    monkeypatch.setenv("FDTD2D_PERSIST", "0")
    name, ref = stepped((STEPS,))
    assert name == "step_tma_kernel<4,3>", name
    for k in ref:
        assert np.array_equal(ref[k], got[k]), k


@pytest.mark.parametrize("rows,nx,ny,P,ca", [
    ("7", 128, 60, 5, 1.0), ("7", 129, 33, 6, 0.999), ("5", 248, 32, 9, 1.0), ("7", 249, 131, 12, 1.0), ("7", 371, 107, 23, 1.0),
    ("7", 372, 108, 24, 1.0), ("5", 500, 149, 30, 0.998), ("7", 502, 210, 52, 1.0), ("7", 613, 163, 20, 1.0), ("5", 490, 185, 2, 1.0)])
def test_tile_partition(gpu, monkeypatch, rows, nx, ny, P, ca):
    """Tiles on the borders and plain tiles moved back: one, two and more columns
    of tiles, widths around them, one and more rows of CPML tiles, points on both
    sides of every 8th row and column where tiles may meet."""
    for v in ("FDTD2D_KERNEL", "FDTD2D_TMA", "FDTD2D_TMAT", "FDTD2D_TB", "FDTD2D_PERSIST", "FDTD2D_RESIDENT"):
        monkeypatch.delenv(v, raising=False)
    n = min((nx - 4) // 8, (ny - 4) // 4) - 1
    prob = F.Problem.from_spec(nx=nx, ny=ny, npml=P, n_steps=STEPS, profile=1, x_lo=nx // 3, x_hi=nx - 3, ne_peak=2e19, nu=3e9,
                               n_elem=n, src_i=3, src_j=2, src_di=8, src_dj=4, n_det=n, det_i=4, det_j=3, det_di=8, det_dj=4)
    prob.setup.ca = prob.setup.da = ca
    st = random_state(None, nx, ny, P, np.random.default_rng(nx))
    monkeypatch.setenv("FDTD2D_TILE", rows)
    name, got = _stepped(gpu, prob, st, CHUNKS)
    assert name == f"step_tmat_kernel<tile,{rows}>", name
    ref = _one_row(gpu, monkeypatch, prob, st, STEPS)
    for k in ref:
        assert np.array_equal(ref[k], got[k]), k
