"""The bytes the benchmark charges a launch of each step kernel."""
import importlib.util
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench", ROOT / "bench.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.mark.parametrize("kernel,steps,passes", [
    ("step_tma_kernel<4,3>", 1, 1), ("step_tmat2_kernel<4,2,2>+step_tma_kernel<2,2>", 2, 1), ("step_tmat_kernel<tile,7>", 4, 1),
    ("step_persist_kernel<0>", 100, 100), ("step_persist_kernel<1>", 7, 7), ("step_persist_kernel<0>/tile<6>", 100, 1),
    ("step_persist_kernel<1>/tile<2>", 4096, 1)])
def test_passes_of_a_launch(bench, kernel, steps, passes):
    """A cell's fields are read and written once per pass: a tile pass once for its
    four steps, the on-chip kernel once per launch, the grid-barrier kernel once per step."""
    assert bench.launch_passes(kernel, steps) == passes
