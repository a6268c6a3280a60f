"""The wavefield that a modelling run leaves behind, however it ran."""
import numpy as np
import pytest

from tests.gpu_cases import engine_for, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("approx,abc", [("acoustic", "cerjan"), ("VTI", "cerjan"), ("TTI", "cerjan"), ("VTI", "CPML")])
@pytest.mark.parametrize("nt", [151, 152, 154])
def test_wavefield_after_a_run_does_not_depend_on_its_loop(approx, abc, nt, monkeypatch):
    """Small runs as tiles publish their fields in either of two sets; a run as
    one-step launches leaves them in the two field buffers.  What is read
    afterwards is the same (nt is even: the last field)."""
    case = make_case(approx, abc, nz=61, nx=133, N=12, nt=nt, nshots=2, seed=5)
    e = engine_for(case)
    for _ in range(2):
        e.forward(case["sz"], case["sx"])
        tiles = e.read_wavefield()
    monkeypatch.setenv("PAM_NO_PERSISTENT", "1")
    e.forward(case["sz"], case["sx"])
    launches = e.read_wavefield()
    assert np.abs(launches).max() > 0
    assert np.array_equal(tiles, launches)
