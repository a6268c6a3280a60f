"""CPML strips launched together in a stream against the forked strips of the step graph.

Both forms evaluate the same expressions, so the seismograms are equal bit for
bit.  Border widths around the shapes that the strips are cut into: odd and even
(cells and pairs along x), the smallest, and beyond the paired z strips.  (The
grids are narrow enough that every tile reaches into a border: the segment
height that the engine picks then changes no rounding.)
"""
import numpy as np
import pytest

from pseudoacousticmodeling_gb300 import Config, Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("approx", ["acoustic", "VTI"])
@pytest.mark.parametrize("border,shots", [(8, 3), (9, 1), (45, 2), (50, 2), (197, 1), (260, 1)])
def test_strips_in_one_launch(approx, border, shots, monkeypatch):
    nz, nx, nt, lag = 37, 61, 140, 60
    cfg = Config(nz=nz, nx=nx, n_abc=border, nt=nt, itlag=lag, dx=10.0, dz=10.0, dt=0.0008, fcut=15.0, max_shots=shots,
                 approximation=approx, boundary="CPML")
    rng = np.random.default_rng(5)
    vp = (2000.0 + 500.0 * rng.random((nz, nx))).astype(np.float32)
    more = () if approx == "acoustic" else (np.full((nz, nx), 0.1, np.float32), np.full((nz, nx), 0.05, np.float32))
    sx = (border + np.linspace(5, nx - 6, shots)).astype(np.int32)
    sz = np.full(shots, border + nz // 2, np.int32)
    rx = (border + np.arange(0, nx, 2)).astype(np.int32)

    def run():
        e = Engine(cfg)
        e.set_models(vp, *more)
        e.set_receivers(np.full(rx.size, border + nz // 2, np.int32), rx)
        return np.array(e.forward(sz, sx))

    monkeypatch.setenv("PAM_NO_PERSISTENT", "1")
    forked = run()
    monkeypatch.setenv("PAM_NO_GRAPH", "1")
    together = run()
    assert np.abs(forked).max() > 0.0
    assert np.array_equal(forked, together)
