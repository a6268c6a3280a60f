"""Small runs as persistent tiles (csrc/pam_tile.cuh) against the one-step
launches, bit for bit: the tiles compute the same cells by the same operations,
whatever the cut of the grid and the number of steps between barriers."""
import numpy as np
import pytest

from pseudoacousticmodeling_gb300 import Config, Engine
from tests.gpu_cases import smooth_field

pytestmark = pytest.mark.gpu


def _engine(approx, nz, nx, N, nt, itlag, shots, seed=1, boundary="cerjan"):
    rng = np.random.default_rng(seed)
    e = Engine(Config(nz=nz, nx=nx, n_abc=N, dz=10.0, dx=8.0, dt=0.0008, nt=nt, itlag=itlag, fcut=30.0,
                      approximation=approx, boundary=boundary, max_shots=shots))
    vp = smooth_field(rng, (nz, nx), 1500.0, 2600.0)
    e.set_models(vp, smooth_field(rng, (nz, nx), 0.0, 0.2), smooth_field(rng, (nz, nx), 0.0, 0.1),
                 smooth_field(rng, (nz, nx), -30.0, 30.0))
    return e, rng


# (nz, nx, border, steps, lag, shots): the smallest grid, one quad of columns
# over a tile's edge, more shots than tiles fit at once, a single step, a step
# count that no group of steps divides, a grid near the largest
SHAPES = [(8, 8, 8, 40, 0, 1), (9, 11, 8, 37, 5, 3), (61, 133, 12, 61, 11, 2), (20, 24, 9, 23, 3, 170),
          (40, 50, 10, 1, 0, 1), (90, 61, 20, 97, 30, 9), (201, 401, 50, 53, 10, 1), (401, 1001, 50, 31, 7, 1)]


@pytest.mark.parametrize("approx", ["acoustic", "VTI", "TTI"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_tiles_are_bitwise_the_one_step_launches(approx, shape, monkeypatch):
    nz, nx, N, nt, itlag, shots = shape
    e, rng = _engine(approx, nz, nx, N, nt, itlag, shots)
    nza, nxa = nz + 2 * N, nx + 2 * N
    sz = rng.integers(4, nza - 4, shots).astype(np.int32)
    sx = rng.integers(4, nxa - 4, shots).astype(np.int32)
    # receivers anywhere on the expanded grid, its frame and coincident cells among them; then a spread per shot
    rz, rx = rng.integers(0, nza, 40).astype(np.int32), rng.integers(0, nxa, 40).astype(np.int32)
    rz[:3], rx[:3] = [0, nza - 1, 7], [0, nxa - 1, 9]
    rz[3], rx[3] = rz[2], rx[2]
    prz, prx = rng.integers(0, nza, (shots, 17)).astype(np.int32), rng.integers(0, nxa, (shots, 17)).astype(np.int32)
    # some near a source, so that large grids record a wave too
    for z, x in ((rz, rx), (prz.T, prx.T)):
        z[8:16] = np.clip(sz[0] + np.arange(8).reshape((8,) + (1,) * (z.ndim - 1)) - 4, 0, nza - 1)
        x[8:16] = sx[0]
    for z, x, per_shot in ((rz, rx, False), (prz, prx, True)):
        e.set_receivers(z, x, per_shot=per_shot)
        tiles = e.forward(sz, sx)
        again = e.forward(sz[:1], sx[:1])
        monkeypatch.setenv("PAM_NO_PERSISTENT", "1")
        one_step = e.forward(sz, sx)
        monkeypatch.delenv("PAM_NO_PERSISTENT")
        assert np.isfinite(one_step).all() and (np.abs(one_step).max() > 0 or nt < 30)
        assert np.array_equal(tiles, one_step)
        assert np.array_equal(again[0], one_step[0])


@pytest.mark.parametrize("approx", ["acoustic", "TTI"])
def test_tiles_in_chunks_with_pinned_output(approx):
    """A pinned output cuts the loop into launches of a few steps each, which
    hand the state over through either published set."""
    torch = pytest.importorskip("torch")
    e, rng = _engine(approx, 61, 133, 12, 83, 9, 2)
    e.set_receivers(np.full(30, 14, np.int32), np.arange(20, 50, dtype=np.int32))
    sz, sx = np.array([14, 40], np.int32), np.array([30, 90], np.int32)
    ref = e.forward(sz, sx)
    out = torch.zeros((2, 74, 30)).pin_memory()
    assert np.array_equal(e.forward(sz, sx, out=out.numpy()), ref)
