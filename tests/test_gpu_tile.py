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


@pytest.mark.parametrize("approx,boundary", [("acoustic", "cerjan"), ("VTI", "cerjan"), ("TTI", "cerjan"),
                                             ("acoustic", "CPML"), ("VTI", "CPML")])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_tiles_are_bitwise_the_one_step_launches(approx, boundary, shape, monkeypatch):
    nz, nx, N, nt, itlag, shots = shape
    e, rng = _engine(approx, nz, nx, N, nt, itlag, shots, boundary=boundary)
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


@pytest.mark.parametrize("approx,boundary", [("acoustic", "cerjan"), ("TTI", "cerjan"), ("acoustic", "CPML")])
def test_tiles_in_chunks_with_pinned_output(approx, boundary):
    """A pinned output cuts the loop into launches of a few steps each, which
    hand the state over through either published set."""
    torch = pytest.importorskip("torch")
    e, rng = _engine(approx, 61, 133, 12, 83, 9, 2, boundary=boundary)
    e.set_receivers(np.full(30, 14, np.int32), np.arange(20, 50, dtype=np.int32))
    sz, sx = np.array([14, 40], np.int32), np.array([30, 90], np.int32)
    ref = e.forward(sz, sx)
    out = torch.zeros((2, 74, 30)).pin_memory()
    assert np.array_equal(e.forward(sz, sx, out=out.numpy()), ref)


# (nz, nx, border, steps, lag, shots): odd sizes, several shots per launch and
# more than fit at once, a step count that no group divides, two segments or more
BACK = [(8, 8, 8, 40, 0, 1), (61, 133, 12, 61, 11, 2), (20, 24, 9, 47, 3, 170), (90, 61, 20, 97, 30, 5),
        (201, 401, 50, 83, 10, 1)]


@pytest.mark.parametrize("job", ["gradient", "rtm"])
@pytest.mark.parametrize("shape", BACK, ids=lambda s: "x".join(map(str, s)))
def test_backward_tiles_match_the_one_step_launches(job, shape, monkeypatch):
    """The fields of the backward tiles are the one-step launches' bit for bit;
    the sums over time and shots are added in another order: each sum has at
    most steps x shots terms in float32, so the two differ by a random walk of
    that many roundings, 2^-24 sqrt(steps x shots) of the sum of magnitudes,
    here held to 16 times that in relative L2 (cancellation within a cell)."""
    nz, nx, N, nt, itlag, shots = shape
    e, rng = _engine("acoustic", nz, nx, N, nt, itlag, shots)
    nza, nxa = nz + 2 * N, nx + 2 * N
    sz, sx = rng.integers(4, nza - 4, shots).astype(np.int32), rng.integers(4, nxa - 4, shots).astype(np.int32)
    rz, rx = rng.integers(4, nza - 4, 60).astype(np.int32), rng.integers(4, nxa - 4, 60).astype(np.int32)
    # one source, and receivers beside it, inside the model, so that its sums are not zero
    sz[0], sx[0] = nza // 2, nxa // 2
    rz[:6], rx[:6] = sz[0] + 1, sx[0] + np.arange(6) - 3
    rz[1], rx[1] = rz[0], rx[0]
    prz, prx = rng.integers(4, nza - 4, (shots, 9)).astype(np.int32), rng.integers(4, nxa - 4, (shots, 9)).astype(np.int32)
    prz[0, :4], prx[0, :4] = rz[:4], rx[:4]
    tol = 16 * 2.0 ** -24 * np.sqrt(nt * shots)

    def run(z, d, K):
        e.rtm_reset()
        if job == "rtm":
            e.rtm(sz, sx, d, ckpt_interval=K)
            return e.rtm_result(norm="none")
        J, g = e.misfit_gradient(sz, sx, d, ckpt_interval=K)
        return g, e.fwi_result()[1], np.array([J])

    def close(a, b):
        for x, y in zip(a, b):
            n = np.linalg.norm(y.astype(np.float64))
            assert np.isfinite(y).all() and n > 0
            assert np.linalg.norm(x.astype(np.float64) - y) <= tol * n

    for z, x, per_shot in ((rz, rx, False), (prz, prx, True)):
        e.set_receivers(z, x, per_shot=per_shot)
        d = (1e-2 * rng.standard_normal((shots, nt - itlag, z.shape[-1]))).astype(np.float32)
        tiles = run(z, d, 0)
        for K in (17, nt - 1):      # the order of the sums does not depend on the segments
            assert all(np.array_equal(a, b) for a, b in zip(run(z, d, K), tiles))
        monkeypatch.setenv("PAM_NO_PERSISTENT", "1")
        one_step = run(z, d, 0)
        monkeypatch.delenv("PAM_NO_PERSISTENT")
        close(tiles, one_step)
    # receivers on the frame stay with the one-step launches
    e.set_receivers(np.array([0, N + 1, sz[0] + 1], np.int32), np.array([N, N + 2, sx[0]], np.int32))
    d = (1e-2 * rng.standard_normal((shots, nt - itlag, 3))).astype(np.float32)
    close(run(rz, d, 0), run(rz, d, 17))


@pytest.mark.parametrize("approx,boundary", [("acoustic", "cerjan"), ("acoustic", "CPML"), ("VTI", "cerjan"), ("TTI", "cerjan")])
@pytest.mark.parametrize("shape", [(9, 9, 8, 61, 7, 2), (61, 133, 12, 150, 11, 2), (90, 61, 21, 97, 30, 5)],
                         ids=lambda s: "x".join(map(str, s)))
def test_migration_strategies_as_tiles(approx, boundary, shape, monkeypatch):
    """Migration with every way of keeping the source field - all steps, bands in
    each storage format, the random border - as tiles against the one-step
    launches: the fields are the same bit for bit, the sums in the order of the
    test above, to the same tolerance (anisotropic images are summed by the same
    kernel, so they are equal)."""
    nz, nx, N, nt, itlag, shots = shape
    e, rng = _engine(approx, nz, nx, N, nt, itlag, shots, boundary=boundary)
    nza, nxa = nz + 2 * N, nx + 2 * N
    sz, sx = np.full(shots, nza // 2, np.int32), (N + np.linspace(2, nx - 3, shots)).astype(np.int32)
    e.set_receivers(np.full(nx - 4, N + 2, np.int32), (N + 2 + np.arange(nx - 4)).astype(np.int32))
    e.set_random_boundary(400.0, 30.0, 3)
    d = (1e-2 * rng.standard_normal((shots, nt - itlag, nx - 4))).astype(np.float32)
    tol = 16 * 2.0 ** -24 * np.sqrt(nt * shots)
    for K, store in ((0, "f32"), (-1, "f32"), (-1, "bf16"), (-1, "f16"), (-2, "f32"), (19, "f16")):
        out = []
        for env in (None, "1"):
            if env:
                monkeypatch.setenv("PAM_NO_PERSISTENT", env)
            e.rtm_reset()
            e.rtm(sz, sx, d, ckpt_interval=K, store=store)
            out.append(e.rtm_result(norm="none"))
            if approx != "acoustic":
                e.fwi_gradient(sz, sx, d, ckpt_interval=K, store=store)
                out[-1] += e.fwi_result()
        monkeypatch.delenv("PAM_NO_PERSISTENT")
        for x, y in zip(*out):
            n = np.linalg.norm(y.astype(np.float64))
            assert np.isfinite(y).all() and n > 0
            assert np.linalg.norm(x.astype(np.float64) - y) <= (tol * n if approx == "acoustic" else 0.0), (K, store)
