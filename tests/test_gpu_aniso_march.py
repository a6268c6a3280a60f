"""The marching anisotropic adjoint (csrc/pam_aniso.cuh) against the FP32
oracle at the sizes where its tiles end: 56 written columns per warp, a pair
of columns per lane, rows in trips of four."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_cases import engine_for, make_case, oracle_models, rel

pytestmark = pytest.mark.gpu

# the image's bar in the migration tests; the anisotropic operator is held to
# three times the FP32 oracle's own distance from FP64 where that is larger
TOL, FP32_FACTOR = 1e-5, 3.0


# expanded widths 8 + 56 k - 1, + 0, + 1, + 2, and heights that leave one to
# three rows to the last trip; the smallest grid
@pytest.mark.parametrize("approx", ["VTI", "TTI"])
@pytest.mark.parametrize("nz,nx,N,nshots", [(8, 8, 8, 1), (31, 95, 12, 1), (32, 96, 12, 3), (33, 97, 12, 2), (34, 98, 12, 5)])
def test_image_at_the_edges_of_the_tiles(approx, nz, nx, N, nshots):
    case = make_case(approx, "cerjan", nz=nz, nx=nx, N=N, nt=200, nshots=nshots, seed=nx, sd_off=True)
    if nz == 8:
        case["sx"], case["sz"] = np.array([11], np.int32), np.array([11], np.int32)
    g, m = case["grid"], oracle_models(case)
    e = engine_for(case)
    d = e.forward(case["sz"], case["sx"])
    e.rtm(case["sz"], case["sx"], d, ckpt_interval=0)
    img, ilum = e.rtm_result(norm="none")
    want = {}
    for dt in (np.float32, np.float64):
        r = [O.rtm_shot(g, m, case["wavelet"], int(sx), int(sz), case["rx"], case["rz"], d[i], dtype=dt)
             for i, (sx, sz) in enumerate(zip(case["sx"], case["sz"]))]
        want[dt] = [sum(np.asarray(v[k], np.float64) for v in r) for k in range(2)]
    for got, ref32, ref64 in zip((img, ilum), want[np.float32], want[np.float64]):
        assert np.isfinite(got).all() and np.abs(ref64).max() > 0
        assert rel(got, ref64) < max(TOL, FP32_FACTOR * rel(ref32, ref64))
