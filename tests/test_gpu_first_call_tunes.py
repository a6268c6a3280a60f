"""The first call for a batch size picks the stepping kernel's segment height,
whichever loop that call itself runs as: a later call into a stream capture
cannot, and would run at the default height."""
import pytest

from tests.gpu_cases import engine_for, make_case

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("approx", ["acoustic", "VTI"])
@pytest.mark.parametrize("device", [False, True])
def test_a_small_modelling_run_tunes(approx, device):
    case = make_case(approx, "CPML", nz=61, nx=133, N=12, nt=150, nshots=2, seed=9)
    e = engine_for(case)
    assert e.segment_height(2) == 0
    if device:
        sz, sx = (torch.as_tensor(case[k], dtype=torch.int32, device="cuda") for k in ("sz", "sx"))
        out = torch.empty((2, case["grid"].nt_data, case["rx"].size), device="cuda")
        torch.cuda.synchronize()
        e.forward_device(sz, sx, out)
        torch.cuda.synchronize()
    else:
        e.forward(case["sz"], case["sx"])
    assert e.tile_workspace() > 0          # it ran as tiles
    assert e.segment_height(2) in (8, 16, 24, 32, 48, 64, 96, 128)
    assert e.segment_height(1) == 0


@pytest.mark.parametrize("job,approx", [("exact", "acoustic"), ("rtm", "acoustic"), ("rtm", "TTI")])
def test_a_small_job_tunes(job, approx):
    case = make_case(approx, "cerjan", nz=61, nx=133, N=12, nt=150, nshots=2, seed=9)
    e = engine_for(case)
    d = e.forward(case["sz"], case["sx"])
    if job == "exact":
        e.misfit_gradient(case["sz"], case["sx"], d)
    else:
        e.rtm(case["sz"], case["sx"], d)
    assert e.tile_workspace() > 0
    assert e.segment_height(2) in (8, 16, 24, 32, 48, 64, 96, 128)
