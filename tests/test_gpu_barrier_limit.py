"""A grid barrier of the persistent tiles that runs into its limit: the blocks
leave, the samples that they have not recorded are NaN, and the host reports it.
One poll is the limit here, so that the first block to arrive gives up; every
wait ends within that poll."""
import numpy as np
import pytest

from pseudoacousticmodeling_gb300 import PamError
from pseudoacousticmodeling_gb300.engine import BOUNDARY_SAVING, RANDOM_BOUNDARY
from tests.gpu_cases import engine_for, make_case

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

POLLS = 1 << 21
GAVE_UP = "PAM_E_CUDA: a grid barrier of the persistent time loop was given up"


@pytest.mark.parametrize("approx,abc", [("acoustic", "cerjan"), ("VTI", "cerjan"), ("TTI", "cerjan"), ("acoustic", "CPML"),
                                        ("VTI", "CPML")])
def test_a_modelling_run_that_gave_up(approx, abc):
    case = make_case(approx, abc, nz=61, nx=133, N=12, nt=150, nshots=2, seed=9)
    e = engine_for(case)
    ref = e.forward(case["sz"], case["sx"])
    assert np.isfinite(ref).all()
    e.set_barrier_polls(1)
    with pytest.raises(PamError, match=GAVE_UP):
        e.forward(case["sz"], case["sx"])
    # device output: NaN in the buffer, and the engine's next call that waits
    sz, sx = (torch.as_tensor(case[k], dtype=torch.int32, device="cuda") for k in ("sz", "sx"))
    out = torch.zeros(ref.shape, device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    e.forward_device(sz, sx, out, stream=st.cuda_stream)
    torch.cuda.synchronize()
    assert torch.isnan(out).any()
    e.set_barrier_polls(POLLS)
    e.forward_device(sz, sx, out, stream=st.cuda_stream)
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), ref)
    with pytest.raises(PamError, match=GAVE_UP):
        e.forward(case["sz"], case["sx"])
    # said once; the engine goes on
    assert np.array_equal(e.forward(case["sz"], case["sx"]), ref)


@pytest.mark.parametrize("job,abc,K", [("exact", "cerjan", 0), ("exact", "cerjan", 40), ("rtm", "cerjan", 0),
                                       ("rtm", "cerjan", BOUNDARY_SAVING), ("rtm", "CPML", BOUNDARY_SAVING),
                                       ("rtm", "cerjan", RANDOM_BOUNDARY), ("reference", "cerjan", RANDOM_BOUNDARY),
                                       ("reference", "cerjan", BOUNDARY_SAVING)])
def test_a_job_that_gave_up(job, abc, K):
    case = make_case("acoustic", abc, nz=61, nx=133, N=12, nt=150, nshots=2, seed=9)
    e = engine_for(case)
    e.set_random_boundary(400.0, 30.0, 3)
    d = 1.01 * e.forward(case["sz"], case["sx"])

    def run():
        e.rtm_reset()
        if job == "exact":
            return e.misfit_gradient(case["sz"], case["sx"], d, ckpt_interval=K)[1]
        if job == "rtm":
            e.rtm(case["sz"], case["sx"], d, ckpt_interval=K)
            return e.rtm_result(norm="none")[0]
        e.fwi_gradient(case["sz"], case["sx"], d, ckpt_interval=K)
        return e.fwi_result()[0]

    ref = run()
    e.set_barrier_polls(1)
    with pytest.raises(PamError, match=GAVE_UP):
        run()
    e.set_barrier_polls(POLLS)
    assert np.array_equal(run(), ref)
