"""The workspace of runs as tiles: it is sized for the batch that runs and not
for max_shots, is bounded and given back, and a run for which it has no room
takes the one-step launches."""
import numpy as np
import pytest

from pseudoacousticmodeling_gb300.engine import BOUNDARY_SAVING, RANDOM_BOUNDARY
from tests.gpu_cases import engine_for, make_case

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

NZ, NX, N = 101, 201, 30


def case_for(approx="acoustic", abc="cerjan", nshots=3, nt=130):
    return make_case(approx, abc, nz=NZ, nx=NX, N=N, nt=nt, nshots=nshots, seed=21)


def shots(case, n):
    return case["sz"][:n], case["sx"][:n]


def test_one_shot_of_an_engine_for_many_takes_the_workspace_of_one(monkeypatch):
    """Boundary saving with the matched layer: 2 + 8 + 4 + 8 + 50 fields per shot."""
    case = case_for(abc="CPML")
    e = engine_for(case, max_shots=48)
    e.set_random_boundary(400.0, 30.0, 3)
    sz, sx = shots(case, 1)
    monkeypatch.setenv("PAM_NO_PERSISTENT", "1")
    d = e.forward(sz, sx)
    e.rtm(sz, sx, d, ckpt_interval=BOUNDARY_SAVING)      # everything but the workspace
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    monkeypatch.delenv("PAM_NO_PERSISTENT")
    e.forward(sz, sx)
    e.rtm(sz, sx, d, ckpt_interval=BOUNDARY_SAVING)
    torch.cuda.synchronize()
    held = before - torch.cuda.mem_get_info()[0]
    # (an allocation takes pages of 2 MiB, and there are eleven arrays, two lists and pinned buffers' tables)
    assert held <= 72 * e.field_bytes() + 16 * (2 << 20), held
    assert 0 < e.tile_workspace() <= 72 * e.field_bytes()
    # another strategy gives the segment's fields back
    e.rtm(sz, sx, d, ckpt_interval=0)
    assert e.tile_workspace() <= 22 * e.field_bytes()
    assert e.tile_workspace(limit_bytes=0) == 0


def jobs(e, case, n, approx, abc):
    """Seismograms, images of every strategy and gradients of the first n shots."""
    sz, sx = shots(case, n)
    out = [e.forward(sz, sx)]
    dev = torch.empty(out[0].shape, device="cuda")
    torch.cuda.synchronize()
    e.forward_device(torch.as_tensor(sz, dtype=torch.int32, device="cuda"),
                     torch.as_tensor(sx, dtype=torch.int32, device="cuda"), dev, stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    out.append(dev.cpu().numpy())
    d = 1.01 * out[0]
    if abc == "cerjan" or approx == "acoustic":
        for K in (0, 40, BOUNDARY_SAVING, RANDOM_BOUNDARY):
            e.rtm_reset()
            e.rtm(sz, sx, d, ckpt_interval=K)
            out += e.rtm_result(norm="none")
            out.append(np.array([e.fwi_gradient(sz, sx, d, ckpt_interval=K)]))
            out += e.fwi_result()
    if abc == "cerjan" and approx == "acoustic":
        for K in (0, 40):
            out += [np.asarray(v) for v in e.misfit_gradient(sz, sx, d, ckpt_interval=K)]
    return out


def same(a, b):
    assert len(a) == len(b)
    for i, (x, y) in enumerate(zip(a, b)):
        assert np.isfinite(y).all()
        assert np.array_equal(x, y), i


@pytest.mark.parametrize("approx,abc", [("acoustic", "cerjan"), ("TTI", "cerjan"), ("acoustic", "CPML"), ("VTI", "CPML")])
def test_no_room_is_the_one_step_launches(approx, abc, monkeypatch):
    case = case_for(approx, abc)
    e = engine_for(case)
    e.set_random_boundary(400.0, 30.0, 3)
    e.tile_workspace(limit_bytes=0)
    none = jobs(e, case, 2, approx, abc)
    assert e.tile_workspace() == 0
    monkeypatch.setenv("PAM_NO_PERSISTENT", "1")
    e2 = engine_for(case)
    e2.set_random_boundary(400.0, 30.0, 3)
    one_step = jobs(e2, case, 2, approx, abc)
    monkeypatch.delenv("PAM_NO_PERSISTENT")
    same(none, one_step)
    # room for a part of it: each sweep that fits runs as tiles (the sums over
    # time of the backward sweeps are in another order there, to the tolerance of
    # the tile tests: 16 roundings of a random walk over steps and shots)
    tol = 16 * 2.0 ** -24 * np.sqrt(case["grid"].nt * 2)
    for fields in (2, 6, 10, 14, 22, 54, 72):
        e.tile_workspace(limit_bytes=2 * fields * e.field_bytes())
        part = jobs(e, case, 2, approx, abc)
        assert 0 < e.tile_workspace() <= 2 * fields * e.field_bytes()
        for i, (x, y) in enumerate(zip(part, one_step)):
            assert np.linalg.norm(x.astype(np.float64) - y) <= tol * np.linalg.norm(y.astype(np.float64)), (fields, i)


@pytest.mark.parametrize("approx,abc", [("acoustic", "cerjan"), ("TTI", "cerjan"), ("acoustic", "CPML")])
def test_batches_that_grow_and_shrink(approx, abc):
    """Each batch gives what a new engine gives it, whatever the workspace was
    sized for before; one that has not fitted does not keep a smaller one out."""
    case = case_for(approx, abc)
    ref = {}
    for n in (1, 2, 3):
        e = engine_for(case)
        e.set_random_boundary(400.0, 30.0, 3)
        ref[n] = jobs(e, case, n, approx, abc)
    e = engine_for(case)
    e.set_random_boundary(400.0, 30.0, 3)
    for n in (1, 3, 2, 1, 3):
        same(jobs(e, case, n, approx, abc), ref[n])
    e.tile_workspace(limit_bytes=80 * e.field_bytes())
    for n in (3, 1):
        jobs(e, case, n, approx, abc)
    same(jobs(e, case, 1, approx, abc), ref[1])
    assert e.tile_workspace() <= 72 * e.field_bytes()


def test_a_batch_that_has_not_fitted_keeps_no_smaller_one_out():
    """Room for the segment's fields of one shot, not of three: three shots migrate
    with the rest of the workspace, and one shot then gets its own."""
    case = case_for()
    e = engine_for(case)
    e.set_random_boundary(400.0, 30.0, 3)
    e.tile_workspace(limit_bytes=80 * e.field_bytes())
    d = e.forward(case["sz"], case["sx"])
    e.rtm(case["sz"], case["sx"], d, ckpt_interval=BOUNDARY_SAVING)
    e.rtm(case["sz"], case["sx"], d, ckpt_interval=0)    # (fits: two arrays more for the receiver side)
    assert e.tile_workspace() == 3 * 6 * e.field_bytes()
    sz, sx = shots(case, 1)
    e.rtm(sz, sx, d[:1], ckpt_interval=RANDOM_BOUNDARY)
    assert e.tile_workspace() == 56 * e.field_bytes()
