"""Runs with device output that are still queued while the caller goes on: what
the engine is told next does not reach them, and queueing does not wait."""
import numpy as np
import pytest

from pseudoacousticmodeling_gb300 import Config, Engine
from tests.gpu_cases import smooth_field

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

WAIT = 400_000_000   # cycles of the kernel that keeps the stream busy (about 0.2 s)


def make_engine(approx, boundary, shots=1, nz=60, nx=110, N=20, nt=160, itlag=20):
    rng = np.random.default_rng(7)
    e = Engine(Config(nz=nz, nx=nx, n_abc=N, dz=10.0, dx=10.0, dt=0.0008, nt=nt, itlag=itlag, fcut=25.0,
                      approximation=approx, boundary=boundary, max_shots=shots))
    e.set_models(smooth_field(rng, (nz, nx), 1600.0, 2600.0), smooth_field(rng, (nz, nx), 0.0, 0.2),
                 smooth_field(rng, (nz, nx), 0.0, 0.1), smooth_field(rng, (nz, nx), -30.0, 30.0))
    rx = np.arange(N, N + nx, 3, dtype=np.int32)
    e.set_receivers(np.full(rx.size, N + 4, np.int32), rx)
    return e, rng


def sources(e, shots):
    g = e.cfg
    x = (g.n_abc + np.linspace(8, g.nx - 9, shots)).astype(np.int32)
    return (torch.full((shots,), g.n_abc + 6, dtype=torch.int32, device="cuda"), torch.as_tensor(x, device="cuda"))


def empty_data(e, shots):
    return torch.zeros((shots, e.cfg.nt_data, e.nrec), dtype=torch.float32, device="cuda")


@pytest.mark.parametrize("approx,boundary", [("acoustic", "cerjan"), ("TTI", "cerjan"), ("acoustic", "CPML"), ("VTI", "CPML")])
def test_a_queued_run_keeps_its_wavelet(approx, boundary):
    """The next wavelet is set while a run that the stream has not begun waits:
    that run models the wavelet it was queued with."""
    e, rng = make_engine(approx, boundary)
    sz, sx = sources(e, 1)
    st = torch.cuda.Stream()
    w = [rng.standard_normal(e.cfg.nt).astype(np.float32) for _ in range(2)]
    alone = []
    for v in w:
        out = empty_data(e, 1)
        torch.cuda.synchronize()
        e.set_wavelet(v)
        e.forward_device(sz, sx, out, stream=st.cuda_stream)
        torch.cuda.synchronize()
        alone.append(out.cpu().numpy())
    assert np.abs(alone[0]).max() > 0 and not np.array_equal(alone[0], alone[1])
    queued = [empty_data(e, 1) for _ in w]
    torch.cuda.synchronize()
    for v, out in zip(w, queued):
        e.set_wavelet(v)
        with torch.cuda.stream(st):
            torch.cuda._sleep(WAIT)
        e.forward_device(sz, sx, out, stream=st.cuda_stream)
    torch.cuda.synchronize()
    for a, b in zip(alone, queued):
        assert np.array_equal(a, b.cpu().numpy())


@pytest.mark.parametrize("per_shot", [False, True])
def test_batches_of_different_sizes_do_not_wait(per_shot):
    """A survey's full batches and its smaller last one, in turn and with new
    receivers in between, are queued while the stream is busy, and give what an
    engine gives that sees one batch and one set of receivers only."""
    shots, sizes = 7, (7, 2, 7, 3, 2)
    st = torch.cuda.Stream()

    def receivers(e, seed):
        rng = np.random.default_rng(seed)
        shape = (shots, 25) if per_shot else (25,)
        e.set_receivers(rng.integers(0, e.cfg.nz_abc, shape).astype(np.int32),
                        rng.integers(0, e.cfg.nx_abc, shape).astype(np.int32), per_shot=per_shot)

    def queue(e, n):
        sz, sx = sources(e, n)
        out = empty_data(e, n)
        torch.cuda.synchronize()
        return sz, sx, out

    ref = {}
    for seed in (1, 2):
        for n in set(sizes):
            e, _ = make_engine("acoustic", "cerjan", shots)
            receivers(e, seed)
            sz, sx, out = queue(e, n)
            e.forward_device(sz, sx, out, stream=st.cuda_stream)
            torch.cuda.synchronize()
            ref[seed, n] = out.cpu().numpy()
    assert all(np.abs(v).max() > 0 for v in ref.values())
    e, _ = make_engine("acoustic", "cerjan", shots)
    receivers(e, 3)
    for n in sizes:                      # each batch size's buffers
        sz, sx, out = queue(e, n)
        e.forward_device(sz, sx, out, stream=st.cuda_stream)
    runs = [(seed, n, *queue(e, n)) for seed in (1, 2) for n in sizes]
    busy = torch.cuda.Event()
    for i, (seed, n, sz, sx, out) in enumerate(runs):
        if i % len(sizes) == 0:
            torch.cuda.synchronize()     # (set_receivers replaces arrays that queued graphs read)
            receivers(e, seed)
            with torch.cuda.stream(st):
                torch.cuda._sleep(WAIT)
            busy.record(st)
        e.forward_device(sz, sx, out, stream=st.cuda_stream)
        assert not busy.query(), (i, n)
    torch.cuda.synchronize()
    for seed, n, _, _, out in runs:
        assert np.array_equal(out.cpu().numpy(), ref[seed, n])
