"""Evaluations on device buffers are in order with the work queued on the stream they are
given, the legacy default stream (torch's own default, handle 0) among them."""
import numpy as np
import pytest

import atmmetaforce as atm
from atmmetaforce import synthetic as S
from atmmetaforce._lib import NUM_RES

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

BUSY = 20_000_000  # clock cycles a stream is kept busy: 10 ms, far more than an evaluation


def _case(seed=31):
    return S.water_ligand_box(2100, 2.8, [13], [(1.3, 1.2, 1.1)], S.PME, 0.9, seed=seed, use_disp_corr=False)


@pytest.mark.parametrize("own_stream", [False, True], ids=["default", "side"])
def test_positions_queued_on_the_stream_are_evaluated(own_stream):
    """Positions that a long chain on the stream has yet to write, and forces that a long
    chain has yet to read, when the call is made."""
    case = _case()
    batch = atm.ReplicaBatch([atm.system_from_case(case)[0]], 0, {"DifferencePath": 1})
    first = torch.as_tensor(case.pos, device="cuda")
    moved = first + 0.01 * torch.sin(torch.arange(first.numel(), device="cuda", dtype=torch.float64)).reshape(-1, 3)
    want = [batch.evaluate(p.cpu().numpy())[1] for p in (first, moved)]
    assert not np.array_equal(want[0], want[1])
    stream = torch.cuda.Stream() if own_stream else torch.cuda.default_stream()
    pos, f = first.clone(), torch.empty_like(first)
    r = torch.empty(1, NUM_RES, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        batch.evaluateDevice(pos.data_ptr(), f.data_ptr(), r.data_ptr(), stream.cuda_stream)
        torch.cuda._sleep(BUSY)
        before = f.clone()
        pos.copy_(moved)
        batch.evaluateDevice(pos.data_ptr(), f.data_ptr(), r.data_ptr(), stream.cuda_stream)
        after = f.clone()
    torch.cuda.synchronize()
    assert np.array_equal(before.cpu().numpy(), want[0])
    assert np.array_equal(after.cpu().numpy(), want[1])


@pytest.mark.parametrize("second", ["host", "default", "side"])
def test_gradients_are_those_of_the_evaluation_before_them(second):
    """Gradients queued behind 10 ms of other work, and an evaluation of other positions
    asked for on another stream meanwhile; gradients on two streams before it."""
    case = _case(32)
    batch = atm.ReplicaBatch([atm.system_from_case(case)[0]], 0, {"DifferencePath": 1, "Adjoint": 1})
    first = torch.as_tensor(case.pos, device="cuda")
    moved = first + 0.01 * torch.cos(torch.arange(first.numel(), device="cuda", dtype=torch.float64)).reshape(-1, 3)
    g = torch.ones(1, dtype=torch.float64, device="cuda")
    f = torch.empty_like(first)
    r = torch.empty(1, NUM_RES, dtype=torch.float64, device="cuda")
    batch.evaluate(case.pos)
    want = batch.backward()
    streams = [torch.cuda.Stream(), torch.cuda.Stream() if second != "side" else torch.cuda.default_stream()]
    dx = [torch.zeros_like(first) for _ in streams]
    dq = [torch.zeros(case.n, dtype=torch.float64, device="cuda") for _ in streams]
    torch.cuda.synchronize()
    for k, s in enumerate(streams):
        with torch.cuda.stream(s):
            torch.cuda._sleep(BUSY)
        batch.backwardDevice(g.data_ptr(), dx[k].data_ptr(), d_dq=dq[k].data_ptr(), stream=s.cuda_stream)
    if second == "host":
        batch.evaluate(moved.cpu().numpy())
    else:
        s = torch.cuda.Stream() if second == "side" else torch.cuda.default_stream()
        batch.evaluateDevice(moved.data_ptr(), f.data_ptr(), r.data_ptr(), s.cuda_stream)
    torch.cuda.synchronize()
    for k in range(2):
        assert np.array_equal(dx[k].cpu().numpy(), want["positions"])
        assert np.array_equal(dq[k].cpu().numpy(), want["charge"])
    assert not np.array_equal(batch.backward()["positions"], want["positions"])
