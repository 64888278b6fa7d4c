"""GPU: the waits of the uneven batch's kernel end beside other work on the GPU, and a
wait that gives up is reported."""
import numpy as np
import pytest

from oracle import oracle
from sip_b200 import fft

pytestmark = pytest.mark.gpu

GROUPS = [(65536, 9), (63000, 8), (40000, 7), (1536, 70), (49152, 5), (8192, 40)]


def _data(plan, seed):
    import torch

    rng = np.random.default_rng(seed)
    x = (rng.uniform(-1, 1, plan.total) + 1j * rng.uniform(-1, 1, plan.total)).astype(np.complex64)
    return x, torch.from_numpy(x).cuda()


@pytest.mark.parametrize("direction", [fft.ASCEND_FFT_FORWARD, fft.ASCEND_FFT_INVERSE])
def test_ends_while_another_kernel_holds_part_of_an_sm(cuda, direction):
    """The grid is as large as an idle GPU holds: with a kernel of one block resident
    (about a second of spinning on the clock, then it ends), some CTA of the batch has no
    place.  The batch ends before that kernel does, with the results of an idle GPU."""
    import torch

    plan = fft.BatchPlan(GROUPS, direction)
    assert "kernel=pairs" in plan.describe()
    x, xd = _data(plan, 1)
    alone, beside = torch.zeros_like(xd), torch.zeros_like(xd)
    plan(xd, alone, use_graph=False)
    plan.synchronize()
    other, mine = torch.cuda.Stream(), torch.cuda.Stream()
    held, ended = torch.cuda.Event(), torch.cuda.Event()
    with torch.cuda.stream(other):
        torch.cuda._sleep(2_000_000_000)
        held.record(other)
    plan(xd, beside, stream=mine, use_graph=False)
    ended.record(mine)
    ended.synchronize()
    assert not held.query()
    torch.cuda.synchronize()
    plan.synchronize(mine)
    assert torch.equal(alone, beside)
    at = 0
    for n, b in GROUPS:
        ref = oracle.c2c(x[at:at + n * b].reshape(b, n), direction == fft.ASCEND_FFT_FORWARD)
        assert oracle.rel_l2(alone[at:at + n * b].cpu().numpy().reshape(b, n), ref) <= oracle.tolerance(n), n
        at += n * b
    plan.close()


def test_a_wait_that_gives_up_is_reported_once(cuda, monkeypatch):
    """With no polls allowed, the first tile whose producer is still running gives up."""
    import torch

    monkeypatch.setenv("ASDSIP_FFT_BATCH_POLLS", "0")
    plan = fft.BatchPlan([(65536, 3)])
    monkeypatch.delenv("ASDSIP_FFT_BATCH_POLLS")
    good = fft.BatchPlan([(65536, 3)])
    x, xd = _data(plan, 2)
    y = torch.zeros_like(xd)
    plan(xd, y)
    torch.cuda.synchronize()
    with pytest.raises(fft.FftError):  # the call before
        plan(xd, y)
    plan(xd, y)
    with pytest.raises(fft.FftError):
        plan.synchronize()
    plan.synchronize()
    # another plan on the device is not affected; the device's error word is an FFT plan's to report
    good(xd, y)
    good.synchronize()
    ref = oracle.c2c(x.reshape(3, 65536), True)
    assert oracle.rel_l2(y.cpu().numpy().reshape(3, 65536), ref) <= oracle.tolerance(65536)
    other = fft.FftPlan([64], fft.ASCEND_FFT_C2C, fft.ASCEND_FFT_FORWARD, 1, stream=torch.cuda.Stream())
    assert fft.asdFftSynchronize(other.handle) == fft.ACL_ERROR_INTERNAL_ERROR
    assert fft.asdFftSynchronize(other.handle) == fft.ACL_SUCCESS
    other.close()
    plan.close()
    good.close()


def test_synchronize_of_an_unknown_plan(lib):
    assert lib.asdFftBatchSynchronize(None, None) == fft.ACL_ERROR_INVALID_PARAM
