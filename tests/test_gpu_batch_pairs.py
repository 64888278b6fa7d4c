"""GPU: uneven batches of smooth lengths, both directions, on the kernel of two transforms
per thread: with and without the captured graph, repeated runs bit for bit the same, and
more segments than the kernel remembers as finished."""
import numpy as np
import pytest

from oracle import oracle
from sip_b200 import fft, workloads

pytestmark = pytest.mark.gpu

FWD, INV = fft.ASCEND_FFT_FORWARD, fft.ASCEND_FFT_INVERSE
SETS = {
    "one tile": [(64, 1)],
    "one pass": [(64, 37), (100, 5), (1024, 9), (1500, 3), (8, 400), (2, 9), (1536, 7)],
    "two passes": [(1452, 3), (4096, 2), (16384, 1), (32768, 2), (3 * 2 ** 13, 1), (49152, 2), (63000, 2)],
    "odd": [(1331, 2), (2197, 5), (6561, 3), (15625, 2), (16807, 1)],
    "three passes": [(2 ** 24, 1), (3 ** 8 * 2 ** 10, 1), (360, 11)],
}


def _run(groups, direction, seed):
    import torch

    rng = np.random.default_rng(seed)
    plan = fft.BatchPlan(groups, direction)
    assert "kernel=pairs" in plan.describe(), plan.describe()
    x = (rng.uniform(-1, 1, plan.total) + 1j * rng.uniform(-1, 1, plan.total)).astype(np.complex64)
    xd = torch.from_numpy(x).cuda()
    outs = []
    for graph in (False, True, True, False):
        y = torch.full_like(xd, float("nan"))
        plan(xd, y, use_graph=graph)
        plan.synchronize()
        outs.append(y)
    for y in outs[1:]:
        assert torch.equal(outs[0], y)
    got = outs[0].cpu().numpy()
    for (n, b), off in zip(plan.groups, plan.offsets):
        ref = oracle.c2c(x[off:off + n * b].reshape(b, n), direction == FWD)
        assert oracle.rel_l2(got[off:off + n * b].reshape(b, n), ref) <= oracle.tolerance(n), (n, b)
    text = plan.describe()
    plan.close()
    return text


@pytest.mark.parametrize("name", list(SETS))
@pytest.mark.parametrize("direction", [FWD, INV])
def test_sets(cuda, name, direction):
    _run(SETS[name], direction, seed=len(name))


@pytest.mark.parametrize("direction", [FWD, INV])
def test_more_segments_than_the_kernel_remembers(cuda, direction):
    lengths = [n for n in workloads.smooth_numbers(1540, 20000)]
    groups = [(lengths[i % len(lengths)], 1 + i % 2) for i in range(1100)]
    text = _run(groups, direction, seed=3)
    assert int(text.split("segments=")[1].split()[0]) > 2048, text[:200]
