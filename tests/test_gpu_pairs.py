"""GPU parity of the kernels that transform two rows or columns per thread: tile
edges (odd and single rows and columns, fewer columns than a tile), every first
radix, column outputs that cross blocks, sources that are 8-byte aligned only, and
the one-kernel Bluestein transform up to its longest convolution."""
import numpy as np
import pytest

from oracle import oracle
from sip_b200 import fft

pytestmark = pytest.mark.gpu

C2C, R2C, C2R = fft.ASCEND_FFT_C2C, fft.ASCEND_FFT_R2C, fft.ASCEND_FFT_C2R
FWD, INV = fft.ASCEND_FFT_FORWARD, fft.ASCEND_FFT_INVERSE


def _check(sizes, typ, direction, batch, seed, vertical=False, shift=0):
    import torch

    rng = np.random.default_rng(seed)
    shape = [batch] + list(sizes) if not vertical else [sizes[0], batch]
    fwd, nd = direction == FWD, len(sizes)
    if typ == R2C:
        x = rng.standard_normal(shape).astype(np.float32)
        ref = oracle.r2c(x, fwd, nd)
    elif typ == C2R:
        shape[-1] = sizes[-1] // 2 + 1
        x = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
        ref = oracle.c2r(x, sizes[-1], fwd, nd)
    else:
        x = (rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape)).astype(np.complex64)
        ref = oracle.c2c(x.T, fwd).T if vertical else oracle.c2c(x, fwd, nd)
    plan = fft.FftPlan(sizes, typ, direction, batch,
                       fft.ASCEND_FFT_VERTICAL if vertical else fft.ASCEND_FFT_HORIZONTAL)
    # shift: the data starts `shift` complex elements into 16-byte aligned buffers
    per = 1 if np.iscomplexobj(x) else 2
    flat = torch.zeros(x.size + 4 * per, dtype=torch.complex64 if per == 1 else torch.float32, device="cuda")
    xd = flat[shift * per:shift * per + x.size].view(x.shape)
    xd.copy_(torch.from_numpy(x))
    od = torch.complex64 if np.iscomplexobj(ref) else torch.float32
    oper = 1 if np.iscomplexobj(ref) else 2
    out = torch.full((ref.size + 4 * oper,), 7.0, dtype=od, device="cuda")
    y = out[shift * oper:shift * oper + ref.size].view(ref.shape)
    plan(xd, y)
    torch.cuda.synchronize()
    n = int(np.prod(sizes))
    assert oracle.rel_l2(y.cpu().numpy(), ref) <= oracle.tolerance(n), plan.describe()
    rest = torch.cat([out[:shift * oper], out[shift * oper + ref.size:]])
    assert bool((rest == 7.0).all())  # nothing written around the outputs
    return plan


@pytest.mark.parametrize("n", [2, 7, 13, 16, 22, 33, 75, 98, 105, 169, 182, 240, 441, 480, 770, 960, 1210, 1536])
@pytest.mark.parametrize("batch", [1, 2, 37])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows(cuda, n, batch, shift):
    for typ, k in ((C2C, n), (R2C, 2 * n), (C2R, 2 * n)):
        _check([k], typ, FWD if batch != 2 else INV, batch, seed=n + batch, shift=shift)


@pytest.mark.parametrize("xy", [(9, 5), (14, 15), (30, 17), (96, 1), (100, 33), (135, 6), (210, 31), (256, 9), (300, 7),
                                (441, 12), (720, 15), (1080, 25), (2000, 3)])
@pytest.mark.parametrize("direction", [FWD, INV])
def test_columns(cuda, xy, direction):
    _check(list(xy), C2C, direction, 3, seed=xy[0], shift=xy[1] % 2)
    if xy[0] * xy[1] > 100:
        _check([xy[0], 2 * xy[1]], R2C, direction, 2, seed=xy[0] + 1)


@pytest.mark.parametrize("n,cols", [(64, 17), (128, 16), (256, 15), (512, 3), (1024, 2), (2048, 5), (375, 9), (4096, 6),
                                    (15000, 3), (65536, 2)])
def test_vertical(cuda, n, cols):
    _check([n], C2C, FWD, cols, seed=n, vertical=True)
    _check([n], C2C, INV, cols, seed=n + 1, vertical=True, shift=1)


@pytest.mark.parametrize("n", [2500, 8748, 16807, 30030, 52920, 59049, 110592, 262144])
@pytest.mark.parametrize("batch", [1, 3])
def test_long_rows(cuda, n, batch):
    _check([n], C2C, FWD, batch, seed=n)
    _check([n], C2C, INV, batch, seed=n + 1, shift=1)


@pytest.mark.parametrize("n", [17, 19, 34, 127, 257, 509, 1021, 1024 - 1, 1031])
@pytest.mark.parametrize("batch", [1, 2, 5, 300])
def test_bluestein(cuda, n, batch):
    for typ in (C2C, R2C, C2R):
        for direction in (FWD, INV):
            plan = _check([n], typ, direction, batch, seed=n + batch)
            if n == 1021 and typ == C2C:
                assert plan.launches() == 1, plan.describe()


def test_bluestein_in_place(cuda):
    import torch

    rng = np.random.default_rng(3)
    x = (rng.uniform(-1, 1, (41, 509)) + 1j * rng.uniform(-1, 1, (41, 509))).astype(np.complex64)
    xd = torch.from_numpy(x).cuda()
    fft.FftPlan([509], C2C, FWD, 41)(xd, xd)
    torch.cuda.synchronize()
    assert oracle.rel_l2(xd.cpu().numpy(), oracle.c2c(x, True)) <= oracle.tolerance(509)


@pytest.mark.parametrize("groups", [[(64, 1)], [(1452, 3), (1331, 2), (2197, 5)], [(4096, 3), (8192, 1), (49152, 2)],
                                    [(65536, 3), (63000, 2), (40000, 1), (2, 9), (1536, 7)]])
def test_uneven_pairs(cuda, groups):
    import torch

    rng = np.random.default_rng(len(groups))
    plan = fft.BatchPlan(groups, FWD)
    assert "kernel=pairs" in plan.describe(), plan.describe()
    x = (rng.uniform(-1, 1, plan.total) + 1j * rng.uniform(-1, 1, plan.total)).astype(np.complex64)
    xd = torch.from_numpy(x).cuda()
    for graph in (False, True, True):
        y = torch.zeros_like(xd)
        plan(xd, y, use_graph=graph)
        torch.cuda.synchronize()
        got, at = y.cpu().numpy(), 0
        for n, b in groups:
            ref = oracle.c2c(x[at:at + n * b].reshape(b, n), True)
            assert oracle.rel_l2(got[at:at + n * b].reshape(b, n), ref) <= oracle.tolerance(n), (n, b)
            at += n * b
    plan.close()
