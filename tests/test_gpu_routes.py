"""GPU: calls that stay off the kernels of two transforms per thread where those lose, each
against the FP64 oracle on the route that its plan names."""
import numpy as np
import pytest

from oracle import oracle
from sip_b200 import fft

pytestmark = pytest.mark.gpu

C2C, R2C, C2R, SEP = fft.ASCEND_FFT_C2C, fft.ASCEND_FFT_R2C, fft.ASCEND_FFT_C2R, fft.ASCEND_FFT_C2C_SEP
FWD, INV = fft.ASCEND_FFT_FORWARD, fft.ASCEND_FFT_INVERSE
VERT, HORI = fft.ASCEND_FFT_VERTICAL, fft.ASCEND_FFT_HORIZONTAL


@pytest.mark.parametrize("n", [4098 + 18, 5000, 7680, 8190])
@pytest.mark.parametrize("direction", [FWD, INV])
def test_separated_long_even_rows_in_one_launch(cuda, n, direction):
    import torch

    rng = np.random.default_rng(n)
    re, im = rng.uniform(-1, 1, (2, 5, n)).astype(np.float32)
    h = fft.asdFftCreate()
    try:
        assert fft.asdFftMakePlan1D(h, n, SEP, direction, 5) == fft.ACL_SUCCESS
        assert fft.launch_count(h) == 1, fft.describe_plan(h)
        assert fft.asdFftGetWorkspaceSize(h) == (fft.ACL_SUCCESS, 0)
        fft.asdFftSetStream(h, torch.cuda.current_stream().cuda_stream or 1)
        x = [torch.from_numpy(v).cuda() for v in (re, im)]
        y = [torch.empty_like(v) for v in x]
        t = [fft.AclTensor.from_torch(v) for v in x + y]
        assert fft.load_library().asdFftExecC2CSeparated(h, *[v.ptr for v in t]) == fft.ACL_SUCCESS
        torch.cuda.synchronize()
        got = y[0].cpu().numpy() + 1j * y[1].cpu().numpy()
        assert oracle.rel_l2(got, oracle.c2c(re + 1j * im, direction == FWD)) <= oracle.tolerance(n)
    finally:
        fft.asdFftDestroy(h)


@pytest.mark.parametrize("n,batch,vertical,steps", [(4116, 5, False, 1), (5000, 4, False, 1), (8190, 3, False, 1),
                                                    (9000, 3, False, 2), (1000000, 1, False, 2), (9000, 7, True, 2)])
@pytest.mark.parametrize("direction", [FWD, INV])
def test_complex32_route(cuda, n, batch, vertical, steps, direction):
    """complex32 data takes the tile kernel's own route (FP16 in and out, FP32 between): the
    result is the FP64 one to the rounding of the outputs, 2^-11 relative each; 1e-3 as for
    the other lengths."""
    import torch

    rng = np.random.default_rng(n + batch)
    shape = (n, batch) if vertical else (batch, n)
    xh = rng.uniform(-1, 1, shape + (2,)).astype(np.float16)
    xd = torch.from_numpy(xh).cuda()
    yd = torch.full_like(xd, float("nan"))
    plan = fft.FftPlan([n], C2C, direction, batch, VERT if vertical else HORI)
    assert "complex32 data" in plan.describe() and f": steps={steps}\n" in plan.describe(), plan.describe()
    a = fft.AclTensor(shape, fft.ACL_COMPLEX32, xd.data_ptr())
    b = fft.AclTensor(shape, fft.ACL_COMPLEX32, yd.data_ptr())
    assert fft.asdFftExecC2C(plan.handle, a, b) == fft.ACL_SUCCESS
    torch.cuda.synchronize()
    y = yd.cpu().numpy().astype(np.float64)
    x = xh.astype(np.float64)
    x, got = x[..., 0] + 1j * x[..., 1], y[..., 0] + 1j * y[..., 1]
    ref = oracle.c2c(x.T, direction == FWD).T if vertical else oracle.c2c(x, direction == FWD)
    assert oracle.rel_l2(got, ref) <= 1e-3
    # interleaved FP32 data of the same plan
    xc = torch.from_numpy(x.astype(np.complex64)).cuda()
    yc = torch.empty_like(xc)
    plan(xc, yc)
    torch.cuda.synchronize()
    assert oracle.rel_l2(yc.cpu().numpy(), ref) <= oracle.tolerance(n)
    for t in (a, b):
        t.close()
    plan.close()


def _check(sizes, typ, direction, batch, seed, vertical=False, shift=0):
    import torch

    rng = np.random.default_rng(seed)
    fwd, nd = direction == FWD, len(sizes)
    shape = [sizes[0], batch] if vertical else [batch] + list(sizes)
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
    plan = fft.FftPlan(sizes, typ, direction, batch, VERT if vertical else HORI)
    y = torch.empty(ref.shape, dtype=torch.complex64 if np.iscomplexobj(ref) else torch.float32, device="cuda")
    # shift: the source starts `shift` complex elements into a 16-byte aligned buffer
    x, skip = torch.from_numpy(np.ascontiguousarray(x)), shift * (1 if np.iscomplexobj(x) else 2)
    xd = torch.empty(x.numel() + skip, dtype=x.dtype, device="cuda")[skip:].view(x.shape)
    xd.copy_(x)
    plan(xd, y)
    torch.cuda.synchronize()
    assert oracle.rel_l2(y.cpu().numpy(), ref) <= oracle.tolerance(int(np.prod(sizes))), plan.describe()
    text = plan.describe()
    plan.close()
    return text


@pytest.mark.parametrize("n", [2, 3, 5, 6, 7, 8, 9, 13, 14, 15])
@pytest.mark.parametrize("direction", [FWD, INV])
def test_short_rows(cuda, n, direction):
    """Many rows of fewer than 14 points (packed points of C2R rows; of R2C rows fewer than 6,
    and 8) on the tile kernel."""
    for typ, k in ((C2C, n), (R2C, 2 * n), (C2R, 2 * n)):
        for batch in (1031, 65536):
            text = _check([k], typ, direction, batch, seed=n)
            pairs = (n >= 6 and n != 8 if typ == R2C else n >= 14) or batch < 65536
            _check([k], typ, direction, batch, seed=n, shift=1)
            assert ("[pair tiles]" in text) == (pairs and "static" not in text), text


@pytest.mark.parametrize("xy", [(3, 7), (8, 8), (8, 33), (9, 16), (9, 17), (16, 12), (16, 24), (30, 9), (32, 16), (33, 9),
                                (36, 2)])
@pytest.mark.parametrize("direction", [FWD, INV])
def test_short_narrow_columns(cuda, xy, direction):
    """Columns of up to 32 points, at most 16 of them (32 below 9 points), on the tile kernel
    beyond one or two waves of tiles."""
    x, y = xy
    for batch in (21, 1300):
        text = _check([x, y], C2C, direction, batch, seed=x)
        columns = [l for l in text.splitlines() if "[1->1]" in l]
        assert len(columns) == 1
        few = x <= 32 and y <= (16 if x >= 9 else 32) and batch > 21
        assert ("[pair tiles]" in columns[0]) == (not few), text
    _check([x, 2 * y], R2C, direction, 1300, seed=x)
    _check([x, 2 * y], C2R, direction, 1300, seed=x)


@pytest.mark.parametrize("n", [17, 23, 31, 34, 37])
@pytest.mark.parametrize("direction", [FWD, INV])
def test_short_bluestein(cuda, n, direction):
    """Convolutions of up to 64 points of many rows in two launches, others in one kernel."""
    for typ in (C2C, R2C, C2R):
        for batch in (3, 333, 16385):
            text = _check([n], typ, direction, batch, seed=n)
            assert ("in one kernel" in text) == (2 * n - 1 > 64 or batch <= (16 if typ == C2R else 16384)), text


@pytest.mark.parametrize("n,batch,passes", [(4374, 8, 2), (4374, 900, 1), (4410, 8, 2), (4410, 900, 1), (4368, 900, 2),
                                            (5082, 800, 1), (5000, 800, 2), (7680, 500, 2), (6561, 40, 1)])
def test_long_rows_without_an_engine(cuda, n, batch, passes):
    """4097..8192 points: one tile or two passes, by length and size of the data; in place and
    from an unaligned source two passes where the length splits."""
    import torch

    text = _check([n], C2C, FWD, batch, seed=n)
    _check([n], C2C, FWD, min(batch, 40), seed=n, shift=1)
    splits = n % 2 == 0
    assert text.startswith(f"steps={2 if splits else 1} "), text
    assert ("out of place from an aligned source: steps=1" in text) == (splits and passes == 1), text
    plan = fft.FftPlan([n], C2C, INV, batch)
    assert plan.launches() == passes
    rng = np.random.default_rng(n)
    x = (rng.uniform(-1, 1, (batch, n)) + 1j * rng.uniform(-1, 1, (batch, n))).astype(np.complex64)
    y = torch.from_numpy(x).cuda()
    plan(y, y)
    torch.cuda.synchronize()
    assert oracle.rel_l2(y.cpu().numpy(), oracle.c2c(x, False)) <= oracle.tolerance(n)
    plan.close()


@pytest.mark.parametrize("xy,batch,one", [((500, 7), 30, True), ((500, 15), 30, True), ((500, 16), 30, False),
                                          ((729, 729), 2, False), ((729, 729), 6, True), ((729, 64), 3, False), ((945, 33), 3, False),
                                          ((1000, 2), 3, True), ((1040, 2), 3, False)])
def test_strided_axis_in_one_or_two_passes(cuda, xy, batch, one):
    text = _check(list(xy), C2C, INV, batch, seed=xy[0])
    assert ("strided x" not in text) == one, text


def test_data_too_large_to_hold_once_more(cuda):
    """Planning only: routes that need a copy of the data as workspace where another route
    does not are taken while input, output and that copy fit the device."""
    import torch

    quarter = torch.cuda.mem_get_info()[1] // 4
    for sizes in ([600, 600], [5000]):
        points = int(np.prod(sizes))
        for batch, fits in ((quarter // (8 * points), True), (quarter // (8 * points) + 1, False)):
            h = fft.asdFftCreate()
            st = (fft.asdFftMakePlan1D(h, sizes[0], C2C, FWD, batch) if len(sizes) == 1 else
                  fft.asdFftMakePlan2D(h, *sizes, C2C, FWD, batch))
            assert st == fft.ACL_SUCCESS
            assert (fft.asdFftGetWorkspaceSize(h)[1] > 0) == fits, fft.describe_plan(h)
            fft.asdFftDestroy(h)
    for rows, fits in ((quarter // (8 * 64), True), (quarter // (8 * 64) + 1, False)):  # 31 points by 64
        h = fft.asdFftCreate()
        assert fft.asdFftMakePlan1D(h, 31, C2C, FWD, rows) == fft.ACL_SUCCESS
        assert (fft.asdFftGetWorkspaceSize(h)[1] > 0) == fits and ("in one kernel" in fft.describe_plan(h)) != fits
        fft.asdFftDestroy(h)
    import ctypes

    lib = fft.load_library()
    for batch, fits in ((quarter // (8 * 2000), True), (quarter // (8 * 2000) + 1, False)):
        h, need = ctypes.c_void_p(), ctypes.c_size_t()
        one = lambda v: (ctypes.c_int64 * 1)(v)
        assert lib.asdFftBatchPlanCreate(ctypes.byref(h), one(2000), one(batch), 1, FWD, None) == fft.ACL_SUCCESS
        assert lib.asdFftBatchGetWorkspaceSize(h, ctypes.byref(need)) == fft.ACL_SUCCESS
        assert (need.value > 0) == fits
        lib.asdFftBatchPlanDestroy(h)


def test_tuned_sequence_without_a_pair_tile(cuda, tmp_path):
    """A cache entry whose radices have no pair tile does not take the whole uneven batch to
    the one-transform kernel: the planner's own radices stand in."""
    import json

    import torch

    path = str(tmp_path / "tune.jsonl")
    entries = {1440: [12, 12, 10], 1296: [9, 12, 12], 1536: [8, 16, 12], 500: [10, 5, 10]}
    with open(path, "w") as f:
        for n, r in entries.items():
            f.write(json.dumps({"gpu": torch.cuda.get_device_name(0), "type": "c2c", "precision": "fp32", "n": n,
                                "radices": r, "maxe": 16, "row_threads": 256, "us": 1.0, "plan_us": 0}) + "\n")
    groups = [(n, 7) for n in entries]
    for direction in (FWD, INV):
        plan = fft.BatchPlan(groups, direction, path)
        text = plan.describe()
        assert "kernel=pairs" in text, text
        assert "n=500 tiles" in text and "radices=10x5x10" in text, text  # (an entry that fits is used)
        rng = np.random.default_rng(5)
        x = (rng.uniform(-1, 1, plan.total) + 1j * rng.uniform(-1, 1, plan.total)).astype(np.complex64)
        y = torch.zeros(plan.total, dtype=torch.complex64, device="cuda")
        plan(torch.from_numpy(x).cuda(), y)
        plan.synchronize()
        for (n, b), off in zip(plan.groups, plan.offsets):
            got = y[off:off + n * b].cpu().numpy().reshape(b, n)
            assert oracle.rel_l2(got, oracle.c2c(x[off:off + n * b].reshape(b, n), direction == FWD)) <= oracle.tolerance(n)
        plan.close()
    # (the choices stay with the process: empty ones give the lengths back to the planner)
    with open(path, "w") as f:
        for n in entries:
            f.write(json.dumps({"gpu": torch.cuda.get_device_name(0), "type": "c2c", "precision": "fp32", "n": n,
                                "radices": [], "maxe": 0, "row_threads": 0, "us": 0, "plan_us": 0}) + "\n")
    assert fft.tune_cache_load(path) == len(entries)


def test_launch_count_of_many_bluestein_rows(cuda):
    """The one-kernel form is one launch whatever the number of rows."""
    plan = fft.FftPlan([37], C2C, FWD, 70000)
    assert "in one kernel" in plan.describe() and plan.launches() == 1
    plan.close()


def test_autotune_takes_the_lengths_that_have_tiles(cuda, tmp_path):
    """The tuner's lengths are those of the launch's tiles: passes as the planner splits them,
    and no rows that are two passes."""
    import json
    import re

    import torch

    path = str(tmp_path / "tune.jsonl")
    groups = [(2200, 40), (4400, 20), (1470, 64), (735, 64), (14300, 9)]
    plan = fft.BatchPlan(groups, INV)
    assert "kernel=pairs" in plan.describe()
    tiles = {int(n) for n in re.findall(r" n=(\d+) tiles=", plan.describe())}
    plan.close()
    assert fft.autotune(groups, INV, path) == fft.ACL_SUCCESS
    lines = [json.loads(l) for l in open(path)]
    assert tiles <= {l["n"] for l in lines}
    assert not {2200, 4400, 14300} & {l["n"] for l in lines}
    plan = fft.BatchPlan(groups, INV, path)
    assert "kernel=pairs" in plan.describe()
    rng = np.random.default_rng(6)
    x = (rng.uniform(-1, 1, plan.total) + 1j * rng.uniform(-1, 1, plan.total)).astype(np.complex64)
    y = torch.zeros(plan.total, dtype=torch.complex64, device="cuda")
    plan(torch.from_numpy(x).cuda(), y)
    plan.synchronize()
    for (n, b), off in zip(plan.groups, plan.offsets):
        got = y[off:off + n * b].cpu().numpy().reshape(b, n)
        assert oracle.rel_l2(got, oracle.c2c(x[off:off + n * b].reshape(b, n), False)) <= oracle.tolerance(n)
    plan.close()
