"""Workloads of the FFT library that its speed is judged on.

``listed()`` names a dozen calls over the range that a program makes of the library: small and
launch-bound batches, the batched real transforms of the benchmark, long rows, 2D and 3D volumes,
lengths that are no power of two, prime lengths, the uneven batch, the inverse STFT, the tensor-core
split form and a burst into the server.  ``draw`` gives more calls of the same ranges.  ``prepare``
builds inputs and plan, ``run`` makes one pass through the public entry points, ``exact`` is the same
pass in FP64 through torch.fft.
"""
import math

import numpy as np
import torch

from sip_b200 import fft
from sip_b200.workloads import smooth_numbers, uneven_batch_set, uneven_flops_bytes

TYPES = {"c2c": fft.ASCEND_FFT_C2C, "r2c": fft.ASCEND_FFT_R2C, "c2r": fft.ASCEND_FFT_C2R}
PRECISIONS = {"fp32": fft.PRECISION_FP32, "fp16x3": fft.PRECISION_FP16X3, "bf16x3": fft.PRECISION_BF16X3}
SERVED = (4096, 8192, 16384, 65536)  # lengths that the server's clients ask for


def plan_case(sizes, batch, typ="c2c", inverse=False, vertical=False, precision="fp32", name=None):
    case = {} if name is None else {"name": name}
    case.update(kind="plan", sizes="x".join(str(s) for s in sizes), batch=batch, type=typ, inverse=inverse,
                vertical=vertical, precision=precision)
    return case


def listed():
    return [
        # one small batch of a radar or comms frame: 4 MB, bound by latency and the launch
        plan_case([1024], 256, name="c2c 1024 x 256"),
        # the benchmark's spectrum of a mixed-radix real batch ...
        plan_case([3000], 4096, "r2c", name="r2c 3000 x 4096"),
        # ... and the way back of its power-of-two one
        plan_case([4096], 4096, "c2r", inverse=True, name="c2r 4096 x 4096"),
        # long rows, two passes over memory: the longest transform that the server's clients ask for
        plan_case([65536], 256, name="c2c 65536 x 256"),
        # images: 2D, strided second axis
        plan_case([2048, 2048], 8, name="c2c 2048^2 x 8"),
        # a volume: 3D, two strided axes
        plan_case([256, 256, 256], 1, inverse=True, name="c2c 256^3 inverse"),
        # video frames, real to half spectrum: both axes mixed radix
        plan_case([1080, 1920], 8, "r2c", name="r2c 1080 x 1920 x 8"),
        # a prime length (chirp convolution)
        plan_case([1021], 4096, name="c2c 1021 x 4096"),
        # the tensor-core split form of batched rows
        plan_case([4096], 4096, precision="fp16x3", name="c2c 4096 x 4096 fp16x3"),
        # many transforms of many lengths in one launch: the uneven-batch workload
        {"name": "uneven 20000", "kind": "uneven", "total": 20000, "lo": 64, "hi": 65536, "set": 2024, "inverse": False},
        # resynthesis of 16 channels of 10 s speech (16 kHz, 25 ms frames, 10 ms hop)
        {"name": "istft 400/160 16 x 1000", "kind": "istft", "n_fft": 400, "hop": 160, "frames": 1000, "channels": 16},
        # a burst of requests of mixed lengths, types and rows into the server, device buffers
        {"name": "serve 16 requests", "kind": "serve", "requests": 16, "rows_min": 64, "rows_max": 1024, "lanes": 4,
         "set": 11},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(rng, lo, hi):
    """A length with prime factors up to 7, log-uniform; a power of two in one of three."""
    if rng.random() < 1 / 3:
        return 1 << rng.randint(math.ceil(math.log2(lo)), int(math.log2(hi)))
    x = _log(rng, lo, hi)
    return min(smooth_numbers(lo, hi), key=lambda s: abs(math.log(s / x)))


def draw(rng):
    what = rng.choice(["rows"] * 6 + ["2d"] * 3 + ["3d"] * 2 + ["vertical", "prime", "uneven", "istft", "split", "serve"])
    points = _log(rng, 1 << 14, 1 << 24)
    inverse = rng.random() < 0.5
    typ = rng.choice(["c2c", "c2c", "r2c", "c2r"])
    if what == "rows":
        n = _smooth(rng, 64, 1 << 18)
        return plan_case([n], max(1, points // n), typ, inverse)
    if what == "2d":
        x, y = _smooth(rng, 16, 4096), _smooth(rng, 32, 4096)
        return plan_case([x, y], max(1, points // (x * y)), typ, inverse)
    if what == "3d":
        x, y, z = (_smooth(rng, 8, 256) for _ in range(3))
        return plan_case([x, y, z], max(1, points // (x * y * z)), typ, inverse)
    if what == "vertical":
        n = 1 << rng.randint(5, 16)
        return plan_case([n], max(2, points // n), "c2c", inverse, vertical=True)
    if what == "prime":
        n = rng.choice([17, 31, 127, 509, 1021, 2039, 4093, 8191, 16381, 65537])
        return plan_case([n], max(1, points // 8 // n), typ, inverse)
    if what == "split":
        n = rng.choice([1024, 2048, 4096])
        return plan_case([n], max(64, points // n), "c2c", inverse, precision=rng.choice(["fp16x3", "bf16x3"]))
    if what == "uneven":
        return {"kind": "uneven", "total": _log(rng, 64, 8000), "lo": 64, "hi": rng.choice([4096, 16384, 65536]),
                "set": rng.randrange(1 << 20), "inverse": inverse}
    if what == "istft":
        n_fft, hop = rng.choice([(256, 64), (400, 160), (512, 128), (1000, 250), (1024, 256), (2048, 512)])
        return {"kind": "istft", "n_fft": n_fft, "hop": hop, "frames": rng.randint(20, 2000), "channels": rng.randint(1, 8)}
    return {"kind": "serve", "requests": rng.randint(4, 16), "rows_min": 64, "rows_max": rng.randint(128, 800),
            "lanes": 4, "set": rng.randrange(1 << 20)}


# ---------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _real(shape, g):
    return torch.randn(shape, device="cuda", generator=g)


def _complex(shape, g):
    """Uniform[-1, 1] real and imaginary parts."""
    return torch.view_as_complex(torch.rand(tuple(shape) + (2,), device="cuda", generator=g).mul_(2).sub_(1))


def _half_spectrum(shape, n, g):
    """Half spectrum of a real signal along the last axis (real first and middle bins)."""
    x = torch.randn(tuple(shape[:-1]) + (n // 2 + 1, 2), device="cuda", generator=g)
    x[..., 0, 1] = 0
    if n % 2 == 0:
        x[..., n // 2, 1] = 0
    return torch.view_as_complex(x)


def _sizes(case):
    return [int(s) for s in case["sizes"].split("x")]


def _plan_input(case, seed):
    sizes, g = _sizes(case), _gen(seed)
    full = [case["batch"]] + sizes
    if case["vertical"]:
        full = [sizes[0], case["batch"]]
    if case["type"] == "r2c":
        return _real(full, g)
    if case["type"] == "c2r":
        x = _half_spectrum(full, sizes[-1], g)
        # several axes: the spectrum of a real volume, so that its edge planes are Hermitian as well
        if len(sizes) > 1:
            v = _real(full, g)
            x = torch.fft.rfftn(v, dim=tuple(range(1, 1 + len(sizes)))).contiguous()
        return x
    return _complex(full, g)


def _groups(case):
    return uneven_batch_set(case["total"], case["lo"], case["hi"], seed=case["set"])


def _requests(case):
    """[(type, length, rows), ...] of a burst."""
    rng = np.random.default_rng(case["set"])
    return [(("c2c", "r2c")[int(rng.integers(2))], SERVED[int(rng.integers(len(SERVED)))],
             int(rng.integers(case["rows_min"], case["rows_max"] + 1))) for _ in range(case["requests"])]


def _served_inputs(case, seed):
    g = _gen(seed)
    return [_complex((rows, n), g) if t == "c2c" else _real((rows, n), g) for t, n, rows in _requests(case)]


def _istft_input(case, seed):
    """Frame spectra, [channel, n_fft, frames], and a Hann window with a small floor."""
    g = _gen(seed)
    x = _complex((case["channels"], case["n_fft"], case["frames"]), g)
    w = torch.hann_window(case["n_fft"], device="cuda") + 0.05
    return x, w


def _istft_length(case):
    return case["n_fft"] + case["hop"] * (case["frames"] - 1) - 2 * (case["n_fft"] // 2)


# ---------------------------------------------------------------------------------------- the call
class _Istft:
    """Handle, workspace and tensor descriptors of an inverse STFT."""

    def __init__(self, case, x, window):
        lib = fft.load_library()
        self.handle = fft.asdFftCreate()
        self.y = torch.empty((case["channels"], _istft_length(case)), dtype=torch.complex64, device="cuda")
        self.args = [fft.AclTensor.from_torch(t) for t in (x, window, self.y)]
        st = lib.asdFftIstftMakePlan(self.handle, self.args[0].ptr, case["n_fft"], case["hop"], case["n_fft"], True,
                                     False, False, 0, True)
        if st != fft.ACL_SUCCESS:
            raise fft.FftError("asdFftIstftMakePlan", st)
        _, need = fft.asdFftGetWorkspaceSize(self.handle)
        self.workspace = torch.empty(max(1, need), dtype=torch.uint8, device="cuda")
        fft.asdFftSetWorkspace(self.handle, self.workspace.data_ptr())
        fft.asdFftSetStream(self.handle, torch.cuda.current_stream().cuda_stream)

    def __call__(self):
        st = fft.load_library().asdFftExecIstft(self.handle, *[a.ptr for a in self.args])
        if st != fft.ACL_SUCCESS:
            raise fft.FftError("asdFftExecIstft", st)
        return self.y

    def __del__(self):
        fft.asdFftDestroy(self.handle)


def prepare(case, seed):
    direction = fft.ASCEND_FFT_INVERSE if case.get("inverse") else fft.ASCEND_FFT_FORWARD
    if case["kind"] == "plan":
        x = _plan_input(case, seed)
        sizes = _sizes(case)
        shape = list(x.shape)
        if case["type"] == "r2c":
            shape[-1] = sizes[-1] // 2 + 1
        if case["type"] == "c2r":
            shape[-1] = sizes[-1]
        y = torch.empty(shape, device="cuda", dtype=torch.float32 if case["type"] == "c2r" else torch.complex64)
        dim = fft.ASCEND_FFT_VERTICAL if case["vertical"] else fft.ASCEND_FFT_HORIZONTAL
        plan = fft.FftPlan(sizes, TYPES[case["type"]], direction, case["batch"], dim,
                           precision=PRECISIONS[case["precision"]])
        return {"kind": "plan", "plan": plan, "in": x, "out": y}
    if case["kind"] == "uneven":
        groups = _groups(case)
        x = _complex((sum(n * b for n, b in groups),), _gen(seed))
        return {"kind": "uneven", "plan": fft.BatchPlan(groups, direction), "in": x, "out": torch.empty_like(x)}
    if case["kind"] == "istft":
        x, w = _istft_input(case, seed)
        return {"kind": "istft", "plan": _Istft(case, x, w), "in": x, "window": w}
    ins = _served_inputs(case, seed)
    reqs, outs = [], []
    for (t, n, rows), x in zip(_requests(case), ins):
        y = torch.empty((rows, n if t == "c2c" else n // 2 + 1), dtype=torch.complex64, device="cuda")
        outs.append(y)
        reqs.append((TYPES[t], n, rows, x.data_ptr(), y.data_ptr()))
    server = fft.Server(lanes=case["lanes"], max_rows=case["rows_max"], device_io=True)
    for t, n in sorted({(r[0], r[1]) for r in reqs}):
        server.warm(t, fft.ASCEND_FFT_FORWARD, n)
    torch.cuda.synchronize()  # the server's own streams read the inputs
    return {"kind": "serve", "server": server, "requests": reqs, "in": ins, "out": outs}


def run(state):
    if state["kind"] in ("plan", "uneven"):
        return state["plan"](state["in"], state["out"])
    if state["kind"] == "istft":
        return state["plan"]()
    server = state["server"]
    for typ, n, rows, src, dst in state["requests"]:
        server.submit(typ, fft.ASCEND_FFT_FORWARD, n, rows, src, dst)
    server.drain(len(state["requests"]))
    return state["out"]


# ---------------------------------------------------------------------------------------- what it needs
def _cost(n_total, rows, typ, line):
    """Bytes and operations of `rows` transforms of n_total points whose last axis is `line` long."""
    half = n_total // line * (line // 2 + 1)
    flops = 5.0 * n_total * math.log2(max(2, n_total)) * rows
    if typ == "c2c":
        return 16 * n_total * rows, flops
    return (4 * n_total + 8 * half) * rows, flops / 2


def work(case):
    if case["kind"] == "plan":
        sizes = _sizes(case)
        by, fl = _cost(math.prod(sizes), case["batch"], case["type"], sizes[-1])
    elif case["kind"] == "uneven":
        fl, by = uneven_flops_bytes(_groups(case))
    elif case["kind"] == "istft":
        n, frames = case["n_fft"], case["frames"] * case["channels"]
        by, fl = _cost(n, frames, "c2c", n)
        by = by // 2 + 4 * n + 8 * case["channels"] * _istft_length(case)
        fl += 4.0 * n * frames
    else:
        costs = [_cost(n, rows, t, n) for t, n, rows in _requests(case)]
        by, fl = sum(c[0] for c in costs), sum(c[1] for c in costs)
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------------------------------- FP64
def _c2c64(x, dims, inverse):
    x = x.to(torch.complex128)
    if inverse:
        return torch.fft.ifftn(x, dim=dims, norm="forward")
    return torch.fft.fftn(x, dim=dims)


def _plan64(case, x):
    """Forward is exp(-i), inverse exp(+i), for every type; nothing is scaled."""
    sizes, inverse = _sizes(case), case["inverse"]
    dims = (0,) if case["vertical"] else tuple(range(1, 1 + len(sizes)))
    if case["type"] == "c2c":
        return _c2c64(x, dims, inverse)
    if case["type"] == "r2c":
        y = torch.fft.rfftn(x.double(), dim=dims)
        if inverse:  # real input: the other sign conjugates the spectrum
            y = torch.conj(y).resolve_conj()
        return y
    x = x.to(torch.complex128)
    if not inverse:  # real output: the other sign conjugates the input
        x = torch.conj(x).resolve_conj()
    return torch.fft.irfftn(x, s=sizes, dim=dims, norm="forward")


def exact(case, seed):
    if case["kind"] == "plan":
        return _plan64(case, _plan_input(case, seed))
    if case["kind"] == "uneven":
        groups = _groups(case)
        x = _complex((sum(n * b for n, b in groups),), _gen(seed))
        y, at = torch.empty(x.numel(), dtype=torch.complex128, device="cuda"), 0
        for n, b in groups:
            y[at:at + n * b] = _c2c64(x[at:at + n * b].view(b, n), (1,), case["inverse"]).reshape(-1)
            at += n * b
        return y
    if case["kind"] == "istft":
        x, w = _istft_input(case, seed)
        n, hop, frames = case["n_fft"], case["hop"], case["frames"]
        t = torch.fft.ifft(x.to(torch.complex128), dim=1) * w.double()[None, :, None]
        at = (torch.arange(n, device="cuda")[:, None] + hop * torch.arange(frames, device="cuda")[None, :]).reshape(-1)
        total = n + hop * (frames - 1)
        y = torch.zeros((case["channels"], total), dtype=torch.complex128, device="cuda")
        y.index_add_(1, at, t.reshape(case["channels"], -1))
        env = torch.zeros(total, dtype=torch.float64, device="cuda")
        env.index_add_(0, at, (w.double() ** 2)[:, None].expand(n, frames).reshape(-1))
        return (y / env)[:, n // 2:n // 2 + _istft_length(case)].contiguous()
    return [_c2c64(x, (1,), False) if t == "c2c" else torch.fft.rfft(x.double())
            for (t, _, _), x in zip(_requests(case), _served_inputs(case, seed))]
