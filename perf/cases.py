"""The transforms whose speed this repository looks after, and how to run them.

Each case is one call (or one call sequence) that a program using the library
makes in its inner loop, through the public entry points: the plan interface
(shafft_b200.FFTND / FFT1D), the real transforms (RPlan) and the batched form
(Batch).  listed() gives the fixed set, draw() more of the same ranges;
prepare() makes what such a program holds before the call (device buffers with
iid uniform [-1, 1) data and a plan), run() one pass, exact() the same result
from torch.fft in 64 bits, work() the bytes and operations a pass cannot do
without.

Kinds:
  c2c    execute on device buffers (the 1/sqrt(N) normalisation fused into the
         execute, or the separate normalize() call of the reference's own
         sequence); the result is left in the plan's data buffer, from which
         the next pass goes on, as in a time-stepping program;
  real   r2c of a real tensor, then c2r back into it;
  batch  one execute over many independent transforms of uneven shapes.
"""
import math
import random

import torch

import shafft_b200 as S
from shafft_b200 import _sm100


def _c2c(name, dims, prec, direction, normalize="fused"):
    return {"name": name, "kind": "c2c", "dims": "x".join(map(str, dims)), "prec": prec, "direction": direction,
            "normalize": normalize}


def listed():
    return [
        # a short signal: the call is nothing but latency
        _c2c("fft1d_1024_c64", (1024,), "c64", "forward"),
        # a small grid that fits L2 many times over; latency and launches again
        _c2c("nd_64x64x32_c64", (64, 64, 32), "c64", "forward"),
        # a small ragged grid in double precision, two prime axes
        _c2c("nd_63x47x31_c128", (63, 47, 31), "c128", "backward"),
        # a prime length: chirp convolution
        _c2c("fft1d_1000003_c64", (1000003,), "c64", "forward"),
        # a mixed-radix length, 3^5 5^3 7^2, in double precision
        _c2c("fft1d_1488375_c128", (1488375,), "c128", "backward"),
        # a long signal of a power-of-two length
        _c2c("fft1d_2p24_c64", (1 << 24,), "c64", "forward"),
        # an image
        _c2c("nd_2048x2048_c64", (2048, 2048), "c64", "backward"),
        # a grid whose extents are not powers of two, with the execute and
        # normalize calls of the reference's interface
        _c2c("nd_384x384x384_c64", (384, 384, 384), "c64", "forward", "separate"),
        # a simulation grid in double precision
        _c2c("nd_256x256x256_c128", (256, 256, 256), "c128", "backward"),
        # the large grid the library is known by
        _c2c("nd_512x512x512_c64", (512, 512, 512), "c64", "forward"),
        # a real field to its half spectrum and back
        {"name": "real_256x256x256_f32", "kind": "real", "dims": "256x256x256", "prec": "c64"},
        # many small 2-D and 3-D transforms of uneven extents
        {"name": "batch_512_c64", "kind": "batch", "count": 512, "shapes_seed": 42, "prec": "c64", "direction": "forward"},
    ]


def _prime(n):
    return n > 1 and all(n % d for d in range(2, math.isqrt(n) + 1))


def _smooth(n, primes=(2, 3, 5, 7)):
    for p in primes:
        while n % p == 0:
            n //= p
    return n == 1


def _near(n, good):
    """The number nearest to n (from below first) that `good` takes."""
    for d in range(n):
        if n - d > 1 and good(n - d):
            return n - d
        if good(n + d):
            return n + d
    return n


def _extent(rng, lo, hi, prime_share):
    """An axis length, log-uniform in [lo, hi]: a power of two, a 7-smooth
    number, any number, or a prime."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    n = max(lo, min(hi, round(v)))
    u = rng.random()
    if u < prime_share:
        return _near(n, _prime)
    if u < prime_share + 0.10:
        return n
    if u < 0.55:
        return min(hi, max(lo, 1 << round(math.log2(n))))
    return _near(n, _smooth)


def draw(rng):
    u = rng.random()
    prec = "c128" if rng.random() < 0.35 else "c64"
    direction = rng.choice(["forward", "backward"])
    normalize = "separate" if rng.random() < 0.3 else "fused"
    if u < 0.12:
        dims = [_extent(rng, 16, 320, 0.0) for _ in range(rng.choice([2, 3, 3]))]
        dims[-1] += dims[-1] % 2
        return {"kind": "real", "dims": "x".join(map(str, dims)), "prec": prec}
    if u < 0.24:
        return {"kind": "batch", "count": round(math.exp(rng.uniform(math.log(8), math.log(384)))),
                "shapes_seed": rng.randrange(1 << 30), "prec": "c64", "direction": direction}
    if u < 0.5:
        # signals of 2^10 to 2^24 points, primes and unfactorable lengths up to 2^21
        n = _extent(rng, 1 << 10, 1 << 24, 0.15)
        if n > 1 << 21 and not _smooth(n, (2, 3, 5, 7, 11, 13)):
            n = _near(n, _smooth)
        dims = [n]
    else:
        # grids: 2-D up to 2048 a side, 3-D up to 384, at most 2^25 points (2^24 in double precision)
        most = 1 << (24 if prec == "c128" else 25)
        while True:
            dims = ([_extent(rng, 64, 2048, 0.08) for _ in range(2)] if rng.random() < 0.4
                    else [_extent(rng, 16, 384, 0.08) for _ in range(3)])
            if math.prod(dims) <= most:
                break
    c = _c2c("", dims, prec, direction, normalize)
    del c["name"]
    return c


def _dims(case):
    return tuple(int(v) for v in case["dims"].split("x"))


def _batch_shapes(case):
    """2-D and 3-D shapes, extents log-uniform in [16, 256] over the 7-smooth
    numbers, one extent in twenty a prime."""
    rng = random.Random(case["shapes_seed"])
    smooth = [n for n in range(16, 257) if _smooth(n)]
    primes = [n for n in range(16, 257) if _prime(n)]
    shapes = []
    for _ in range(case["count"]):
        dims = []
        for _ in range(rng.choice([2, 3])):
            v = rng.uniform(math.log(16), math.log(256))
            dims.append(rng.choice(primes) if rng.random() < 0.05 else min(smooth, key=lambda n: abs(math.log(n) - v)))
        shapes.append(tuple(dims))
    return shapes


def _batch_offsets(shapes):
    """Element offset of each transform in one packed array (256-byte steps), and its length."""
    off, at = [], 0
    for s in shapes:
        off.append(at)
        at += -(-math.prod(s) // 32) * 32
    return off, at


def _rdtype(case):
    return torch.float64 if case["prec"] == "c128" else torch.float32


def _cdtype(case):
    return torch.complex128 if case["prec"] == "c128" else torch.complex64


def _uniform(shape, dtype, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return torch.rand(shape, dtype=dtype, device="cuda", generator=gen).mul_(2).sub_(1)


def _input(case, seed):
    if case["kind"] == "real":
        return _uniform(_dims(case), _rdtype(case), seed)
    if case["kind"] == "batch":
        shapes = _batch_shapes(case)
        off, n = _batch_offsets(shapes)
        x = torch.zeros((n,), dtype=_cdtype(case), device="cuda")
        u = torch.view_as_complex(_uniform((n, 2), _rdtype(case), seed))
        for o, s in zip(off, shapes):
            x[o:o + math.prod(s)] = u[o:o + math.prod(s)]
        return x
    return torch.view_as_complex(_uniform(_dims(case) + (2,), _rdtype(case), seed))


def prepare(case, seed):
    x = _input(case, seed)
    prec = S.Z2Z if case["prec"] == "c128" else S.C2C
    if case["kind"] == "real":
        plan = _sm100.RPlan(_dims(case), prec)
        dims = _dims(case)
        spec = torch.empty(dims[:-1] + (dims[-1] // 2 + 1,), dtype=_cdtype(case), device="cuda")
        return {"kind": "real", "plan": plan, "x": x, "spec": spec, "scale": 1.0 / math.prod(dims)}
    if case["kind"] == "batch":
        shapes = _batch_shapes(case)
        off, _ = _batch_offsets(shapes)
        y = torch.zeros_like(x)
        es = x.element_size()
        plan = _sm100.Batch(shapes, prec)
        return {"kind": "batch", "plan": plan, "x": x, "y": y,
                "src": [x.data_ptr() + o * es for o in off], "dst": [y.data_ptr() + o * es for o in off],
                "direction": S.FORWARD if case["direction"] == "forward" else S.BACKWARD}
    dims = _dims(case)
    if len(dims) == 1:
        plan = S.FFT1D()
        S.check(plan.init(dims[0], precision=prec), "init")
    else:
        plan = S.FFTND()
        S.check(plan.init([1] * len(dims), list(dims), prec), "init")
    S.check(plan.plan(), "plan")
    w = torch.empty_like(x)
    S.check(plan.set_buffers(x.data_ptr(), w.data_ptr()), "setBuffers")
    return {"kind": "c2c", "plan": plan, "x": x, "w": w, "separate": case["normalize"] == "separate",
            "direction": S.FORWARD if case["direction"] == "forward" else S.BACKWARD}


def run(state):
    plan = state["plan"]
    if state["kind"] == "real":
        plan.r2c(state["x"].data_ptr(), state["spec"].data_ptr())
        plan.c2r(state["spec"].data_ptr(), state["x"].data_ptr(), state["scale"])
        return {"spectrum": state["spec"], "x": state["x"]}
    if state["kind"] == "batch":
        plan.execute(state["src"], state["dst"], state["direction"])
        return state["y"]
    if state["separate"]:
        S.check(plan.execute(state["direction"]), "execute")
        S.check(plan.normalize(), "normalize")
    else:
        S.check(plan.execute_normalized(state["direction"]), "execute")
    rc, data, _ = plan.get_buffers()
    S.check(rc, "getBuffers")
    return state["x"] if data == state["x"].data_ptr() else state["w"]


def exact(case, seed):
    x = _input(case, seed)
    if case["kind"] == "real":
        x = x.double()
        return {"spectrum": torch.fft.rfftn(x), "x": x}
    x = x.to(torch.complex128)
    inverse = case["direction"] == "backward"
    if case["kind"] == "batch":
        y = torch.zeros_like(x)
        shapes = _batch_shapes(case)
        for o, s in zip(_batch_offsets(shapes)[0], shapes):
            v = x[o:o + math.prod(s)].view(s)
            v = torch.fft.ifftn(v, norm="forward") if inverse else torch.fft.fftn(v)
            y[o:o + math.prod(s)] = v.reshape(-1)
        return y
    return torch.fft.ifftn(x, norm="ortho") if inverse else torch.fft.fftn(x, norm="ortho")


def work(case):
    """Each input read once and each output written once; 5 N log2 N
    operations a complex transform, half of that a real one."""
    es = 16 if case["prec"] == "c128" else 8
    if case["kind"] == "batch":
        ns = [math.prod(s) for s in _batch_shapes(case)]
        return {"bytes": 2 * es * sum(ns), "flops": sum(5 * n * math.log2(n) for n in ns)}
    dims = _dims(case)
    n = math.prod(dims)
    if case["kind"] == "real":
        spec = n // dims[-1] * (dims[-1] // 2 + 1)
        return {"bytes": 2 * (n * es // 2 + spec * es), "flops": 5 * n * math.log2(n)}
    return {"bytes": 2 * es * n, "flops": 5 * n * math.log2(n)}
