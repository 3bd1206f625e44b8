"""The work that users of this library have it do, as cases that can be timed.

A case is one call (or one batched launch) on device buffers: compress or
decompress, float32 or float64, lossless or with an absolute error bound, on one
of five kinds of data, from a few KB to the 302 MB field of the benchmark.

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) what a program holds before the call: values or a stream, buffers, a plan
  run(state)          the call
  work(case)          the bytes that the call has to read and write
  exact(case, seed)   the decoded values by their definition, in 64 bits
"""
import math

import numpy as np
import torch

from sleek_b200 import api
from sleek_b200.batch import BatchPlan

TORCH = {"f32": torch.float32, "f64": torch.float64}
NUMPY = {"f32": np.float32, "f64": np.float64}
WIDTH = {"f32": 4, "f64": 8}

#: The kinds of data, each with the magnitude that sets the width of its quantized values.
KINDS = {
    "signal": 700.0,      # a measured time series: sinusoids, noise, 0.1 % NaN, infinities and denormals
    "turbulence": 3.5,    # a simulation's 3-D field: Fourier modes of a k^(-5/3) spectrum and a gradient
    "latlon": 0.7,        # a climate model's 2-D field: smooth, noisy in 1 % of the points
    "density": 32.0,      # a lognormal 3-D density
    "particles": 150.0,   # coordinates in [0, 256), sorted in blocks of 4096
}

LARGEST = 256 * 384 * 384 * 8  # bytes of the largest listed array
BATCH = 60                     # arrays of a batch


def listed():
    def one(name, op, dtype, kind, n, eb=0.0, first=0):
        return {"name": name, "op": op, "dtype": dtype, "kind": kind, "n": n, "eb": eb, "first": first}

    return [
        # the smallest requests of a service: a few KB, where the call itself is the cost
        one("compress_f32_4k", "compress", "f32", "latlon", 1001),
        # a variable of a small block of a simulation, read back
        one("decompress_f64_eb_200k", "decompress", "f64", "turbulence", 25003, eb=1e-3),
        # one time step of a 2-D climate variable (1800 x 3600), both ways, with the usual bound
        one("compress_f32_eb_26m", "compress", "f32", "latlon", 1800 * 3600, eb=1e-3),
        one("decompress_f32_eb_26m", "decompress", "f32", "latlon", 1800 * 3600, eb=1e-3),
        # a long 1-D record kept exactly, both ways
        one("compress_f32_64m", "compress", "f32", "signal", 1 << 24),
        one("decompress_f32_64m", "decompress", "f32", "signal", 1 << 24),
        # a ragged slab in the middle of a larger array, which starts at any element
        one("compress_f32_eb_slab_40m", "compress", "f32", "density", 10_000_019, eb=1e-3, first=1),
        # the 3-D double field of a simulation's checkpoint: exact, then with a bound, both ways
        one("compress_f64_302m", "compress", "f64", "turbulence", 256 * 384 * 384),
        one("compress_f64_eb_302m", "compress", "f64", "turbulence", 256 * 384 * 384, eb=1e-4),
        one("decompress_f64_eb_302m", "decompress", "f64", "turbulence", 256 * 384 * 384, eb=1e-4),
        # many variables of uneven sizes, types and bounds at once (4 KB to 16 MB each)
        {"name": "compress_batch", "op": "compress_batch", "arrays": BATCH, "least": 4 << 10, "most": 16 << 20, "sizes": 1},
        {"name": "decompress_batch", "op": "decompress_batch", "arrays": BATCH, "least": 4 << 10, "most": 16 << 20, "sizes": 1},
    ]


def draw(rng):
    op = rng.choice(["compress"] * 5 + ["decompress"] * 5 + ["compress_batch", "decompress_batch"])
    if op.endswith("batch"):
        return {"op": op, "arrays": rng.randint(8, BATCH), "least": 4 << 10,
                "most": int(math.exp(rng.uniform(math.log(256 << 10), math.log(16 << 20)))), "sizes": rng.randint(2, 1 << 30)}
    dtype = rng.choice(["f32", "f64"])
    kind = rng.choice(sorted(KINDS))
    n = int(math.exp(rng.uniform(math.log(1 << 10), math.log(LARGEST)))) // WIDTH[dtype]
    eb = 10.0 ** rng.uniform(-6, -1) if rng.random() < 0.5 else 0.0
    first = rng.choice([0, 0, 0, 1, 3]) if op == "compress" else 0
    return {"op": op, "dtype": dtype, "kind": kind, "n": max(1, n - first), "eb": eb, "first": first}


# ---- data -----------------------------------------------------------------------

def field(kind, dtype, n, seed):
    """`n` values of one kind, on the GPU, made from the seed alone."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    f64 = {"device": "cuda", "dtype": torch.float64}
    tau = 2 * math.pi

    def uniform(*shape):
        return torch.rand(*shape, generator=g, **f64)

    if kind == "signal":
        freq, phase = 10 ** (uniform(4) * 3 - 5), uniform(4) * tau
        i = torch.arange(n, **f64)
        x = 1e-3 * torch.randn(n, generator=g, **f64)
        for k in range(4):
            x += 1e3 * torch.sin(tau * freq[k] * i + phase[k])
        x = x.to(TORCH[dtype])
        at = torch.randint(0, n, (n // 1000,), generator=g, device="cuda").unique()
        odd = torch.tensor([math.nan, math.inf, -math.inf, 3e-41 if dtype == "f32" else 5e-320], device="cuda", dtype=x.dtype)
        x[at] = odd[torch.arange(at.numel(), device="cuda") % 4]
        return x
    if kind == "turbulence":
        side = max(1, min(384, round(n ** (1 / 3))))
        shape = (-(-n // (side * side)), side, side)
        k = torch.randint(1, 33, (3, 64), generator=g, device="cuda").to(torch.float64)
        amp = k.square().sum(0) ** (-5 / 6)
        amp = amp / (0.5 * amp.square().sum()).sqrt()
        phase = uniform(64) * tau
        a = [torch.arange(s, **f64)[:, None] * (tau / max(s, 64)) * k[d] for d, s in enumerate(shape)]
        a[0] = a[0] + phase
        yx = (a[1][:, None, :] + a[2][None, :, :]).reshape(side * side, 64)
        x = (amp * a[0].cos()) @ yx.cos().T - (amp * a[0].sin()) @ yx.sin().T
        x = x.reshape(-1)[:n]
        x += (0.1 / 256) * (torch.arange(n, **f64) % side)
        return x.to(TORCH[dtype])
    if kind == "latlon":
        rows = max(1, math.isqrt(n // 2))
        cols = -(-n // rows)
        l, p, q = torch.arange(9, **f64), uniform(9, 9) * tau, uniform(9, 9) * tau
        a = torch.randn(9, 9, generator=g, **f64) / (1 + l[:, None] + l[None, :])
        lat = torch.linspace(-math.pi / 2, math.pi / 2, rows, **f64)
        lon = torch.arange(cols, **f64) * (tau / cols)
        s = a * torch.sin(l[:, None] * lat[:, None, None] + p)
        c = torch.cos(l * lon[:, None, None] + q)
        x = (s.reshape(rows, 81) @ c.reshape(cols, 81).T).reshape(-1)[:n]
        x += 0.01 * torch.randn(n, generator=g, **f64) * (uniform(n) < 0.01)
        return x.to(TORCH[dtype])
    if kind == "density":
        side = max(2, math.ceil(n ** (1 / 3)))
        w = torch.fft.rfftn(torch.randn(side, side, side, generator=g, device="cuda"))
        f, h = torch.fft.fftfreq(side, device="cuda"), torch.fft.rfftfreq(side, device="cuda")
        k2 = f[:, None, None].square() + f[None, :, None].square() + h.square()
        k2[0, 0, 0] = math.inf
        x = torch.fft.irfftn(w * k2 ** -0.75, s=(side, side, side)).reshape(-1)[:n]
        x = (x - x.mean()) / x.std().clamp_min(1e-6) if n > 1 else x
        return torch.exp(1.5 * x.to(torch.float64)).to(TORCH[dtype])
    x = torch.rand(n, generator=g, device="cuda", dtype=TORCH[dtype]) * 256.0
    head = n // 4096 * 4096
    return torch.cat([x[:head].view(-1, 4096).sort(dim=1).values.reshape(-1), x[head:].sort().values])


def members(case):
    """The arrays of a batch: (kind, type, values, bound), half of them exact."""
    rng = np.random.default_rng(case["sizes"])
    kinds = sorted(KINDS)
    out = []
    for i in range(case["arrays"]):
        size = math.exp(rng.uniform(math.log(case["least"]), math.log(case["most"])))
        dtype = "f32" if rng.random() < 0.5 else "f64"
        bound = 10.0 ** rng.uniform(-6, -1)
        out.append((kinds[i % len(kinds)], dtype, int(size) // WIDTH[dtype], bound if i % 2 else 0.0))
    return out


# ---- the calls ------------------------------------------------------------------

def stream_of(x, eb):
    """The stream of an array, at its exact size."""
    return api.compress(x, eb or None).clone()


def prepare(case, seed):
    if case["op"].endswith("batch"):
        made = members(case)
        arrays = [field(kind, dtype, n, seed * 1000 + i) for i, (kind, dtype, n, _) in enumerate(made)]
        ebs = [eb or None for *_, eb in made]
        if case["op"] == "compress_batch":
            plan = BatchPlan.compress(arrays, ebs)
            for o in plan.outputs:
                o.zero_()  # what lies behind a stream is the same in every run
        else:
            streams = [stream_of(x, eb) for x, eb in zip(arrays, ebs)]
            plan = BatchPlan.decompress(streams, [NUMPY[m[1]] for m in made], ebs, [m[2] for m in made])
        return {"plan": plan}
    dtype, n, eb = case["dtype"], case["n"], case["eb"]
    x = field(case["kind"], dtype, n + case["first"], seed)[case["first"]:]
    size = torch.zeros(1, dtype=torch.int64, device="cuda")
    args = (api.sleek_error_bound(eb, NUMPY[dtype]),) if eb else ()
    if case["op"] == "compress":
        out = torch.zeros(api.sleek_upper_bound_size(n * WIDTH[dtype]), dtype=torch.uint8, device="cuda")
        return {"compress": True, "args": args + (x, n, out, size), "out": out, "size": size}
    stream = stream_of(x, eb)
    out = torch.empty(n, dtype=TORCH[dtype], device="cuda")
    return {"compress": False, "args": args + (stream, out, size), "out": out, "size": size, "length": stream.numel()}


def run(state):
    plan = state.get("plan")
    if plan is not None:
        plan.run()
        return plan.outputs, plan.sizes
    if state["compress"]:
        api.sleek_compress_gpu(0, *state["args"])
    else:
        api.sleek_decompress_gpu(0, *state["args"], encoded_bytes=state["length"])
    return state["out"], state["size"]


# ---- what a pass cannot do without, and what it returns -------------------------

def stream_bytes(kind, dtype, n, eb):
    """About the bytes of the stream of one array."""
    bits = 8 * WIDTH[dtype]
    if eb:
        bits = min(bits, max(1.0, 1 + math.log2(KINDS[kind]) - math.floor(math.log2(eb)) - 1))
    else:
        bits *= 0.9
    return int(n * bits / 8 + -(-n * WIDTH[dtype] // 16384) * 36 + 8)


def work(case):
    if case["op"].endswith("batch"):
        every = members(case)
    else:
        every = [(case["kind"], case["dtype"], case["n"], case["eb"])]
    return {"bytes": sum(n * WIDTH[d] + stream_bytes(k, d, n, eb) for k, d, n, eb in every), "flops": 0}


def decoded(x, eb):
    """The values that come back: the ones that went in, or the nearest multiples of twice the bound's power of two."""
    v = x.to(torch.float64)
    if not eb:
        return v
    step = 2.0 ** (math.floor(math.log2(eb)) + 1)
    limit = step * 2.0 ** (23 if x.dtype == torch.float32 else 52)  # from here on the values are kept as they are
    y = v.abs() / step
    q = y.floor()
    q = (q + (y - q >= 0.5)) * step
    return torch.where(v.abs() < limit, torch.where(v < 0, -q, q), v)


def exact(case, seed):
    if case["op"] == "compress" or case["op"] == "compress_batch":
        return None
    if case["op"] == "decompress_batch":
        made = members(case)
        return [decoded(field(k, d, n, seed * 1000 + i), eb) for i, (k, d, n, eb) in enumerate(made)], None
    x = field(case["kind"], case["dtype"], case["n"] + case["first"], seed)[case["first"]:]
    return decoded(x, case["eb"]), None
