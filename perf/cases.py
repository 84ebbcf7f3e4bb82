"""Workloads whose speed is tracked, through the package's public calls.

Each case is one round of work of a program that keeps its arrays on the
GPU: a forward transform and the inverse of its result (the reference's own
benchmark loop does both), through ``dfft.fft/ifft/rfft/irfft``, a
``dfft.Batch`` or the distributed-array drivers ``dfft.gpu_fft_`` /
``dfft.gpu_ifft_``.  Sizes are those of the configured workloads (bench.py,
bench_configs.py), of the serving mix (cubic edges 64..384) and of the
parity tests (ragged, odd, prime and long axes).

A case is a dict of plain values:
  kind    "c2c" | "rfft" | "dct" | "batch" | "darray"
  n1..n3  extents, dim 1 first (1-D arrays have n2 = n3 = 0)
  double  True: ComplexF64 / Float64, False: ComplexF32 / Float32
  order   "F" column-major (Julia's layout) or "C" row-major (torch's own)
  slab    c2c: decomp=Slab() instead of Pencil()
  dist    input distribution: "normal", "uniform01", "uniform11"
  grids, shapes_seed   batch: how many grids, and the seed of their edges
  chunk   darray: block edge c of Blocks(n1, c, c) and its two partners
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "daggerfft.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import dfft  # noqa: E402

# edges of the batched workload and of the serving mix
BATCH_EDGES = (48, 64, 80, 96, 120, 128, 160, 192)
SERVE_EDGES = (64, 96, 128, 192, 256, 384)


def _case(name, kind, n1, n2, n3, double=False, order="F", slab=False, dist="normal", **more):
    return dict(name=name, kind=kind, n1=n1, n2=n2, n3=n3, double=double, order=order, slab=slab, dist=dist, **more)


def listed():
    return [
        # the headline: 512^3 ComplexF32, Slab; the largest call
        _case("c2c32_512_slab", "c2c", 512, 512, 512, slab=True),
        # the configured 128^3 ComplexF64 Pencil transform
        _case("c2c64_128_pencil", "c2c", 128, 128, 128, double=True, dist="uniform01"),
        # the configured 256^3 real transforms, both precisions
        _case("rfft64_256", "rfft", 256, 256, 256, double=True, dist="uniform01"),
        _case("rfft32_256", "rfft", 256, 256, 256, dist="uniform01"),
        # the configured stack of 32 planes: 2-D DCT-II, then DCT-III
        _case("dct64_256x256x32", "dct", 256, 256, 32, double=True, dist="uniform01"),
        # the configured batch: 64 uneven grids, one call
        _case("batch64_uneven", "batch", 0, 0, 0, dist="uniform11", grids=64, shapes_seed=4),
        # the serving mix's largest cube (not a power of two), and one of its
        # small ones as a row-major torch tensor (the README's own call)
        _case("c2c32_384_pencil", "c2c", 384, 384, 384),
        _case("c2c32_96_roworder", "c2c", 96, 96, 96, order="C"),
        # the smallest calls: launch and call latency
        _case("c2c32_32x24x16", "c2c", 32, 24, 16),
        # ragged axes: a prime, a 5-smooth and a 7-smooth length
        _case("c2c32_251x100x98", "c2c", 251, 100, 98, order="C"),
        # one long axis (a signal rather than a grid)
        _case("c2c32_1d_2e20", "c2c", 1 << 20, 0, 0),
        # the distributed-array Pencil driver on one GPU: the chunks' stage
        # transforms and the two redistributions between blockings
        _case("darray32_256_pencil", "darray", 256, 256, 256, chunk=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _edges(rng, lo, hi, most):
    """Three extents of a grid: configured edges, powers of two, or any
    integers (odd and prime ones among them), at most `most` elements."""
    while True:
        style = rng.random()
        if style < 0.35:
            e = [rng.choice(SERVE_EDGES)] * 3
        elif style < 0.6:
            e = [rng.choice(BATCH_EDGES + SERVE_EDGES) for _ in range(3)]
        else:
            e = [_log_int(rng, lo, hi) for _ in range(3)]
        cap = most if style < 0.6 else most // 32  # ragged grids are the smaller ones
        if e[0] * e[1] * e[2] <= cap:
            return e


def draw(rng):
    kind = rng.choice(("c2c", "c2c", "rfft", "rfft", "dct", "batch", "long", "darray"))
    double = rng.random() < 0.4
    order = rng.choice(("F", "C"))
    if kind == "long":
        # up to 2^21: powers of two, 5-smooth lengths and any integer
        style = rng.random()
        if style < 0.4:
            n = 1 << rng.randint(16, 21)
        elif style < 0.7:
            n = 2 ** rng.randint(10, 12) * 3 ** rng.randint(1, 3) * 5 ** rng.randint(1, 2)
        else:
            n = _log_int(rng, 1 << 16, 1 << 20)
        return dict(kind="c2c", n1=n, n2=0, n3=0, double=double, order="F", slab=False, dist="normal")
    if kind == "dct":
        n1, n2 = rng.choice(((64, 48), (128, 128), (256, 256), (256, 512), (512, 512), (100, 75),
                             (_log_int(rng, 16, 300), _log_int(rng, 16, 300))))
        n3 = _log_int(rng, 1, 64)
        return dict(kind="dct", n1=n1, n2=n2, n3=n3, double=double, order=order, slab=False, dist="uniform01")
    if kind == "batch":
        return dict(kind="batch", n1=0, n2=0, n3=0, double=False, order="F", slab=False, dist="uniform11",
                    grids=_log_int(rng, 4, 64), shapes_seed=rng.randint(0, 1 << 20))
    if kind == "darray":
        n = rng.choice((64, 96, 128, 192, 256))
        return dict(kind="darray", n1=n, n2=n, n3=n, double=double, order="F", slab=False, dist="normal",
                    chunk=rng.choice((n // 2, n // 4, n // 2 + 5)))
    e = _edges(rng, 12, 400, 1 << (25 if double else 26))
    return dict(kind=kind, n1=e[0], n2=e[1], n3=e[2], double=double, order=order,
                slab=kind == "c2c" and rng.random() < 0.5, dist=rng.choice(("normal", "uniform01")))


# ---------------------------------------------------------------------------


def _shape(case):
    return tuple(case[k] for k in ("n1", "n2", "n3") if case[k] > 0)


def _batch_shapes(case):
    rng = np.random.default_rng(case["shapes_seed"])
    return [tuple(int(e) for e in rng.choice(BATCH_EDGES, 3)) for _ in range(case["grids"])]


def _fill(shape, dtype, dist, order, gen):
    """A seeded tensor of logical shape `shape` in the requested memory order."""
    mem = tuple(reversed(shape)) if order == "F" else shape
    real = torch.empty(0, dtype=dtype).abs().dtype

    def one():
        if dist == "normal":
            return torch.randn(mem, dtype=real, device="cuda", generator=gen)
        t = torch.rand(mem, dtype=real, device="cuda", generator=gen)
        return t if dist == "uniform01" else t * 2 - 1

    t = torch.complex(one(), one()) if dtype.is_complex else one()
    return t.permute(*reversed(range(len(mem)))) if order == "F" else t


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    cplx = torch.complex128 if case["double"] else torch.complex64
    real = torch.float64 if case["double"] else torch.float32
    if case["kind"] == "batch":
        return [_fill(s, cplx, case["dist"], "F", gen) for s in _batch_shapes(case)]
    return _fill(_shape(case), real if case["kind"] in ("rfft", "dct") else cplx, case["dist"], case["order"], gen)


class _Batch:
    def __init__(self, ins):
        self.ins = ins
        plans = [dfft.gpu_plan_transform(dfft.FFT(), x, (1, 2, 3)) for x in ins]
        self.outs = [dfft.empty_like_layout(p.out_shape, x.dtype, x) for p, x in zip(plans, ins)]
        self.batch = dfft.Batch(plans)

    def __call__(self):
        return self.batch.execute(self.ins, self.outs)


class _DArrays:
    """The reference's Pencil layouts: Blocks(n1,c,c), Blocks(c,n2,c) and
    Blocks(c,c,n3), with the workspaces of the four redistributions."""

    def __init__(self, a, c):
        n = tuple(a.shape)
        self.source = dfft.distribute(a, dfft.Blocks(n[0], c, c))
        self.A = dfft.empty_darray(n, dfft.Blocks(n[0], c, c), a.dtype)
        self.B = dfft.empty_darray(n, dfft.Blocks(c, n[1], c), a.dtype)
        self.C = dfft.empty_darray(n, dfft.Blocks(c, c, n[2]), a.dtype)
        ws = dfft.create_gpu_workspace
        self.ab, self.bc = ws(self.A, self.B), ws(self.B, self.C)
        self.cb, self.ba = ws(self.C, self.B), ws(self.B, self.A)

    def __call__(self):
        dims, pencil = (1, 2, 3), dfft.Pencil()
        # the drivers work in place on A's chunks: this round's field
        for dst, src in zip(self.A.chunks, self.source.chunks):
            dst.copy_(src)
        dfft.gpu_fft_(self.C, self.A, self.B, self.ab, self.bc, (dfft.FFT_(),) * 3, dims, pencil)
        spectrum = [c.clone() for c in self.C.chunks]  # what the program uses before the inverse overwrites C
        dfft.gpu_ifft_(self.A, self.C, self.B, self.cb, self.ba, (dfft.IFFT_(),) * 3, dims, pencil)
        return {"spectrum": spectrum, "back": list(self.A.chunks)}


def prepare(case, seed):
    kind = case["kind"]
    a = _inputs(case, seed)
    if kind == "batch":
        return _Batch(a)
    if kind == "darray":
        return _DArrays(a, case["chunk"])
    dims = tuple(range(1, a.dim() + 1))
    if kind == "c2c":
        decomp = dfft.Slab() if case["slab"] else dfft.Pencil()

        def call():
            f = dfft.fft(a, decomp=decomp, dims=dims)
            return {"f": f, "x": dfft.ifft(f, decomp=decomp, dims=dims)}
    elif kind == "rfft":
        n = a.shape[0]

        def call():
            f = dfft.rfft(a, dims=dims)
            return {"f": f, "x": dfft.irfft(f, n, dims=dims)}
    else:
        ii = dfft.R2R((dfft.REDFT10, dfft.REDFT10))
        iii = dfft.R2R((dfft.REDFT01, dfft.REDFT01))

        def call():
            f = dfft.fft(a, transforms=(ii,), dims=(1, 2))
            return {"f": f, "x": dfft.ifft(f, transforms=(iii,), dims=(1, 2))}
    return call


def run(state):
    return state()


def work(case):
    csz = 16 if case["double"] else 8
    if case["kind"] == "batch":  # forward only
        n = [math.prod(s) for s in _batch_shapes(case)]
        return {"bytes": sum(2 * csz * k for k in n), "flops": sum(5 * k * math.log2(k) for k in n)}
    s = _shape(case)
    n = math.prod(s)
    if case["kind"] == "rfft":
        half = (s[0] // 2 + 1) * s[1] * s[2]
        return {"bytes": 2 * (n * csz // 2 + half * csz), "flops": 2 * 2.5 * n * math.log2(n)}
    if case["kind"] == "dct":
        return {"bytes": 4 * n * csz // 2, "flops": 2 * 2.5 * n * math.log2(s[0] * s[1])}
    # forward: field in, spectrum out; inverse: spectrum in, field out
    return {"bytes": 4 * n * csz, "flops": 2 * 5 * n * math.log2(n)}


def _dct2_matrix(n, device):
    k = torch.arange(n, dtype=torch.float64, device=device)
    return 2 * torch.cos(math.pi / n * k[:, None] * (k[None, :] + 0.5))


def _dct3_matrix(n, device):
    k = torch.arange(n, dtype=torch.float64, device=device)
    m = 2 * torch.cos(math.pi / n * (k[:, None] + 0.5) * k[None, :])
    m[:, 0] = 1
    return m


def _blocks(t, b):
    """The chunks of Blocks(*b), dim 1 of the block grid fastest."""
    s = t.shape
    return [t[x:x + b[0], y:y + b[1], z:z + b[2]] for z in range(0, s[2], b[2]) for y in range(0, s[1], b[1])
            for x in range(0, s[0], b[0])]


def exact(case, seed):
    kind = case["kind"]
    a = _inputs(case, seed)
    if kind == "batch":
        return [torch.fft.fftn(x.to(torch.complex128)) for x in a]
    if kind == "c2c":
        w = a.to(torch.complex128)
        f = torch.fft.fftn(w)
        return {"f": f, "x": w}
    if kind == "rfft":
        w = a.to(torch.float64)
        # rfft halves the first dim: the last of the axes given
        return {"f": torch.fft.rfftn(w, dim=(2, 1, 0)), "x": w}
    if kind == "dct":
        w = a.to(torch.float64)
        f = torch.einsum("ka,lb,abz->klz", _dct2_matrix(w.shape[0], w.device), _dct2_matrix(w.shape[1], w.device), w)
        return {"f": f, "x": w * (4.0 * w.shape[0] * w.shape[1])}
    w = a.to(torch.complex128)
    c = case["chunk"]
    n = tuple(w.shape)
    return {"spectrum": _blocks(torch.fft.fftn(w), (c, c, n[2])), "back": _blocks(w, (n[0], c, c))}
