"""Passes of up to 96 MB are launched while the kernel before them in the
stream still runs, and wait for it in the kernel (programmatic stream
serialization).  The results of chains of calls without a synchronisation, in
turn with ordinary kernels that write their inputs and read their outputs,
captured into a graph, and on several streams, are the ones that the same
calls give one at a time."""
import pytest
import torch

import dfft

pytestmark = pytest.mark.gpu


def _c2c(dims):
    return (lambda x: dfft.fft(x, dims=dims)), (lambda y: dfft.ifft(y, dims=dims))


def _dct():
    ii, iii = dfft.R2R((dfft.REDFT10, dfft.REDFT10)), dfft.R2R((dfft.REDFT01, dfft.REDFT01))
    return (lambda x: dfft.fft(x, transforms=(ii,), dims=(1, 2))), (lambda y: dfft.fft(y, transforms=(iii,), dims=(1, 2)))


def _real(n):
    return (lambda x: dfft.rfft(x, dims=(1, 2, 3))), (lambda y: dfft.irfft(y, n, dims=(1, 2, 3)))


# forward, inverse, shape, type: one-tile, TMA, slab (with its memset), prime,
# four-step, real and DCT passes
CASES = {
    "tiny": _c2c((1, 2, 3)) + ((32, 24, 16), torch.complex64),
    "direct": _c2c((1, 2, 3)) + ((96, 96, 96), torch.complex64),
    "feed": _c2c((1, 2, 3)) + ((128, 160, 120), torch.complex64),
    "slab": _c2c((1, 2, 3)) + ((256, 256, 12), torch.complex64),
    "double": _c2c((1, 2, 3)) + ((128, 128, 32), torch.complex128),
    "prime": _c2c((1, 2, 3)) + ((251, 100, 14), torch.complex64),
    "four-step": _c2c((1,)) + ((1 << 17, 2), torch.complex64),
    "long-prime": _c2c((1,)) + ((20011, 2), torch.complex64),
    "real": _real(128) + ((128, 64, 48), torch.float32),
    "real-odd": _real(75) + ((75, 40, 22), torch.float64),
    "dct": _dct() + ((256, 256, 6), torch.float64),
}
ROUNDS = 6


def _inputs(name, n=ROUNDS):
    shape, dtype = CASES[name][2:]
    g = torch.Generator(device="cuda").manual_seed(len(name))
    mem = tuple(reversed(shape))
    return [torch.randn(mem, dtype=dtype, device="cuda", generator=g).permute(*reversed(range(len(shape))))
            for _ in range(n)]


def _one_at_a_time(name, xs):
    fwd, inv = CASES[name][:2]
    want = []
    for x in xs:
        torch.cuda.synchronize()
        y = fwd(x)
        torch.cuda.synchronize()
        z = y * 0.5
        torch.cuda.synchronize()
        w = inv(z)
        torch.cuda.synchronize()
        want.append((y, w))
    return want


def _check(want, got):
    torch.cuda.synchronize()
    assert dfft.device_error() == 0
    for (y, w), (gy, gw) in zip(want, got):
        assert torch.equal(y, gy) and torch.equal(w, gw)


@pytest.mark.parametrize("name", CASES)
def test_chain_with_other_kernels_on_one_stream(name):
    fwd, inv = CASES[name][:2]
    xs = _inputs(name)
    want = _one_at_a_time(name, xs)
    buf = torch.empty_like(xs[0])
    got = []
    for x in xs * 2:
        buf.copy_(x)  # writes what the pass before may still be reading
        y = fwd(buf)
        z = y * 0.5  # reads what the pass has just written
        buf.zero_()  # the input is gone as soon as the transform is through
        got.append((y, inv(z)))
        z.zero_()
    _check(want * 2, got)


@pytest.mark.parametrize("name", CASES)
def test_captured_into_a_graph(name):
    fwd, inv = CASES[name][:2]
    xs = _inputs(name)
    want = _one_at_a_time(name, xs)  # also builds the plans
    buf = xs[0].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = fwd(buf)
        z = y * 0.5
        w = inv(z)
    got = []
    for x in xs * 2:
        buf.copy_(x)
        graph.replay()
        got.append((y.clone(), w.clone()))
    _check(want * 2, got)


@pytest.mark.parametrize("name", CASES)
def test_plan_executed_in_a_capture(name):
    # Plan.execute with a plan that holds its workspace, in place where it can be
    shape, dtype = CASES[name][2:]
    if not dtype.is_complex:
        pytest.skip("complex plans only")
    dims = (1,) if name in ("four-step", "long-prime") else (1, 2, 3)
    xs = _inputs(name)
    buf = xs[0].clone()
    p = dfft.gpu_plan_transform(dfft.FFT_(), buf, dims)
    want = []
    for x in xs:
        t = x.clone()
        torch.cuda.synchronize()
        p.execute(t, t)
        torch.cuda.synchronize()
        want.append((x, t))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        p.execute(buf, buf)
    got = []
    for x in xs:
        buf.copy_(x)
        graph.replay()
        got.append((x, buf.clone()))
    _check(want, got)


@pytest.mark.parametrize("name", CASES)
def test_several_streams(name):
    fwd, inv = CASES[name][:2]
    xs = _inputs(name)
    want = _one_at_a_time(name, xs)
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    got = [None] * len(xs)
    for rep in range(3):
        for i, x in enumerate(xs):
            with torch.cuda.stream(streams[i % len(streams)]):
                y = fwd(x)
                got[i] = (y, inv(y * 0.5))
    _check(want, got)


def test_events_between_streams():
    # a pass on one stream waits for an event of another: the kernel before it
    # in its own stream is not what it depends on
    fwd, inv = CASES["direct"][:2]
    xs = _inputs("direct")
    want = _one_at_a_time("direct", xs)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    got = []
    for x in xs:
        with torch.cuda.stream(a):
            y = fwd(x)
            z = y * 0.5
        b.wait_stream(a)
        with torch.cuda.stream(b):
            w = inv(z)
        a.wait_stream(b)
        got.append((y, w))
        for t in (y, z):
            t.record_stream(b)
    _check(want, got)
