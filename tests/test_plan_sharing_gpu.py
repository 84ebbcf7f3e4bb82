"""Calls that hide their plan (dfft.fft and the others) share it between
streams and threads: the cached plan holds no workspace, every execution
brings its own.  Checked for each use of a workspace: the fused slab pass's
job counters, the scratch of a four-step axis, the intermediate of irfft."""
import threading

import numpy as np
import pytest
import torch

import dfft
from dfft import _lib

pytestmark = pytest.mark.gpu

# (call, input shape, real input)
CASES = {
    "slab-192": (lambda x: dfft.fft(x, dims=(1, 2)), (192, 192, 120), torch.complex128),
    "slab-256": (lambda x: dfft.fft(x, dims=(1, 2)), (256, 256, 64), torch.complex64),
    "four-step": (lambda x: dfft.fft(x, dims=(1,)), (1 << 17, 4), torch.complex64),
    "irfft": (lambda x: dfft.irfft(x, 128, dims=(1, 2, 3)), (65, 96, 80), torch.complex64),
}


def _input(shape, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(tuple(reversed(shape)) + (2,), device="cuda", generator=g,
                    dtype=torch.float64 if dtype == torch.complex128 else torch.float32)
    return torch.view_as_complex(x).permute(*reversed(range(len(shape))))


@pytest.mark.parametrize("name", CASES)
def test_hidden_plans_hold_no_workspace(name):
    call, shape, dtype = CASES[name]
    dfft.gpu_cleanup_plans()
    call(_input(shape, dtype, 1))
    plans = [p for p in dfft.GPU_PLAN_CACHE.values() if p.workspace_bytes]
    assert plans and all(p._bring == p.workspace_bytes for p in plans)


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("threads", [False, True])
def test_same_call_on_several_streams(name, threads):
    call, shape, dtype = CASES[name]
    xs = [_input(shape, dtype, 10 + i) for i in range(3)]
    want = [call(x) for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    got = [[] for _ in xs]

    def one(i):
        with torch.cuda.stream(streams[i]):
            got[i].append(call(xs[i]))

    for _ in range(8):
        if threads:
            ts = [threading.Thread(target=one, args=(i,)) for i in range(len(xs))]
            for t in ts:
                t.start()
            for t in ts:
                t.join()
        else:
            for i in range(len(xs)):
                one(i)
    torch.cuda.synchronize()
    assert dfft.device_error() == 0
    for w, ys in zip(want, got):
        assert len(ys) == 8 and all(torch.equal(w, y) for y in ys)


def test_threads_on_one_stream():
    call, shape, dtype = CASES["slab-256"]
    xs = [_input(shape, dtype, 20 + i) for i in range(3)]
    want = [call(x) for x in xs]
    got = [None] * len(xs)

    def one(i):
        for _ in range(16):
            got[i] = call(xs[i])

    ts = [threading.Thread(target=one, args=(i,)) for i in range(len(xs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    assert dfft.device_error() == 0
    assert all(torch.equal(w, y) for w, y in zip(want, got))


def test_plans_a_caller_holds_keep_their_workspace():
    call, shape, dtype = CASES["four-step"]
    x = _input(shape, dtype, 3)
    want = call(x)
    p = dfft.get_or_create_gpu_plan(dfft.FFT(), x, (1,))
    assert p.workspace_bytes and not p._bring
    q = dfft.gpu_plan_transform(dfft.FFT(), x, (1,), flags=_lib.FLAG_CALLER_WORKSPACE)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    for plan, stream in ((p, None), (q, None), (q, s), (q, s.cuda_stream)):
        out = dfft.empty_like_layout(p.out_shape, dtype, x)
        plan.execute(x, out, stream)
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    # a plan without a workspace is one plan for both uses
    small = _input((32, 24), dtype, 4)
    dfft.fft(small, dims=(1,))
    assert dfft.get_or_create_gpu_plan(dfft.FFT(), small, (1,)) in dfft.GPU_PLAN_CACHE.values()
    assert len({id(v) for v in dfft.GPU_PLAN_CACHE.values() if v.shape == (32, 24)}) == 1


def test_workspace_is_checked():
    x = _input((1 << 17,), torch.complex64, 5)
    p = dfft.gpu_plan_transform(dfft.FFT(), x, (1,), flags=_lib.FLAG_CALLER_WORKSPACE)
    out = torch.empty_like(x)
    L = dfft.lib()
    assert L.dfft_execute(p._h, x.data_ptr(), out.data_ptr(), 0) == _lib.ERROR_INVALID_VALUE
    assert L.dfft_execute_workspace(p._h, x.data_ptr(), out.data_ptr(), 0, None) == _lib.ERROR_INVALID_VALUE
    w = torch.empty(p.workspace_bytes + 256, dtype=torch.uint8, device="cuda")
    assert L.dfft_execute_workspace(p._h, x.data_ptr(), out.data_ptr(), 0, w.data_ptr() + 16) == \
        _lib.ERROR_INVALID_VALUE
