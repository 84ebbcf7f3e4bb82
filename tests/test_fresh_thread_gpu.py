"""A call whose passes need TMA descriptors as the first CUDA work of a new
thread: the descriptor encoder is a driver call, and nothing before it has
bound the device's context to that thread."""
import threading

import numpy as np
import pytest
import torch

import dfft
import dfft_oracle as oracle
from helpers import rand, rel, to_gpu, to_np, tol_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["slab", "strided-feed", "strided-pipe", "tiled-strided", "mixed"])
def test_first_work_of_a_thread(name):
    kind = {}
    if name == "tiled-strided":
        a = rand((16, 128, 8), np.float64, seed=1)
        tr = (dfft.R2R((dfft.REDFT10,)),)
        g, call = to_gpu(a), lambda x: dfft.fft(x, dims=(2,), transforms=tr)
        ref, tag, dims = oracle.fft(a, dims=(2,), transforms=(oracle.R2R((dfft.REDFT10,)),)), tr[0], (2,)
    else:
        shape, dims = {"slab": ((256, 256, 4), (1, 2)), "strided-feed": ((256, 256, 40), (3,)),
                       "strided-pipe": ((320, 180, 80), (2,)), "mixed": ((16, 512, 8), (2,))}[name]
        if name == "strided-feed":
            shape, dims = (256, 256, 64), (2,)
        a = rand(shape, np.complex64, seed=2)
        if name == "mixed":
            kind["method"] = "mixed"
        g, call = to_gpu(a), lambda x: dfft.fft(x, dims=dims, **kind)
        ref, tag = oracle.fft(a, dims=dims), dfft.FFT()
    d = dfft.gpu_plan_transform(tag, g, dims, **kind).describe()
    assert d.startswith(name), d
    call(g)  # the plan is built, and the allocator holds the output's size
    torch.cuda.synchronize()
    got, err = [], []

    def work():
        try:
            got.append(call(g))
        except Exception as e:  # reported below, in the test's own thread
            err.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert not err, err[0]
    assert rel(to_np(got[0]), ref) <= tol_for(a.dtype)
