"""Lengths with a prime factor above 13 run Bluestein's algorithm in one
launch while the convolution length fits one CTA: a compiled length (up to
4096 ComplexF32 / 2048 ComplexF64) or one of the run-time-radix kernel
(to 16384 / 8192).  Edges of those ranges, contiguous and strided axes,
column counts that do not fill a tile, and the real and r2r sides, against
the FP64 oracle."""
import numpy as np
import pytest
import torch

import dfft
import dfft_oracle as oracle
from helpers import rand, rel, to_gpu, to_np, tol_for

pytestmark = pytest.mark.gpu


def _one_launch(transform, g, dims, **kw):
    p = dfft.gpu_plan_transform(transform, g, dims, **kw)
    assert p.launches == len(dims) and "bluestein" in p.describe(), p.describe()
    return p


@pytest.mark.parametrize("n,dtype", [
    # the longest prime of each two-radix convolution length, and the first past the last one
    *[(n, np.complex64) for n in (17, 31, 47, 61, 89, 127, 191, 251, 383, 509, 521)],
    *[(n, np.complex128) for n in (17, 31, 47, 61, 89, 127, 191, 251, 257)],
    # compiled lengths of the general kernel, then its run-time radices
    (2039, np.complex64), (2053, np.complex64), (8191, np.complex64),
    (1021, np.complex128), (1031, np.complex128), (4093, np.complex128)])
@pytest.mark.parametrize("strided", [False, True])
def test_c2c_edges(n, dtype, strided):
    shape, dims = ((5, n, 3), (2,)) if strided else ((n, 7), (1,))
    a = rand(shape, dtype, seed=n)
    g = to_gpu(a)
    _one_launch(dfft.FFT(), g, dims)
    F = dfft.fft(g, dims=dims)
    assert rel(to_np(F), oracle.fft(a, dims=dims)) <= tol_for(dtype)
    assert rel(to_np(dfft.ifft(F, dims=dims)), a) <= tol_for(dtype)


@pytest.mark.parametrize("n", [14, 22, 26, 98, 182, 343, 1001, 1014])
@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
def test_compiled_lengths_with_7_11_13(n, dtype):
    a = rand((5, n, 7), dtype, seed=n)
    g = to_gpu(a)
    assert "dynamic" not in dfft.gpu_plan_transform(dfft.FFT(), g, (2,)).describe()
    F = dfft.fft(g, dims=(2,))
    assert rel(to_np(F), oracle.fft(a, dims=(2,))) <= tol_for(dtype)
    assert rel(to_np(dfft.ifft(F, dims=(2,))), a) <= tol_for(dtype)


@pytest.mark.parametrize("n", [31, 37, 158, 509])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape_of", [lambda n: ((n, 5), (1,)), lambda n: ((3, n, 4), (2,))])
def test_real_and_r2r_sides(n, dtype, shape_of):
    shape, dims = shape_of(n)
    a = rand(shape, dtype, seed=n)
    g = to_gpu(a)
    F = dfft.rfft(g, dims=dims)
    assert rel(to_np(F), oracle.rfft(a, dims=dims)) <= tol_for(dtype)
    assert rel(to_np(dfft.irfft(F, n, dims=dims)), a) <= tol_for(dtype)
    for kind in (dfft.REDFT10, dfft.RODFT01, dfft.REDFT11, dfft.RODFT00, dfft.DHT):
        y = dfft.fft(g, dims=dims, transforms=(dfft.R2R((kind,)),))
        ref = oracle.r2r_direct(a.astype(np.longdouble), kind, dims[0] - 1)
        assert rel(to_np(y), ref) <= tol_for(dtype)


def test_in_place_and_infinities_stay_in_their_column():
    a = rand((34, 31, 8), np.complex64, seed=1)
    a[0, 3, 2] = np.inf  # one column of axis 2 is not finite; the others are untouched
    g = to_gpu(a)
    dfft.fft_(g, dims=(2,))
    torch.cuda.synchronize()
    y = to_np(g)
    b = a.copy()
    b[0, :, 2] = 0
    ref = oracle.fft(b, dims=(2,))
    keep = np.ones((34, 8), bool)
    keep[0, 2] = False
    assert not np.isfinite(y[0, :, 2]).any()
    assert rel(y.transpose(0, 2, 1)[keep], np.asarray(ref).transpose(0, 2, 1)[keep]) <= 1e-5


@pytest.mark.parametrize("n,dtype", [(2053, np.complex64), (5003, np.complex64), (6007, np.complex64),
                                     (1031, np.complex128), (2503, np.complex128)])
def test_one_launch_takes_the_shortest_convolution(n, dtype):
    # beyond the compiled lengths the one-launch kernel runs the smallest
    # 5-smooth length, not the longer one a four-step pair would split into
    shortest = next(k for k in range(2 * n - 1, 4 * n) if _smooth5(k))
    a = rand((n, 3), dtype, seed=n)
    p = _one_launch(dfft.FFT(), to_gpu(a), (1,))
    assert f" L={shortest} " in p.describe(), p.describe()
    F = dfft.fft(to_gpu(a), dims=(1,))
    assert rel(to_np(F), oracle.fft(a, dims=(1,))) <= tol_for(dtype)


def _smooth5(k):
    for q in (2, 3, 5):
        while k % q == 0:
            k //= q
    return k == 1


@pytest.mark.parametrize("n", [17, 23, 37, 73, 137, 151, 311, 613, 1123, 1217, 1531, 1777])
@pytest.mark.parametrize("strided", [False, True])
def test_every_compiled_convolution_on_real_sides(n, strided):
    # one length behind each convolution of the general kernel that the
    # complex two-radix kernels do not use
    shape, dims = ((5, n, 3), (2,)) if strided else ((n, 7), (1,))
    for dtype in (np.float32, np.float64):
        a = rand(shape, dtype, seed=n)
        g = to_gpu(a)
        F = dfft.rfft(g, dims=dims)
        assert rel(to_np(F), oracle.rfft(a, dims=dims)) <= tol_for(dtype)
        assert rel(to_np(dfft.irfft(F, n, dims=dims)), a) <= tol_for(dtype)
