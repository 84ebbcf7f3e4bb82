"""Tile-staged R2R passes (tiled_pass): every FFTW kind the reference lists
(src/fft.jl:1-11) along the contiguous axis (whole pencils) and a strided
axis (column tiles), at extents whose FFT length is 128, 256 or 512, checked
against the oracle's direct sums / FFTW definitions."""
import numpy as np
import pytest

import dfft
import dfft_oracle as oracle
from helpers import rand, rel, to_gpu, to_np, tol_for

pytestmark = pytest.mark.gpu

# kind -> data extents N whose FFT length (N, 2N, 2(N-1), 2(N+1)) is 128 / 256 / 512
EXTENTS = {dfft.REDFT10: [128, 256, 512], dfft.REDFT01: [128, 256, 512], dfft.RODFT10: [128, 256],
           dfft.RODFT01: [128, 256], dfft.DHT: [128, 512], dfft.REDFT11: [64, 128, 256],
           dfft.RODFT11: [64, 128], dfft.REDFT00: [65, 129], dfft.RODFT00: [63, 127]}
CASES = [(k, n) for k, ns in EXTENTS.items() for n in ns]


@pytest.mark.parametrize("kind,n", CASES)
@pytest.mark.parametrize("axis", [1, 2])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_tiled_kinds(kind, n, axis, dtype):
    shape = (n, 16, 4) if axis == 1 else (16, n, 4)
    a = rand(shape, dtype, seed=kind * 997 + n + axis)
    g = to_gpu(a)
    tr = (dfft.R2R((kind,)),)
    p = dfft.gpu_plan_transform(dfft.R2R((kind,)), g, (axis,))
    y = dfft.fft(g, dims=(axis,), transforms=tr)
    ref = oracle.fft(a, dims=(axis,), transforms=(oracle.R2R((kind,)),))
    assert rel(to_np(y), ref) <= tol_for(dtype), p.describe()
    assert dfft.device_error() == 0


@pytest.mark.parametrize("order", ["F", "C"])
def test_dct_stack_uses_tiles(order):
    # the DCT-II / DCT-III stack of the batched configuration, 256 x 256 x 32
    a = rand((256, 256, 32), np.float64, seed=3, kind="uniform01")
    g = to_gpu(a, order)
    for kind in (dfft.REDFT10, dfft.REDFT01):
        p = dfft.gpu_plan_transform(dfft.R2R((kind, kind)), g, (1, 2))
        kinds = [ln.split()[0] for ln in p.describe().strip().splitlines()]
        assert kinds and all(k.startswith("tiled") for k in kinds), p.describe()
    F = dfft.fft(g, dims=(1, 2), transforms=(dfft.R2R((dfft.REDFT10, dfft.REDFT10)),))
    ref = oracle.fft(a, dims=(1, 2), transforms=(oracle.R2R((oracle.REDFT10, oracle.REDFT10)),))
    assert rel(to_np(F), ref) <= 1e-12
    B = dfft.fft(F, dims=(1, 2), transforms=(dfft.R2R((dfft.REDFT01, dfft.REDFT01)),))
    assert rel(to_np(B), a * (2 * 256) ** 2) <= 1e-12


@pytest.mark.parametrize("n", [128, 256, 512])
@pytest.mark.parametrize("cols", [1, 4, 13])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", [dfft.REDFT10, dfft.REDFT01])
def test_column_counts_that_do_not_fill_a_tile(n, cols, dtype, kind):
    # contiguous pencils whose last tile is partial, and few strided columns;
    # an infinity stays in its own column
    a = rand((n, cols), dtype, seed=n + cols)
    tr = (dfft.R2R((kind,)),)
    p = dfft.gpu_plan_transform(dfft.R2R((kind,)), to_gpu(a), (1,))
    assert p.describe().startswith("tiled-contig"), p.describe()
    ref = oracle.fft(a, dims=(1,), transforms=(oracle.R2R((kind,)),))
    assert rel(to_np(dfft.fft(to_gpu(a), dims=(1,), transforms=tr)), ref) <= tol_for(dtype)
    b = np.ascontiguousarray(a.T)
    y = to_np(dfft.fft(to_gpu(b), dims=(2,), transforms=tr))
    assert rel(y, np.asarray(ref).T) <= tol_for(dtype)
    if cols > 1:
        a[3, cols - 1] = np.inf
        y = to_np(dfft.fft(to_gpu(a), dims=(1,), transforms=tr))
        assert np.isfinite(y[:, :-1]).all() and not np.isfinite(y[:, -1]).all()
        assert rel(y[:, :-1], np.asarray(ref)[:, :-1]) <= tol_for(dtype)


@pytest.mark.parametrize("n", [128, 256, 512])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", [dfft.REDFT10, dfft.REDFT01])
@pytest.mark.parametrize("shape_of", [lambda n: ((n, 9479), (1,)), lambda n: ((20, n, 300), (2,))])
def test_several_rounds_of_tiles(n, dtype, kind, shape_of):
    # more tiles than CTAs, in rounds that are not full
    shape, dims = shape_of(n)
    a = rand(shape, dtype, seed=n)
    p = dfft.gpu_plan_transform(dfft.R2R((kind,)), to_gpu(a), dims)
    assert p.describe().startswith("tiled"), p.describe()
    y = to_np(dfft.fft(to_gpu(a), dims=dims, transforms=(dfft.R2R((kind,)),)))
    k, m = np.arange(n)[:, None], np.arange(n)[None, :]
    if kind == dfft.REDFT10:
        t = 2 * np.cos(np.pi / n * k * (m + 0.5))
    else:
        t = 2 * np.cos(np.pi / n * (k + 0.5) * m)
        t[:, 0] = 1
    ref = np.moveaxis(np.tensordot(t, a.astype(np.float64), axes=(1, dims[0] - 1)), 0, dims[0] - 1)
    assert rel(y, ref) <= tol_for(dtype)
    assert dfft.device_error() == 0
