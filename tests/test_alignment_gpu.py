"""Arrays that start in the middle of a larger buffer: a contiguous view at an
odd element offset is aligned to its own type only.  Real sides read and
write pairs of such a view element by element; a complex address that is not
a multiple of the element size is an error status, before any launch."""
import ctypes

import numpy as np
import pytest
import torch

import dfft
import dfft_oracle as oracle
from dfft import _lib
from helpers import rand, rel, to_np, tol_for

pytestmark = pytest.mark.gpu


def offset_view(a, order="F", skip=1):
    """Device copy of `a` whose first element is `skip` elements into its buffer."""
    flat = np.concatenate([np.zeros(skip, a.dtype), a.ravel(order=order)])
    t = torch.from_numpy(flat).cuda()[skip:]
    assert t.data_ptr() % (2 * a.itemsize) == (skip % 2) * a.itemsize
    if order == "C":
        return t.view(a.shape)
    return t.view(tuple(reversed(a.shape))).permute(*reversed(range(a.ndim)))


@pytest.mark.parametrize("shape,dims", [((1000, 3), (1,)), ((250, 7), (1,)), ((20, 22, 5), (1, 2, 3)), ((74, 5), (1,)),
                                        ((40002, 2), (1,)), ((6, 250), (2,))])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_rfft_and_irfft_of_offset_views(shape, dims, dtype):
    a = rand(shape, dtype, seed=shape[0])
    x = offset_view(a)
    ref = oracle.rfft(a, dims=dims)
    F = dfft.rfft(x, dims=dims)
    assert rel(to_np(F), ref) <= tol_for(dtype)
    n = shape[dims[0] - 1]
    p = dfft.gpu_plan_transform(dfft.IRFFT(), F, dims, n=n)
    out = offset_view(np.zeros_like(a))
    p.execute(F, out)
    assert rel(to_np(out), a) <= tol_for(dtype)


@pytest.mark.parametrize("dtype,off", [(torch.complex64, 4), (torch.complex128, 8)])
@pytest.mark.parametrize("n", [64, 251, 1200, 5000, 1 << 17])
def test_complex_address_between_elements_is_refused(dtype, off, n):
    x = torch.zeros(2 * n + 2, dtype=dtype, device="cuda")
    p = dfft.gpu_plan_transform(dfft.FFT(), x[:n], (1,))
    L = dfft.lib()
    a, b = x.data_ptr(), x[n + 1:].data_ptr()
    for i, o in ((a + off, b), (a, b + off)):
        assert L.dfft_execute(p._h, i, o, 0) == _lib.ERROR_CUDA
    for persistent in (False, True):
        batch = dfft.Batch([p], persistent=persistent)
        ins, outs = (ctypes.c_void_p * 1)(a + off), (ctypes.c_void_p * 1)(b)
        assert L.dfft_batch_execute(batch._h, ins, outs, None) == _lib.ERROR_CUDA
    torch.cuda.synchronize()
    assert float(x.abs().sum()) == 0
    p.execute(x[:n], x[n:2 * n])
    torch.cuda.synchronize()


def test_no_alloc_entry_point_on_offset_arrays():
    f = dfft.lib().dfft_irfft_noalloc_f32
    f.restype, f.argtypes = ctypes.c_int, [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int,
                                           ctypes.POINTER(ctypes.c_int64), ctypes.c_void_p]
    a = rand((250, 6), np.float32, seed=3)
    F = torch.from_numpy(np.ascontiguousarray(oracle.rfft(a, dims=(1,)).T.astype(np.complex64))).cuda()
    out = offset_view(np.zeros_like(a))
    shape = (ctypes.c_int64 * 2)(250, 6)
    assert f(F.data_ptr() + 4, out.data_ptr(), 2, shape, None) == _lib.ERROR_INVALID_VALUE
    ref = to_np(dfft.irfft(F.permute(1, 0), 250, dims=(1, 2)))
    assert f(F.data_ptr(), out.data_ptr(), 2, shape, None) == 0
    torch.cuda.synchronize()
    assert rel(to_np(out), ref) <= 1e-5


@pytest.mark.parametrize("n", [128, 256, 512])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", [dfft.REDFT10, dfft.REDFT01])
@pytest.mark.parametrize("cols,strided", [(1, False), (13, False), (16, False), (4, True), (16, True)])
def test_dct_of_offset_views(n, dtype, kind, cols, strided):
    shape, dims = ((cols, n, 3), (2,)) if strided else ((n, cols), (1,))
    a = rand(shape, dtype, seed=n + cols)
    x = offset_view(a)
    tr = (dfft.R2R((kind,)),)
    p = dfft.gpu_plan_transform(tr[0], x, dims)
    if cols != 4 or n == 512:  # (four columns: narrower than the tiles of 128 and 256)
        assert p.describe().startswith("tiled"), p.describe()
    ref = oracle.fft(a, dims=dims, transforms=(oracle.R2R((kind,)),))
    assert rel(to_np(dfft.fft(x, dims=dims, transforms=tr)), ref) <= tol_for(dtype)  # input between 16 bytes
    out = offset_view(np.zeros_like(a))
    p.execute(offset_view(a, skip=0), out)
    assert rel(to_np(out), ref) <= tol_for(dtype)  # output
    p.execute(x, x)
    assert rel(to_np(x), ref) <= tol_for(dtype)  # in place


@pytest.mark.parametrize("shape,dims", [((1 << 17,), (1,)), ((1 << 20,), (1,)), ((45000, 3), (1,)), ((3, 20480, 2), (2,)),
                                        ((143 * 128, 2), (1,)), ((20011, 2), (1,)), ((2, 40009), (2,))])
def test_long_axes_of_offset_views(shape, dims):
    a = rand(shape, np.complex64, seed=len(shape))
    x = offset_view(a)
    ref = oracle.fft(a, dims=dims)
    p = dfft.gpu_plan_transform(dfft.FFT(), x, dims)
    assert "four-step" in p.describe(), p.describe()
    out = offset_view(np.zeros_like(a))
    p.execute(x, out)
    assert rel(to_np(out), ref) <= tol_for(np.complex64)
    dfft.fft_(x, dims=dims)
    assert rel(to_np(x), ref) <= tol_for(np.complex64)
    dfft.ifft_(x, dims=dims)
    assert rel(to_np(x), a) <= tol_for(np.complex64)
