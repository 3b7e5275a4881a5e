"""Periodic line solves at the lengths where the segment length, the number
of scan batches or the kernel changes."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

A = 2.5
# the system's condition number is below 1 + 4 a = 11; tens of roundings per cell
TOL = {"f64": 1e-13, "f32": 1e-5}


def reference(c, axis, eaxis):
    """(1 - 2a) c + a (neighbours along eaxis), then the solve, by FFT."""
    if eaxis >= 0:
        c = (1 - 2 * A) * c + A * (np.roll(c, 1, eaxis) + np.roll(c, -1, eaxis))
    n = c.shape[axis]
    lam = 1 + 2 * A * (1 - np.cos(2 * np.pi * np.arange(n // 2 + 1) / n))
    lam = lam.reshape([-1 if k == axis else 1 for k in range(c.ndim)])
    return np.fft.irfft(np.fft.rfft(c, axis=axis) / lam, n=n, axis=axis)


def solve(c0, axis, eaxis, f, offset=0):
    import torch
    from pyphasefield_gb300 import _lib as L
    dt = torch.float32 if f == "f32" else torch.float64
    g = L.PpfGrid(ndim=c0.ndim, pitch=(c0.shape[-1] + 3) // 4 * 4)
    for i, n in enumerate(c0.shape):
        g.shape[i] = n
    dims = c0.shape[:-1] + (g.pitch,)
    bufs = [torch.full((int(np.prod(dims)) + 8,), float("nan"), dtype=dt, device="cuda")
            [offset:offset + int(np.prod(dims))] for _ in range(2)]
    src, dst = (b.view(dims)[..., :c0.shape[-1]] for b in bufs)
    src.copy_(torch.from_numpy(c0))
    nb = C.c_size_t()
    L.call("ppf_implicit_scratch_bytes", C.byref(g), src.element_size(), C.byref(nb))
    sc = torch.empty(max(16, nb.value), dtype=torch.uint8, device="cuda")
    L.call(f"ppf_line_solve_{f}", C.byref(g), axis, C.c_double(A), eaxis, C.c_double(A),
           C.c_void_p(bufs[0].data_ptr()), C.c_void_p(bufs[1].data_ptr()),
           C.c_void_p(sc.data_ptr()), C.c_size_t(sc.numel()),
           C.c_void_p(torch.cuda.current_stream().cuda_stream))
    return dst.double().cpu().numpy()


@pytest.mark.parametrize("n", [3, 7, 8, 9, 31, 33, 257, 264, 265, 512, 513, 1023, 1040, 1041, 1536,
                               1537, 2048, 2049, 2081, 4095, 4096, 4097])
@pytest.mark.parametrize("f", ["f32", "f64"])
def test_line_lengths(cuda, n, f):
    rng = np.random.default_rng(n)
    for shape, axis in (((n, 13), 0), ((13, n), 1), ((n, 4, 9), 0), ((3, n, 5), 1), ((3, 4, n), 2)):
        c0 = rng.random(shape)
        for eaxis in range(-1, len(shape)):
            if eaxis >= 0 and shape[eaxis] < 3:
                continue
            got, ref = solve(c0, axis, eaxis, f), reference(c0, axis, eaxis)
            err = np.linalg.norm(got - ref) / np.linalg.norm(ref)
            assert err < TOL[f], (shape, axis, eaxis, err)


@pytest.mark.parametrize("f", ["f32", "f64"])
@pytest.mark.parametrize("shape", [(300, 1030), (1030, 1100), (1600, 2700), (70, 256, 256)])
def test_grid_sizes(cuda, f, shape):
    """Cell counts on both sides of the segment-length rule."""
    c0 = np.random.default_rng(1).random(shape)
    for axis in range(len(shape)):
        for eaxis in (-1, axis):
            got, ref = solve(c0, axis, eaxis, f), reference(c0, axis, eaxis)
            assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < TOL[f], (axis, eaxis)


@pytest.mark.parametrize("f", ["f32", "f64"])
def test_misaligned_rows(cuda, f):
    """Rows off the 16-byte boundary are copied cell by cell."""
    c0 = np.random.default_rng(2).random((21, 133))
    for eaxis in (-1, 0, 1):
        np.testing.assert_array_equal(solve(c0, 1, eaxis, f), solve(c0, 1, eaxis, f, offset=1))
