"""Periodic line solves over the whole range of alpha, on both sides of the
limits of the one-launch kernel and of its divided half step."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = {"f32": 2.0 ** -24, "f64": 2.0 ** -53}
# tens of roundings per cell, none amplified by the implicit part (sums of
# positive terms, scaled by their own gain)
TOL = {"f32": 1e-5, "f64": 1e-13}


def reference(c, axis, a, eaxis, ea):
    c = c.astype(np.longdouble)
    if eaxis >= 0:
        c = c + ea * ((np.roll(c, 1, eaxis) - c) + (np.roll(c, -1, eaxis) - c))
    n = c.shape[axis]
    lam = 1 + 4 * np.longdouble(a) * np.sin(np.pi * np.arange(n // 2 + 1, dtype=np.longdouble) / n) ** 2
    lam = lam.reshape([-1 if k == axis else 1 for k in range(c.ndim)])
    return np.fft.irfft(np.fft.rfft(c, axis=axis) / lam, n=n, axis=axis).astype(np.float64)


def solve(c0, axis, a, eaxis, ea, f):
    import torch
    from pyphasefield_gb300 import _lib as L
    g = L.PpfGrid(ndim=2, pitch=(c0.shape[1] + 3) // 4 * 4)
    g.shape[0], g.shape[1] = c0.shape
    bufs = [torch.zeros(c0.shape[0], g.pitch, device="cuda",
                        dtype=torch.float32 if f == "f32" else torch.float64) for _ in range(2)]
    bufs[0][:, :c0.shape[1]] = torch.from_numpy(c0)
    nb = C.c_size_t()
    L.call("ppf_implicit_scratch_bytes", C.byref(g), bufs[0].element_size(), C.byref(nb))
    sc = torch.empty(max(16, nb.value), dtype=torch.uint8, device="cuda")
    L.call(f"ppf_line_solve_{f}", C.byref(g), axis, C.c_double(a), eaxis, C.c_double(ea),
           C.c_void_p(bufs[0].data_ptr()), C.c_void_p(bufs[1].data_ptr()),
           C.c_void_p(sc.data_ptr()), C.c_size_t(sc.numel()),
           C.c_void_p(torch.cuda.current_stream().cuda_stream))
    return bufs[1][:, :c0.shape[1]].double().cpu().numpy()


def field(shape, f):
    c = np.random.default_rng(sum(shape)).random(shape)
    return c.astype(np.float32).astype(np.float64) if f == "f32" else c


def bound(f, a, eaxis, axis, ea):
    # the root is formed in double: 1 - r to sqrt(a) ulps, the gain to twice that
    tol = TOL[f] + 8 * EPS["f64"] * np.sqrt(a)
    if eaxis == axis:
        # the half step's roundings, ea |c| ulps in every mode, against a result
        # that the solve has brought back to the size of c
        tol += 16 * EPS[f] * ea
    return tol


@pytest.mark.parametrize("a", [0.0, 1e-6, 2e-3, 0.5, 3.9, 4.1, 60.0, 127.0, 129.0, 1e4, 3e5, 2e7, 1e12,
                               1e16, 1e18])
@pytest.mark.parametrize("f", ["f32", "f64"])
def test_any_alpha(cuda, f, a):
    for shape, axis in (((300, 20), 0), ((20, 300), 1), ((19, 1100), 1), ((5, 4100), 1)):
        c0 = field(shape, f)
        for eaxis in (-1, 0, 1):
            got, ref = solve(c0, axis, a, eaxis, a, f), reference(c0, axis, a, eaxis, a)
            assert np.isfinite(got).all(), (shape, axis, eaxis)
            err = np.linalg.norm(got - ref) / np.linalg.norm(ref)
            assert err < bound(f, a, eaxis, axis, a), (shape, axis, eaxis, err)


@pytest.mark.parametrize("ea", [1e-3, 1.0, 4.0, 12345.0, 12345678.9, 1e12, 1e16])
@pytest.mark.parametrize("f", ["f32", "f64"])
def test_explicit_weight_of_its_own(cuda, f, ea):
    """The explicit part's weight far from the implicit one's; a uniform field
    comes back as it was."""
    for shape, axis in (((300, 20), 0), ((20, 300), 1)):
        for eaxis in (0, 1):
            c0 = field(shape, f)
            got, ref = solve(c0, axis, 2.5, eaxis, ea, f), reference(c0, axis, 2.5, eaxis, ea)
            err = np.linalg.norm(got - ref) / np.linalg.norm(ref)
            assert err < TOL[f], (shape, axis, eaxis, err)
            one = np.full(shape, 0.75)
            np.testing.assert_allclose(solve(one, axis, 2.5, eaxis, ea, f), one, rtol=TOL[f])
