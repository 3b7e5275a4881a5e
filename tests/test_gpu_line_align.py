"""Line solves on fields off the boundary of the kernels' vectors, in one launch and
in three: the same bits as on it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve(c0, axis, a, eaxis, f, off_in=0, off_out=0, off_scratch=0, inplace=False):
    import torch
    from pyphasefield_gb300 import _lib as L
    dt = torch.float32 if f == "f32" else torch.float64
    g = L.PpfGrid(ndim=c0.ndim, pitch=(c0.shape[-1] + 3) // 4 * 4)
    for i, n in enumerate(c0.shape):
        g.shape[i] = n
    dims = c0.shape[:-1] + (g.pitch,)
    n = int(np.prod(dims))
    flat = [torch.full((n + 8,), float("nan"), dtype=dt, device="cuda") for _ in range(2)]
    src, dst = flat[0][off_in:off_in + n], flat[1][off_out:off_out + n]
    if inplace:
        dst = src
    src.view(dims)[..., :c0.shape[-1]] = torch.from_numpy(c0)
    nb = C.c_size_t()
    L.call("ppf_implicit_scratch_bytes", C.byref(g), src.element_size(), C.byref(nb))
    sc = torch.empty(nb.value + 64, dtype=torch.uint8, device="cuda")
    L.call(f"ppf_line_solve_{f}", C.byref(g), axis, C.c_double(a), eaxis, C.c_double(a),
           C.c_void_p(src.data_ptr()), C.c_void_p(dst.data_ptr()),
           C.c_void_p(sc.data_ptr() + off_scratch), C.c_size_t(sc.numel() - 64),
           C.c_void_p(torch.cuda.current_stream().cuda_stream))
    out = dst.view(dims)[..., :c0.shape[-1]].cpu().numpy()
    if not inplace:  # nothing written beside the rows
        assert torch.isnan(flat[1][:off_out]).all() and torch.isnan(flat[1][off_out + n:]).all()
    return out


# alpha 300: three launches; 2.5: one, but for the columns of 4500 and 2100 cells
@pytest.mark.parametrize("a", [2.5, 300.0])
@pytest.mark.parametrize("shape, axis", [((33, 21), 0), ((21, 33), 1), ((4500, 5), 0), ((5, 4500), 1),
                                         ((2100, 6), 0), ((6, 2100), 1), ((40, 3, 7), 0),
                                         ((3, 40, 7), 1), ((3, 4, 131), 2)], ids=str)
@pytest.mark.parametrize("f", ["f32", "f64"])
def test_fields_off_the_boundary(cuda, a, shape, axis, f):
    c0 = np.random.default_rng(4).random(shape)
    for eaxis in range(-1, len(shape)):
        ref = solve(c0, axis, a, eaxis, f)
        assert np.isfinite(ref).all()
        for off_in, off_out in ((1, 0), (0, 1), (3, 2)):
            np.testing.assert_array_equal(solve(c0, axis, a, eaxis, f, off_in, off_out), ref)
        if eaxis < 0:
            np.testing.assert_array_equal(solve(c0, axis, a, eaxis, f, off_in=1, inplace=True), ref)


@pytest.mark.parametrize("f", ["f32", "f64"])
def test_scratch_off_the_boundary(cuda, f):
    """Not used by the one launch; the three refuse it."""
    from pyphasefield_gb300 import _lib as L
    c0 = np.random.default_rng(5).random((33, 21))
    np.testing.assert_array_equal(solve(c0, 0, 2.5, -1, f, off_scratch=4), solve(c0, 0, 2.5, -1, f))
    with pytest.raises(L.PpfError, match="aligned"):
        solve(c0, 0, 300.0, -1, f, off_scratch=4)
