"""A native run of steps that a pass refuses half way."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_passes_before_the_refused_one_are_reported(cuda):
    import torch
    from pyphasefield_gb300 import _lib as L
    params = L.PpfDiffusionParams(1.0, 0.1, 1.0)
    grid = L.PpfGrid(ndim=2, pitch=64)
    grid.shape[0] = grid.shape[1] = 64
    bc, tiling = L.PpfBoundary(), L.PpfTiling()
    a = torch.rand(64, 64, device="cuda")
    b, a1, b1 = (torch.zeros_like(a) for _ in range(3))
    a1.copy_(a)
    s = torch.cuda.current_stream().cuda_stream

    def run(x, y, depths):
        r = L.PpfRun(model=L.PPF_RUN_DIFFUSION, elem_bytes=4)
        r.params, r.grid = C.addressof(params), C.pointer(grid)
        r.boundary, r.tiling = C.pointer(bc), C.pointer(tiling)
        r.a[0], r.b[0] = x.data_ptr(), y.data_ptr()
        n = len(depths)
        L.call("ppf_run", C.byref(r), (C.c_int32 * n)(*depths), n, None, s)

    done = C.c_int32()
    run(a1, b1, [3])
    L.call("ppf_run_passes", C.byref(done))
    assert done.value == 1
    with pytest.raises(L.PpfError, match="depth=9"):
        run(a, b, [3, 9])
    L.call("ppf_run_passes", C.byref(done))
    assert done.value == 1
    assert torch.equal(b, b1) and torch.equal(a, a1)
