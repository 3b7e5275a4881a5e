"""The engines' watch: a non-finite cell anywhere raises its bit, padding never does."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def watch(fields, grid, prec):
    import torch
    from pyphasefield_gb300 import _lib as L
    status, counter = (torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(2))
    host = torch.zeros(1, dtype=torch.int32, pin_memory=True)
    L.call("ppf_watch_" + prec, (C.c_void_p * len(fields))(*[f.data_ptr() for f in fields]),
           len(fields), C.byref(grid), C.c_void_p(status.data_ptr()),
           C.c_void_p(counter.data_ptr()), C.c_void_p(host.data_ptr()),
           C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert int(counter) == 0 and int(status) == int(host)
    return int(host)


# whole vectors and ragged rows, a shifted pointer (single cells), planes,
# more cells than one sweep of the launch holds
@pytest.mark.parametrize("shape,pitch,shift", [((1, 3), 32, 0), ((7, 64), 64, 0), ((5, 37), 64, 0),
                                               ((5, 37), 40, 0), ((5, 37), 64, 1),
                                               ((3, 4, 21), 32, 0), ((1700, 1501), 1504, 0)])
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_watch_finds_every_cell(cuda, shape, pitch, shift, prec):
    import torch
    from pyphasefield_gb300 import _lib as L
    grid = L.PpfGrid(ndim=len(shape), pitch=pitch)
    for i, n in enumerate(shape):
        grid.shape[i] = n
    ny, nx = shape[-2:]
    nz = shape[0] if len(shape) == 3 else 1
    plane = pitch * ny
    dtype = torch.float32 if prec == "f32" else torch.float64
    bufs = [torch.full((nz * plane + 4,), float("nan"), dtype=dtype, device="cuda")[shift:]
            for _ in range(2)]
    views = [b[:nz * plane].view(nz, ny, pitch)[:, :, :nx] for b in bufs]
    for v in views:
        v.fill_(1.0)
    assert watch(bufs, grid, prec) == 0
    for z, y, x in {(0, 0, 0), (nz - 1, ny - 1, nx - 1), (0, ny - 1, 0), (nz - 1, 0, nx - 1),
                    (nz // 2, ny // 2, nx // 2)}:
        for f, bad in ((0, float("inf")), (1, float("nan"))):
            views[f][z, y, x] = bad
            assert watch(bufs, grid, prec) == L.PPF_STATUS_NONFINITE
            views[f][z, y, x] = 1.0
    assert watch(bufs, grid, prec) == 0
