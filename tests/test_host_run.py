"""Argument checks of the native run of steps (no GPU)."""
import ctypes as C

import pytest


@pytest.mark.parametrize("change, message", [
    (dict(elem_bytes=2), "elem_bytes"), (dict(model=99), "unknown"), (dict(params=None), "NULL"),
    (dict(depth=0), "depth")])
def test_run_rejects_bad_arguments(change, message):
    from pyphasefield_gb300 import _lib as L
    if not L.LIB_PATH.exists():
        pytest.skip("library not built")
    params = L.PpfDiffusionParams(1.0, 0.1, 1.0)
    grid = L.PpfGrid(ndim=2, pitch=8)
    grid.shape[0] = grid.shape[1] = 8
    run = L.PpfRun(model=L.PPF_RUN_DIFFUSION, elem_bytes=4)
    run.params, run.grid = C.addressof(params), C.pointer(grid)
    depth = change.pop("depth", 1)
    for k, v in change.items():
        setattr(run, k, v)
    with pytest.raises(L.PpfError, match=message):
        L.call("ppf_run", C.byref(run), (C.c_int32 * 1)(depth), 1, None, None)
