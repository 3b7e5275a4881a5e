"""Depths of a native run of steps: models of one step per pass (no GPU)."""
import ctypes as C

import pytest


@pytest.mark.parametrize("depths", [(2,), (1, 3)])
@pytest.mark.parametrize("model", ["CAHN_HILLIARD", "WARREN1995", "DIFFUSION_IMPLICIT",
                                   "PHASE_IMPLICIT", "NCGPU"])
def test_more_than_one_step_per_pass_is_refused(model, depths):
    """Before any launch: the noise step would run ahead of the steps taken."""
    from pyphasefield_gb300 import _lib as L
    if not L.LIB_PATH.exists():
        pytest.skip("library not built")
    params = (C.c_char * 512)()
    grid = L.PpfGrid(ndim=2, pitch=8)
    grid.shape[0] = grid.shape[1] = 8
    run = L.PpfRun(model=getattr(L, "PPF_RUN_" + model), elem_bytes=4)
    run.params, run.grid = C.addressof(params), C.pointer(grid)
    n = len(depths)
    with pytest.raises(L.PpfError, match=f"one step per pass .depth={max(depths)}") as e:
        L.call("ppf_run", C.byref(run), (C.c_int32 * n)(*depths), n, None, None)
    assert e.value.code == L.PPF_ERR_UNSUPPORTED
