"""3-D steps (and 2-D Cahn-Hilliard) with an output off the 16-byte boundary:
the same bits as with an aligned one. An input off it is refused."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import make_structs

pytestmark = pytest.mark.gpu

MODELS = {"diffusion": dict(D=1.0), "allen_cahn": dict(M=0.1, epsilon=1.0, W=1.0),
          "cahn_hilliard": dict(M=1.0, epsilon=1.0)}


def step(model, sfx, shape, bc, off_in, off_out):
    import torch
    from pyphasefield_gb300 import _lib as L
    dtype = torch.float32 if sfx == "f32" else torch.float64
    g, b, kshape, pitch = make_structs(shape, bc)
    dims = kshape[:-1] + (pitch,)
    n = int(np.prod(dims))
    c0 = np.random.default_rng(9).uniform(-0.05, 0.05, kshape)
    bufs = [torch.zeros(n + 4, dtype=dtype, device="cuda")[o:o + n].view(dims)
            for o in (off_in, off_out)]
    bufs[0][..., :kshape[-1]] = torch.from_numpy(c0)
    kw = MODELS[model]
    args = [C.c_void_p(t.data_ptr()) for t in bufs]
    if model == "diffusion":
        p = L.PpfDiffusionParams(1.0, 0.1, kw["D"])
    elif model == "allen_cahn":
        p = L.PpfAllenCahnParams(1.0, 0.1, kw["M"], kw["epsilon"], kw["W"])
    else:
        p = L.PpfCahnHilliardParams(1.0, 0.01, kw["M"], kw["epsilon"],
                                    2.0 ** -24 if sfx == "f32" else 0.0)
        p.centered = 1
        args += [None, None]
    L.call(f"ppf_{model}_step_{sfx}", C.byref(p), C.byref(g), C.byref(b), *args,
           C.byref(L.PpfTiling()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    return bufs[1][..., :kshape[-1]].cpu().numpy()


@pytest.mark.parametrize("model, shape", [
    ("diffusion", (5, 18, 131)), ("diffusion", (3, 40, 20)), ("allen_cahn", (5, 33, 130)),
    ("cahn_hilliard", (5, 18, 131)), ("cahn_hilliard", (3, 17, 256)),
    ("cahn_hilliard", (40, 130))], ids=str)
@pytest.mark.parametrize("sfx", ["f32", "f64"])
@pytest.mark.parametrize("bc", ["PERIODIC", "NEUMANN"])
def test_output_off_the_boundary(cuda, model, shape, sfx, bc):
    from pyphasefield_gb300 import _lib as L
    ref = step(model, sfx, shape, bc, 0, 0)
    np.testing.assert_array_equal(step(model, sfx, shape, bc, 0, 1), ref)
    with pytest.raises(L.PpfError, match="16-byte aligned"):
        step(model, sfx, shape, bc, 1, 0)
