"""3-D Diffusion / Allen-Cahn steps at the sizes where the default kernel's
edge handling changes (a vector, a strip, a warp's rows, a chunk of planes),
against the tile kernel, whose edge cells go through the per-cell rule (bit for
bit), and the float64 oracle."""
import numpy as np
import pytest

from oracle import restate
from tests.helpers import rel_l2, run_single_gpu

pytestmark = pytest.mark.gpu

BCS = ["PERIODIC", "NEUMANN", "DIRCHLET", ["NEUMANN", "DIRCHLET", "PERIODIC"],
       ["PERIODIC", "NEUMANN", "DIRCHLET"]]


@pytest.mark.parametrize("shape", [(1, 1, 4), (2, 3, 5), (3, 4, 127), (4, 5, 128), (5, 16, 129),
                                   (9, 17, 63), (8, 33, 131), (3, 2, 260), (17, 15, 64)])
@pytest.mark.parametrize("bc", BCS, ids=str)
def test_single_step_edges(cuda, shape, bc):
    c0 = np.random.default_rng(5).random(shape)
    bcs = [bc] * 3 if isinstance(bc, str) else bc
    vals = [[[0.25, 0.5] if b != "PERIODIC" else [0.0, 0.0] for b in bcs]]
    for model, kw in (("diffusion", dict(D=1.0)), ("allen_cahn", dict(M=0.1, epsilon=1.0, W=1.0))):
        for prec in ("fp32", "fp64"):
            a = run_single_gpu(model, c0, 3, bc, 1.0, 0.1, values=vals, precision=prec, **kw)
            for z in (1, 3):
                np.testing.assert_array_equal(
                    a, run_single_gpu(model, c0, 3, bc, 1.0, 0.1, values=vals, precision=prec,
                                      zchunk=z, **kw))
            b = run_single_gpu(model, c0, 3, bc, 1.0, 0.1, values=vals, precision=prec,
                               tile=(64, 8), **kw)
            np.testing.assert_array_equal(a, b)
        ref = restate.run_single(model, c0, 3, bc, 1.0, 0.1, values=vals, **kw)
        assert rel_l2(a, ref) < 1e-12


# short rows: groups of 16 and 8 lanes (float and double change over at different
# widths), ragged in x and with the last groups past the grid in y
@pytest.mark.parametrize("shape", [(3, 37, 24), (5, 70, 17), (4, 90, 40), (3, 61, 34), (2, 83, 140),
                                   (3, 45, 64), (4, 129, 90)])
@pytest.mark.parametrize("bc", BCS, ids=str)
def test_short_rows(cuda, shape, bc):
    test_single_step_edges(cuda, shape, bc)
