"""A chunk length below 1 leaves the choice to the kernels that choose it
themselves; the tile kernel refuses it."""
import numpy as np
import pytest

from tests.helpers import run_single_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model, kw", [("diffusion", dict(D=1.0)),
                                       ("cahn_hilliard", dict(M=1.0, epsilon=1.0, centered=1))])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_chunk_below_one(cuda, model, kw, precision):
    c0 = np.random.default_rng(3).random((6, 20, 70))
    ref = run_single_gpu(model, c0, 2, "PERIODIC", 1.0, 0.01, precision=precision, **kw)
    got = run_single_gpu(model, c0, 2, "PERIODIC", 1.0, 0.01, precision=precision, zchunk=-1, **kw)
    np.testing.assert_array_equal(got, ref)


def test_tiles_refuse_it(cuda):
    from pyphasefield_gb300 import _lib as L
    with pytest.raises(L.PpfError, match="zchunk"):
        run_single_gpu("diffusion", np.zeros((6, 20, 70)), 1, "PERIODIC", 1.0, 0.1, zchunk=-1,
                       tile=(64, 8), D=1.0)
