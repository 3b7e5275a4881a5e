"""3-D steps (and 2-D Cahn-Hilliard, one plane) on grids with more row bands, or
more chunks of planes, than one dimension of a launch holds (65535)."""
import numpy as np
import pytest

from oracle import restate
from tests.helpers import rel_l2, run_single_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape, precision", [
    ((1, 600001, 6), "fp64"),    # 8 to 32 rows a block
    ((2, 1100003, 4), "fp32"),   # 16 to 64
    ((700001, 1, 3), "fp32"),    # 8 planes a chunk
    ((700001, 2, 3), "fp64")], ids=str)
@pytest.mark.parametrize("bc", ["PERIODIC", "NEUMANN"])
def test_long_axes(cuda, shape, precision, bc):
    c0 = np.random.default_rng(6).random(shape)
    got = run_single_gpu("diffusion", c0, 2, bc, 1.0, 0.1, precision=precision, D=1.0)
    ref = restate.run_single("diffusion", c0, 2, bc, 1.0, 0.1, D=1.0)
    # a dozen roundings a step
    assert rel_l2(got, ref) < (1e-6 if precision == "fp32" else 1e-14)


def test_rows_of_32_lanes(cuda):
    """Eight rows a block in double."""
    shape = (1, 524400, 64)
    c0 = np.random.default_rng(7).random(shape)
    got = run_single_gpu("diffusion", c0, 1, "NEUMANN", 1.0, 0.1, precision="fp64", D=1.0)
    ref = restate.run_single("diffusion", c0, 1, "NEUMANN", 1.0, 0.1, D=1.0)
    assert rel_l2(got, ref) < 1e-14


@pytest.mark.parametrize("shape", [(1100003, 4), (1, 1050007, 3), (2, 1048600, 4)], ids=str)
def test_cahn_hilliard_long_axes(cuda, shape):
    q = 2.0 ** -24
    c0 = 0.5 + np.rint(np.random.default_rng(8).uniform(-0.05, 0.05, shape) / q) * q
    got = run_single_gpu("cahn_hilliard", c0, 2, "PERIODIC", 1.0, 0.01, precision="fp32", quantum=q,
                         centered=1, M=1.0, epsilon=1.0)
    ref = restate.run_single("cahn_hilliard", c0, 2, "PERIODIC", 1.0, 0.01, M=1.0, epsilon=1.0)
    assert rel_l2(got, ref) < 2.5e-6
    assert np.sum(got - 0.5) == np.sum(c0 - 0.5)
