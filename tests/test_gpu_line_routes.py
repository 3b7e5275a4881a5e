"""Periodic line solves at the edges of the one-launch kernel's rules."""
import numpy as np
import pytest

from tests.test_gpu_line_alpha import TOL, solve
from tests.test_gpu_line_fused import A, reference

pytestmark = pytest.mark.gpu


def check(shape, axis, f, eaxes=(-1, 0, 1)):
    c0 = np.random.default_rng(shape[0] + shape[1]).random(shape)
    if f == "f32":
        c0 = c0.astype(np.float32).astype(np.float64)
    for eaxis in eaxes:
        got, ref = solve(c0, axis, A, eaxis, A, f), reference(c0, axis, eaxis)
        err = np.linalg.norm(got - ref) / np.linalg.norm(ref)
        assert err < TOL[f], (shape, axis, eaxis, err)


# eight segments (a thread per line closes the carries) and nine, of 8 and of 16 cells
@pytest.mark.parametrize("n, lines", [(3, 300), (63, 7), (64, 130), (65, 33), (128, 9000), (129, 9000)])
@pytest.mark.parametrize("f", ["f32", "f64"])
def test_short_lines(cuda, n, lines, f):
    check((n, lines), 0, f)
    check((lines, n), 1, f)


# the half step along another axis: vectors, a row's ragged end, rows off the boundary
# (a pitch that is a multiple of 4 keeps every row of a 16-byte aligned field on it)
@pytest.mark.parametrize("n", [4, 5, 127, 128, 130, 1100, 2047])
@pytest.mark.parametrize("f", ["f32", "f64"])
def test_half_step_along_another_axis(cuda, n, f):
    check((37, n), 1, f, eaxes=(0,))


# lines of 1537 to 2048 cells by 16 (below 300 lines) and by 32 cells; longer ones on
# both sides of the three launches' rule
@pytest.mark.parametrize("n, lines", [(1600, 299), (1600, 300), (2048, 3), (2049, 1), (2049, 2),
                                      (2100, 63), (2100, 64), (2100, 99), (2100, 100), (2100, 601),
                                      (2561, 255), (2561, 256), (3501, 127), (3501, 128),
                                      (1201, 7000), (801, 10500)])
@pytest.mark.parametrize("f", ["f32", "f64"])
def test_long_lines(cuda, n, lines, f):
    eaxes = (-1, 0, 1) if lines >= 3 else (-1,)
    check((n, lines), 0, f, eaxes=eaxes)
    check((lines, n), 1, f, eaxes=eaxes)
