"""2-D Diffusion / Allen-Cahn kernels at the sizes where their edge handling
changes: rows and columns around a vector, a warp's strip and its bands."""
import ctypes as C

import numpy as np
import pytest

from oracle import restate
from tests.helpers import make_structs, rel_l2, run_single_gpu

pytestmark = pytest.mark.gpu

BCS = ["PERIODIC", "NEUMANN", "DIRCHLET", ["DIRCHLET", "PERIODIC"], ["NEUMANN", "DIRCHLET"]]


def face_values(bc, nd=2):
    bcs = [bc] * nd if isinstance(bc, str) else bc
    return [[[0.25, 0.5] if b != "PERIODIC" else [0.0, 0.0] for b in bcs]]


@pytest.mark.parametrize("shape", [(1, 4), (2, 5), (3, 1), (15, 127), (16, 128), (17, 129),
                                   (18, 258), (33, 63), (5, 64), (4, 65)])
@pytest.mark.parametrize("bc", BCS, ids=str)
def test_single_step_edges(cuda, shape, bc):
    """Depth 1 against the tile kernel, whose every edge cell goes through the
    per-cell rule (bit for bit), and the float64 oracle; gradients and fixed
    values on the faces."""
    c0 = np.random.default_rng(5).random(shape)
    vals = face_values(bc)
    kw = dict(M=0.1, epsilon=1.0, W=1.0)
    for prec in ("fp32", "fp64"):
        a = run_single_gpu("allen_cahn", c0, 3, bc, 1.0, 0.1, values=vals, precision=prec, **kw)
        b = run_single_gpu("allen_cahn", c0, 3, bc, 1.0, 0.1, values=vals, precision=prec,
                           tile=(64, 8), **kw)
        np.testing.assert_array_equal(a, b)
    ref = restate.run_single("allen_cahn", c0, 3, bc, 1.0, 0.1, values=vals, **kw)
    assert rel_l2(a, ref) < 1e-12


@pytest.mark.parametrize("offset", [1, 2, 4])
def test_single_step_misaligned_rows(cuda, offset):
    """Field pointers off the 16-byte boundary take scalar loads and stores,
    with the same result."""
    import torch
    from pyphasefield_gb300 import _lib as L
    shape = (37, 131)
    g, b, _, pitch = make_structs(shape, "NEUMANN")
    c0 = np.random.default_rng(6).random(shape)
    p = L.PpfDiffusionParams(1.0, 0.1, 1.0)
    t = L.PpfTiling(depth=1)
    got = []
    for off in (0, offset):
        bufs = [torch.zeros(shape[0] * pitch + 8, device="cuda")[off:off + shape[0] * pitch]
                for _ in range(2)]
        bufs[0].view(shape[0], pitch)[:, :shape[1]] = torch.from_numpy(c0)
        L.call("ppf_diffusion_step_f32", C.byref(p), C.byref(g), C.byref(b),
               C.c_void_p(bufs[0].data_ptr()), C.c_void_p(bufs[1].data_ptr()), C.byref(t),
               C.c_void_p(torch.cuda.current_stream().cuda_stream))
        got.append(bufs[1].view(shape[0], pitch)[:, :shape[1]].cpu().numpy())
    np.testing.assert_array_equal(got[0], got[1])


# one grid per block shape of the several-step kernel, odd sides
@pytest.mark.parametrize("shape", [(3, 7), (61, 203), (501, 301), (777, 515), (1101, 2103)])
@pytest.mark.parametrize("depth", [2, 5, 8])
def test_block_kernel_equals_single_steps(cuda, shape, depth):
    """Passes of several steps (float) equal single steps bit for bit."""
    c0 = np.random.default_rng(7).random(shape)
    for model, kw in (("diffusion", dict(D=1.0)), ("allen_cahn", dict(M=0.1, epsilon=1.0, W=1.0))):
        for bc in BCS:
            vals = [[v if b == "DIRCHLET" else [0.0, 0.0]
                     for v, b in zip(face_values(bc)[0], [bc] * 2 if isinstance(bc, str) else bc)]]
            a = run_single_gpu(model, c0, depth + 2, bc, 1.0, 0.1, values=vals, precision="fp32", **kw)
            b = run_single_gpu(model, c0, depth + 2, bc, 1.0, 0.1, values=vals, precision="fp32",
                               depth=depth, **kw)
            np.testing.assert_array_equal(a, b)


# grids of the tallest blocks (8 warps of twelve rows at one and at more blocks per SM,
# 16 of four, 12 of six)
@pytest.mark.parametrize("shape", [(1021, 1030), (1303, 1999), (1203, 1190), (1303, 1301)])
@pytest.mark.parametrize("bc", ["PERIODIC", ["NEUMANN", "DIRCHLET"]], ids=str)
def test_tall_blocks_equal_single_steps(cuda, shape, bc):
    c0 = np.random.default_rng(8).random(shape)
    vals = [[v if b == "DIRCHLET" else [0.0, 0.0]
             for v, b in zip(face_values(bc)[0], [bc] * 2 if isinstance(bc, str) else bc)]]
    kw = dict(M=0.1, epsilon=1.0, W=1.0, values=vals, precision="fp32")
    a = run_single_gpu("allen_cahn", c0, 11, bc, 1.0, 0.1, **kw)
    b = run_single_gpu("allen_cahn", c0, 11, bc, 1.0, 0.1, depth=8, **kw)
    np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("steps", [1, 7, 50, 100, 131])
@pytest.mark.parametrize("gradient", [0.0, 0.5])
def test_engine_default_depth_equals_single_steps(cuda, steps, gradient):
    """The engine's own steps per pass (graphs and the remainder) against
    one launch per step; a face gradient keeps single steps."""
    from pyphasefield_gb300 import DiffusionGB300
    c0 = np.random.default_rng(8).random((70, 150))
    vals = [[[gradient, 0.0], [0.0, 0.0]]]
    sim = DiffusionGB300(dimensions=[70, 150], dx=1.0, dt=0.1, boundary_conditions="NEUMANN",
                         user_data={"D": 1.0, "graph_chunk": 24})
    sim.initialize_fields_and_imported_data()
    sim._boundary_conditions_array[0][0, :] = gradient
    sim.fields[0].data[1:-1, 1:-1] = c0
    sim.simulate(steps)
    assert sim._ppf_auto_depth() == (8 if gradient == 0 else 1)
    sim.retrieve_fields_from_GPU()
    ref = run_single_gpu("diffusion", c0, steps, "NEUMANN", 1.0, 0.1, values=vals,
                         precision="fp32", D=1.0)
    np.testing.assert_array_equal(sim.fields[0].get_cells(), ref)
