"""The float Cahn-Hilliard kernel at the sizes where its edge handling changes
(a vector, a strip, a warp's rows, a chunk of planes, one plane)."""
import numpy as np
import pytest

from oracle import restate
from tests.helpers import rel_l2, run_single_gpu

pytestmark = pytest.mark.gpu

Q = 2.0 ** -24
KW = dict(M=1.0, epsilon=1.0)


@pytest.mark.parametrize("shape", [(3, 3), (5, 130), (18, 127), (17, 256), (1, 5, 126), (2, 4, 125),
                                   (3, 5, 128), (5, 6, 129), (9, 17, 131), (40, 3, 259)])
@pytest.mark.parametrize("bc", ["PERIODIC", "NEUMANN", "MIXED"])
def test_march_edges(cuda, shape, bc):
    """Against the float64 oracle (2.5e-6: a few hundred roundings of 2^-25 on
    a field of about 1/2 in four steps), bit-identical for every chunk length,
    and the mass of the quantised steps exactly conserved."""
    bc = [["NEUMANN", "PERIODIC", "NEUMANN"][a] for a in range(len(shape))] if bc == "MIXED" else bc
    rng = np.random.default_rng(3)
    c0 = 0.5 + np.rint(rng.uniform(-0.05, 0.05, shape) / Q) * Q
    ref = restate.run_single("cahn_hilliard", c0, 4, bc, 1.0, 0.01, **KW)
    for quantum, centered in ((Q, 1), (0.0, 1), (0.0, 0)):
        out = run_single_gpu("cahn_hilliard", c0, 4, bc, 1.0, 0.01, precision="fp32",
                             quantum=quantum, centered=centered, **KW)
        assert rel_l2(out, ref) < 2.5e-6, (quantum, centered)
        for z in (1, 2, 3):
            np.testing.assert_array_equal(out, run_single_gpu(
                "cahn_hilliard", c0, 4, bc, 1.0, 0.01, precision="fp32", quantum=quantum,
                centered=centered, zchunk=z, **KW))
        if quantum:
            assert np.sum(out - 0.5) == np.sum(c0 - 0.5)


@pytest.mark.parametrize("shape", [(70, 300), (20, 30, 140)])
def test_mass_history_is_exact(cuda, shape):
    from pyphasefield_gb300 import CahnHilliardGB300
    rng = np.random.default_rng(4)
    sim = CahnHilliardGB300(dimensions=list(shape), dx=1.0, dt=0.01, boundary_conditions="NEUMANN",
                            user_data=dict(KW, graph_chunk=10))
    sim.initialize_fields_and_imported_data()
    u = np.rint(rng.uniform(-0.05, 0.05, shape) / Q) * Q
    sim.fields[0].data[(slice(1, -1),) * len(shape)] = 0.5 + u
    sim.simulate(25)
    m = sim.collect_mass_history()
    assert len(m) == 25 and np.all(m == np.sum(u) + 0.5 * u.size)
