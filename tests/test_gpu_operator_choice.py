"""The CG operator that a handle keeps when its preconditioner changes: the two-level preconditioner's
one-launch solve has operator 0, whichever one the tuner took for the diagonal preconditioner; a pinned
operator stays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu(nn):
    if nn.device_count() < 1:
        pytest.skip("no CUDA device")
    return nn


@pytest.mark.parametrize("n", [20, 40, 64, 80])
def test_operator_after_the_diagonal_preconditioner(gpu, n):
    nn = gpu
    inp = nn.synth(1, n, 3)
    sims = []
    for jacobi_first in (True, False):
        sim = nn.Simulation.from_synth(inp)
        sim.build_neighbours()
        sim.set_solver(1e-12)
        if jacobi_first:
            sim.set_preconditioner(nn.PRECOND_JACOBI)
            sim.forward(2, nn.MIXED)
            print(n, "operator under the diagonal preconditioner", sim.tuning()[2])
            sim.set_preconditioner(nn.PRECOND_TWO_LEVEL)
            sim.reset()
        sim.forward(2, nn.MIXED)
        assert sim.tuning()[2] == 0
        sims.append(sim)
    (c, phi, ph), (c1, phi1, ph1) = (s.state() for s in sims)
    assert np.array_equal(ph, ph1)
    assert np.abs(c - c1).max() <= 1e-8 * np.abs(c1).max()
    assert np.abs(phi - phi1).max() <= 1e-8 * np.abs(phi1).max()


def test_pinned_operator_stays(gpu):
    nn = gpu
    sim = nn.Simulation.from_synth(nn.synth(1, 20, 3))
    sim.build_neighbours()
    sim.set_preconditioner(nn.PRECOND_JACOBI)
    sim.set_tuning(4, 8, 3)
    sim.forward(1, nn.MIXED)
    sim.set_preconditioner(nn.PRECOND_TWO_LEVEL)
    sim.forward(1, nn.MIXED)
    assert sim.tuning() == (4, 8, 3)
