"""One-off evaluations on other inputs (nnpp_solve_potential and nnpp_residuals with phases of their own)
between the steps of a run leave it as it was: the operator's arrays and a coarse operator formed for those
phases are not the run's.  The states are the bits of the run without them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu(nn):
    if nn.device_count() < 1:
        pytest.skip("no CUDA device")
    return nn


@pytest.mark.parametrize("n", [12, 28])
@pytest.mark.parametrize("precond", [0, 1])
@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("replaced", [False, True])  # the state replaced just before: a coarse rebuild is due
def test_evaluations_leave_the_run(gpu, n, precond, mixed, replaced):
    nn = gpu
    prec = nn.MIXED if mixed else nn.FP64
    states = []
    for probe in (None, "solve", "residuals"):
        sim = nn.Simulation.from_synth(nn.synth(1, n, 1))
        sim.build_neighbours()
        sim.set_preconditioner(precond)
        sim.set_tuning(4, 8, 0)
        sim.forward(4, prec)
        c, phi, ph = sim.state()
        other = ph.copy()
        other[::3] = 0
        if replaced:
            sim.set_state(c, phi, ph)
        if probe == "solve":
            sim.solve_potential(c, other, precision=prec)
        elif probe == "residuals":
            sim.residuals(c, phi, other, precision=prec)
        sim.forward(4, prec)
        states.append(sim.state())
    for other in states[1:]:
        for a, b in zip(states[0], other):
            assert np.array_equal(a, b)
