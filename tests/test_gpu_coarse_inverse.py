"""The coarse operator's direct inverse (block cyclic reduction over planes of aggregates): boxes
whose longest axis is each of the three (planes along it), one plane only, aggregates without
unknowns, and a potential without any Dirichlet value, whose singular operator must fall back to the
Newton-Schulz iteration.  The solves meet the tolerance either way, so the check is the potential
against the oracle's (the bound of test_solve_potential), which inverse was used, and that the
coarse correction cuts the iterations as it should."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu(nn):
    if nn.device_count() < 1:
        pytest.skip("no CUDA device")
    return nn


def _box(nn, shape, dirichlet, seed=3):
    """A jittered lattice box in the first lattice's parameters, its two ends along x Dirichlet (or
    none), a solid ball in the middle."""
    inp = nn.synth(0, 16, 1)
    p = inp["params"].copy()
    rng = np.random.default_rng(seed)
    i = np.stack(np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")).reshape(3, -1)
    x = (i + 0.5 + rng.uniform(-0.2, 0.2, i.shape)) * p.dx
    N = x.shape[1]
    end = (i[0] < 3) | (i[0] >= shape[0] - 3)
    mid = np.array(shape)[:, None] * p.dx / 2
    solid = (((x - mid) ** 2).sum(0) < (0.3 * min(shape) * p.dx) ** 2) & ~end
    ic = np.full((5, N), 0.1) + 0.01 * rng.uniform(size=(5, N))
    ic[:4, solid] = np.array([1.0, 0.0, 0.0, 0.0])[:, None]
    ic[4] = 0.0
    bc = -np.ones((5, N))
    if dirichlet:
        bc[:4, end] = 0.1
        bc[4, end] = 0.0
    return p, np.ascontiguousarray(x), np.where(end & dirichlet, 0, 1).astype(np.int32), bc, ic, solid.astype(np.int32)


@pytest.mark.parametrize("shape", [(40, 13, 10), (13, 40, 10), (12, 10, 40), (20, 16, 5), (33, 33, 33)])
def test_direct_inverse_shapes(gpu, orc, shape):
    nn = gpu
    p, x, bt, bc, ic, ph = _box(nn, shape, True)
    sim = nn.Simulation(p, x, bt, bc, ic, ph)
    sim.build_neighbours()
    o = orc.Oracle(p, x, bt, bc, ic, ph)
    o.build_neighbours()
    o.set_solver(1e-13)
    phi_o = o.solve_potential(ic[:4], ph)[0]
    sim.set_solver(1e-11)
    phi, its, _ = sim.solve_potential(ic[:4], ph, precision=nn.MIXED)
    assert np.linalg.norm(phi - phi_o) <= 1e-8 * np.linalg.norm(phi_o)
    stats = sim.coarse_stats()
    assert stats["rebuilds"] == 1 and stats["last_ns_steps"] == 0
    sim.set_preconditioner(nn.PRECOND_JACOBI)
    _, its_jacobi, _ = sim.solve_potential(ic[:4], ph, precision=nn.MIXED)
    assert its < its_jacobi


def test_singular_operator_takes_newton_schulz(gpu):
    nn = gpu
    p, x, bt, bc, ic, ph = _box(nn, (20, 14, 12), False)
    sim = nn.Simulation(p, x, bt, bc, ic, ph)
    sim.build_neighbours()
    sim.set_solver(1e-10, 50)
    sim.forward(2, nn.MIXED)
    assert sim.coarse_stats()["last_ns_steps"] == 18
    c, phi, _ = sim.state()
    assert np.isfinite(c).all() and np.isfinite(phi).all()
