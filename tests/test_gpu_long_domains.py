"""Long, thin domains (wires, struts) through the two-level preconditioner: hundreds to thousands of planes
of aggregates along one axis, each axis in turn.  The potential against the oracle's to 1e-8 (the bound of
the other solves: the tolerances 1e-11 and 1e-13 times the condition number), the directly inverted coarse
operator, and fewer iterations than the diagonal preconditioner alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu(nn):
    if nn.device_count() < 1:
        pytest.skip("no CUDA device")
    return nn


def _wire(nn, shape, seed=5):
    """A jittered lattice with a solid ball in the middle.  One edge line along the long axis has Dirichlet
    values, which vary along it."""
    inp = nn.synth(0, 16, 1)
    p = inp["params"].copy()
    rng = np.random.default_rng(seed)
    axis = int(np.argmax(shape))
    i = np.stack(np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")).reshape(3, -1)
    x = (i + 0.5 + rng.uniform(-0.1, 0.1, i.shape)) * p.dx
    N = x.shape[1]
    line = np.all(np.delete(i, axis, axis=0) == 0, axis=0)
    mid = np.array(shape)[:, None] * p.dx / 2
    solid = (((x - mid) ** 2).sum(0) < (3.0 * p.dx) ** 2) & ~line
    ic = np.full((5, N), 0.1) + 0.01 * rng.uniform(size=(5, N))
    ic[:4, solid] = np.array([1.0, 0.0, 0.0, 0.0])[:, None]
    ic[4] = 0.0
    bc = -np.ones((5, N))
    bc[:4, line] = 0.1
    bc[4, line] = np.sin(i[axis, line] * (20.0 / max(shape)))
    return p, np.ascontiguousarray(x), np.where(line, 0, 1).astype(np.int32), bc, ic, solid.astype(np.int32)


def _solve_and_step(nn, orc, shape, planes):
    p, x, bt, bc, ic, ph = _wire(nn, shape)
    sim = nn.Simulation(p, x, bt, bc, ic, ph)
    sim.build_neighbours()
    o = orc.Oracle(p, x, bt, bc, ic, ph)
    o.build_neighbours()
    o.set_solver(1e-13)
    phi_o = o.solve_potential(ic[:4], ph)[0]
    sim.set_solver(1e-11)
    for prec in (nn.MIXED, nn.FP64):
        phi, its, _ = sim.solve_potential(ic[:4], ph, precision=prec)
        assert np.linalg.norm(phi - phi_o) <= 1e-8 * np.linalg.norm(phi_o)
        stats = sim.coarse_stats()
        assert stats["rebuilds"] >= 1 and stats["last_ns_steps"] == 0
        assert planes <= sim.preconditioner()[1] <= 3000
        if prec == nn.MIXED:
            its_two = its
    sim.forward(2, nn.MIXED)
    c, phi, _ = sim.state()
    assert np.isfinite(c).all() and np.isfinite(phi).all()
    sim.set_preconditioner(nn.PRECOND_JACOBI)
    _, its_jacobi, _ = sim.solve_potential(ic[:4], ph, precision=nn.MIXED)
    print(shape, "iterations", its_two, "jacobi", its_jacobi, "aggregates", stats)
    assert its_two < its_jacobi


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_more_than_512_planes(gpu, orc, axis):
    """4 x 4 x 1560 nodes: 2 x 2 x 517 one-bin aggregates, 258 x 259 plane pairs in the inverse's growth."""
    shape = [4, 4, 4]
    shape[axis] = 1560
    _solve_and_step(gpu, orc, tuple(shape), 4 * 512)


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_1024_bins_along_an_axis(gpu, orc, axis):
    """3 x 3 x 3086 nodes: 1024 one-bin aggregates on one axis, the most that the lists take (and what the
    coarse operator's node words hold, 10 bits an axis)."""
    shape = [3, 3, 3]
    shape[axis] = 3086
    _solve_and_step(gpu, orc, tuple(shape), 1024)


def test_more_bins_are_refused(gpu):
    """3 x 3 x 3100 nodes: 1028 bins on one axis are an error before any coarse operator is formed."""
    nn = gpu
    for axis in range(3):
        shape = [3, 3, 3]
        shape[axis] = 3100
        sim = nn.Simulation(*_wire(nn, tuple(shape)))
        with pytest.raises(nn.NNPPError) as e:
            sim.build_neighbours()
        assert e.value.status == 6
