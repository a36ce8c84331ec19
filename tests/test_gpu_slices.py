"""The sliced step kernels where they can go wrong: node counts off the slices of 32 rows and the
quads of bonds, each number of warps that share a slice (8, 4, 2, 1 by size), and a handle that
changes precision between steps (the FP64 weights are laid out by its first FP64 run and the CG rows
refilled by each) -- against the oracle's steps.  The states differ by the solves' tolerances (1e-12 of
the right-hand side, times the condition number: 1e-8 of the largest value) in FP64; mixed steps round
each bond sum to FP32 and the increment dt F is ~1e-3 of c, so 1e-8 there too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu(nn):
    if nn.device_count() < 1:
        pytest.skip("no CUDA device")
    return nn


def _pair(nn, orc, n, N):
    inp = nn.synth(1, n, 7)
    args = [inp["params"]] + [np.ascontiguousarray(inp[k][..., :N])
                              for k in ("nodes", "bctypes", "bcvalues", "icvalues", "phase0")]
    sim, o = nn.Simulation(*args), orc.Oracle(*args)
    sim.build_neighbours()
    o.build_neighbours()
    sim.set_solver(1e-12)
    o.set_solver(1e-13)
    return sim, o


def _check(sim, o):
    c, phi, ph = sim.state()
    co, phio, pho, _ = o.state()
    assert np.array_equal(ph, pho)
    assert np.abs(c - co).max() <= 1e-8 * np.abs(co).max()
    assert np.abs(phi - phio).max() <= 1e-8 * max(np.abs(phio).max(), 1e-30)


@pytest.mark.parametrize("n,N", [(10, 1), (10, 33), (10, 997), (20, 8000), (28, 21951), (38, 54871),
                                 (56, 175615), (64, 262143)])
@pytest.mark.parametrize("order", ["fp64", "mixed", "switch"])
def test_sliced_steps(gpu, orc, n, N, order):
    nn = gpu
    sim, o = _pair(nn, orc, n, N)
    for prec in dict(fp64=[nn.FP64] * 2, mixed=[nn.MIXED] * 2, switch=[nn.MIXED, nn.FP64, nn.MIXED])[order]:
        sim.forward(2, prec)
        o.forward(2)
        _check(sim, o)
