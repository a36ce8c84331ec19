"""The implicit step's sliced operator and device-side GMRES where they can go wrong: node counts off
the slices of 32 rows, a size above the line below which four warps share a slice, whose potential
system passes a GMRES restart -- against the oracle's step: the same Newton iterations, the states to 1e-9 (the bound of the other implicit tests: the GMRES tolerance's rounding),
identical masks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu(nn):
    if nn.device_count() < 1:
        pytest.skip("no CUDA device")
    return nn


@pytest.mark.parametrize("n,N,dt_scale", [(10, 33, 10.0), (10, 997, 10.0), (50, 125000, 10.0)])
def test_implicit_slices(gpu, orc, n, N, dt_scale):
    nn = gpu
    inp = nn.synth(1, n, 9)
    p = inp["params"].copy()
    p.dt *= dt_scale
    args = [np.ascontiguousarray(inp[k][..., :N]) for k in ("nodes", "bctypes", "bcvalues", "icvalues", "phase0")]
    sim = nn.Simulation(p, *args)
    sim.build_neighbours()
    o = orc.Oracle(p, *args)
    o.build_neighbours()
    ng, kg = sim.forward_implicit(1)
    no, ko = o.implicit_forward(1)
    print("newton gpu %d oracle %d, gmres gpu %d oracle %d" % (ng, no, kg, ko))
    assert ng == no
    assert abs(kg - ko) <= max(2, 0.02 * ko)
    if N > 100000:
        assert kg > 60 * ng  # the potential's system passes a restart every 30 iterations
    c_g, phi_g, ph_g = sim.state()
    c_o, phi_o, ph_o, _ = o.state()
    assert np.linalg.norm(c_g - c_o) <= 1e-9 * np.linalg.norm(c_o)
    assert np.linalg.norm(phi_g - phi_o) <= 1e-9 * np.linalg.norm(phi_o)
    assert np.array_equal(ph_g, ph_o)


@pytest.mark.parametrize("n,most_mb", [(20, 512), (50, 320)])
def test_memory_kept_between_calls(gpu, n, most_mb):
    """What nnpp_forward_implicit leaves on the device: at 125,000 nodes the Arnoldi basis (155 MB) and the
    off-diagonals (590 MB) go back on return (330 bytes a node and 12 a bond slot, 220 MB, stay); small
    handles keep theirs.  A second call continues as one call of two steps does."""
    nn = gpu
    torch = pytest.importorskip("torch")
    inp = nn.synth(1, n, 9)
    sims = []
    for _ in range(2):
        sim = nn.Simulation.from_synth(inp)
        sim.build_neighbours()
        sims.append(sim)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    sims[0].forward_implicit(1)
    torch.cuda.synchronize()
    held = before - torch.cuda.mem_get_info()[0]
    print("held %.1f MB" % (held / 1e6))
    assert held <= most_mb * 1e6
    sims[0].forward_implicit(1)
    sims[1].forward_implicit(2)
    for a, b in zip(sims[0].state(), sims[1].state()):
        assert np.array_equal(a, b)
