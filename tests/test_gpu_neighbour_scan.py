"""The neighbour scan's FP32 decisions with their FP64 fallback: nodes exactly on the horizon
(lattices of a spacing that FP64 holds, r a whole number of spacings: every tie is decided by the
reference's FP64 test), cells much smaller and much larger than the radius (larger than about 10^5
radii every test is the FP64 one) and flat extents, against the oracle's lists, order included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu(nn):
    if nn.device_count() < 1:
        pytest.skip("no CUDA device")
    return nn


def _oracle_lists(nn, orc, nodes, r, cell):
    N = nodes.shape[1]
    inp = nn.synth(0, 4, 1)
    o = orc.Oracle(inp["params"], nodes, np.ones(N, dtype=np.int32), -np.ones((5, N)), np.zeros((5, N)),
                   np.zeros(N, dtype=np.int32))
    ml = o.build_neighbours(1024, r, cell)
    lengths, ptr, cols = o.clouds()
    expect = -np.ones((N, 1024), dtype=np.int32)
    for i in range(N):
        expect[i, :lengths[i]] = cols[ptr[i]:ptr[i + 1]]
    return ml, lengths, expect


@pytest.mark.parametrize("shape,r_cells,cell_factor", [
    ((11, 10, 9), 3.0, 3.25),       # ties, cells a little wider than the radius
    ((11, 10, 9), 3.0, 0.5),        # ties, a dozen cells along the diameter
    ((17, 31, 1), 2.0, 10.0),       # a flat extent
    ((12, 11, 7), 3.0, 1.0e7),      # one cell: every test falls back to FP64
])
def test_scan_ties_and_cells(gpu, orc, shape, r_cells, cell_factor):
    nn = gpu
    dx = 0.125
    g = np.stack(np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")).reshape(3, -1).astype(np.float64) * dx
    g = np.ascontiguousarray(g[:, np.random.default_rng(4).permutation(g.shape[1])])
    cell = (cell_factor * dx, cell_factor * dx * 1.5, cell_factor * dx)
    clouds, lengths, ml = nn.build_clouds_hash(1024, r_cells * dx, *cell, g)
    ml_o, len_o, expect = _oracle_lists(nn, orc, g, r_cells * dx, cell)
    assert ml == ml_o
    assert np.array_equal(lengths, len_o)
    assert np.array_equal(clouds, expect)


@pytest.mark.parametrize("offset", [0.0, 2.0 ** 20, 2.0 ** 38])
def test_scan_far_from_the_origin(gpu, orc, offset):
    """Ties on a lattice far from the origin (every coordinate exact).  The cell side is chosen so that at
    2^38 three sides in FP64 lie halfway between two coordinates: the fourth column's corner then differs
    by a coordinate's last place, 1.6e-4 radii, with the product rounded or not."""
    nn = gpu
    dx = 0.125
    side = float.fromhex("0x1.a2d2aaaaaaaaap-2")
    g = np.stack(np.meshgrid(*[np.arange(n) for n in (11, 10, 9)], indexing="ij")).reshape(3, -1).astype(np.float64) * dx
    g = np.ascontiguousarray(g[:, np.random.default_rng(4).permutation(g.shape[1])] + offset)
    cell = (side, 4.1 * dx, 3.28 * dx)
    clouds, lengths, ml = nn.build_clouds_hash(1024, 3.0 * dx, *cell, g)
    ml_o, len_o, expect = _oracle_lists(nn, orc, g, 3.0 * dx, cell)
    assert ml == ml_o
    assert np.array_equal(lengths, len_o)
    assert np.array_equal(clouds, expect)


@pytest.mark.parametrize("N", [1, 33, 1000])
def test_one_scan_and_two_scans_agree(gpu, N):
    """The one-scan build (rows of max_node_no - 1 columns, packed) against the two-scan build that a
    max_node_no too large for such rows takes: the same lists."""
    nn = gpu
    inp = nn.synth(1, 10, seed=2)
    args = [inp["params"]] + [np.ascontiguousarray(inp[k][..., :N])
                              for k in ("nodes", "bctypes", "bcvalues", "icvalues", "phase0")]
    out = []
    for most in (200, (1 << 29) // N + 2):
        sim = nn.Simulation(*args)
        sim.build_neighbours(most)
        out.append(sim.neighbours_csr())
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])


def test_build_where_rows_and_lists_do_not_fit_together(gpu):
    """103,823 nodes of up to 4,168 neighbours with 2.8 GB of device memory left: the one-scan build's rows
    take 2.08 GB and the lists 1.4, so the rows are given back and the two-scan build runs.  (The test's
    own allocation is what fills the device.)"""
    nn = gpu
    torch = pytest.importorskip("torch")
    n, most = 47, 5001
    g = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij")).reshape(3, -1).astype(np.float64)
    args = (most, 10.0, 10.0, 10.0, 10.0, np.ascontiguousarray(g))
    _, expect, ml = nn.build_clouds_hash(*args, want_clouds=False)
    bonds = int(expect.sum()) - expect.size
    rows = 4 * (most - 1) * g.shape[1]
    left = int(2.8e9)
    assert rows < left < rows + 4 * bonds - 200e6 and 4 * bonds < left - 500e6
    torch.cuda.synchronize()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        _, lengths, ml2 = nn.build_clouds_hash(*args, want_clouds=False)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert ml2 == ml
    assert np.array_equal(lengths, expect)
