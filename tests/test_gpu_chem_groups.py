"""The ten-species residual's grouped kernel where it can go wrong: node counts off the groups of 32
(down to one node), both sides of the line below which four warps share a group, and coefficients
that need the general kernel (a migration ratio that differs within a charge group) -- against the
oracle's restatement, whose sums the kernel reorders: 1e-12 of each field's largest value, the bound
of the other residual tests (about 100 terms a row at 2.2e-16 each leave it 40 times over)."""
import os

import numpy as np
import pytest

import chem_case

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "chemistry.npz")


@pytest.fixture(scope="module")
def gpu(nn):
    if nn.device_count() < 1:
        pytest.skip("no CUDA device")
    return nn


@pytest.mark.parametrize("n,N,ratio", [(12, 1, False), (12, 31, False), (12, 33, False), (12, 127, False),
                                       (12, 1000, True), (16, 4095, False), (62, 233440, False),
                                       (62, 233473, False)])
def test_grouped_residual_sizes(gpu, orc, n, N, ratio):
    nn = gpu
    g = np.load(GOLDEN)
    d2, dc, d11 = chem_case.reactive_data2(g["data2"]), g["datac"].copy(), g["datac11"]
    if ratio:
        dc[4, 6] *= 1.5  # one species' migration factor apart from its charge group's
    nodes, phase, Un1, Un, r, cell = chem_case.case_inputs(nn.synth, 1, n, 4, g["data2"])
    nodes, phase, Un1, Un = (np.ascontiguousarray(a[..., :N]) for a in (nodes, phase, Un1, Un))
    clouds, lengths, ml = nn.build_clouds_hash(160, r, cell, cell, cell, nodes)
    F = nn.residuals_full(nodes, clouds[:, :ml], lengths, Un1, Un, phase, chem_case.VOLN1REL, d2, dc, d11)
    ptr = np.zeros(N + 1, dtype=np.int64)
    ptr[1:] = np.cumsum(lengths)
    cols = clouds[:, :ml][np.arange(ml)[None, :] < lengths[:, None]].astype(np.int32)
    Fr = orc.residuals_full(nodes, ptr, cols, Un1, Un, phase, chem_case.VOLN1REL, d2, dc, d11)
    for k in range(11):
        assert np.abs(F[k] - Fr[k]).max() <= 1e-12 * np.abs(Fr[k]).max(), k
    assert np.array_equal(F[10] == 0.0, Fr[10] == 0.0)


@pytest.mark.parametrize("n", [12, 62])
def test_grouped_residual_phases_other_than_solid_and_liquid(gpu, orc, n):
    """The reference tests phases for 1 and for 0: a bond of any other value is neither solid-solid nor
    liquid-liquid.  Both forms of the grouped kernel."""
    nn = gpu
    g = np.load(GOLDEN)
    d2, dc, d11 = chem_case.reactive_data2(g["data2"]), g["datac"], g["datac11"]
    nodes, phase, Un1, Un, r, cell = chem_case.case_inputs(nn.synth, 1, n, 4, g["data2"])
    N = nodes.shape[1]
    phase = phase.copy()
    phase[np.random.default_rng(2).permutation(N)[:N // 4]] = 2
    clouds, lengths, ml = nn.build_clouds_hash(160, r, cell, cell, cell, nodes)
    F = nn.residuals_full(nodes, clouds[:, :ml], lengths, Un1, Un, phase, chem_case.VOLN1REL, d2, dc, d11)
    ptr = np.zeros(N + 1, dtype=np.int64)
    ptr[1:] = np.cumsum(lengths)
    cols = clouds[:, :ml][np.arange(ml)[None, :] < lengths[:, None]].astype(np.int32)
    Fr = orc.residuals_full(nodes, ptr, cols, Un1, Un, phase, chem_case.VOLN1REL, d2, dc, d11)
    for k in range(11):
        assert np.abs(F[k] - Fr[k]).max() <= 1e-12 * np.abs(Fr[k]).max(), k
