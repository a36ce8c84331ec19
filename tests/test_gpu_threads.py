"""Distinct handles stepped from several threads at once, as a program with a thread a handle steps them:
the one-launch inner solves (cooperative launches of all or part of the SMs) of several streams meet on one
chip.  Each handle's state is the bits of its run alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu(nn):
    if nn.device_count() < 1:
        pytest.skip("no CUDA device")
    return nn


@pytest.mark.parametrize("sides", [(20, 20, 20, 20, 20, 20, 20, 20), (12, 20, 28, 40), (50, 64, 28, 50)])
def test_handles_from_several_threads(gpu, sides):
    nn = gpu
    sims, expect = [], []
    for q, n in enumerate(sides):
        sim = nn.Simulation.from_synth(nn.synth(1, n, q + 1))
        sim.build_neighbours()
        sim.set_tuning(4, 8, 0)  # the timings of a tuner that runs beside others would choose for it
        sims.append(sim)
    work = [(20, nn.MIXED), (6, nn.FP64), (20, nn.MIXED)]
    errors = []

    def run(sim):
        try:
            for steps, prec in work:
                sim.forward(steps, prec)
        except Exception as e:  # noqa: BLE001 -- reported by the test's thread
            errors.append(e)

    for sim in sims:
        run(sim)
        expect.append(sim.state())
        sim.reset()
    assert not errors
    threads = [threading.Thread(target=run, args=(sim,)) for sim in sims]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for sim, ref in zip(sims, expect):
        for a, b in zip(sim.state(), ref):
            assert np.array_equal(a, b)
