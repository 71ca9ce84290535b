"""Fused steps of the batched form against one launch per domain and step: the same bits, for every
remainder of three steps, domains at and off window and segment edges, and after a tuning that
moves the state; a missing arrival is reported, and the batch's kernel is not left half set up."""
import numpy as np
import pytest

from simuverse_gb300 import BatchSimulator
from simuverse_gb300 import _native as nat

pytestmark = pytest.mark.gpu

DOMAINS = [dict(nx=64, ny=8, scene="cavity", tau=0.6, speed=0.08), dict(nx=65, ny=97, scene="channel", tau=0.7, speed=0.05),
           dict(nx=121, ny=64, scene="channel", tau=0.56, speed=0.03), dict(nx=257, ny=130, scene="cavity", tau=0.9, speed=0.1),
           dict(nx=180, ny=201, scene="channel", tau=0.8, speed=0.07),
           # with this one the batch is large enough for fused steps
           dict(nx=1500, ny=1400, scene="channel", tau=0.65, speed=0.06)]


def test_fused_passes_equal_single_steps(gpu):
    a, b = BatchSimulator(DOMAINS), BatchSimulator(DOMAINS)
    b.configure(method="domain_loop")
    for n in (1, 2, 3, 4, 5, 30):
        a.step(n)
        a.status()
        b.step(n)
        for i in range(len(DOMAINS)):
            fluid = ~np.isin(a.info(i)["material"], (2, 4))
            x, y = a.read_populations(i)[:, fluid], b.read_populations(i)[:, fluid]
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (n, i)
            for x, y in zip(a.read_macro(i), b.read_macro(i)):
                assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (n, i)


def test_missing_arrival_in_a_fused_pass(gpu):
    a = BatchSimulator(DOMAINS)
    assert a.inject_missing_arrival(nsteps=7, block=1, step=4, timeout_ns=200_000_000) == nat.LBM_ERR_TIMEOUT
    b = BatchSimulator(DOMAINS)
    assert b.tune(trial_steps=3)["ms_per_step"] > 0
    b.step(6)
    b.status()
