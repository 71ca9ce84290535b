"""Tuned batches: the cached settings of one batch must suit the next one of its class, and the state is that of
as many single steps as the counter says."""
import numpy as np
import pytest

from simuverse_gb300 import BatchSimulator

pytestmark = pytest.mark.gpu

# with a domain of 64 columns the batch takes fused steps, with one of 48 (another scene, the same size class) it
# does not
BIG = dict(nx=1500, ny=1400, scene="channel", tau=0.65, speed=0.06)
WIDE = dict(nx=64, ny=72, scene="cavity", tau=0.6, speed=0.08)
NARROW = dict(nx=48, ny=96, scene="cavity", tau=0.6, speed=0.08)
MORE = dict(nx=130, ny=64, scene="channel", tau=0.8, speed=0.03)


def _check(batch, domains):
    """The batch against one launch per domain and step, after the steps it has taken."""
    batch.status()
    steps = batch.counters[0]
    single = BatchSimulator(domains)
    single.configure(method="domain_loop")
    single.step(steps)
    for i in range(len(domains)):
        for a, b in zip(batch.read_macro(i), single.read_macro(i)):
            # the tile forms of a tuning round differently: some roundings of numbers of about 1 a step
            assert np.max(np.abs(a.astype(np.float64) - b)) <= steps * 2.0 ** -23, (i, steps)
    single.close()


@pytest.mark.parametrize("first,second,others", [(NARROW, WIDE, [BIG]), (WIDE, NARROW, [BIG, MORE])],
                         ids=["narrow first", "wide first"])
def test_two_batches_of_one_class(gpu, first, second, others):
    for small in (first, second):
        domains = [small] + others
        b = BatchSimulator(domains)
        b.tune(trial_steps=3)
        b.step(7)
        _check(b, domains)
        # a second batch takes the cached settings
        c = BatchSimulator(domains)
        assert c.tune(trial_steps=3) == b.config
        assert c.counters[0] == 0
        c.step(11)
        _check(c, domains)
        for x in (b, c):
            x.close()
