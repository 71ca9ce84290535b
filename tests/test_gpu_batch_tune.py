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


def test_fused_steps_have_a_grid_of_their_own(gpu):
    """A tile form of one block per SM does not take warps from the fused steps: a block of the second half of their
    grid exists, and its absence is noticed."""
    import torch

    from simuverse_gb300 import _native as nat

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    b = BatchSimulator([WIDE, BIG])
    b.configure(blocks_per_sm=1)
    assert b.inject_missing_arrival(nsteps=7, block=2 * sms, step=4, timeout_ns=200_000_000) == nat.LBM_ERR_TIMEOUT
    b.close()
    # and the time reported is that of the setting that runs: at most a few times the time of a long call
    b = BatchSimulator([WIDE, BIG, MORE, MORE])
    ms = b.tune(trial_steps=3)["ms_per_step"]
    e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    stream = torch.cuda.Stream()
    b.set_stream(stream.cuda_stream)
    b.step(300)
    e[0].record(stream)
    b.step(300)
    e[1].record(stream)
    stream.synchronize()
    assert e[0].elapsed_time(e[1]) / 300 <= 1.5 * ms
    b.close()


def _takes_fused_steps(batch, nsteps):
    """Whether a call of nsteps does: the tile form of one block per SM has no block 2 x SMs, whose absence would be
    noticed (the state is of no use afterwards)."""
    import torch

    from simuverse_gb300 import _native as nat

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    batch.configure(blocks_per_sm=1)
    rc = batch.inject_missing_arrival(nsteps=nsteps, block=2 * sms, step=0, timeout_ns=200_000_000)
    assert rc in (0, nat.LBM_ERR_TIMEOUT)
    return rc != 0


def _equal(n, nx, ny, scene):
    return [dict(nx=nx, ny=ny, scene=scene, tau=0.7, speed=0.05)] * n


@pytest.mark.parametrize("domains,pays", [
    (_equal(1000, 64, 64, "channel"), False), (_equal(512, 64, 64, "channel"), False), (_equal(260, 64, 128, "cavity"), False), (_equal(64, 121, 300, "channel"), False),
    (_equal(128, 181, 181, "cavity"), False), (_equal(128, 1024, 16, "channel"), False),
    (_equal(40, 300, 200, "cavity"), True), (_equal(4, 1000, 700, "cavity"), True), ([BIG], True)])
def test_where_fused_steps_pay(gpu, domains, pays):
    b = BatchSimulator(domains)
    assert _takes_fused_steps(b, 3) == pays
    assert not _takes_fused_steps(b, 2)
    b.close()
    if len(domains) > 1:  # (the two forms tie on the one channel)
        b = BatchSimulator(domains)
        b.tune(trial_steps=10)
        assert _takes_fused_steps(b, 3) == pays
        b.close()
