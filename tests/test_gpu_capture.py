"""Steps that a caller captures into a CUDA graph of its own, replayed between edits and plain calls: the state is that
of single steps (kernel="cell").  A replay reads the buffer that the captured call read, so an even number of
steps must end in it, and what a record counts down is known on the device only."""
import numpy as np
import pytest

from test_gpu_fused import _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,scene,form,n", [(1300, 1250, "cavity", dict(mode="physics"), 2), (1300, 1250, "channel", dict(mode="physics", collision="kbc"), 8),
                                                (1700, 1650, "poiseuille", dict(mode="reference", arith="fast"), 2),
                                                (128, 128, "channel", dict(mode="physics"), 16)])
def test_captured_steps(gpu, nx, ny, scene, form, n):
    import torch

    from simuverse_gb300 import FluidSimulator

    if form["mode"] == "physics":
        form = dict(form, lid_speed=0.05, inlet_speed=0.03, solid_fraction=0.0)
    a, b = (FluidSimulator(nx, ny, scene=scene, tau=0.62, kernel=k, **form) for k in ("auto", "cell"))
    stream = torch.cuda.Stream()
    a.set_stream(stream.cuda_stream)
    for s in (a, b):
        s.step(n)
        s.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        a.step(n)

    def replay(times):
        with torch.cuda.stream(stream):
            for _ in range(times):
                graph.replay()
        for _ in range(times):  # (a call's last step writes the field, in the reference's rules with bits of its own)
            b.step(n)

    replay(3)
    _same(a, b, "replayed")
    for s in (a, b):  # 90 steps of a force, some of them replayed
        s.add_external_force((nx + 40.0, ny + 30.0), (nx - 40.0, ny - 30.0))
    replay(2)
    _same(a, b, "force")
    for s in (a, b):
        s.step(2 * n)
        s.add_obstacle(29, ny // 2)
    replay(2)
    for s in (a, b):
        s.step(100)
    replay(1)
    for s in (a, b):
        s.step(1)
    _same(a, b, "plain calls between")
    assert np.array_equal(a.info(), b.info())
