"""Fused steps where planes are further apart than 32 bits count: the states themselves, compared on the device, and a frame of
two steps of the reference's own scene."""
import numpy as np
import pytest

from test_gpu_f64_precision import _View
from test_gpu_fused import _same

pytestmark = pytest.mark.gpu


def test_states_beyond_32_bits(gpu):
    import torch

    from simuverse_gb300 import FluidSimulator

    if torch.cuda.mem_get_info()[0] < 150 << 30:
        pytest.skip("not enough device memory")
    nx, ny = 32768, 16400
    row = (0.02 * np.random.default_rng(6).standard_normal(nx + 64)).astype(np.float32)
    u = np.stack([row[k % 61:k % 61 + nx] for k in range(ny)])
    sims, views = [], []
    for kernel in ("auto", "cell"):
        s = FluidSimulator(nx, ny, mode="physics", scene="periodic", tau=0.6, kernel=kernel)
        s.init_equilibrium(None, u, u[::-1])
        s.step(3)
        s.sync()
        v = _View(s, s.device_populations()[0], 9 * s.N)
        v.__cuda_array_interface__["typestr"] = "<i4"  # bits
        sims.append(s)
        views.append(torch.as_tensor(v, device="cuda").view(9, -1))
    for j in range(9):
        assert torch.equal(views[0][j], views[1][j]), j
    for s in sims:
        s.close()


def test_reference_frames(gpu):
    """One launch a frame where the walls agree (as after creation), state and field of two single steps."""
    from simuverse_gb300 import FluidSimulator

    a, b = (FluidSimulator(1801, 1600, arith="fast", tau=0.62, kernel=k) for k in ("auto", "cell"))
    for frame in range(3):
        before = a.kernel_launches
        for s in (a, b):
            s.compute()
        assert a.kernel_launches == before + 1
        _same(a, b, frame)
