"""The reciprocal of lbm_core.cuh (hardware approximation and one Newton step) where it is used: the velocity of cells whose
momentum is a power of two is the reciprocal of their density, scaled.  All 2^24 densities of [0.5, 2) against the IEEE
quotient, and the packed form of the fused steps against the scalar one on the same lattice."""
import numpy as np
import pytest

from test_gpu_f64_precision import _View

pytestmark = pytest.mark.gpu

SIDE = 4096


def _densities():
    k = np.arange(2 ** 23, dtype=np.uint32)
    return np.concatenate([(np.uint32(e << 23) | k).view(np.float32) for e in (126, 127)]).reshape(SIDE, SIDE)


def _lattice(kernel, collision, state):
    import torch

    from simuverse_gb300 import FluidSimulator

    s = FluidSimulator(SIDE, SIDE, mode="physics", scene="periodic", tau=0.8, kernel=kernel, collision=collision)
    s.sync()
    view = _View(s, s.device_populations()[0], 9 * s.N)
    view.__cuda_array_interface__["typestr"] = "<f4"
    torch.as_tensor(view, device="cuda").view(9, SIDE, SIDE).copy_(state)
    torch.cuda.synchronize()
    return s


@pytest.mark.parametrize("collision", ["bgk", "kbc"])
def test_every_significand(gpu, collision):
    import torch

    rho, j = _densities(), np.float32(2.0 ** -6)
    state = torch.zeros(9, SIDE, SIDE, device="cuda")
    state[0] = torch.from_numpy((rho - np.float32(1)) - j)  # exact, as are the sums that the step forms of these two
    state[1] = float(j)
    one = _lattice("cell", collision, state)
    one.step(1)
    got_rho, ux, uy = one.read_macro()
    assert np.array_equal(got_rho, rho) and not uy.any()
    want = j / rho  # (rounded once; the scaling is exact)
    assert np.array_equal(ux.view(np.uint32), want.view(np.uint32))
    one.step(2)
    many = _lattice("auto", collision, state)
    before = many.kernel_launches
    many.step(3)
    assert many.kernel_launches == before + 1
    for a, b in zip(one.read_macro(), many.read_macro()):
        assert np.isfinite(a).all() and np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_reference_rules(gpu):
    """Densities all over the shaders' range of 0.8 to 1.2: fused frames against single steps, whose reciprocal is CUDA's."""
    from simuverse_gb300 import FluidSimulator

    w = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4, np.float32)[:, None, None]
    rng = np.random.default_rng(3)
    f = w * rng.uniform(0.75, 1.25, (1, SIDE, SIDE)).astype(np.float32) * rng.uniform(0.98, 1.02, (9, SIDE, SIDE)).astype(np.float32)
    out = []
    for kernel in ("auto", "cell"):
        s = FluidSimulator(SIDE, SIDE, scene="custom", arith="fast", tau=0.9, kernel=kernel)
        s.write_populations(f)
        before = s.kernel_launches
        s.step(3)
        assert s.kernel_launches - before == (1 if kernel == "auto" else 3)
        out.append(s.read_macro() + (s.read_populations(),))
        s.close()
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
