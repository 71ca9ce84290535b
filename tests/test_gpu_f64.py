"""FP64 BGK (lbm_cell64.cuh) against the FP64 oracle: densities far from 1 (the reciprocal), rates on both
sides of 0.5 and 1 (the constants that must close), every boundary rule and a force that counts down."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

STEPS = 60
# some twenty roundings of populations below 1 a cell step (2^-53 each, on both sides), carried with gain 1
TOL = 2 * STEPS * 20 * 2.0 ** -53


@pytest.mark.parametrize("tau", [0.505, 0.6, 1.0, 2.7])
@pytest.mark.parametrize("scene,nx,ny", [("cavity", 129, 67), ("channel", 200, 45), ("periodic", 64, 33)])
def test_f64_bgk_matches_oracle(gpu, scene, nx, ny, tau):
    from simuverse_gb300 import FluidSimulator

    sim = FluidSimulator(nx, ny, mode="physics", dtype="f64", scene=scene, tau=tau, lid_speed=0.05,
                         inlet_speed=0.03, disk_radius=(3.0, 6.0), seed=4)
    info = sim.info()
    x, y = np.meshgrid(np.arange(nx), np.arange(ny))
    fluid = info["material"] == 1
    fluid[0] = fluid[-1] = fluid[:, 0] = fluid[:, -1] = False
    ys, xs = np.nonzero(fluid)
    for i, count in ((len(ys) // 3, 7), (len(ys) // 2, -1)):
        info[ys[i], xs[i]] = (6, count, 0.004, -0.003)
    sim.set_info(info)
    # even and odd waves, density from 0.6 to 1.7
    wave = np.sin(2 * np.pi * x / nx) * np.cos(2 * np.pi * y / ny)
    fields = [a.astype(np.float32) for a in (1.15 + 0.55 * wave, 0.03 * wave, -0.02 * wave * wave)]
    sim.init_equilibrium(*fields)
    ref = oracle.PhysOracle(info, tau, np.float64)
    ref.init_equilibrium(*fields)
    sim.step(STEPS)
    ref.step(STEPS)
    got, want = sim.read_populations(np.float64), ref.populations()
    wet = ~np.isin(info["material"], (2, 4))
    assert np.isfinite(want).all()
    assert np.max(np.abs(got - want)[:, wet]) <= TOL
    if scene == "periodic":  # forces move momentum, nothing moves mass
        assert abs(sim.conservation()[0] - ref.conservation()[0]) <= 1e-13 * nx * ny
