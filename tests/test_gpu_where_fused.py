"""Where steps are fused: launches of a call on both sides of each line of the rules (march_pays, cluster_steps), and the
state of single steps on either."""
import numpy as np
import pytest

from test_gpu_fused import _same

pytestmark = pytest.mark.gpu


def _records(info, kind):
    ny, nx = info.shape
    rng = np.random.default_rng(1)
    at = (rng.random((ny, nx)) < (0.1 if kind in ("solid", "moving") else 0.01)) & (info["material"] == 1)
    if kind in ("solid", "moving"):
        info["material"][at] = 4
        info["vx"][at] = 0.01 if kind == "moving" else 0.0
    if kind == "column":
        at[:] = False
        at[1:-1, 5] = True
    if kind in ("force", "column"):
        info["material"][at] = 6
        info["block_iter"][at] = -1
        info["vx"][at] = 1e-3
    return info


REF = dict(mode="reference", arith="fast")
KBC = dict(collision="kbc")


@pytest.mark.parametrize("nx,ny,scene,form,kind,steps,launches", [
    # widths, faces and walls
    (1000, 900, "periodic", {}, None, 3, 1), (1000, 1000, "channel", {}, None, 3, 1), (1000, 1000, "cavity", {}, None, 2, 1),
    (240, 4000, "channel", {}, None, 3, 1), (421, 2300, "channel", {}, None, 4, 2), (301, 2800, "channel", {}, None, 3, 3),
    (121, 20000, "channel", {}, None, 3, 3), (100, 9000, "channel", {}, None, 3, 3), (64, 20000, "cavity", {}, None, 3, 3),
    (100, 9000, "cavity", {}, None, 3, 1), (150, 6000, "periodic", {}, None, 2, 1), (121, 7000, "periodic", {}, None, 2, 2),
    (60000, 20, "cavity", {}, None, 3, 3), (60000, 20, "periodic", {}, None, 3, 1), (64, 12504, "channel", {}, None, 3, 3),
    (181, 5000, "periodic", KBC, None, 3, 1), (181, 5000, "cavity", KBC, None, 3, 3), (300, 3000, "cavity", KBC, None, 3, 1),
    (300, 3000, "channel", KBC, None, 3, 3), (300, 4200, "channel", KBC, None, 3, 1), (420, 2100, "channel", KBC, None, 3, 1),
    (1300, 700, "custom", REF, None, 2, 1), (301, 2700, "custom", REF, None, 2, 2), (240, 4000, "poiseuille", REF, None, 2, 1),
    (100, 9000, "poiseuille", REF, None, 2, 2), (1001, 900, "poiseuille", REF, None, 3, 1), (800, 999, "custom", REF, None, 3, 3),
    # forcing cells, moving walls, walls inside
    (1000, 1000, "periodic", {}, "column", 3, 3), (1500, 1500, "periodic", {}, "column", 3, 1), (1500, 1500, "periodic", {}, "force", 3, 3),
    (1500, 1500, "periodic", KBC, "moving", 2, 2), (1500, 1500, "periodic", {}, "solid", 3, 1), (1032, 780, "channel", {}, "solid", 3, 1),
    # small lattices
    (128, 128, "periodic", {}, None, 20, 1), (128, 128, "periodic", {}, "force", 20, 1), (128, 128, "periodic", KBC, "force", 20, 20),
    (64, 64, "periodic", KBC, "force", 20, 1), (192, 192, "periodic", {}, "force", 20, 20), (192, 192, "periodic", KBC, "moving", 20, 20),
    (192, 192, "periodic", {}, "moving", 20, 1), (256, 256, "periodic", {}, "moving", 20, 20), (256, 256, "periodic", {}, "solid", 20, 1),
    (256, 256, "periodic", {}, None, 20, 1)])
def test_launches(gpu, nx, ny, scene, form, kind, steps, launches):
    from simuverse_gb300 import FluidSimulator

    if "mode" not in form:
        form = dict(form, mode="physics", lid_speed=0.05, inlet_speed=0.03, solid_fraction=0.0)
    a, b = (FluidSimulator(nx, ny, scene=scene, tau=0.62, kernel=k, **form) for k in ("auto", "cell"))
    for s in (a, b):
        if kind:
            s.set_info(_records(s.info(), kind))
            s.init_equilibrium()
    for _ in range(2):
        before = a.kernel_launches
        for s in (a, b):
            s.step(steps)
        assert a.kernel_launches - before == launches
    _same(a, b, (nx, ny, scene))
