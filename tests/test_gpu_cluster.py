"""Many steps of a small lattice in one launch (lbm_step_cluster.cu) against the one-step kernels
(kernel="cell"): the same bits for every boundary rule, band and window shape, odd and even step
counts, both layouts of the populations between steps; records and outflow cells that the launch does
not take stay on single steps.  In the bounds-checked build no index leaves its buffer."""
import os
import subprocess
import sys

import numpy as np
import pytest

from test_gpu_fused import ROOT, _mask, _same

pytestmark = pytest.mark.gpu

# bands of one row and of many, of like and unlike height; one window to 16, of every width modulo 4
SIZES = [(192, 192), (64, 64), (65, 131), (33, 17), (4, 16), (30, 700), (700, 48), (1024, 47), (1001, 33), (126, 370),
         (257, 70)]
SCENES = [(s, c) for c in ("bgk", "kbc") for s in ("cavity", "channel", "periodic")]


def _lattice(nx, ny, scene, block_iter=-1, far_outlet=False, **kw):
    from simuverse_gb300 import FluidSimulator

    s = FluidSimulator(nx, ny, mode="physics", scene=scene, tau=0.6, lid_speed=0.05, inlet_speed=0.03,
                       solid_fraction=0.0, **kw)
    if nx >= 16:
        info = s.info()
        if nx >= 64:
            info = _mask(info, nx + ny, block_iter)
        else:
            info[ny // 2, nx // 2] = info[1, nx - 2] = (4, -1, 0.0, 0.0)
            info[ny // 2 - 2, nx // 2] = (6, block_iter, 0.01, -0.02)
        # moving obstacles, one beside the last column; a wall in that column, and a fluid cell across from it
        info[ny // 3, nx - 2] = info[ny // 4, nx // 3] = (4, -1, 0.02, -0.01)
        if nx >= 64:  # inlets away from the first column, in both halves of a window
            info[ny // 5, 5] = info[ny // 5, 40] = (3, -1, 0.02, 0.01)
        if scene == "channel":
            info[ny // 2, nx - 1] = info[2 * ny // 3, nx - 1] = (4, -1, 0.0, 0.01)
            info[ny // 2 - 1:ny // 2 + 2, 0] = (1, -1, 0.0, 0.0)
        if far_outlet:
            info[ny // 2, nx // 2] = (5, -1, 0.0, 0.0)
        s.set_info(info)
    rng = np.random.default_rng(nx + 1)
    s.init_equilibrium(*((a + 0.02 * rng.standard_normal((ny, nx))).astype(np.float32) for a in (1.0, 0.03, 0.0)))
    return s


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("scene,collision", SCENES)
def test_one_launch_equals_single_steps(gpu, nx, ny, scene, collision):
    a, b = (_lattice(nx, ny, scene, collision=collision, **kw) for kw in ({}, {"kernel": "cell"}))
    for n in (16, 17, 32, 1041 if nx == 64 else 33):
        launches = a.kernel_launches
        a.step(n)
        assert a.kernel_launches == launches + (2 if n > 1024 else 1)
        b.step(n)
        _same(a, b, (n, scene, collision))
    # walls whose slots differ between the buffers
    f = a.read_populations() + np.float32(1e-3) * np.random.default_rng(5).random((9, ny, nx), np.float32)
    for s in (a, b):
        s.write_populations(f)
    for n in (16, 1, 17):
        a.step(n)
        b.step(n)
        _same(a, b, (n, "written"))


def test_what_stays_on_single_steps(gpu):
    for kw in (dict(block_iter=5), dict(far_outlet=True)):
        a, b = _lattice(200, 100, "channel", **kw), _lattice(200, 100, "channel", kernel="cell", **kw)
        for n in (4, 20):
            launches = a.kernel_launches
            a.step(n)
            # five steps while records count down, then one launch for the rest
            assert a.kernel_launches - launches == (2 if n == 20 and "block_iter" in kw else n)
            b.step(n)
            _same(a, b, (n, kw))
            assert np.array_equal(a.info(), b.info())


@pytest.mark.parametrize("scene", ["poiseuille", "custom"])
def test_other_scenes(gpu, scene):
    """The reference's masks in physics mode: their outflow is not in the last column.  A reset brings them back."""
    from simuverse_gb300 import FluidSimulator

    a, b = (FluidSimulator(130, 60, mode="physics", scene=scene, tau=0.7, **kw) for kw in ({}, {"kernel": "cell"}))
    for s in (a, b):
        info = s.info()
        info[info["material"] == 5] = (1, -1, 0.0, 0.0)
    for again in range(2):
        a.step(20)
        b.step(20)
        _same(a, b, scene)
        for s in (a, b):
            s.set_info(info) if again == 0 else None
            s.reset()


@pytest.mark.parametrize("nx,ny,scene,collision,steps,launches", [
    (256, 256, "cavity", "bgk", 10, 1), (256, 256, "cavity", "bgk", 9, 9), (256, 256, "channel", "bgk", 100, 100),
    (256, 256, "periodic", "kbc", 100, 100), (300, 300, "periodic", "bgk", 100, 100), (128, 128, "channel", "bgk", 6, 1),
    (128, 128, "channel", "bgk", 5, 5), (64, 15, "periodic", "bgk", 50, 50)])
def test_where_the_line_lies(gpu, nx, ny, scene, collision, steps, launches):
    from simuverse_gb300 import FluidSimulator

    kw = dict(mode="physics", scene=scene, collision=collision, tau=0.6, lid_speed=0.05, inlet_speed=0.03)
    a, b = FluidSimulator(nx, ny, **kw), FluidSimulator(nx, ny, kernel="cell", **kw)
    before = a.kernel_launches
    a.step(steps)
    assert a.kernel_launches - before == launches
    b.step(steps)
    _same(a, b, (nx, ny, scene, collision, steps))


def child_main():
    import ctypes

    from simuverse_gb300 import _native as nat

    lib = nat.load()
    assert nat.LIB_PATH.endswith("liblbm_bounds.so")
    runs = 0
    for nx, ny in SIZES:
        for scene, collision in SCENES:
            s = _lattice(nx, ny, scene, collision=collision)
            for n in (16, 17):
                s.step(n)
            s.sync()
            s.close()
            n, i, lim, site = ctypes.c_uint64(), ctypes.c_uint64(), ctypes.c_uint64(), ctypes.c_int32()
            assert lib.lbm_bounds_report(ctypes.byref(n), ctypes.byref(i), ctypes.byref(lim), ctypes.byref(site)) == 0
            assert n.value == 0, (nx, ny, scene, collision, n.value, i.value, lim.value, site.value)
            runs += 1
    print("small lattices: %d runs without a record" % runs)


def test_no_index_leaves_its_buffer(gpu):
    from simuverse_gb300 import build

    build.build(variant="bounds")
    env = dict(os.environ, SIMUVERSE_LBM_VARIANT="bounds", PYTHONPATH=ROOT)
    code = "import sys; sys.path.insert(0, %r); import test_gpu_cluster as t; t.child_main()" % os.path.join(ROOT, "tests")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "without a record" in r.stdout
