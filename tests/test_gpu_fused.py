"""Fused time steps (lbm_step_fused.cu) against the one-step kernels (kernel="cell"): the state and the
macro field after a call of n steps are the same bits, at window and segment edges, for every
boundary rule, and where fusing must not happen (records that count down, walls whose unwritten
slots differ between the buffers).  In the bounds-checked build no index leaves its buffer."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# all above the size from which steps are fused; widths of and off a multiple of four, one window to many
SIZES = [(64, 12504), (65, 12401), (121, 6700), (841, 960), (1032, 780), (60004, 14)]


def _mask(info, seed, block_iter):
    """Obstacles beside walls, in corners and scattered, and forcing cells with that countdown."""
    ny, nx = info.shape
    rng = np.random.default_rng(seed)
    at = [(1, 1), (nx - 2, 1), (1, ny - 2), (nx - 2, ny - 2), (nx // 2, 1), (61, ny // 2), (62, ny // 2)]
    at += [(int(rng.integers(1, nx - 1)), int(rng.integers(1, ny - 1))) for _ in range(nx * ny // 150)]
    for x, y in at:
        info[y, x] = (4, -1, 0.0, 0.0)
    for _ in range(4):
        x, y = int(rng.integers(1, nx - 1)), int(rng.integers(1, ny - 1))
        if info[y, x]["material"] == 1:
            info[y, x] = (6, block_iter, 0.01, -0.02)
    return info


def _lattice(nx, ny, scene, seed, block_iter=-1, **kw):
    from simuverse_gb300 import FluidSimulator

    if "mode" not in kw:
        kw.update(mode="physics", lid_speed=0.05, inlet_speed=0.03, solid_fraction=0.0)
    s = FluidSimulator(nx, ny, scene=scene, tau=0.6, **kw)
    s.set_info(_mask(s.info(), seed, block_iter))
    if kw["mode"] == "physics":
        rng = np.random.default_rng(seed + 1)
        s.init_equilibrium(*((a + 0.02 * rng.standard_normal((ny, nx))).astype(np.float32) for a in (1.0, 0.03, 0.0)))
    else:
        s.reset() if scene != "poiseuille" else None  # (a reset would rebuild that scene's mask)
    return s


def _same(a, b, label):
    # the populations the next step reads, as stored: solid cells and both layouts included
    assert np.array_equal(a.read_populations().view(np.uint32), b.read_populations().view(np.uint32)), label
    for x, y in zip(a.read_macro(), b.read_macro()):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), label


def _forms():
    physics = [(s, dict(collision=c)) for c in ("bgk", "kbc") for s in ("cavity", "channel", "periodic")]
    return physics + [(s, dict(mode="reference", arith="fast")) for s in ("poiseuille", "cavity", "custom")]


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("scene,form", _forms(), ids=lambda v: v if isinstance(v, str) else "-".join(v.values()))
def test_fused_steps_equal_single_steps(gpu, nx, ny, scene, form):
    a, b = _lattice(nx, ny, scene, nx, **form), _lattice(nx, ny, scene, nx, kernel="cell", **form)
    for n in (2, 3, 4, 5, 7):
        launches = a.kernel_launches
        a.step(n)
        assert a.kernel_launches - launches == {2: 1, 3: 1, 4: 2, 5: 2, 7: 3}[n] or scene == "poiseuille"
        b.step(n)
        _same(a, b, (n, form))


@pytest.mark.parametrize("scene,form", [("cavity", {}), ("channel", {}), ("poiseuille", dict(mode="reference", arith="fast")),
                                        ("custom", dict(mode="reference", arith="fast"))])
def test_counting_records_and_unlike_walls(gpu, scene, form):
    a, b = _lattice(1100, 800, scene, 3, 5, **form), _lattice(1100, 800, scene, 3, 5, kernel="cell", **form)
    for n in (4, 2, 6):
        a.step(n)
        b.step(n)
        _same(a, b, n)
        assert np.array_equal(a.info(), b.info())
    # solid cells too: the buffers differ there now
    f = a.read_populations() + np.float32(1e-3) * np.random.default_rng(5).random((9, 800, 1100), np.float32)
    for s in (a, b):
        s.write_populations(f)
    for n in (2, 4, 3, 5):
        a.step(n)
        b.step(n)
        _same(a, b, n)


def test_planes_beyond_32_bits(gpu):
    """2^29 cells and more: eight planes are further apart than 32 bits count."""
    import torch

    from simuverse_gb300 import FluidSimulator

    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("not enough device memory")
    nx, ny = 32768, 16400
    row = (0.02 * np.random.default_rng(6).standard_normal(nx + 64)).astype(np.float32)
    u = np.stack([row[k % 61:k % 61 + nx] for k in range(ny)])
    sums = []
    for kernel in ("auto", "cell"):
        s = FluidSimulator(nx, ny, mode="physics", scene="periodic", tau=0.6, kernel=kernel)
        s.init_equilibrium(None, u, u[::-1])
        s.step(3)
        sums.append(s.conservation())
        s.close()
    assert sums[0] == sums[1]  # FP64 sums in a fixed order over the same bits


def child_main():
    import ctypes

    from simuverse_gb300 import _native as nat

    lib = nat.load()
    assert nat.LIB_PATH.endswith("liblbm_bounds.so")
    runs = 0
    for nx, ny in SIZES:
        for scene, form in _forms():
            s = _lattice(nx, ny, scene, nx + ny, **form)
            for n in (3, 2, 4):
                s.step(n)
            s.sync()
            s.close()
            n, i, lim, site = ctypes.c_uint64(), ctypes.c_uint64(), ctypes.c_uint64(), ctypes.c_int32()
            assert lib.lbm_bounds_report(ctypes.byref(n), ctypes.byref(i), ctypes.byref(lim), ctypes.byref(site)) == 0
            assert n.value == 0, (nx, ny, scene, form, n.value, i.value, lim.value, site.value)
            runs += 1
    print("fused steps: %d runs without a record" % runs)


def test_no_index_leaves_its_buffer(gpu):
    from simuverse_gb300 import build

    build.build(variant="bounds")
    env = dict(os.environ, SIMUVERSE_LBM_VARIANT="bounds", PYTHONPATH=ROOT)
    code = "import sys; sys.path.insert(0, %r); import test_gpu_fused as t; t.child_main()" % os.path.join(ROOT, "tests")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "without a record" in r.stdout
