"""Edits between calls that take several steps per launch: the state after them is that of single steps
(kernel="cell") bit for bit, solid cells included.  A cell that turns solid keeps what each of the two
population buffers holds, which outer-ring cells of the reference's rules pull from, and which comes back when the
cell turns into fluid again; so the buffers must hold what single steps leave there."""
import os
import subprocess
import sys

import numpy as np
import pytest

from test_gpu_fused import ROOT, _same

pytestmark = pytest.mark.gpu

# lattices of fused steps (march), of two of them as well, and, in physics mode, of one cluster
LARGE, SMALL = (1300, 1250), (128, 128)
FORMS = [((1700, 1650), "poiseuille", dict(mode="reference", arith="fast")),
         ((1500, 1350), "custom", dict(mode="reference", arith="fast"))]
FORMS += [(size, scene, dict(mode="physics", collision=c)) for size in (LARGE, SMALL)
          for scene, c in (("channel", "bgk"), ("periodic", "bgk"), ("cavity", "kbc"))]
IDS = ["%s %s %s" % (s[0], sc, f.get("collision", "reference")) for s, sc, f in FORMS]


def _pair(size, scene, form):
    from simuverse_gb300 import FluidSimulator

    nx, ny = size
    out = []
    for kernel in ("auto", "cell"):
        kw = dict(form, kernel=kernel, tau=0.62)
        if form["mode"] == "physics":
            kw.update(lid_speed=0.05, inlet_speed=0.03, solid_fraction=0.0)
        s = FluidSimulator(nx, ny, scene=scene, **kw)
        if form["mode"] == "physics":
            rng = np.random.default_rng(nx)
            s.init_equilibrium(*((a + 0.02 * rng.standard_normal((ny, nx))).astype(np.float32) for a in (1.0, 0.03, 0.0)))
        out.append(s)
    return out


def _both(pair, f):
    for s in pair:
        f(s)


def _fused(pair, n):
    """Steps of both; the first takes more than one of them in some launch."""
    before = pair[0].kernel_launches
    _both(pair, lambda s: s.step(n))
    return pair[0].kernel_launches - before < n


# (a large lattice's last launch is one of 2 or 3 steps; a small one takes some ten steps in one)
CALLS = [(f, n) for f in FORMS for n in ((2, 3, 4, 7, 16, 17) if f[0] == SMALL else (2, 3, 4, 7))]


@pytest.mark.parametrize("size,scene,form,n", [f + (n,) for f, n in CALLS], ids=["%s %d" % (IDS[FORMS.index(f)], n) for f, n in CALLS])
def test_edits_between_calls(gpu, size, scene, form, n):
    nx, ny = size
    pair = _pair(size, scene, form)
    fused = _fused(pair, n)
    assert fused or size == SMALL and n < 16
    x, y = 29, ny // 2  # reaches columns 1 and 0
    _both(pair, lambda s: s.add_obstacle(x, y))
    _both(pair, lambda s: s.step(5))
    _same(*pair, "obstacle")
    # a force stroke through it: some of its cells are fluid again, with what the wall has kept
    _both(pair, lambda s: s.add_external_force((2.0 * x + 20.0, 2.0 * y), (4.0, 2.0 * y - 20.0)))
    _both(pair, lambda s: s.step(4))
    _same(*pair, "stroke")
    _both(pair, lambda s: s.step(100))  # the stroke's records end after 90
    _fused(pair, n)
    _both(pair, lambda s: s.set_tau(0.7))  # what is made up for was computed at the former rate
    _both(pair, lambda s: s.apply_edits([("obstacle", nx - 30, ny // 2), ("obstacle", nx // 2, 28)]))
    _both(pair, lambda s: s.step(5))
    _same(*pair, "edit list")
    _fused(pair, n)
    info = pair[0].info()
    assert np.array_equal(info, pair[1].info())
    info[ny // 2 - 10:ny // 2, 1:60] = (1, -1, 0.0, 0.0)  # uncovers half of the first obstacle
    info[ny // 2 + 40:ny // 2 + 44, nx // 3] = (4, -1, 0.0, 0.0)
    _both(pair, lambda s: s.set_info(info))
    for k in (1, 4, n):
        _both(pair, lambda s: s.step(k))
        _same(*pair, "mask")


@pytest.mark.parametrize("size,scene,form", FORMS, ids=IDS)
@pytest.mark.parametrize("n", [2, 3, 16])
def test_what_else_keeps_the_other_buffer(gpu, tmp_path, size, scene, form, n):
    """Checkpoints hold both buffers; a reset and new populations leave cells of the other one."""
    nx, ny = size
    pair, other = _pair(size, scene, form), _pair(size, scene, form)
    obstacle = lambda s: s.add_obstacle(29, ny // 2)
    _fused(pair, n)
    for k, s in enumerate(pair):
        s.save(str(tmp_path / ("%d" % k)))
    with open(tmp_path / "0", "rb") as a, open(tmp_path / "1", "rb") as b:
        assert a.read() == b.read()
    for k, s in enumerate(other):
        s.load(str(tmp_path / ("%d" % k)))
    _both(other, obstacle)
    for k in (1, 2, 3, n):
        _both(other, lambda s: s.step(k))
        _same(*other, "loaded")
    f = pair[0].read_populations() * np.float32(1.01)
    _both(pair, lambda s: s.write_populations(f))
    _both(pair, obstacle)
    for k in (1, 4):
        _both(pair, lambda s: s.step(k))
        _same(*pair, "written")
    _fused(pair, n)
    _both(pair, lambda s: s.reset())
    _both(pair, lambda s: s.add_obstacle(nx // 2, ny // 2))
    for k in (1, 4):
        _both(pair, lambda s: s.step(k))
        _same(*pair, "reset")


@pytest.mark.parametrize("size,scene,form", FORMS, ids=IDS)
@pytest.mark.parametrize("stroke", ["call", "list"])
def test_records_that_change_before_the_walls(gpu, tmp_path, size, scene, form, stroke):
    """A stroke, then an obstacle or a checkpoint, without a step between: its records have counted nothing yet, and what is
    made up for was computed without them."""
    nx, ny = size
    pair = _pair(size, scene, form)
    line = (nx + 90.0, ny + 40.0, nx - 90.0, ny - 40.0)
    force = (lambda s: s.add_external_force(line[:2], line[2:])) if stroke == "call" else (lambda s: s.apply_edits([("force",) + line]))
    assert _fused(pair, 19)
    _both(pair, force)
    for k, s in enumerate(pair):
        s.save(str(tmp_path / ("%d" % k)))
    with open(tmp_path / "0", "rb") as a, open(tmp_path / "1", "rb") as b:
        assert a.read() == b.read()
    _both(pair, lambda s: s.add_obstacle(nx // 2 + 20, ny // 2))
    assert np.array_equal(pair[0].info(), pair[1].info())
    for k in (1, 4):
        _both(pair, lambda s: s.step(k))
        _same(*pair, "obstacle")


@pytest.mark.parametrize("size,scene,form", [FORMS[1], (LARGE, "cavity", dict(mode="physics"))], ids=["reference", "physics"])
def test_unlike_walls_do_not_outlive_their_cause(gpu, tmp_path, size, scene, form):
    """New records that leave the walls as they were, and a checkpoint of a lattice whose walls agree: a frame of two
    steps is one launch."""
    a, b = _pair(size, scene, form)
    _both((a, b), lambda s: s.step(3))
    info = a.info()
    info["vx"][5, 5] = 0.01
    _both((a, b), lambda s: s.set_info(info))
    before = a.kernel_launches
    _both((a, b), lambda s: s.compute())
    assert a.kernel_launches == before + 1
    _same(a, b, "records")
    path = str(tmp_path / "walls")
    b.save(path)
    c = _pair(size, scene, form)[0]
    c.load(path)
    before = c.kernel_launches
    _both((c, b), lambda s: s.compute())
    assert c.kernel_launches == before + 1
    _same(c, b, "checkpoint")


def child_main():
    import ctypes

    from simuverse_gb300 import _native as nat

    lib = nat.load()
    assert nat.LIB_PATH.endswith("liblbm_bounds.so")
    for size, scene, form in FORMS:
        for n in (16,) if size == SMALL else (2, 3):
            test_edits_between_calls(lib, size, scene, form, n)
    n = ctypes.c_uint64()
    assert lib.lbm_bounds_report(ctypes.byref(n), None, None, None) == 0 and n.value == 0
    print("edits: no record")


def test_without_device_scratch(gpu):
    """The bounds-checked build takes the steps again through host memory, as where the device has none left."""
    from simuverse_gb300 import build

    build.build(variant="bounds")
    env = dict(os.environ, SIMUVERSE_LBM_VARIANT="bounds", PYTHONPATH=ROOT)
    code = "import sys; sys.path.insert(0, %r); import test_gpu_edits_fused as t; t.child_main()" % os.path.join(ROOT, "tests")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "no record" in r.stdout
