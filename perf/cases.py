"""Workloads whose speed is followed: what a user of the library has it do, through its Python
entry points, from one frame of a window-sized lattice to steps of an 8192 x 8192 one.

Kinds of case (the "kind" of a case's dict):

step      ``FluidSimulator.step`` of a lattice that lives on the GPU, physics rules or the
          reference's; the macro field and the populations stay on the device.
frame     one frame of the interactive simulator: step, particles, step, particles, present.
run       a whole run as a batch job makes it: create, step, read the macro field into
          page-locked host memory, close.
batch     many lattices of uneven size advanced together, every field read back.
coarse    the coarse lattice of the learned closure: k steps, one closure application, repeated.
train     Adam iterations of the closure on stored pairs.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from simuverse_gb300 import INFO_DTYPE, BatchSimulator, FluidSimulator, generate_domains
from simuverse_gb300.closure import Closure
from simuverse_gb300.view import Particles

DTYPE_BYTES = {"f32": 4, "f64": 8, "f16": 2, "bf16": 2}
EX = (0, 1, 0, -1, 0, 1, -1, -1, 1)
EY = (0, 0, -1, 0, 1, -1, -1, 1, 1)
INV = (0, 3, 4, 1, 2, 7, 8, 5, 6)
W = (4 / 9,) + (1 / 9,) * 4 + (1 / 36,) * 4
BULK, BOUNDARY, INLET, OBSTACLE, OUTLET = 1, 2, 3, 4, 5


def listed():
    return [
        # the lid-driven cavity every solver is checked on, a hundred steps a call: launches count
        dict(name="cavity_256", kind="step", nx=256, ny=256, scene="cavity", dtype="f32", tau=0.6, steps=100),
        # the interactive simulator in a 1200 x 750 window: one frame, as the reference draws it
        dict(name="frame_600x375", kind="frame", nx=600, ny=375, particles=10000),
        # channel flow around seeded disks, the benchmark's own size and step count
        dict(name="channel_4096", kind="step", nx=4096, ny=4096, scene="channel", dtype="f32", tau=0.56, steps=20),
        # half-precision storage with stochastic rounding, for the largest lattices
        dict(name="channel_8192_f16_sr", kind="step", nx=8192, ny=8192, scene="channel", dtype="f16",
             rounding="stochastic", tau=0.6, steps=10),
        # bfloat16 storage on a lattice that is no multiple of a tile
        dict(name="channel_3002x1701_bf16", kind="step", nx=3002, ny=1701, scene="channel", dtype="bf16", tau=0.6,
             steps=20),
        # the double-precision run that the others are judged by
        dict(name="channel_2048_f64", kind="step", nx=2048, ny=2048, scene="channel", dtype="f64", tau=0.6, steps=10),
        # the reference's rules at the size its roofline is quoted at: one frame of two steps
        dict(name="reference_8192", kind="step", nx=8192, ny=8192, scene="poiseuille", mode="reference", arith="fast",
             dtype="f32", tau=0.62, steps=2),
        # decaying turbulence near tau = 1/2 with the entropic collision, as the closure's fine run
        dict(name="turbulence_2048_kbc", kind="step", nx=2048, ny=2048, scene="periodic", dtype="f32",
             collision="kbc", tau=0.5005, steps=16),
        # a parameter study: cavities and channels of 64 to 1024 cells a side
        dict(name="batch_64", kind="batch", domains=64, sizes=1, steps=1000),
        # the coarse lattice with the learned closure every fourth step
        dict(name="coarse_1024", kind="coarse", n=1024, steps=16, every=4),
        # training it: batches of eight 256 x 256 windows
        dict(name="train_8x256", kind="train", n=512, crop=256, batch=8, pairs=24, iters=10),
        # the benchmark's end-to-end figure
        dict(name="run_4096", kind="run", nx=4096, ny=4096, scene="channel", dtype="f32", tau=0.56, steps=20),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "step", "step", "frame", "batch", "coarse", "train", "run"))
    if kind == "step":
        mode = rng.choice(("physics", "physics", "physics", "reference"))
        if mode == "reference":
            nx, ny = _logint(rng, 96, 6000), _logint(rng, 96, 6000)
            return dict(kind="step", nx=nx, ny=ny, scene=rng.choice(("poiseuille", "cavity")), mode="reference",
                        arith=rng.choice(("exact", "fast")), dtype="f32", tau=round(rng.uniform(0.55, 1.0), 3),
                        steps=_logint(rng, 1, max(1, min(100, 10 ** 8 // (nx * ny)))))
        scene = rng.choice(("cavity", "channel", "channel", "periodic"))
        dtype = rng.choice(("f32", "f32", "f32", "f16", "bf16", "f64"))
        top = 2048 if dtype == "f64" else 6000
        nx, ny = _logint(rng, 64, top), _logint(rng, 64, top)
        if rng.random() < 0.4:
            nx = max(64, nx // 64 * 64)
        c = dict(kind="step", nx=nx, ny=ny, scene=scene, dtype=dtype, tau=round(rng.uniform(0.55, 1.0), 3),
                 steps=_logint(rng, 1, max(1, min(100, (2 * 10 ** 7 if dtype == "f64" else 2 * 10 ** 8) // (nx * ny)))))
        if DTYPE_BYTES[dtype] == 2:
            c["rounding"] = rng.choice(("nearest", "stochastic"))
        if scene == "periodic" and dtype == "f32":
            c["collision"] = rng.choice(("bgk", "kbc"))
        return c
    if kind == "frame":
        return dict(kind="frame", nx=_logint(rng, 160, 1920), ny=_logint(rng, 120, 1080),
                    particles=_logint(rng, 1000, 60000))
    if kind == "batch":
        return dict(kind="batch", domains=rng.randint(8, 64), sizes=rng.randint(2, 999), steps=_logint(rng, 50, 800))
    if kind == "coarse":
        return dict(kind="coarse", n=16 * _logint(rng, 8, 64), steps=rng.choice((4, 8, 16)), every=rng.choice((2, 4)))
    if kind == "train":
        return dict(kind="train", n=512, crop=rng.choice((64, 128, 256)), batch=rng.choice((4, 8)), pairs=24,
                    iters=rng.randint(2, 10))
    return dict(kind="run", nx=_logint(rng, 256, 4000), ny=_logint(rng, 256, 4000), scene="channel", dtype="f32",
                tau=round(rng.uniform(0.55, 1.0), 3), steps=_logint(rng, 4, 20))


# ---- inputs -----------------------------------------------------------------------------
def _smooth(nx, ny, gen, amp, cell=24):
    """A smooth random field of RMS about `amp` that varies over `cell` cells (FP32, on the GPU)."""
    low = torch.randn(1, 1, max(4, ny // cell), max(4, nx // cell), generator=gen, device="cuda")
    return F.interpolate(low, size=(ny, nx), mode="bilinear", align_corners=True)[0, 0] * (1.3 * amp)


def _flow(case, seed):
    """Density and velocity a running simulation of the scene has: the scene's mean flow with
    smooth disturbances (three FP32 planes on the GPU)."""
    nx, ny = case["nx"], case["ny"]
    g = torch.Generator(device="cuda").manual_seed(7919 * seed + 1)
    cell = 24 if min(nx, ny) > 200 else 8
    ux, uy, r = (_smooth(nx, ny, g, a, cell) for a in (0.01, 0.01, 0.003))
    if case["scene"] == "channel":
        ux = ux + _parabola(ny, 0.05).to(torch.float32)[:, None]
    return 1.0 + r, ux, uy


def _parabola(ny, peak):
    s = torch.arange(ny, device="cuda", dtype=torch.float64) - 0.5
    h = float(ny - 2)
    return (4.0 * peak * s * (h - s) / (h * h)).clamp_min(0.0)


def _disks(nx, ny, seed):
    """Solid disks, radius 8 to 32 cells, about 5 % of the cells, none touching another: one in
    each square of a grid, moved at random inside it.  True where a cell is solid."""
    pitch = 168
    g = torch.Generator(device="cuda").manual_seed(104729 * seed + 2)
    gx, gy = (nx + pitch - 1) // pitch, (ny + pitch - 1) // pitch
    u = torch.rand(3, gy, gx, generator=g, device="cuda")
    r = 8.0 + 24.0 * u[0]
    off = 36.0 + (pitch - 72.0) * u[1:]
    x, y = torch.arange(nx, device="cuda"), torch.arange(ny, device="cuda")
    ix, iy = (x // pitch)[None, :].expand(ny, nx), (y // pitch)[:, None].expand(ny, nx)
    dx = (x % pitch)[None, :] - off[0][iy, ix]
    dy = (y % pitch)[:, None] - off[1][iy, ix]
    solid = dx * dx + dy * dy <= (r * r)[iy, ix]
    solid[:, :2] = False
    solid[:, -2:] = False
    return solid


def _mask(case, seed):
    """(material, vx) planes of a physics-mode scene: int32 and FP32."""
    nx, ny = case["nx"], case["ny"]
    m = torch.full((ny, nx), BULK, dtype=torch.int32, device="cuda")
    v = torch.zeros(ny, nx, dtype=torch.float32, device="cuda")
    if case["scene"] == "cavity":
        m[0], m[-1], m[:, 0], m[:, -1] = (BOUNDARY,) * 4
        v[0, 1:-1] = 0.1
    elif case["scene"] == "channel":
        m[:, 0], m[:, -1] = INLET, OUTLET
        v[:, 0] = _parabola(ny, 0.05).to(torch.float32)
        m[_disks(nx, ny, seed)] = OBSTACLE
        m[0], m[-1] = BOUNDARY, BOUNDARY
        v[0], v[-1] = 0.0, 0.0
    return m, v


def _info(m, v):
    t = torch.stack((m, torch.full_like(m, -1), v.view(torch.int32), torch.zeros_like(m)), dim=-1)
    return t.cpu().numpy().view(INFO_DTYPE).reshape(m.shape)


class _View:
    """A device buffer of the library as a tensor, without a copy; the tensor keeps its owner."""

    def __init__(self, owner, ptr, count, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 2}


def _view(owner, ptr, shape, dtype):
    kind = {"f32": "<f4", "f64": "<f8", "f16": "<f2", "bf16": "<i2"}[dtype]
    t = torch.as_tensor(_View(owner, ptr, math.prod(shape), kind), device="cuda")
    return (t.view(torch.bfloat16) if dtype == "bf16" else t).view(shape)


def _outputs(sim, views):
    """The macro planes and the current populations, in place (the population buffer alternates)."""
    key = sim.device_populations()[0]
    if key not in views:
        views[key] = _view(sim, key, (9 * sim.N,), sim.dtype)
    return views["macro"] + (views[key],)


def _macro_views(sim):
    return tuple(_view(sim, p, (sim.ny, sim.nx), "f32") for p in sim.device_macro())


def _lattice(case, seed):
    if case.get("mode") == "reference":
        sim = FluidSimulator(case["nx"], case["ny"], mode="reference", scene=case["scene"], tau=case["tau"],
                             arith=case["arith"])
        sim.write_populations(_reference_start(case, seed).cpu().numpy())
        return sim
    more = {k: case[k] for k in ("collision", "rounding") if k in case}
    sim = FluidSimulator(case["nx"], case["ny"], mode="physics", scene=case["scene"], dtype=case["dtype"],
                         tau=case["tau"], lid_speed=0.1, inlet_speed=0.05, solid_fraction=0.0, **more)
    if case["scene"] == "channel":
        sim.set_info(_info(*_mask(case, seed)))
    sim.init_equilibrium(*(t.cpu().numpy() for t in _flow(case, seed)))
    return sim


def _reference_start(case, seed):
    """Populations of a running reference-mode lattice: equilibrium of the flow, inside the
    shaders' clamps (FP32, absolute).  A wall holds what it hands back to a fluid cell inside
    the outer ring, and nothing else."""
    rho, ux, uy = (t.double() for t in _flow(dict(case, scene="channel"), seed))
    f = torch.stack(_equilibrium(rho, ux, uy)).to(torch.float32)
    solid, _ = _reference_mask(case["nx"], case["ny"], case["scene"])
    takes = ~solid
    takes[0], takes[-1], takes[:, 0], takes[:, -1] = (False,) * 4
    for j in range(9):
        f[j][solid & ~torch.roll(takes, (-EY[j], -EX[j]), (0, 1))] = 0.0
    return f


def _equilibrium(rho, ux, uy):
    usq = 1.5 * (ux * ux + uy * uy)
    out = []
    for i in range(9):
        eu = EX[i] * ux + EY[i] * uy
        out.append(W[i] * rho * (1.0 + 3.0 * eu + 4.5 * eu * eu - usq))
    return out


def _turbulent(n, seed, amp=0.04):
    """A divergence-free random velocity field on a periodic square (two FP32 planes)."""
    g = torch.Generator(device="cuda").manual_seed(15485863 * seed + 3)
    k = torch.fft.fftfreq(n, 1.0 / n, device="cuda")
    kk = torch.sqrt(k[None, :] ** 2 + k[:, None] ** 2)
    psi = torch.fft.fft2(torch.randn(n, n, generator=g, device="cuda")) * torch.exp(-(kk / 8.0) ** 2) * kk
    ux = torch.fft.ifft2(1j * k[:, None] * psi).real
    uy = torch.fft.ifft2(-1j * k[None, :] * psi).real
    s = amp / torch.sqrt((ux * ux + uy * uy).mean())
    return ux * s, uy * s


def _coarse_lattice(n, seed):
    sim = FluidSimulator(n, n, mode="physics", scene="periodic", tau=0.500125, collision="kbc")
    sim.init_equilibrium(None, *(t.cpu().numpy() for t in _turbulent(n, seed)))
    return sim


def _domains(case, seed):
    """The study's lattices (their sizes belong to the case), each at parameters of its own."""
    rng = np.random.default_rng(seed)
    return [dict(d, tau=round(rng.uniform(0.55, 1.0), 4), speed=round(rng.uniform(0.02, 0.1), 4))
            for d in generate_domains(case["domains"], case["sizes"])]


def _network(seed):
    """Weights and biases of the closure's three layers, of the size training starts from."""
    rng = np.random.default_rng(seed)
    out = []
    for cin, cout in ((9, 32), (32, 32), (32, 9)):
        out.append(rng.standard_normal(9 * cin * cout) * math.sqrt(2.0 / (9 * cin)))
        out.append(0.02 * rng.standard_normal(cout))
    return np.concatenate(out).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "step":
        s["sim"] = sim = _lattice(case, seed)
        s["views"] = {"macro": _macro_views(sim)}
    elif kind == "frame":
        s["sim"] = sim = FluidSimulator(case["nx"], case["ny"], tau=0.62, pixel_size=2)
        sim.write_populations(_reference_start(dict(case, scene="poiseuille"), seed).cpu().numpy())
        s["particles"] = p = Particles(sim, count=case["particles"], seed=seed)
        s["views"] = {"macro": _macro_views(sim), "rgba": _view(p, p.present(), (p.canvas_h, p.canvas_w, 4), "f32")}
    elif kind == "run":
        s["seed"] = seed
        s["host"] = tuple(torch.empty(case["ny"], case["nx"], pin_memory=True).numpy() for _ in range(3))
    elif kind == "batch":
        s["sim"] = sim = BatchSimulator(_domains(case, seed))
        sim.tune(trial_steps=4)
    elif kind == "coarse":
        s["sim"] = sim = _coarse_lattice(case["n"], seed)
        s["closure"] = c = Closure(case["n"], case["n"], seed=seed, s_in=20.0, s_out=1e4, inputs="eq", target="stress")
        c.params = _network(seed)
        s["views"] = {"macro": _macro_views(sim)}
    else:
        n = case["n"]
        rng = np.random.default_rng(seed)
        s["closure"] = c = Closure(n, n, seed=seed, s_in=20.0, s_out=300.0, inputs="eq", target="stress")
        c.params = _network(seed)
        c.set_stress_factor(16.0)
        c.reserve(case["pairs"], case["crop"], case["batch"])
        pred, target = _coarse_lattice(n, 2 * seed), _coarse_lattice(n, 2 * seed + 1)
        u, v = _turbulent(n, 2 * seed), _turbulent(n, 2 * seed + 1, 0.004)
        target.init_equilibrium(None, *((a + b).cpu().numpy() for a, b in zip(u, v)))
        for _ in range(case["pairs"]):
            c.add_pair(pred, target, int(rng.integers(0, n)), int(rng.integers(0, n)))
        s["seed"] = seed
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        if case["steps"] == 2:
            s["sim"].compute()  # the interactive simulator's frame
        else:
            s["sim"].step(case["steps"])
        return _outputs(s["sim"], s["views"])
    if kind == "frame":
        s["particles"].compute()
        s["particles"].present()
        return _outputs(s["sim"], s["views"]) + (s["views"]["rgba"],)
    if kind == "run":
        with FluidSimulator(case["nx"], case["ny"], mode="physics", scene=case["scene"], dtype=case["dtype"],
                            tau=case["tau"], inlet_speed=0.05, seed=s["seed"]) as sim:
            sim.step(case["steps"])
            return sim.read_macro(out=s["host"])
    if kind == "batch":
        s["sim"].step(case["steps"])
        return np.concatenate([np.ravel(a) for i in range(case["domains"]) for a in s["sim"].read_macro(i)])
    if kind == "coarse":
        for _ in range(case["steps"] // case["every"]):
            s["sim"].step(case["every"])
            s["closure"].apply(s["sim"])
        return _outputs(s["sim"], s["views"])
    loss = s["closure"].train(case["iters"], lr=1e-3, seed=s["seed"])
    return loss, s["closure"].params


def work(case):
    """A pass reads its state once and leaves the new state and what it returns; the operations
    are the collisions' (about 110 a cell and step), the convolutions' and the pixels'."""
    kind = case["kind"]
    if kind in ("step", "run"):
        cells, b = case["nx"] * case["ny"], DTYPE_BYTES[case["dtype"]]
        kbc = case.get("collision") == "kbc"
        state = cells * (18 * b + 2) if kind == "step" else cells * (9 * b + 2)
        return {"bytes": state + 12 * cells, "flops": cells * case["steps"] * (190 if kbc else 110)}
    if kind == "frame":
        cells, px = case["nx"] * case["ny"], 4 * case["nx"] * case["ny"]
        return {"bytes": cells * (72 + 2 + 24) + px * (12 + 16 + 4) + case["particles"] * 96,
                "flops": cells * 2 * 110 + px * 30 + case["particles"] * 200}
    if kind == "batch":
        cells = sum(d["nx"] * d["ny"] for d in generate_domains(case["domains"], case["sizes"]))
        return {"bytes": cells * (72 + 2 + 12), "flops": cells * case["steps"] * 110}
    conv = 2 * 9 * (9 * 32 + 32 * 32 + 32 * 9)
    if kind == "coarse":
        cells, calls = case["n"] ** 2, case["steps"] // case["every"]
        return {"bytes": cells * (72 + 2 + 12), "flops": cells * (case["steps"] * 190 + calls * conv)}
    cells = case["batch"] * case["crop"] ** 2 * case["iters"]
    return {"bytes": cells * 4 * (9 + 9), "flops": cells * 3 * conv}


# ---- the same in 64 bits, in plain torch -------------------------------------------------
def exact(case, seed):
    """FP64 results.  None: a training run (its batches come from the library's generator), a
    whole run (so do its disks), a frame (the particles' jitter too), and more cell updates than
    plain torch does in some seconds."""
    kind = case["kind"]
    if kind == "step" and case["nx"] * case["ny"] * case["steps"] <= 7 * 10 ** 8:
        if case.get("mode") == "reference":
            # (the walls' own slots in the populations depend on the order of the boundary pass)
            return _exact_reference(_reference_start(case, seed), case) + (None,)
        m, v = _mask(case, seed)
        rho, ux, uy = (t.double() for t in _flow(case, seed))
        f = torch.stack(_equilibrium(rho, ux, uy))
        f, macro = _exact_physics(f, m, v, 1.0 / _tau32(case["tau"]), case["steps"], case.get("collision", "bgk"))
        return macro + (_stored(f, m, case),)
    if kind == "batch" and case["domains"] * case["steps"] <= 4000:
        return _exact_batch(case, seed)
    if kind == "coarse":
        return _exact_coarse(case, seed)
    return None


def _tau32(tau):
    return float(np.float32(tau))


def _stored(f, m, case):
    """Deviations f - w as the lattice stores them: zero in solid cells, FP16 times 2^10, and
    16-bit rows of a multiple of 64 cells in tiles that keep their nine planes together."""
    d = f - torch.tensor(W, dtype=torch.float64, device="cuda")[:, None, None]
    d[:, (m == BOUNDARY) | (m == OBSTACLE)] = 0.0
    if case["dtype"] == "f16":
        d = d * 1024.0
    nx, ny = case["nx"], case["ny"]
    if DTYPE_BYTES[case["dtype"]] == 2 and nx % 64 == 0:
        d = d.view(9, ny, nx // 64, 64).permute(1, 2, 0, 3)
    return d.reshape(-1)


def _exact_physics(f, m, v, omega, steps, collision):
    """Pull streaming with half-way bounce-back (moving lid), Zou-He inlet on the west face,
    outflow anchored at unit density on the east face, BGK or entropic collision."""
    w = torch.tensor(W, dtype=torch.float64, device="cuda")
    solid = (m == BOUNDARY) | (m == OBSTACLE)
    inlet, outlet = m[:, 0] == INLET, m[:, -1] == OUTLET
    v = v.double()
    back, lid = [], []
    for j in range(9):
        src = torch.roll(solid, (EY[j], EX[j]), (0, 1)) & ~solid
        if EX[j] == -1 and bool(outlet.any()):  # the outflow pulls from its own column
            own = torch.roll(solid, EY[j], 0)[:, -1]
            src[:, -1] = torch.where(outlet, own & ~solid[:, -1], src[:, -1])
        back.append(src)
        lid.append(torch.where(src & solid.roll((EY[j], EX[j]), (0, 1)),
                               torch.roll(v, (EY[j], EX[j]), (0, 1)) * (6.0 * W[j] * EX[j]), 0.0))
    f = f.clone()
    f[:, solid] = w[:, None]
    macro = None
    for _ in range(steps):
        p = []
        for j in range(9):
            s = torch.roll(f[j], (EY[j], EX[j]), (0, 1))
            if EX[j] == -1 and bool(outlet.any()):
                s[:, -1] = torch.where(outlet, torch.roll(f[j][:, -1], EY[j], 0), s[:, -1])
            if j:
                s = torch.where(back[j], f[INV[j]] + lid[j], s)
            p.append(s)
        if bool(inlet.any()):
            c = [q[:, 0].clone() for q in p]
            u = v[:, 0]
            r = (c[0] + c[2] + c[4] + 2.0 * (c[3] + c[6] + c[7])) / (1.0 - u)
            n1 = c[3] + 2.0 / 3.0 * r * u
            n5 = c[7] + 0.5 * (c[4] - c[2]) + r * u / 6.0
            n8 = c[6] + 0.5 * (c[2] - c[4]) + r * u / 6.0
            for j, n in ((1, n1), (5, n5), (8, n8)):
                p[j][:, 0] = torch.where(inlet, n, c[j])
        if bool(outlet.any()):
            tot = sum(q[:, -1] for q in p)
            for q in p:
                q[:, -1] = torch.where(outlet, q[:, -1] / tot, q[:, -1])
        rho = sum(p)
        ux = (p[1] + p[5] + p[8] - p[3] - p[6] - p[7]) / rho
        uy = (p[4] + p[7] + p[8] - p[2] - p[5] - p[6]) / rho
        eq = _equilibrium(rho, ux, uy)
        if collision == "kbc":
            n = [p[j] - eq[j] for j in range(9)]
            dn, dp = 0.25 * (n[1] + n[3] - n[2] - n[4]), 0.25 * (n[8] + n[6] - n[5] - n[7])
            ds = (None, dn, -dn, dn, -dn, -dp, dp, -dp, dp)
            sh = sum(ds[j] * (n[j] - ds[j]) / eq[j] for j in range(1, 9))
            hh = sum((n[j] - (ds[j] if j else 0.0)) ** 2 / eq[j] for j in range(9))
            beta = 0.5 * omega
            gamma = torch.where(hh > 1e-30, 1.0 / beta - (2.0 - 1.0 / beta) * sh / hh, 2.0)
            o = [p[j] - beta * (2.0 * ds[j] + gamma * (n[j] - ds[j])) for j in range(1, 9)]
            o = [rho - sum(o)] + o
        else:
            o = [p[j] + omega * (eq[j] - p[j]) for j in range(9)]
        f = torch.stack([torch.where(solid, W[j], o[j]) for j in range(9)])
        macro = tuple(torch.where(solid, 0.0, t) for t in (rho, ux, uy))
    return f, macro


def _reference_mask(nx, ny, scene):
    """(solid, forcing speed) of the reference's scenes (simuverse/src/fluid/lattice.rs:52-83)."""
    solid = torch.zeros(ny, nx, dtype=torch.bool, device="cuda")
    force = torch.zeros(ny, nx, dtype=torch.float64, device="cuda")
    solid[-1] = True
    if scene == "cavity":
        solid[:, 0], solid[:, -1] = True, True
        force[1, 1:-1] = float(np.float32(0.13))
        return solid, force
    x, y = torch.arange(nx, device="cuda", dtype=torch.float32), torch.arange(ny, device="cuda", dtype=torch.float32)
    n = np.float32
    at = ((n(nx) / n(7) - n(28), n(ny) / n(2)), (n(nx) / n(5), n(ny) / n(4)), (n(nx) / n(5), n(ny) * n(0.75)))
    for cx, cy in at:
        dx, dy = (x - float(cx))[None, :], (y - float(cy))[:, None]
        solid |= torch.sqrt(dx * dx + dy * dy) <= 28.0
    solid[:, :2], solid[:, -2:] = False, False
    solid[0], solid[-1] = True, True
    force[1:-1, 1] = float(np.float32(0.12))
    return solid, force


def _exact_reference(f, case):
    """The shaders' rules: clamped density and populations, truncated weights, forcing rows,
    walls that hand populations back in the next step's buffer."""
    f = f.double()
    wt = [float(np.float32(t)) for t in [0.444444] + [0.111111] * 4 + [0.0277777] * 4]
    top = [float(np.float32(t)) for t in [0.6] + [0.2222] * 4 + [0.1111] * 4]
    lo, hi = float(np.float32(0.8)), float(np.float32(1.2))
    om = 1.0 / _tau32(case["tau"])
    solid, force = _reference_mask(case["nx"], case["ny"], case["scene"])
    inside = torch.zeros_like(solid)
    inside[1:-1, 1:-1] = True
    acts = force != 0.0
    other = torch.zeros_like(f)  # the buffer that the first step writes
    macro = None
    for _ in range(case["steps"]):
        p = [torch.roll(f[j], (EY[j], EX[j]), (0, 1)) for j in range(9)]
        rho = sum(p).clamp(lo, hi)
        ux = (p[1] + p[5] + p[8] - p[3] - p[6] - p[7]) / rho
        uy = (p[4] + p[7] + p[8] - p[2] - p[5] - p[6]) / rho
        ux, uy = torch.where(acts, 0.5 * force / rho, ux), torch.where(acts, 0.0, uy)
        usq = 1.5 * (ux * ux + uy * uy)
        g = []
        for j in range(9):
            eu = EX[j] * ux + EY[j] * uy
            eq = rho * wt[j] * (1.0 + 3.0 * eu + 4.5 * eu * eu - usq)
            t = (p[j] - om * (p[j] - eq) + 3.0 * wt[j] * EX[j] * force).clamp(0.0, top[j])
            g.append(torch.where(solid, other[j], t))
        n = [t.clone() for t in g]
        for j in range(1, 9):
            gives = inside & ~solid & torch.roll(solid, (-EY[j], -EX[j]), (0, 1))
            takes = torch.roll(gives, (EY[j], EX[j]), (0, 1))
            n[INV[j]] = torch.where(takes, torch.roll(g[j], (EY[j], EX[j]), (0, 1)), n[INV[j]])
            n[j] = torch.where(gives, 0.0, n[j])
        f, other = torch.stack(n), f
        macro = tuple(torch.where(solid, 0.0, t) for t in (rho, ux, uy))
    return macro


def _exact_coarse(case, seed):
    """The entropic collision with the closure's stress form after every few steps: features of
    the equilibrium, three convolutions, the divergence of their projected outputs."""
    n = case["n"]
    v = torch.zeros(n, n, device="cuda")
    m = torch.full((n, n), BULK, dtype=torch.int32, device="cuda")
    ux, uy = (t.double() for t in _turbulent(n, seed))
    f = torch.stack(_equilibrium(torch.ones_like(ux), ux, uy))
    w = torch.tensor(W, dtype=torch.float64, device="cuda")[:, None, None]
    layers, at = [], 0
    prm = torch.from_numpy(_network(seed)).double().cuda()
    for cin, cout in ((9, 32), (32, 32), (32, 9)):
        k = prm[at:at + 9 * cin * cout].view(3, 3, cin, cout).permute(3, 2, 0, 1).contiguous()
        at += 9 * cin * cout
        layers.append((k, prm[at:at + cout]))
        at += cout
    for _ in range(case["steps"] // case["every"]):
        f, macro = _exact_physics(f, m, v, 1.0 / _tau32(0.500125), case["every"], "kbc")
        rho = f.sum(0)
        ux = (f[1] + f[5] + f[8] - f[3] - f[6] - f[7]) / rho
        uy = (f[4] + f[7] + f[8] - f[2] - f[5] - f[6]) / rho
        y = (20.0 * (torch.stack(_equilibrium(rho, ux, uy)) - w))[None]
        for i, (k, b) in enumerate(layers):
            y = F.conv2d(F.pad(y, (1, 1, 1, 1), mode="circular"), k, b)
            y = y.relu() if i < 2 else y
        y = y[0]
        s = y.sum(0)
        sx = sum(EX[j] * y[j] for j in range(9))
        sy = sum(EY[j] * y[j] for j in range(9))
        y = [y[j] - W[j] * (s + 3.0 * (EX[j] * sx + EY[j] * sy)) for j in range(9)]
        y = [torch.roll(y[j], (EY[j], EX[j]), (0, 1)) * (-0.5 / 1e4) for j in range(9)]
        jx, jy = (sum(e[j] * y[j] for j in range(9)) for e in (EX, EY))
        f = torch.stack([f[j] + 3.0 * W[j] * (EX[j] * jx + EY[j] * jy) for j in range(9)])
    return macro + ((f - w).reshape(-1),)


def _exact_batch(case, seed):
    """Every domain of the batch from rest: (rho, ux, uy) planes one after the other."""
    out = []
    for d in _domains(case, seed):
        nx, ny = d["nx"], d["ny"]
        m = torch.full((ny, nx), BULK, dtype=torch.int32, device="cuda")
        v = torch.zeros(ny, nx, dtype=torch.float32, device="cuda")
        if d["scene"] == "cavity":
            m[0], m[-1], m[:, 0], m[:, -1] = (BOUNDARY,) * 4
            v[0, 1:-1] = d["speed"]
        else:
            m[:, 0], m[:, -1] = INLET, OUTLET
            v[:, 0] = _parabola(ny, d["speed"]).to(torch.float32)
            m[0], m[-1] = BOUNDARY, BOUNDARY
            v[0], v[-1] = 0.0, 0.0
        one = torch.ones(ny, nx, dtype=torch.float64, device="cuda")
        f = torch.stack(_equilibrium(one, 0 * one, 0 * one))
        _, macro = _exact_physics(f, m, v, 1.0 / _tau32(d["tau"]), case["steps"], "bgk")
        out.extend(t.reshape(-1) for t in macro)
    return torch.cat(out)
