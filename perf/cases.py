"""What a user has this package do, as cases that can be timed and compared.

Every case is one pass through the public entry points (World, Ferromagnet,
TimeSolver, FieldQuantity, StrayField, the batched solves, and their engine
handle for device pointers): evaluating a quantity of a magnet, integrating the
equation of motion from a given state for a given time, advancing many solves
together, and serving one whole solve from its admission to its result.

  listed()            the named cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) the world, magnets and inputs of a case, on the GPU
  run(state)          one pass; its outputs
  work(case)          bytes and operations that a pass cannot do without
  exact(case, seed)   the outputs of the first pass in 64 bits, plain torch

A pass always starts from the state that `prepare` made (set again through the
engine, device to device) and from the time step it found, so that every pass
does the same work.
"""
import math

import numpy as np
import torch

import mumaxplus_b200 as mpx
from mumaxplus_b200 import _abi, batch

GAMMA = 1.7595e11
MU0 = 1.25663706212e-6

# The materials of the workloads: the field-driven film, the skyrmion
# multilayer (interfacial DMI, perpendicular anisotropy, periodic in x and y) and
# the same multilayer material with open edges.
MATERIALS = {
    "film": dict(cell=(3e-9, 3e-9, 3e-9), msat=8.6e5, aex=1.3e-11, alpha=0.02, bias=(-0.030, 0.005, 0.0), dmi=0.0,
                 ku1=0.0, pbc=(0, 0, 0)),
    "multilayer": dict(cell=(2e-9, 2e-9, 1e-9), msat=5.8e5, aex=1.5e-11, alpha=0.1, bias=(0.0, 0.0, 0.2), dmi=3e-3,
                       ku1=8e5, pbc=(2, 2, 0)),
    "patch": dict(cell=(2e-9, 2e-9, 1e-9), msat=5.8e5, aex=1.5e-11, alpha=0.1, bias=(0.0, 0.0, 0.2), dmi=3e-3,
                  ku1=8e5, pbc=(0, 0, 0)),
}

QUANTITIES = {
    "torque": _abi.Q_TORQUE,
    "demag_field": _abi.Q_DEMAG_FIELD,
    "effective_field": _abi.Q_EFFECTIVE_FIELD,
    "total_energy_density": _abi.Q_TOTAL_ENERGY_DENSITY,
}


def listed():
    return [
        # The smallest call: the torque of a strip, as a script asks for it
        # between steps.  Launches and latency.
        dict(name="strip_torque", kind="eval", quantity="torque", material="film", nx=128, ny=32, nz=1),
        # <m>(t) of a film at 20 time points: the hysteresis / switching study,
        # one small solve alone on the device.
        dict(name="film_solve", kind="solve", material="film", nx=256, ny=64, nz=1, method="DormandPrince",
             duration=5e-12, points=20),
        # A skyrmion disc: geometry mask and a damping that grows towards the
        # edge (per-cell parameter), the default Runge-Kutta method, a size
        # that is no power of two.
        dict(name="disc_run", kind="run", material="patch", nx=200, ny=200, nz=1, method="Fehlberg", disc=True,
             duration=4e-13),
        # The large periodic multilayer, integrated: the production run.
        dict(name="multilayer_run", kind="run", material="multilayer", nx=512, ny=512, nz=8, method="DormandPrince",
             disc=False, duration=4e-13),
        # A medium sample whose sides are what its device's are (open edges,
        # three layers): ragged lengths along every axis.
        dict(name="ragged_run", kind="run", material="patch", nx=300, ny=180, nz=3, method="DormandPrince",
             disc=False, duration=4e-13),
        # A thick block: many layers.
        dict(name="block_run", kind="run", material="film", nx=80, ny=80, nz=40, method="DormandPrince", disc=False,
             duration=1e-12),
        # The demagnetising field of a large sample of random unit vectors.
        dict(name="demag_large", kind="eval", quantity="demag_field", material="film", nx=1024, ny=1024, nz=4),
        # An energy-density map of an odd-sized sample.
        dict(name="energy_odd", kind="eval", quantity="total_energy_density", material="patch", nx=437, ny=291, nz=2),
        # Two films in one world, ten layers apart, acting on each other.
        dict(name="pair_run", kind="pair", material="film", nx=256, ny=256, nz=1, gap=10, method="DormandPrince",
             duration=2e-12),
        # The stray field of a magnet on a grid above it (an MFM image).
        dict(name="stray_image", kind="stray", material="film", nx=192, ny=160, nz=2, dx=240, dy=200, gap=12),
        # The relaxation batch: independent solves of many sizes, advanced together.
        dict(name="batch_run", kind="batch", count=24, seed=4, lo=32, hi=256, duration=1e-12),
        # One served solve: admitted (its kernel built), integrated for a short
        # time, its result fetched, its memory given back.
        dict(name="served_solve", kind="serve", material="film", nx=170, ny=170, nz=2, method="DormandPrince",
             duration=1e-12),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eval", "solve", "run", "run", "thick", "pair", "stray", "batch", "serve"])
    if kind == "eval":
        nz = rng.choice([1, 1, 2, 3, 4])
        nx = _log_uniform(rng, 64, 1024)
        ny = max(16, min(1024, int(nx * rng.uniform(0.3, 1.6))))
        return dict(kind="eval", quantity=rng.choice(sorted(QUANTITIES)), material=rng.choice(["film", "patch"]),
                    nx=nx, ny=ny, nz=nz)
    if kind == "solve":
        return dict(kind="solve", material="film", nx=_log_uniform(rng, 64, 400), ny=_log_uniform(rng, 32, 128), nz=1,
                    method=rng.choice(["DormandPrince", "Fehlberg"]), duration=4e-12, points=rng.randint(5, 20))
    if kind == "run":
        nz = rng.choice([1, 1, 2, 3, 5, 8])
        nx = _log_uniform(rng, 64, 512)
        ny = max(32, min(512, int(nx * rng.uniform(0.4, 1.4))))
        methods = ["DormandPrince", "DormandPrince", "Fehlberg", "BogackiShampine"]
        return dict(kind="run", material=rng.choice(["film", "multilayer", "patch"]), nx=nx, ny=ny, nz=nz,
                    method=rng.choice(methods if nx * ny * nz <= 200_000 else methods[:3]),
                    disc=rng.random() < 0.3, duration=3e-13)
    if kind == "thick":
        return dict(kind="run", material="film", nx=_log_uniform(rng, 32, 128), ny=_log_uniform(rng, 32, 128),
                    nz=rng.randint(9, 48), method="DormandPrince", disc=False, duration=5e-13)
    if kind == "pair":
        return dict(kind="pair", material="film", nx=_log_uniform(rng, 96, 320), ny=_log_uniform(rng, 96, 320),
                    nz=rng.choice([1, 1, 2]), gap=rng.randint(1, 20), method="DormandPrince", duration=1e-12)
    if kind == "stray":
        return dict(kind="stray", material="film", nx=_log_uniform(rng, 48, 400), ny=_log_uniform(rng, 48, 400),
                    nz=rng.choice([1, 2, 4]), dx=_log_uniform(rng, 48, 400), dy=_log_uniform(rng, 48, 400),
                    gap=rng.randint(1, 40))
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(8, 32), seed=rng.randrange(1 << 20), lo=32, hi=rng.randint(128, 256),
                    duration=6e-13)
    return dict(kind="serve", material="film", nx=_log_uniform(rng, 64, 320), ny=_log_uniform(rng, 64, 320),
                nz=rng.choice([1, 2, 4]), method="DormandPrince", duration=5e-13)


# ------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _smooth_unit(shape, seed, passes=3):
    """Random unit vectors smoothed over the face neighbours, float32 (3, nz, ny, nx)."""
    m = torch.randn((3, *shape), generator=_generator(seed), device="cuda")
    for _ in range(passes):
        acc, cnt = m.clone(), torch.ones(shape, device="cuda")
        for ax in range(3):
            n = shape[ax]
            if n < 2:
                continue
            lo, hi = m.narrow(ax + 1, 0, n - 1), m.narrow(ax + 1, 1, n - 1)
            acc.narrow(ax + 1, 0, n - 1).add_(hi)
            acc.narrow(ax + 1, 1, n - 1).add_(lo)
            cnt.narrow(ax, 0, n - 1).add_(1)
            cnt.narrow(ax, 1, n - 1).add_(1)
        m = acc / cnt
    return (m / m.norm(dim=0)).contiguous()


def _bubbles(shape, seed):
    """Up domain with reversed discs, tilted a little by a smooth random field."""
    nz, ny, nx = shape
    rng = np.random.default_rng(seed)
    m = torch.zeros((3, nz, ny, nx), device="cuda")
    m[2] = 1.0
    Y, X = torch.meshgrid(torch.arange(ny, device="cuda"), torch.arange(nx, device="cuda"), indexing="ij")
    for _ in range(max(2, nx * ny // 6500)):
        cx, cy, r = rng.uniform(0, nx), rng.uniform(0, ny), rng.integers(5, 16)
        dx, dy = (X - cx).abs(), (Y - cy).abs()
        dx, dy = torch.minimum(dx, nx - dx), torch.minimum(dy, ny - dy)
        m[2][:, dx * dx + dy * dy < r * r] = -1.0
    m = m + 0.3 * _smooth_unit(shape, seed + 77)
    return (m / m.norm(dim=0)).contiguous()


def _initial(case, seed, which=0):
    shape = (case["nz"], case["ny"], case["nx"])
    if case.get("quantity") == "demag_field":
        return _smooth_unit(shape, seed, passes=0)
    if MATERIALS[case["material"]]["ku1"]:
        return _bubbles(shape, seed + 1000 * which)
    return _smooth_unit(shape, seed + 1000 * which)


def _disc(case):
    """Elliptic mask and a damping that grows towards its edge."""
    ny, nx = case["ny"], case["nx"]
    y, x = np.mgrid[0:ny, 0:nx]
    r = np.sqrt(((x - (nx - 1) / 2) / (nx / 2)) ** 2 + ((y - (ny - 1) / 2) / (ny / 2)) ** 2)
    shape = (case["nz"], ny, nx)
    alpha = 0.1 + 0.4 * np.clip((r - 0.8) / 0.2, 0, 1)
    return np.broadcast_to(r <= 1.0, shape).copy(), np.broadcast_to(alpha, shape).astype(np.float32).copy()


def _world(case):
    p = MATERIALS[case["material"]]
    mg = tuple(n if r else 0 for n, r in zip((case["nx"], case["ny"], case["nz"]), p["pbc"]))
    return mpx.World(p["cell"], pbc_repetitions=p["pbc"], mastergrid=mpx.Grid(mg)), p


def _magnet(world, p, case, origin=(0, 0, 0)):
    geometry = alpha = None
    if case.get("disc"):
        geometry, alpha = _disc(case)
    magnet = mpx.Ferromagnet(world, mpx.Grid((case["nx"], case["ny"], case["nz"]), origin), geometry=geometry)
    magnet.msat, magnet.aex = p["msat"], p["aex"]
    magnet.alpha = p["alpha"] if alpha is None else alpha[None]
    if p["ku1"]:
        magnet.ku1, magnet.anisU = p["ku1"], (0.0, 0.0, 1.0)
    if p["dmi"]:
        magnet.dmi_tensor.set_interfacial_dmi(p["dmi"])
    return magnet


def _instances(case, seed):
    """Relaxation solves: square sides log-uniform, one or two layers, random
    cubic cell, material, damping and applied field; a random state each."""
    rng = np.random.default_rng(case["seed"])
    ws, ms = [], []
    for k in range(case["count"]):
        side = int(np.floor(case["lo"] * (case["hi"] / case["lo"]) ** rng.uniform()))
        nz, c = int(rng.integers(1, 3)), float(rng.uniform(2e-9, 4e-9))
        b = rng.standard_normal(3)
        b *= rng.uniform(0, 0.1) / np.linalg.norm(b)
        ws.append(dict(name=f"solve_{k}", size=(side, side, nz), cellsize=(c, c, c), msat=float(rng.uniform(4e5, 1e6)),
                       aex=float(rng.uniform(5e-12, 2e-11)), alpha=float(rng.uniform(0.01, 0.5)),
                       world_bias=tuple(float(v) for v in b)))
        ms.append(_smooth_unit((nz, side, side), 10000 * int(seed) + k))
    return ws, ms


class State:
    """What a program holds between calls."""


def prepare(case, seed):
    s = State()
    s.case = case
    kind = case["kind"]
    if kind == "batch":
        ws, s.m0 = _instances(case, seed)
        s.batch = batch.Batch()
        s.engine = s.batch.engine
        s.solves = [s.batch.add(w, m0=m.cpu().numpy()) for w, m in zip(ws, s.m0)]
        s.dt = [s.engine.get_timestep(v.group) for v in s.solves]
        s.out = [torch.empty_like(m) for m in s.m0]
        return s
    if kind == "serve":
        p = MATERIALS[case["material"]]
        s.batch = batch.Batch(method=case["method"])
        s.w = dict(name="request", size=(case["nx"], case["ny"], case["nz"]), cellsize=p["cell"], msat=p["msat"],
                   aex=p["aex"], alpha=p["alpha"], world_bias=p["bias"])
        s.m0 = _initial(case, seed).cpu().numpy()
        return s
    world, p = _world(case)
    s.world, s.engine, s.solver = world, world._engine, world.timesolver
    s.magnets = [_magnet(world, p, case)]
    s.m0 = [_initial(case, seed)]
    if kind == "pair":
        s.magnets.append(_magnet(world, p, case, origin=(0, 0, case["nz"] + case["gap"])))
        s.m0.append(_initial(case, seed, 1))
    world.bias_magnetic_field = p["bias"]
    torch.cuda.synchronize()
    for magnet, m in zip(s.magnets, s.m0):
        s.engine.set_m_device(magnet._id, m.data_ptr())
    if kind == "eval":
        ncomp = 1 if case["quantity"].endswith("density") else 3
        s.out = torch.empty((ncomp, *s.m0[0].shape[1:]), device="cuda")
        s.q = QUANTITIES[case["quantity"]]
    elif kind == "stray":
        s.field = mpx.StrayField(s.magnets[0], mpx.Grid((case["dx"], case["dy"], 1), (-8, -8, case["nz"] + case["gap"])))
    else:
        s.solver.set_method(case["method"])
        s.dt = s.solver.sensible_timestep
        s.out = [torch.empty_like(m) for m in s.m0]
        if kind == "solve":
            n = case["points"]
            s.times = [case["duration"] * (k + 1) / n for k in range(n)]
            s.table = {"m": s.magnets[0].magnetization.average}
    return s


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "eval":
        s.engine.eval_device(s.magnets[0]._id, s.q, s.out.data_ptr())
        return s.out
    if kind == "stray":
        return s.field.eval()
    if kind == "batch":
        for v, m, dt in zip(s.solves, s.m0, s.dt):
            s.engine.set_m_device(v.magnet, m.data_ptr())
            s.engine.set_timestep(v.group, dt)
            s.batch.start(v, case["duration"])
        running = 1
        while running:
            s.batch.advance(4)
            _, running = s.batch.poll()
        for v, o in zip(s.solves, s.out):
            s.engine.get_m_device(v.magnet, o.data_ptr())
        return s.out
    if kind == "serve":
        v = s.batch.add(s.w, m0=s.m0)
        s.batch.start(v, case["duration"])
        running = 1
        while running:
            s.batch.advance(4)
            _, running = s.batch.poll()
        return s.batch.finish(v).m
    for magnet, m in zip(s.magnets, s.m0):
        s.engine.set_m_device(magnet._id, m.data_ptr())
    s.solver.timestep = s.dt
    if kind == "solve":
        s.solver.time = 0.0
        rows = s.solver.solve(s.times, s.table)
        s.engine.get_m_device(s.magnets[0]._id, s.out[0].data_ptr())
        return {"table": np.asarray(rows["m"], dtype=np.float32), "m": s.out[0]}
    s.solver.run(case["duration"])
    for magnet, o in zip(s.magnets, s.out):
        s.engine.get_m_device(magnet._id, o.data_ptr())
    return s.out


# -------------------------------------------------------------------- work
# Time steps of about this length are what the step control settles at.
STEP = {"film": 1.5e-13, "multilayer": 4e-14, "patch": 4e-14}
EVALS = {"Heun": 2, "BogackiShampine": 4, "CashKarp": 6, "Fehlberg": 6, "DormandPrince": 6}


def _evaluation(nx, ny, nz, out_words=3):
    """One evaluation of the field of an nx x ny x nz magnet: m read, the result
    written, the distinct values of its kernel read; the linear convolution by
    FFTs of twice the size and the local terms."""
    cells = nx * ny * nz
    padded = cells
    for n in (nx, ny, nz):
        padded *= 2 if n > 1 else 1
    kernel = (nx + 1) * (ny + 1) * ((nz + 1) * 6 if nz > 1 else 4)
    return 4.0 * ((3 + out_words) * cells + kernel), 2 * 3 * 2.5 * padded * math.log2(padded) + 150.0 * cells


def work(case):
    kind = case["kind"]
    if kind == "batch":
        rng = np.random.default_rng(case["seed"])
        total = [0.0, 0.0]
        for _ in range(case["count"]):
            side = int(np.floor(case["lo"] * (case["hi"] / case["lo"]) ** rng.uniform()))
            nz = int(rng.integers(1, 3))
            rng.uniform(2e-9, 4e-9), rng.standard_normal(3), [rng.uniform() for _ in range(4)]
            n = EVALS["DormandPrince"] * max(1.0, case["duration"] / STEP["film"])
            b, f = _evaluation(side, side, nz)
            total[0] += n * b
            total[1] += n * f
        return {"bytes": total[0], "flops": total[1]}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if kind == "eval":
        b, f = _evaluation(nx, ny, nz, 1 if case["quantity"].endswith("density") else 3)
        return {"bytes": b, "flops": f}
    if kind == "stray":
        kx, ky, kz = nx + case["dx"] - 1, ny + case["dy"] - 1, nz
        pts = kx * ky * kz
        return {"bytes": 4.0 * (3 * nx * ny * nz + 3 * case["dx"] * case["dy"] + 6 * pts),
                "flops": 2 * 3 * 2.5 * pts * math.log2(pts)}
    n = EVALS[case["method"]] * max(1.0, case["duration"] / STEP[case["material"]])
    b, f = _evaluation(nx, ny, nz)
    k = 4 if kind == "pair" else 1  # two magnets and the field of each on the other
    return {"bytes": n * b * k, "flops": n * f * k}


# ------------------------------------------------------------------- exact
def _newell_diag(x, y, z):
    """Newell's indefinite integral of N_xx (Newell, Williams and Dunlop 1993, eq. 27)."""
    R = torch.sqrt(x * x + y * y + z * z)
    xz, xy = torch.sqrt(x * x + z * z), torch.sqrt(x * x + y * y)
    zero = torch.zeros_like(R)
    f = (y / 2) * (z * z - x * x) * torch.where(xz > 0, torch.asinh(y / xz), zero)
    f = f + (z / 2) * (y * y - x * x) * torch.where(xy > 0, torch.asinh(z / xy), zero)
    f = f - torch.where(x != 0, x * y * z * torch.atan(y * z / (x * R)), zero)
    return f + (2 * x * x - y * y - z * z) * R / 6


def _newell_off(x, y, z):
    """Newell's indefinite integral of N_xy (eq. 32)."""
    R = torch.sqrt(x * x + y * y + z * z)
    xy, yz, xz = torch.sqrt(x * x + y * y), torch.sqrt(y * y + z * z), torch.sqrt(x * x + z * z)
    zero = torch.zeros_like(R)
    g = x * y * z * torch.where(xy > 0, torch.asinh(z / xy), zero)
    g = g + (y / 6) * (3 * z * z - y * y) * torch.where(yz > 0, torch.asinh(x / yz), zero)
    g = g + (x / 6) * (3 * z * z - x * x) * torch.where(xz > 0, torch.asinh(y / xz), zero)
    g = g - torch.where(z != 0, (z * z * z / 6) * torch.atan(x * y / (z * R)), zero)
    g = g - torch.where(y != 0, (z * y * y / 2) * torch.atan(x * z / (y * R)), zero)
    g = g - torch.where(x != 0, (z * x * x / 2) * torch.atan(y * z / (x * R)), zero)
    return g - x * y * R / 3


class _Convolution:
    """Field of the cells of a source grid on a destination grid `shift` cells away."""

    def __init__(self, nsrc, ndst, shift, cell, period=(0, 0, 0), images=(0, 0, 0)):
        self.nsrc, self.ndst = nsrc, ndst
        self.k = [a + b - 1 for a, b in zip(nsrc, ndst)]
        lo = [s - (a - 1) for s, a in zip(shift, nsrc)]
        axes = []  # lattice around every displacement of every image, x last
        for a in range(3):
            reach = period[a] * images[a]
            axes.append(torch.arange(lo[a] - reach - 1, lo[a] + self.k[a] + reach + 1, device="cuda",
                                     dtype=torch.float64) * cell[a])
        z, y, x = torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
        self.spectrum = []
        for fn, (u, v, w) in ((_newell_diag, (x, y, z)), (_newell_diag, (y, z, x)), (_newell_diag, (z, x, y)),
                              (_newell_off, (x, y, z)), (_newell_off, (x, z, y)), (_newell_off, (y, z, x))):
            f = torch.nan_to_num(fn(u, v, w))
            for ax in range(3):
                n = f.shape[ax]
                f = f.narrow(ax, 2, n - 2) - 2 * f.narrow(ax, 1, n - 2) + f.narrow(ax, 0, n - 2)
            f = -f / (4 * math.pi * cell[0] * cell[1] * cell[2])
            table = torch.zeros(self.k[::-1], device="cuda", dtype=torch.float64)
            for i in range(2 * images[0] + 1):
                for j in range(2 * images[1] + 1):
                    for l in range(2 * images[2] + 1):
                        o = (l * period[2], j * period[1], i * period[0])
                        table += f[o[0]:o[0] + self.k[2], o[1]:o[1] + self.k[1], o[2]:o[2] + self.k[0]]
            self.spectrum.append(torch.fft.rfftn(table))

    def __call__(self, magnetization):
        xx, yy, zz, xy, xz, yz = self.spectrum
        m = [torch.fft.rfftn(c, s=self.k[::-1]) for c in magnetization]
        rows = ((xx, xy, xz), (xy, yy, yz), (xz, yz, zz))
        cut = tuple(slice(self.nsrc[a] - 1, self.nsrc[a] - 1 + self.ndst[a]) for a in (2, 1, 0))
        return torch.stack([-MU0 * torch.fft.irfftn(sum(k * c for k, c in zip(row, m)), s=self.k[::-1])[cut]
                            for row in rows])


class _Magnet:
    """Right-hand side of one magnet with uniform parameters (but for the damping) in 64 bits."""

    def __init__(self, n, cell, msat, aex, alpha, bias, dmi=0.0, ku1=0.0, pbc=(0, 0, 0), geometry=None):
        self.n, self.cell, self.msat, self.aex, self.alpha, self.dmi, self.ku1, self.pbc = (n, cell, msat, aex, alpha,
                                                                                           dmi, ku1, pbc)
        shape = (n[2], n[1], n[0])
        self.inside = (torch.ones(shape, dtype=torch.bool, device="cuda") if geometry is None
                       else torch.as_tensor(geometry, device="cuda"))
        self.bias = torch.tensor(bias, device="cuda", dtype=torch.float64).view(3, 1, 1, 1)
        self.demag = _Convolution(n, n, (0, 0, 0), cell, [v if r else 0 for v, r in zip(n, pbc)], pbc)
        self.stray = []  # (convolution, index of the source magnet)

    def _local(self, m):
        exch, dm = torch.zeros_like(m), torch.zeros_like(m)
        for ax in range(3):
            dim = 3 - ax
            for d in (-1, 1):
                mn = torch.roll(m, -d, dim)
                there = torch.roll(self.inside, -d, dim - 1).clone()
                if not self.pbc[ax]:
                    there.select(dim - 1, 0 if d < 0 else self.n[ax] - 1).fill_(False)
                # the Neumann ghost of a missing neighbour, tilted by the DMI
                ghost = m
                if self.dmi and ax < 2:
                    g = torch.zeros_like(m)
                    g[ax], g[2] = -self.dmi * m[2], self.dmi * m[ax]
                    ghost = m + d * self.cell[ax] / (2 * self.aex) * g
                mn = torch.where(there, mn, ghost)
                exch += 2 * self.aex / self.cell[ax] ** 2 * (mn - m)
                if self.dmi and ax < 2:
                    dm[ax] += self.dmi * mn[2] * d / self.cell[ax]
                    dm[2] -= self.dmi * mn[ax] * d / self.cell[ax]
        return exch / self.msat, dm / self.msat

    def parts(self, m, states=None):
        exch, dm = self._local(m)
        anis = torch.zeros_like(m)
        anis[2] = 2 * self.ku1 / self.msat * m[2]
        ext = self.bias.expand_as(m)
        for conv, j in self.stray:
            ext = ext + conv(states[j][1] * states[j][0])
        demag = self.demag(self.msat * torch.where(self.inside, m, torch.zeros_like(m)))
        return exch, anis, ext, dm, demag

    def torque(self, m, states=None):
        h = sum(self.parts(m, states))
        mxh = torch.linalg.cross(m, h, dim=0)
        t = -GAMMA / (1 + self.alpha ** 2) * (mxh + self.alpha * torch.linalg.cross(m, mxh, dim=0))
        return torch.where(self.inside, t, torch.zeros_like(t))


# (a, b, b of the embedded method, orders)
TABLEAUS = {
    "BogackiShampine": ([[], [1 / 2], [0, 3 / 4], [2 / 9, 1 / 3, 4 / 9]], [2 / 9, 1 / 3, 4 / 9, 0],
                        [7 / 24, 1 / 4, 1 / 3, 1 / 8], (3, 2)),
    "Fehlberg": ([[], [1 / 4], [3 / 32, 9 / 32], [1932 / 2197, -7200 / 2197, 7296 / 2197],
                  [439 / 216, -8, 3680 / 513, -845 / 4104], [-8 / 27, 2, -3544 / 2565, 1859 / 4104, -11 / 40]],
                 [16 / 135, 0, 6656 / 12825, 28561 / 56430, -9 / 50, 2 / 55],
                 [25 / 216, 0, 1408 / 2565, 2197 / 4104, -1 / 5, 0], (5, 4)),
    "DormandPrince": ([[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
                       [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
                       [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
                       [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]],
                      [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84, 0],
                      [5179 / 57600, 0, 7571 / 16695, 393 / 640, -92097 / 339200, 187 / 2100, 1 / 40], (5, 4)),
}


class _Solver:
    """The adaptive Runge-Kutta integration of the magnets of one world."""

    def __init__(self, magnets, states, method, max_error=1e-5):
        self.magnets, self.max_error = magnets, max_error
        self.a, self.b, self.b2, self.order = TABLEAUS[method]
        self.m = [s.double() / s.double().norm(dim=0) for s in states]
        self.m = [torch.where(g.inside, v, s.double()) for g, v, s in zip(magnets, self.m, states)]
        self.t = 0.0
        self.dt = 0.01 / max(float(k.norm(dim=0).max()) for k in self._slope(self.m))

    def _slope(self, m):
        pairs = [(torch.where(g.inside, v, torch.zeros_like(v)), g.msat) for g, v in zip(self.magnets, m)]
        return [g.torque(v, pairs) for g, v in zip(self.magnets, m)]

    def _moved(self, k, row):
        out = []
        for j, (g, m) in enumerate(zip(self.magnets, self.m)):
            v = m + self.dt * sum(c * ks[j] for c, ks in zip(row, k) if c)
            out.append(torch.where(g.inside, v / v.norm(dim=0), m))
        return out

    def step(self):
        """Attempts until one is accepted."""
        while True:
            k = []
            for row in self.a:
                k.append(self._slope(self._moved(k, row) if row else self.m))
            err = 0.0
            for j in range(len(self.m)):
                e = sum((c - d) * ks[j] for c, d, ks in zip(self.b, self.b2, k))
                err = max(err, self.dt * float(e.norm(dim=0).max()))
            ok, dt = err < self.max_error, self.dt
            if ok:
                self.m = self._moved(k, self.b)
                self.t += dt
            c = (self.max_error / err) ** (1 / ((self.order[1] if ok else self.order[0]) + 1)) if err else math.inf
            self.dt = dt * min(2.0, max(0.5, 0.8 * c))
            if ok:
                return

    def run(self, until):
        while self.t < until - self.dt:
            self.step()
        self.dt = until - self.t
        self.step()


def _exact_magnet(case):
    p = MATERIALS[case["material"]]
    geometry, alpha = None, p["alpha"]
    if case.get("disc"):
        geometry, alpha = _disc(case)
        alpha = torch.as_tensor(alpha, device="cuda").double()
    return _Magnet((case["nx"], case["ny"], case["nz"]), p["cell"], p["msat"], p["aex"], alpha, p["bias"], p["dmi"],
                   p["ku1"], p["pbc"], geometry)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ws, ms = _instances(case, seed)
        out = []
        for w, m in zip(ws, ms):
            g = _Magnet(w["size"], w["cellsize"], w["msat"], w["aex"], w["alpha"], w["world_bias"])
            solver = _Solver([g], [m], "DormandPrince")
            solver.run(case["duration"])
            out.append(solver.m[0])
        return out
    p = MATERIALS[case["material"]]
    n = (case["nx"], case["ny"], case["nz"])
    if kind == "stray":
        m = _initial(case, seed).double()
        conv = _Convolution(n, (case["dx"], case["dy"], 1), (-8, -8, case["nz"] + case["gap"]), p["cell"])
        return conv(p["msat"] * m / m.norm(dim=0))
    magnets, states = [_exact_magnet(case)], [_initial(case, seed)]
    if kind == "eval":
        g, m = magnets[0], states[0].double() / states[0].double().norm(dim=0)
        if case["quantity"] == "torque":
            return g.torque(m)
        exch, anis, ext, dm, demag = g.parts(m)
        if case["quantity"] == "demag_field":
            return demag
        if case["quantity"] == "effective_field":
            return exch + anis + ext + dm + demag
        half = -0.5 * p["msat"] * (m * (exch + dm + demag)).sum(0) - p["msat"] * (m * ext).sum(0)
        return (half - p["ku1"] * m[2] ** 2)[None]
    if kind == "pair":
        magnets.append(_exact_magnet(case))
        states.append(_initial(case, seed, 1))
        up = (0, 0, case["nz"] + case["gap"])
        magnets[1].stray.append((_Convolution(n, n, up, p["cell"]), 0))
        magnets[0].stray.append((_Convolution(n, n, tuple(-v for v in up), p["cell"]), 1))
    solver = _Solver(magnets, states, case["method"])
    if kind == "solve":
        rows = []
        for k in range(case["points"]):
            solver.run(case["duration"] * (k + 1) / case["points"])
            rows.append(solver.m[0].reshape(3, -1).mean(1))
        return {"table": torch.stack(rows), "m": solver.m[0]}
    solver.run(case["duration"])
    return solver.m[0] if kind == "serve" else solver.m
