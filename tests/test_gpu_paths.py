"""Edges of the launch paths that magnets take by size and options, against the
FP64 oracle: the warp-column forms of the split y/z path, the one-column-per-warp
transforms of small solves, the lean epilogue with a geometry mask and per-cell
damping, the octant construction of the demag kernel, and the stray fields of
several magnets sharing their launches.

Tolerances as tests/test_gpu_parity.py: fields <= 1e-5 of max|B| (FP32 transforms of
a few thousand points: about 1e-6), 5e-5 for the demag field alone at 150,000 cells
and more (the bound of tests/test_gpu_configs.py there; the oracle convolves the
GPU's kernel values), one explicit step of m <= 2e-6 absolute (rounding of m, dt k and
their sum, 3 x 6e-8 of 1, with a factor of ten)."""
import numpy as np
import pytest

import oracle as O
from spec import MagnetSpec, max_rel, random_m

pytestmark = pytest.mark.gpu
abi = O.abi
FIELD_TOL = 1e-5


def _demag(mpx, spec, seed=3):
    m0 = random_m(spec.shape, seed=seed, smooth=2)
    ow, q = spec.oracle_world(m0)
    world, magnet = spec.product(mpx, m0)
    got = magnet._engine.eval(magnet._id, abi.Q_DEMAG_FIELD, (3, *spec.shape))
    return max_rel(got, ow.eval(q, abi.Q_DEMAG_FIELD))


# nx, ny, nz: y lengths 64 .. 1024 and z lengths 32 .. 256 at the ends of their ranges (2 n - 1 just below and
# above a power of two), column counts that leave the last warp and the last block partly filled, and the
# lengths outside (y 32, z 512), which keep the block-wide passes
@pytest.mark.parametrize("size", [(5, 17, 9), (9, 32, 16), (6, 33, 17), (3, 64, 32), (7, 65, 33), (2, 128, 64),
                                  (5, 129, 10), (3, 40, 65), (2, 257, 12), (3, 18, 128), (4, 16, 12), (2, 20, 130)])
def test_split_path_lengths(mpx, size):
    assert _demag(mpx, MagnetSpec(size=size, cellsize=(2e-9, 1.5e-9, 1e-9), msat=8e5)) < FIELD_TOL


def test_split_path_periodic_z(mpx):
    spec = MagnetSpec(size=(10, 40, 20), cellsize=(2e-9, 2e-9, 2e-9), msat=8e5, mastergrid_size=(10, 0, 20),
                      pbc=(1, 0, 1))
    assert _demag(mpx, spec) < FIELD_TOL


# x rows and y columns of 512 points with 1 .. 4 rows, odd row counts, and y lengths 64 .. 512 with 3 and 6
# columns: as many columns as warps or fewer
@pytest.mark.parametrize("size", [(129, 1, 1), (256, 2, 1), (200, 3, 1), (130, 20, 2), (17, 32, 1), (9, 64, 2),
                                  (33, 100, 1), (5, 256, 1), (4, 250, 3)])
def test_small_solve_transforms(mpx, size):
    assert _demag(mpx, MagnetSpec(size=size, cellsize=(2e-9, 1.5e-9, 1e-9), msat=8e5)) < FIELD_TOL


def _disc(shape):
    nz, ny, nx = shape
    y, x = np.mgrid[0:ny, 0:nx]
    r = ((x - nx / 2 + 0.5) / (nx / 2)) ** 2 + ((y - ny / 2 + 0.5) / (ny / 2)) ** 2
    return np.broadcast_to(r <= 1, shape).copy()


@pytest.mark.parametrize("kind", ["geometry", "alpha", "frozen", "all", "openbc", "periodic", "odd"])
@pytest.mark.parametrize("method", ["Heun", "DormandPrince"])
def test_masked_stage_epilogue(mpx, kind, method):
    """One explicit step of a magnet with uniform field parameters and a mask, per-cell damping or frozen spins."""
    size = (45, 30, 2) if kind == "odd" else (44, 30, 2)
    shape = size[::-1]
    rng = np.random.default_rng(5)
    extra = {}
    if kind in ("geometry", "all", "openbc", "periodic", "odd"):
        extra["geometry"] = _disc(shape)
    if kind in ("alpha", "all", "odd"):
        extra["alpha"] = rng.uniform(0.05, 0.5, shape).astype(np.float32)[None]
    if kind in ("frozen", "all"):
        extra["frozen"] = (rng.uniform(size=shape) < 0.2).astype(np.float32)[None]
    if kind == "openbc":
        extra["enable_openbc"] = True
    if kind == "periodic":
        extra.update(mastergrid_size=(44, 30, 0), pbc=(1, 1, 0))
    s = MagnetSpec(size=size, cellsize=(2e-9, 2e-9, 1e-9), msat=5.8e5, aex=1.5e-11, ku1=6e5, anisU=(0, 0, 1),
                   dmi={"xxz": 2e-3, "yyz": 2e-3}, world_bias=(0.01, 0.0, 0.1), **{"alpha": 0.1, **extra})
    m0 = random_m(s.shape, seed=11, smooth=2)
    ow, q = s.oracle_world(m0)
    ow.set_method(method)
    world, magnet = s.product(mpx, m0)
    world.timesolver.set_method(method)
    world.timesolver.adaptive_timestep = False
    ow.set_solver(adaptive=0)
    dt = 0.5 * ow.sensible_timestep()
    ow.timestep = dt
    world.timesolver.timestep = dt
    ow.steps(2)
    world.timesolver.steps(2)
    assert np.max(np.abs(magnet.magnetization.eval() - ow.get_m(q))) < 2e-6


# lattices over both signs, one sign, periodic images, a single layer, and sides of one cell
@pytest.mark.parametrize("size,pbc", [((6, 5, 4), (0, 0, 0)), ((6, 5, 1), (2, 0, 0)), ((1, 7, 3), (0, 1, 1)),
                                      ((9, 1, 1), (0, 0, 0)), ((33, 17, 2), (1, 1, 0))])
def test_kernel_construction(mpx, size, pbc):
    mg = tuple(n if p else 0 for n, p in zip(size, pbc))
    assert _demag(mpx, MagnetSpec(size=size, cellsize=(1e-9, 2e-9, 1.5e-9), msat=8e5, mastergrid_size=mg,
                                  pbc=pbc)) < FIELD_TOL


# The demag kernel and the FP32 table of the real-space kernel are built apart, from lattices of different room:
# the images of the kernel's lattice one at a time along x, along x and y, along all axes, with the table's all
# together; and the table's one at a time.  The oracle convolves the table's values: with its own the distant images
# would compare the FP64 cancellation of two tensor codes instead.
@pytest.mark.parametrize("size,pbc", [((60, 60, 1), (9, 9, 0)), ((24, 60, 4), (0, 8, 9)), ((36, 36, 8), (0, 0, 60)),
                                      ((200, 2, 3), (4200, 0, 0))])
def test_kernel_construction_in_parts(mpx, size, pbc):
    nx, ny, nz = size
    mg = tuple(n if p else 0 for n, p in zip(size, pbc))
    spec = MagnetSpec(size=size, cellsize=(1e-9, 2e-9, 1.5e-9), msat=8e5, mastergrid_size=mg, pbc=pbc)
    m0 = random_m(spec.shape, seed=3, smooth=2)
    world, magnet = spec.product(mpx, m0)
    K = magnet._engine.demag_kernel(magnet._id)  # displacement 0 at index K - n
    ow, q = spec.oracle_world(m0)
    ow.set_kernel_octant(q, np.ascontiguousarray(K[:, K.shape[1] - nz:, K.shape[2] - ny:, K.shape[3] - nx:]))
    got = magnet._engine.eval(magnet._id, abi.Q_DEMAG_FIELD, (3, *spec.shape))
    assert max_rel(got, ow.eval(q, abi.Q_DEMAG_FIELD)) < FIELD_TOL


def test_three_magnets_share_launches(mpx):
    """Every destination has two sources; two of the three pairs of sizes share a launch shape, one takes the
    direct sum (below 2^22 interactions)."""
    cs = (2e-9, 3e-9, 2.5e-9)
    specs = [MagnetSpec(size=(60, 48, 1), cellsize=cs, msat=8e5, aex=1e-11, alpha=0.1),
             MagnetSpec(size=(60, 48, 1), origin=(0, 0, 5), cellsize=cs, msat=6e5, aex=1e-11, alpha=0.1),
             MagnetSpec(size=(20, 14, 2), origin=(80, 10, 0), cellsize=cs, msat=7e5, aex=1e-11, alpha=0.1)]
    ms = [random_m(s.shape, seed=70 + k, smooth=2) for k, s in enumerate(specs)]
    ow = O.OracleWorld()
    keep = []
    qs = [ow.add_magnet(s.desc(keep)) for s in specs]
    world = mpx.World(cs)
    mags = []
    for s, m, q in zip(specs, ms, qs):
        ow.set_m(q, m)
        mag = mpx.Ferromagnet(world, mpx.Grid(s.size, s.origin))
        mag.msat, mag.aex, mag.alpha = s.msat, s.aex, s.alpha
        mag.magnetization = m
        mags.append(mag)
    for q, mag, s in zip(qs, mags, specs):
        got = mag._engine.eval(mag._id, abi.Q_EXTERNAL_FIELD, (3, *s.shape))
        assert max_rel(got, ow.eval(q, abi.Q_EXTERNAL_FIELD)) < FIELD_TOL
    ow.set_method("DormandPrince")
    world.timesolver.set_method("DormandPrince")
    world.timesolver.adaptive_timestep = False
    ow.set_solver(adaptive=0)
    dt = 0.5 * ow.sensible_timestep()
    ow.timestep = dt
    world.timesolver.timestep = dt
    ow.steps(2)
    world.timesolver.steps(2)
    for q, mag in zip(qs, mags):
        assert np.max(np.abs(mag.magnetization.eval() - ow.get_m(q))) < 2e-6


# lengths 3 2^k (magnets of at least 150,000 cells): y lengths 96 .. 768 at z lengths 1, 4, 8, 16 and on the split
# path, x lengths 384 and 768, sides at the ends of their ranges (2 n - 1 just below the length and just above the
# power of two below it), odd row counts, one and several columns per warp
@pytest.mark.parametrize("size", [(1000, 160, 1), (500, 340, 1), (384, 392, 1), (1024, 192, 1), (610, 257, 1),
                                  (420, 180, 2), (1000, 96, 2), (192, 400, 2), (129, 601, 2), (150, 350, 3),
                                  (385, 129, 4), (1000, 40, 4), (400, 95, 4), (300, 130, 4), (193, 384, 3),
                                  (150, 140, 8), (130, 260, 5), (1000, 33, 5), (160, 48, 20), (100, 96, 16),
                                  (90, 180, 10), (60, 300, 9), (30, 65, 80), (257, 193, 4)])
def test_lengths_with_a_factor_three(mpx, size):
    nx, ny, nz = size
    assert nx * ny * nz >= 150000
    spec = MagnetSpec(size=size, cellsize=(2e-9, 1.5e-9, 1e-9), msat=8e5)
    m0 = random_m(spec.shape, seed=3, smooth=2)
    world, magnet = spec.product(mpx, m0)
    eng = magnet._engine
    K = eng.demag_kernel(magnet._id)  # displacement 0 at index K - n
    octant = np.ascontiguousarray(K[:, K.shape[1] - nz:, K.shape[2] - ny:, K.shape[3] - nx:].astype(np.float64))
    ow, q = spec.oracle_world(m0)
    ow.set_kernel_octant(q, octant)  # the same kernel values: the convolution alone is compared
    got = eng.eval(magnet._id, abi.Q_DEMAG_FIELD, (3, *spec.shape))
    assert max_rel(got, ow.eval(q, abi.Q_DEMAG_FIELD)) < 5e-5


@pytest.mark.parametrize("size", [(150, 350, 3), (301, 167, 3), (1000, 160, 1), (160, 48, 20)])
def test_stages_with_a_factor_three(mpx, size):
    """Stage combination, the three passes and the lean epilogue over two Dormand-Prince steps."""
    s = MagnetSpec(size=size, cellsize=(3e-9, 3e-9, 3e-9), msat=8e5, aex=1.3e-11, alpha=0.1,
                   world_bias=(0.0, 0.01, 0.0))
    m0 = random_m(s.shape, seed=8, smooth=3)
    ow, q = s.oracle_world(m0)
    ow.set_method("DormandPrince")
    ow.set_solver(adaptive=0)
    world, magnet = s.product(mpx, m0)
    world.timesolver.set_method("DormandPrince")
    world.timesolver.adaptive_timestep = False
    dt = 2 * ow.sensible_timestep()
    ow.timestep = dt
    world.timesolver.timestep = dt
    ow.steps(2)
    world.timesolver.steps(2)
    assert np.max(np.abs(magnet.magnetization.eval() - ow.get_m(q))) < 2e-6


def test_factor_three_solves_in_a_batch(mpx):
    """Solves with and without these lengths together end as each does alone."""
    from mumaxplus_b200 import batch, workloads as W

    ws = []
    for k, (side, nz) in enumerate([(40, 1), (190, 5), (100, 1), (280, 2), (60, 1), (390, 1)]):
        ws.append(dict(name=f"s{k}", size=(side, side, nz), cellsize=(3e-9, 3e-9, 3e-9), msat=8e5, aex=1.3e-11,
                       alpha=0.3, world_bias=(0.0, 0.01, 0.0),
                       m0=lambda s=side, z=nz, k=k: W.smoothed_random_m((z, s, s), 100 + k)))
    together, _, _ = batch.relax_batch(batch.Batch(), ws, duration=1e-12, torque_stop=0.0, autotune=False)
    alone, _, _ = batch.run_plain(batch.Batch(), ws, duration=1e-12, torque_stop=0.0)
    for a, b in zip(together, alone):
        assert a.steps == b.steps and np.array_equal(a.m, b.m)
