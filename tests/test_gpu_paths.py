"""Edges of the launch paths that magnets take by size and options, against the
FP64 oracle: the warp-column forms of the split y/z path, the one-column-per-warp
transforms of small solves, the lean epilogue with a geometry mask and per-cell
damping, the octant construction of the demag kernel, and the stray fields of
several magnets sharing their launches.

Tolerances as tests/test_gpu_parity.py: fields <= 1e-5 of max|B| (FP32 transforms of
a few thousand points: about 1e-6; also at 150,000 cells and more, where the oracle
convolves the GPU's kernel values, as in tests/test_gpu_configs.py), one explicit step of m <= 2e-6 absolute (rounding of m, dt k and
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


def _masked_spec(size, kind):
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
    return MagnetSpec(size=size, cellsize=(2e-9, 2e-9, 1e-9), msat=5.8e5, aex=1.5e-11, ku1=6e5, anisU=(0, 0, 1),
                      dmi={"xxz": 2e-3, "yyz": 2e-3}, world_bias=(0.01, 0.0, 0.1), **{"alpha": 0.1, **extra})


def _two_steps(mpx, s, method):
    """Largest difference of m from the oracle's after two explicit steps."""
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
    return np.max(np.abs(magnet.magnetization.eval() - ow.get_m(q)))


@pytest.mark.parametrize("kind", ["geometry", "alpha", "frozen", "all", "openbc", "periodic", "odd"])
@pytest.mark.parametrize("method", ["Heun", "DormandPrince"])
def test_masked_stage_epilogue(mpx, kind, method):
    """One explicit step of a magnet with uniform field parameters and a mask, per-cell damping or frozen spins."""
    assert _two_steps(mpx, _masked_spec((45, 30, 2) if kind == "odd" else (44, 30, 2), kind), method) < 2e-6


# the masked epilogue in every form of the inverse x pass: rows of 512 points one per warp, of 1024, of 2048 (warp
# pairs), of 384 (one per warp) and 768, and a magnet whose other rows are powers of two beside them
@pytest.mark.parametrize("size,method", [((140, 31, 2), "DormandPrince"), ((201, 9, 1), "Heun"),
                                         ((300, 30, 2), "DormandPrince"), ((513, 24, 2), "DormandPrince"),
                                         ((192, 400, 2), "Heun"), ((330, 231, 2), "DormandPrince")])
def test_masked_stage_epilogue_by_row_length(mpx, size, method):
    assert _two_steps(mpx, _masked_spec(size, "all"), method) < 2e-6


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
    """Every destination has two sources: the two directions of the pair of equal magnets share the launches of the
    FFT form, the small magnet's pairs take the direct sum (below 2^22 interactions)."""
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


def _worlds(mpx, specs):
    ow = O.OracleWorld()
    keep = []
    qs = [ow.add_magnet(s.desc(keep)) for s in specs]
    world = mpx.World(specs[0].cellsize)
    mags = []
    for k, (s, q) in enumerate(zip(specs, qs)):
        m = random_m(s.shape, seed=70 + k, smooth=2)
        ow.set_m(q, m)
        mag = mpx.Ferromagnet(world, mpx.Grid(s.size, s.origin))
        mag.msat, mag.aex, mag.alpha = s.msat, s.aex, s.alpha
        mag.magnetization = m
        mags.append(mag)
    return ow, qs, world, mags


# Magnets of which every pair takes the FFT form (at least 2^22 interactions): three whose pairs differ in their
# padded x and y lengths and so in the blocks and the shared memory of a common launch; three with pair z lengths of
# 16, whose y and z passes are apart; and nine, more destinations than one launch takes.  Every destination has two
# sources or more, so the fields of later rounds are added.
@pytest.mark.parametrize("sizes", [[(60, 48, 1), (150, 40, 1), (20, 210, 1)], [(40, 40, 5), (40, 30, 5), (30, 44, 6)],
                                   [(64, 32, 1)] * 9], ids=["lengths", "five_passes", "nine"])
def test_magnets_of_one_world_share_pair_launches(mpx, sizes):
    cs = (2e-9, 3e-9, 2.5e-9)
    cells = [nx * ny * nz for nx, ny, nz in sizes]
    assert min(a * b for i, a in enumerate(cells) for b in cells[:i]) >= 1 << 22
    specs, z = [], 0
    for k, size in enumerate(sizes):
        specs.append(MagnetSpec(size=size, origin=(3 * k, 2 * k, z), cellsize=cs, msat=8e5 - 3e4 * k, aex=1e-11, alpha=0.1))
        z += size[2] + 2
    ow, qs, world, mags = _worlds(mpx, specs)
    for q, mag, s in list(zip(qs, mags, specs))[:3]:
        got = mag._engine.eval(mag._id, abi.Q_EXTERNAL_FIELD, (3, *s.shape))
        assert max_rel(got, ow.eval(q, abi.Q_EXTERNAL_FIELD)) < FIELD_TOL
    ow.set_method("Heun")
    world.timesolver.set_method("Heun")
    world.timesolver.adaptive_timestep = False
    ow.set_solver(adaptive=0)
    ow.timestep = world.timesolver.timestep = 1e-14
    ow.steps(1)
    world.timesolver.steps(1)
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
    assert max_rel(got, ow.eval(q, abi.Q_DEMAG_FIELD)) < FIELD_TOL


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


def test_many_yz_classes_in_a_batch(mpx):
    """Solves of eight y/z launch classes, more than there are side streams, end together as each does alone."""
    from mumaxplus_b200 import batch, workloads as W

    sizes = [(40, 32, 1), (40, 32, 2), (40, 32, 4), (40, 32, 6), (16, 300, 1), (16, 16, 1), (8, 600, 1), (400, 190, 2),
             (20, 40, 12)]
    ws = [dict(name=f"c{k}", size=n, cellsize=(3e-9, 3e-9, 3e-9), msat=8e5, aex=1.3e-11, alpha=0.3,
               world_bias=(0.0, 0.01, 0.0), m0=lambda n=n, k=k: W.smoothed_random_m(n[::-1], 200 + k))
          for k, n in enumerate(sizes)]
    together, _, _ = batch.relax_batch(batch.Batch(), ws, duration=1e-12, torque_stop=0.0, autotune=False)
    alone, _, _ = batch.run_plain(batch.Batch(), ws, duration=1e-12, torque_stop=0.0)
    for a, b in zip(together, alone):
        assert a.steps == b.steps > 0 and np.array_equal(a.m, b.m)
