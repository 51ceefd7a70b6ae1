"""The FP64 form's ordered reduction and banded SOR at the sizes where they
can go wrong, bit for bit against the CPU checker.

* The ordered deposition and charge removal sum each node's particles in
  particle order; the kernel takes 32 entries a warp and follows a run that
  goes on behind them 32 at a time, so runs of 1, 31, 32, 33, ... entries at
  every offset, and meshes with one, two and four entries a particle.
* The SOR with its rows in shared memory: bands of two rows and of many, the
  narrowest meshes, rows of one and of several warps, and both kinds of ends.
"""
import numpy as np
import pytest

from spiffe_b200 import abi, geometry, gpu, workloads
from helpers import MODES, QoMC

pytestmark = pytest.mark.gpu


def pillbox(nz, nr, modes=MODES, **bcs):
    cfg = workloads.PillboxConfig(nz=nz, nr=nr)
    f = geometry.fields_for(nz, nr, cfg.zmin, cfg.zmax, cfg.rmax, cfg.geo_text(), modes=modes, **bcs)
    f.mesh.dt = cfg.dt
    return f


def crowded_beam(f, counts, seed=3):
    """Particles counts[k] of which lie around node (5 + k % 20, 1 + k // 20), shuffled."""
    rng = np.random.default_rng(seed)
    n, m = int(sum(counts)), f.mesh
    k = rng.permutation(np.repeat(np.arange(len(counts)), counts))
    a = {"z": (5 + k % 20 + rng.uniform(-0.49, 0.49, n)) * m.dz, "r": (1 + k // 20 + rng.uniform(-0.49, 0.49, n)) * m.dr}
    for name in ("vz", "vr", "vphi"):
        a[name] = rng.normal(size=n) * 1e8
    b = abi.Beam(n + 16)
    b.set(n, Q=-rng.uniform(0.5, 1.5, n) * 1e-15, particleID=np.arange(1, n + 1), status=np.ones(n, np.uint64), **a)
    b.npActive, b.nextParticleID, b.QoMC = n, n + 1, QoMC
    return b


@pytest.mark.parametrize("smear", [0, abi.FL_RADIAL_SMEAR, abi.FL_LONGIT_SMEAR,
                                   abi.FL_RADIAL_SMEAR | abi.FL_LONGIT_SMEAR])
@pytest.mark.parametrize("counts", [[1], [31], [32, 1, 1], [33, 31, 65, 64, 2, 1, 96], [5000] + [1] * 200 + [7] * 90])
def test_ordered_sums_in_particle_order(oracle, counts, smear):
    f = pillbox(60, 50, MODES | smear)
    b = crowded_beam(f, counts)
    g = gpu.GpuInstance(f, capacity=b.capacity)
    g.set_deposit_order(1)
    g.upload_beam(b)
    g.zero_currents()
    g.deposit()
    g.deposit()  # a second time on top of the first: the sums start from the arrays' values
    ref = f.copy()
    oracle.zero_currents(ref)
    oracle.deposit(ref, b)
    oracle.deposit(ref, b)
    out = g.fields(f)
    for n in ("Jz", "Jr"):
        assert np.array_equal(out[n], ref[n]), n
    # the particles' charge leaves Q the same way (the solve is a few sweeps)
    opts = abi.poisson_options(step_interval=1, accuracy=1e-300, maximum_iterations=4)
    g.poisson_correction(1, opts)
    ref = f.copy()
    oracle.poisson_correction(ref, b, 1, opts)
    out = g.fields(f)
    for n in ("Q", "Psi", "Ez", "Er"):
        assert np.array_equal(out[n], ref[n]), n


@pytest.mark.parametrize("smear", [0, abi.FL_RADIAL_SMEAR, abi.FL_RADIAL_SMEAR | abi.FL_LONGIT_SMEAR])
@pytest.mark.parametrize("modes", [MODES | abi.FL_TE_FIELDS, (MODES | abi.FL_TE_FIELDS) & ~abi.FL_TM_FIELDS])
def test_ordered_sums_of_every_component(oracle, modes, smear):
    """Components sorted together, or one by one where the buffers do not hold all."""
    f = pillbox(60, 50, modes | smear)
    b = crowded_beam(f, [700, 33, 64] + [3] * 150)
    g = gpu.GpuInstance(f, capacity=b.capacity)
    g.set_deposit_order(1)
    g.upload_beam(b)
    ref = f.copy()
    for _ in range(2):
        g.zero_currents()
        oracle.zero_currents(ref)
        g.deposit()
        oracle.deposit(ref, b)
        out = g.fields(f)
        for n in ("Jz", "Jr", "Jphi"):
            if n in f.a and (n == "Jphi" or modes & abi.FL_TM_FIELDS):
                assert np.array_equal(out[n], ref[n]), n


@pytest.mark.parametrize("ends", [(abi.NEUMANN, abi.NEUMANN), (abi.DIRICHLET, abi.DIRICHLET),
                                  (abi.NEUMANN, abi.DIRICHLET)])
@pytest.mark.parametrize("nz, nr", [(6, 5), (7, 6), (40, 9), (41, 66), (300, 67), (307, 34), (90, 259), (700, 130),
                                    (24, 1030), (601, 321)])
def test_sor_is_the_serial_iteration(oracle, nz, nr, ends):
    f = pillbox(nz, nr, left_bc=ends[0], right_bc=ends[1])
    rng = np.random.default_rng(nz * 1000 + nr)
    f["Q"] = rng.normal(size=f.shape) * 1e6
    f["Psi"] = np.where(rng.uniform(size=f.shape) < 0.5, 0.0, rng.normal(size=f.shape))
    g = gpu.GpuInstance(f)
    for limit in (2, 37):  # exactly this many half-sweeps
        g.upload_fields(f)
        assert g.solve_poisson(0, 1e-300, limit) == -1
        ref = f.copy()
        n, _, _ = oracle.solve_poisson(ref, ref["Psi"], ref["Q"], 1e-300, limit)
        assert n == -1 and np.array_equal(g.fields(f)["Psi"], ref["Psi"]), limit
    g.upload_fields(f)
    n = g.solve_poisson(0, 0.2, 500)  # the stop rule inside the run
    ref = f.copy()
    m, _, _ = oracle.solve_poisson(ref, ref["Psi"], ref["Q"], 0.2, 500)
    assert n == m and np.array_equal(g.fields(f)["Psi"], ref["Psi"])


@pytest.mark.parametrize("nz, nr", [(12, 12), (20, 33), (106, 162), (301, 83), (700, 64), (769, 33),  # one cluster
                                    (770, 100), (300, 411)])  # just too large for one
def test_sor_of_one_cluster_and_of_the_grid(oracle, nz, nr):
    """Meshes of two to sixteen bands in one thread-block cluster, with one
    and with two rows a thread and a short last band, and their neighbours."""
    test_sor_is_the_serial_iteration(oracle, nz, nr, (abi.NEUMANN, abi.DIRICHLET))


def test_sor_follows_ends_set_after_setup(oracle):
    """set_mesh may change the end conditions, and with them the update rows."""
    f = pillbox(60, 40)
    f["Q"] = np.random.default_rng(4).normal(size=f.shape) * 1e6
    g = gpu.GpuInstance(f)
    g.solve_poisson(0, 1e-300, 4)
    fd = f.copy()
    fd.mesh.left_bc = abi.DIRICHLET
    m = g.get_mesh()
    m.left_bc = abi.DIRICHLET
    g.set_mesh(m)
    g.upload_fields(fd)
    g.solve_poisson(0, 1e-300, 20)
    ref = fd.copy()
    oracle.solve_poisson(ref, ref["Psi"], ref["Q"], 1e-300, 20)
    assert np.array_equal(g.fields(fd)["Psi"], ref["Psi"])


@pytest.mark.parametrize("n, n_lost", [(1, 1), (2, 1), (40, 39), (1500, 1024), (9000, 4096), (20000, 6000), (40000, 33000),
                                       (32769, 1024), (32769, 1025), (32784, 32783), (50001, 50001), (99999, 50000),
                                       (300000, 1500), (300000, 298000), (1100000, 400000)])
def test_swap_compaction_pairs_holes_with_the_last_survivors(n, n_lost):
    """The j-th lost slot takes the j-th survivor counted from the end, whatever
    the number of losses (none, a block's, more than are sorted, a burst shared
    by two and by all blocks, everything), and the counts are ready for the next
    push."""
    f = pillbox(60, 50)
    m = f.mesh
    rng = np.random.default_rng(n)
    lost = np.sort(rng.choice(n, n_lost, replace=False))
    z = np.full(n, 0.5 * (m.zmin + m.zmax))
    z[lost] = m.zmax - 0.1 * m.dz  # leaves the mesh in one step at pz = 10
    pz = np.zeros(n)
    pz[lost] = 10.0
    vz = np.where(pz > 0, 2.98e8, 0.0)
    b = abi.Beam(n + 16)
    b.QoMC = QoMC
    b.set(n, z=z, r=np.full(n, 10.0 * m.dr), pz=pz, vz=vz, Q=np.full(n, -1e-16), particleID=np.arange(1, n + 1),
          status=np.full(n, abi.PART_ACTIVE, np.uint64))
    b.npActive = n
    g = gpu.GpuInstance(f, capacity=b.capacity)
    g.upload_beam(b)
    g.configure_run(space_charge=0, push=abi.push_options(abi.COMPACT_SWAP, abi.SCREEN_PARTICLE))
    new_np = n - n_lost
    gone = np.isin(np.arange(n), lost)
    expect = np.arange(1, n + 1)[:new_np]
    holes, donors = lost[lost < new_np], np.nonzero(~gone[new_np:])[0] + new_np
    expect[holes] = donors[::-1] + 1
    for _ in range(2):  # the second step loses nothing
        g.run_steps(1)
        got = g.download_beam(abi.Beam(b.capacity))
        assert got.np == got.npActive == new_np
        assert np.array_equal(got["particleID"], expect)
    g.close()


def test_current_is_cleared_and_read_where_it_lies(oracle):
    """Currents left by an upload, by deposits on top of one another and by
    earlier, wider deposits: the clearing, and the field update that reads J
    only in its box, against the checker's whole arrays."""
    f = pillbox(60, 50)
    rng = np.random.default_rng(8)
    for n in ("Ez", "Er", "Bphi", "Jz", "Jr"):
        f[n] = rng.normal(size=f.shape) * (1e3 if n[0] == "J" else 1.0)
    ref = f.copy()
    g = gpu.GpuInstance(f, capacity=4096)
    g.set_deposit_order(1)
    wide, narrow = crowded_beam(f, [3] * 200), crowded_beam(f, [5])

    def same(names=("Jz", "Jr", "Ez", "Er", "Bphi")):
        out = g.fields(f)
        for n in names:
            assert np.array_equal(out[n], ref[n]), n

    g.upload_fields(f)
    g.advance_fields()  # with the uploaded current
    oracle.advance_fields(ref)
    same()
    for beams in ([wide], [narrow], [wide, narrow], [], [narrow]):
        g.zero_currents()
        oracle.zero_currents(ref)
        for b in beams:
            g.upload_beam(b)
            g.deposit()
            oracle.deposit(ref, b)
        g.advance_fields()
        oracle.advance_fields(ref)
        same()
    g.close()


@pytest.mark.parametrize("nz, nr, spread", [(60, 50, 1.0), (300, 200, 0.1), (300, 200, 1.0)])
@pytest.mark.parametrize("n", [196608, 196609, 200000])
def test_unordered_sums_of_many_particles(nz, nr, spread, n):
    """From 3 2^16 particles a block sums its particles in shared memory before
    they go to J, where their nodes span few enough (the beam of a tenth of the
    mesh; the others go to J one by one)."""
    f = pillbox(nz, nr)
    m = f.mesh
    rng = np.random.default_rng(n + nr)
    z = (0.45 + spread * rng.uniform(-0.45, 0.55, n)) * (m.zmax - m.zmin) + m.zmin
    r = spread * rng.uniform(0, 1, n) ** 2 * m.dr * (nr - 1)
    unordered_is_ordered(f, z, r, np.where(rng.uniform(size=n) < 0.9, abi.PART_ACTIVE, 0), rng)


@pytest.mark.parametrize("modes", [MODES, MODES | abi.FL_TE_FIELDS, (MODES | abi.FL_TE_FIELDS) & ~abi.FL_TM_FIELDS])
@pytest.mark.parametrize("rows, cols, a_cell, order", [(32, 64, 0, "random"), (33, 63, 0, "random"), (32, 65, 0, "random"),
                                                       (1, 1, 0, "random"), (300, 2, 0, "random"), (32, 64, 0, "cells"),
                                                       (500, 60, 6, "cells"), (500, 60, 16, "cells"), (40, 40, 200, "cells")])
def test_unordered_sums_of_a_block(rows, cols, a_cell, order, modes):
    """Blocks of 2048 particles that span 2048 nodes (the most that a block sums
    itself) and a few more, in random order and in the order of their cells,
    where whole warps or groups of two to thirty lanes of a warp add to one
    node; a tenth of the particles is inactive."""
    n = 200000
    f = pillbox(520, 70, modes)
    rng = np.random.default_rng(rows * cols + a_cell)
    if order == "random":
        cell = rng.integers(0, rows * cols, n)
    elif a_cell:  # about a_cell particles in each of the first cells
        cell = np.repeat(np.arange(n), rng.integers(a_cell // 2, a_cell * 3 // 2 + 1, n))[:n] % (rows * cols)
    else:
        cell = np.sort(rng.integers(0, rows * cols, n))
    # the nearest nodes of both components' stencils are the cell's own
    z, r = 3 + cell % rows + rng.uniform(0.1, 0.4, n), cell // rows + rng.uniform(0.1, 0.4, n)
    unordered_is_ordered(f, z * f.mesh.dz + f.mesh.zmin, r * f.mesh.dr,
                         np.where(rng.uniform(size=n) < 0.9, abi.PART_ACTIVE, 0), rng)


def unordered_is_ordered(f, z, r, status, rng):
    """The deposition against the ordered sums.  Either order of n additions is
    within n eps / 2 of the exact sum of the contributions' magnitudes, which
    the same beam with positive velocities deposits."""
    n, status = len(z), status.astype(np.uint64)
    b = abi.Beam(n)
    v = rng.normal(size=(3, n)) * 1e8
    got = {}
    for name, order, vel in (("sum", 0, v), ("ordered", 1, v), ("size", 1, np.abs(v))):
        b.set(n, z=z, r=r, vz=vel[0], vr=vel[1], vphi=vel[2], Q=np.full(n, -1e-15), particleID=np.arange(1, n + 1), status=status)
        b.npActive, b.nextParticleID, b.QoMC = int((status > 0).sum()), n + 1, QoMC
        g = gpu.GpuInstance(f, capacity=n)
        g.set_deposit_order(order)
        g.upload_beam(b)
        g.zero_currents()
        g.deposit()
        got[name] = g.fields(f)
        g.close()
    names = ("Jz", "Jr") * bool(f.mesh.modes & abi.FL_TM_FIELDS) + ("Jphi",) * bool(f.mesh.modes & abi.FL_TE_FIELDS)
    for k in names:
        assert np.any(got["ordered"][k] != 0)
        assert np.all(np.abs(got["sum"][k] - got["ordered"][k]) <= n * 2.3e-16 * np.abs(got["size"][k])), k


# numerators of the divisions by dr, dz, eps0 and the SOR's diagonals: ordinary
# ones; quotients that are subnormal, or lie half way between two subnormals
# (powers of two apart); near overflow
SCALES = [1.0, 2.0 ** -941, 1e-290, 1e-305, 2.0 ** -1030, 2.0 ** -1074, 2.0 ** 899, 2.0 ** 950, 1e300]


def scaled(rng, shape, scale):
    """Random values around a scale (whole multiples of the smallest subnormal
    where that is the scale), zeros of both signs among them."""
    x = np.round(rng.normal(size=shape) * 64) * scale
    return np.where(rng.uniform(size=shape) < 0.05, np.copysign(0.0, x), x)


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("dz, dr", [(None, None), (4.0, 2.0), (6.0, 3.0), (2.0 ** -60, 2.0 ** 60), (2.0 ** -61, 2.0 ** 61)])
def test_field_update_divides_as_the_reference_does(oracle, scale, dz, dr):
    """The update's quotients are formed from reciprocals: the same bits at
    every size of numerator, infinities and NaN among them, for the divisors
    that take that way and for those beyond them."""
    f = pillbox(33, 29)
    if dz:
        f.mesh.dz, f.mesh.dr = dz, dr
    f.mesh.dt = 0.25 if scale > 1e200 or scale < 1e-200 else 1e-13
    rng = np.random.default_rng(7)
    for n in ("Ez", "Er", "Bphi", "Jz", "Jr"):
        f[n] = scaled(rng, f.shape, scale)
    f["Ez"][11, 7], f["Jz"][13, 9], f["Er"][20, 11] = np.inf, -np.inf, np.nan
    g = gpu.GpuInstance(f)
    g.upload_fields(f)
    ref = f.copy()
    for _ in range(2):
        g.advance_fields()
        oracle.advance_fields(ref)
    out = g.fields(f)
    for n in ("Ez", "Er", "Bphi", "Bphi2"):
        assert np.array_equal(out[n], ref[n], equal_nan=True), n
    g.close()


@pytest.mark.parametrize("nz, nr", [(40, 31), (300, 411)])  # one cluster, the grid
@pytest.mark.parametrize("dz, dr, scale", [(None, None, s) for s in SCALES] +
                         # beyond the divisors of the reciprocal's way: quotients are subnormal where the numerators
                         # are not, here half way between two subnormals in one of twenty nodes
                         [(2.0 ** -70, 2.0 ** -71, 2.0 ** k) for k in (-881, -890, -900)])
def test_sor_divides_as_the_reference_does(oracle, nz, nr, dz, dr, scale):
    f = pillbox(nz, nr)
    if dz:
        f.mesh.dz, f.mesh.dr = dz, dr
    rng = np.random.default_rng(9)
    f["Q"] = scaled(rng, f.shape, scale) if not dz else rng.integers(1, 1 << 53, f.shape) * (scale * 2.0 ** -53)
    f["Psi"] = np.zeros(f.shape)
    g = gpu.GpuInstance(f)
    for limit in (2, 9):
        g.upload_fields(f)
        ref = f.copy()
        n, _, _ = oracle.solve_poisson(ref, ref["Psi"], ref["Q"], 1e-300, limit)
        assert g.solve_poisson(0, 1e-300, limit) == n
        assert np.array_equal(g.fields(f)["Psi"], ref["Psi"], equal_nan=True), limit
    g.close()
