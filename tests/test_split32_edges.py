"""The split form's push and deposition at the places where their fast paths
end, against the FP64 form of the same library (itself bit-exact with the
CPU checker): particles in every cell of small meshes, next to the walls, the
axis, the irises and the last rows and columns, where some take the interior
gather and deposit and their warp's neighbours the general ones; and the
particles' order, which must change no result."""
import numpy as np
import pytest

from spiffe_b200 import abi, geometry, gpu, workloads
from helpers import MODES, QoMC

pytestmark = pytest.mark.gpu


def state(kind, nz, nr, per_cell=3, seed=1):
    cfg = (workloads.PillboxConfig if kind == "pillbox" else workloads.Gun16Config)(nz=nz, nr=nr, n_macro=1)
    f = geometry.fields_for(nz, nr, cfg.zmin, cfg.zmax, cfg.rmax, cfg.geo_text(), modes=MODES | abi.FL_SPACE_CHARGE)
    f.mesh.dt = cfg.dt
    rng = np.random.default_rng(seed)
    for n, scale in (("Ez", 1e7), ("Er", 1e7), ("Bphi", 1e-2), ("Bphi2", 1e-2), ("EzImposed", 1e6), ("ErImposed", 1e6)):
        f[n] = scale * rng.normal(size=f.shape)
    f["BzImposed"], f["BrImposed"] = 0.1 * rng.normal(size=f.shape), 0.1 * rng.normal(size=f.shape)
    n = nz * nr * per_cell
    z = rng.uniform(0, nz - 1, n) * f.mesh.dz + f.mesh.zmin
    r = np.abs(rng.uniform(-0.5, nr - 1, n)) * f.mesh.dr
    r[:: 97] = 0.0
    p = rng.normal(size=(3, n)) * 0.3
    p[2][r == 0] = 0.0
    g = np.sqrt(1 + (p ** 2).sum(0))
    b = abi.Beam(n + 16)
    b.set(n, z=z, r=r, pz=p[0], pr=p[1], r_pphi=p[2] * r, vz=workloads.C_MKS * p[0] / g, vr=workloads.C_MKS * p[1] / g,
          vphi=np.where(r > 0, workloads.C_MKS * p[2] / g, 0), Q=-rng.uniform(0.5, 1, n) * 1e-15,
          particleID=np.arange(1, n + 1), status=np.ones(n, np.uint64), zmax=z, zmin=z, rmax=r, rmin=r)
    b.npActive, b.nextParticleID, b.QoMC, b.stiffness = n, n + 1, QoMC, 1.0
    return f, b


def by_id(b):
    order = np.argsort(b["particleID"], kind="stable")
    return {k: b[k][order] for k in ("particleID", "z", "r", "pz", "pr", "r_pphi", "zmax", "rmax")}


def deposited(f, b, velocity):
    """Jz and Jr that the FP64 form deposits of the particles b."""
    c = abi.Beam(b.np)
    c.set(b.np, **{k: b[k][: b.np] for k in ("z", "r", "pz", "pr", "r_pphi", "Q", "particleID", "status")},
          **{k: velocity(b[k][: b.np]) for k in ("vz", "vr", "vphi")})
    c.npActive, c.nextParticleID, c.QoMC = b.np, b.nextParticleID, QoMC
    g = gpu.GpuInstance(f, capacity=c.capacity)
    g.upload_beam(c)
    g.zero_currents()
    g.deposit()
    out = g.fields(f)
    g.close()
    return out


@pytest.mark.parametrize("kind, nz, nr", [("pillbox", 5, 5), ("pillbox", 8, 6), ("pillbox", 33, 41), ("gun", 151, 42),
                                          ("gun", 77, 90)])
def test_push_and_deposit_in_every_cell(kind, nz, nr):
    f, b = state(kind, nz, nr)
    push = abi.push_options(abi.COMPACT_SWAP, abi.SCREEN_PARTICLE)
    out = {}
    for prec in (gpu.PRECISION_F64, gpu.PRECISION_SPLIT32):
        g = gpu.GpuInstance(f, capacity=b.capacity, precision=prec)
        g.upload_beam(b)
        g.configure_run(space_charge=1, push=push)
        g.run_steps(1)  # the split form deposits the pushed particles at the end of the step
        ob = g.download_beam(abi.Beam(b.capacity))
        out[prec] = by_id(ob)
    fused = g.fields(f)
    x, y = out[gpu.PRECISION_F64], out[gpu.PRECISION_SPLIT32]
    # a particle within rounding of a cell's edge may be lost on one side only
    both = np.intersect1d(x["particleID"], y["particleID"])
    assert len(both) >= 0.999 * max(len(x["particleID"]), len(y["particleID"]))
    x = {k: v[np.isin(x["particleID"], both)] for k, v in x.items()}
    y = {k: v[np.isin(y["particleID"], both)] for k, v in y.items()}
    m = f.mesh
    for k, unit in (("z", m.dz), ("r", m.dr), ("zmax", m.dz), ("rmax", m.dr)):
        assert np.max(np.abs(x[k] - y[k])) <= 1e-5 * nz * unit, k
    for k in ("pz", "pr", "r_pphi"):
        # FP32 fields and weights: a particle next to an edge of a stencil may
        # use the neighbouring node with a weight of rounding size
        d = np.abs(x[k] - y[k])
        assert np.quantile(d, 0.999) <= 1e-5 * np.max(np.abs(x[k])), k
    # the current that the push left, node by node, against the FP64 form's of
    # the very particles that it left: FP32 velocities and shares, and the
    # fixed point's quantum (2^-38 of the charge a node can hold)
    ref, size = deposited(f, ob, lambda v: v), deposited(f, ob, np.abs)
    g.zero_currents()
    g.deposit()  # the general path, of the same particles in the same form
    general = g.fields(f)
    for k in ("Jz", "Jr"):
        quantum = 1e-9 * np.max(np.abs(size[k]))
        assert np.all(np.abs(fused[k] - ref[k]) <= 2e-6 * np.abs(size[k]) + quantum), k
        assert np.all(np.abs(fused[k] - general[k]) <= 1e-6 * np.abs(size[k]) + quantum), k


@pytest.mark.parametrize("modes", [0, abi.FL_RADIAL_SMEAR | abi.FL_LONGIT_SMEAR])
@pytest.mark.parametrize("kind, nz, nr", [("pillbox", 33, 41), ("gun", 1200, 12), ("gun", 60, 900)])
def test_order_of_particles_changes_nothing(kind, nz, nr, modes):
    """Sorted on every step or never: the same bits (the deposition is exact)."""
    f, b = state(kind, nz, nr, per_cell=1)
    f.mesh.modes |= modes
    out = []
    for interval in (0, 1, 3):
        g = gpu.GpuInstance(f, capacity=b.capacity, precision=gpu.PRECISION_SPLIT32)
        g.set_sort_interval(interval)
        g.upload_beam(b)
        g.configure_run(space_charge=1, push=abi.push_options(abi.COMPACT_SWAP, abi.SCREEN_PARTICLE))
        g.run_steps(7)
        out.append((by_id(g.download_beam(abi.Beam(b.capacity))), g.fields(f)))
    for beam, fields in out[1:]:
        for k, v in out[0][0].items():
            assert np.array_equal(v, beam[k]), k
        for k in ("Ez", "Er", "Bphi", "Jz", "Jr"):
            assert np.array_equal(out[0][1][k], fields[k]), k


@pytest.mark.parametrize("n, n_lost", [(1, 1), (40, 39), (257, 200), (5000, 2047), (262145, 4000), (262145, 5000)])
def test_the_lost_leave_in_index_order_and_the_counts_are_reset(n, n_lost):
    """One block removes the lost, with few enough of them to be sorted and
    with more: the k-th hole takes the k-th survivor above the new count, and
    the counts are ready for the next push."""
    cfg = workloads.PillboxConfig()
    f = geometry.fields_for(cfg.nz, cfg.nr, cfg.zmin, cfg.zmax, cfg.rmax, cfg.geo_text(), modes=MODES)
    f.mesh.dt = cfg.dt
    rng = np.random.default_rng(n + n_lost)
    lost = np.sort(rng.choice(n, n_lost, replace=False))
    z = np.full(n, 0.5 * (cfg.zmin + cfg.zmax))
    z[lost] = cfg.zmax - 0.1 * cfg.dz  # leaves the mesh in one step at pz = 10
    pz = np.zeros(n)
    pz[lost] = 10.0
    b = abi.Beam(n + 16)
    b.QoMC = QoMC
    b.set(n, z=z, r=np.full(n, 0.2 * cfg.rmax), pz=pz, Q=np.full(n, -1e-16), particleID=np.arange(1, n + 1),
          status=np.full(n, abi.PART_ACTIVE, np.uint64))
    b.npActive = n
    g = gpu.GpuInstance(f, capacity=b.capacity, precision=gpu.PRECISION_SPLIT32)
    g.set_sort_interval(0)
    g.upload_beam(b)
    g.configure_run(space_charge=0, push=abi.push_options(abi.COMPACT_SWAP, abi.SCREEN_PARTICLE))
    new_np = n - n_lost
    gone = np.isin(np.arange(n), lost)
    expect = np.arange(1, n + 1)[:new_np]
    expect[lost[lost < new_np]] = np.nonzero(~gone[new_np:])[0] + new_np + 1
    for _ in range(2):  # the second step loses nothing
        g.run_steps(1)
        got = g.download_beam(abi.Beam(b.capacity))
        assert got.np == got.npActive == new_np
        assert np.array_equal(got["particleID"], expect)
    assert g.work_counters()["particle_steps"] == n + new_np
    g.close()
