"""The multigrid solver's kernels at the sizes where they can go wrong: a few
rows a band and many, level rows of one warp, of as many columns as fit shared
memory and of more, more column pairs than a CTA has threads, coarsening of
one direction only, a coarsest level solved by its inverse and one that can
be coarsened no further and is swept, and all end conditions.

The check is the stop rule, evaluated here in FP64 from the returned
potential: sum |rhs - A Psi| < accuracy sum |rhs|.  (The residual's own
rounding, some 10 eps |Psi| / h^2 a node, is 1e-11 of the sum at the most.)"""
import numpy as np
import pytest

from spiffe_b200 import abi, geometry, gpu, workloads
from helpers import MODES, poisson_residual
from test_split32 import split

pytestmark = pytest.mark.gpu

NN, DN, ND, DD = [(a, b) for b in (abi.NEUMANN, abi.DIRICHLET) for a in (abi.NEUMANN, abi.DIRICHLET)]
SMALL = [(17, 33, 1), (40, 30, 1), (41, 64, 1),          # nz, nr, dz/dr: the next level is solved by its inverse
         (301, 83, 1)]                                   # one pair a thread on the next level
LARGE = [(700, 300, 1), (1000, 700, 1),                  # two and more
         (64, 1903, 1), (60, 1930, 1), (48, 2030, 1),    # rows that just fit shared memory, and wider ones
         (300, 2000, 0.25), (900, 150, 0.25),            # z alone is coarsened first
         (2000, 60, 4), (200, 800, 4)]                   # r alone


# (a mirrored right end that lies on no coarser level's row, as in most of the
# large meshes, slows the convergence: a property of the interpolation)
@pytest.mark.parametrize("mesh, ends", [(m, e) for m in SMALL + LARGE for e in (NN, DN)] +
                         [(m, e) for m in SMALL for e in (ND, DD)])
def test_solves_meet_the_stop_rule(mesh, ends):
    check(mesh, ends)


@pytest.mark.parametrize("mesh", [(6, 1500, 1), (1500, 6, 1), (5000, 6, 1)])
def test_a_coarsest_level_too_large_for_its_inverse(mesh):
    """Four rows or columns cannot be coarsened: swept in shared memory, and
    where that is too small in global memory."""
    check(mesh, NN)


def check(mesh, ends):
    nz, nr, ratio = mesh
    cfg = workloads.PillboxConfig(nz=nz, nr=nr, R=1e-4 * (nr - 1), L=1e-4 * ratio * (nz - 1))
    f = geometry.fields_for(nz, nr, cfg.zmin, cfg.zmax, cfg.rmax, cfg.geo_text(), modes=MODES, left_bc=ends[0],
                            right_bc=ends[1])
    f.mesh.dt = cfg.dt
    rng = np.random.default_rng(nz + nr)
    z, r = np.arange(f.shape[0])[:, None] / nz, np.arange(f.shape[1])[None, :] / nr
    f["Q"] = (np.exp(-((z - 0.4) ** 2 + r ** 2) / 0.02) + 0.1 * rng.normal(size=f.shape)) * 1e6
    f["Psi"] = np.zeros(f.shape)
    g = split(f)
    g.configure_run(space_charge=0, poisson=abi.poisson_options(step_interval=1))
    n = g.solve_poisson(0, 1e-6, 100)
    res, drive = poisson_residual(f, g.fields(f)["Psi"], f["Q"])
    print(mesh, ends, n, "cycles", res / drive)
    assert 0 < n <= 40 and res < 1e-6 * drive
    g.close()
