"""Work buffers that could not be allocated: the calls that need them return
an error before they launch anything, and the instance stays usable."""
import ctypes as C

import numpy as np
import pytest

from spiffe_b200 import abi, geometry, gpu, workloads
from helpers import MODES, QoMC


class Mesh(C.Structure):  # the first members of DevMesh (common.cuh)
    _fields_ = [("nz", C.c_int), ("nr", C.c_int), ("pitch", C.c_int), ("doubles", C.c_double * 6), ("bc", C.c_int * 4),
                ("modes", C.c_uint), ("rest", C.c_char * 1024)]


class Work(C.Structure):  # Particles64Work (modules.cuh)
    _fields_ = [(n, C.c_void_p) for n in ("lost", "lost_list", "holes", "donors", "keys", "keys_alt", "vals",
                                          "vals_alt", "cub_tmp")] + [("cub_bytes", C.c_size_t),
                                                                      ("capacity", C.c_longlong), ("met_none", C.c_bool)]


def zeros(n=4096):
    return C.byref(C.create_string_buffer(n))


@pytest.mark.parametrize("modes", [abi.FL_TM_FIELDS, abi.FL_TM_FIELDS | abi.FL_TE_FIELDS, abi.FL_TE_FIELDS])
def test_ordered_deposition_without_its_buffers_launches_nothing(modes):
    lib = gpu.load()
    m = Mesh(nz=60, nr=50, pitch=51, modes=modes)
    before = lib.spiffe_gpu_launch_count()
    for w in (Work(), Work(capacity=1000)):
        rc = lib.spiffe_deposit64(C.byref(m), zeros(), zeros(), None, C.c_longlong(1000), C.c_bool(True), C.byref(w), None)
        assert rc != 0
    # buffers that are there but too small for both components' entries (the
    # address is never used)
    w = Work(keys=256, vals=256, capacity=999)
    m.modes |= abi.FL_RADIAL_SMEAR | abi.FL_LONGIT_SMEAR
    rc = lib.spiffe_deposit64(C.byref(m), zeros(), zeros(), None, C.c_longlong(1000), C.c_bool(True), C.byref(w), None)
    assert rc != 0
    assert lib.spiffe_gpu_launch_count() == before


def test_pushes_without_their_buffers_launch_nothing():
    lib = gpu.load()
    before = lib.spiffe_gpu_launch_count()
    m = Mesh(nz=60, nr=50, pitch=51, modes=abi.FL_TM_FIELDS)
    w = Work(met_none=True)
    assert lib.spiffe_push64(C.byref(m), zeros(), zeros(), zeros(), zeros(), None, C.c_longlong(10), C.byref(w), None) != 0
    # zeroed Particles32Work
    assert lib.s32_push(C.byref(m), zeros(), zeros(), zeros(), zeros(), None, C.c_longlong(10), 0, zeros(), zeros(), None) != 0
    assert lib.s32_sort(C.byref(m), zeros(), None, C.c_longlong(10), zeros(), None) != 0
    assert lib.spiffe_gpu_launch_count() == before


@pytest.mark.parametrize("ordered", [False, True])
def test_a_failed_allocation_leaves_no_capacity(ordered):
    """With no device every allocation fails."""
    import torch

    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    lib = gpu.load()
    w = Work()
    assert lib.spiffe_particles64_work(C.byref(w), C.c_longlong(5000), C.c_bool(ordered)) != 0
    assert w.capacity == 0 and not w.lost and not w.keys


@pytest.mark.gpu
def test_ordered_mode_is_on_only_once_its_buffers_are_there():
    import torch

    n = 1 << 22
    cfg = workloads.PillboxConfig(nz=60, nr=50)
    f = geometry.fields_for(60, 50, cfg.zmin, cfg.zmax, cfg.rmax, cfg.geo_text(), modes=MODES)
    b = abi.Beam(n)
    rng = np.random.default_rng(1)
    b.set(n, z=rng.uniform(0.2, 0.8, n) * f.mesh.zmax, r=rng.uniform(0.1, 0.8, n) * f.mesh.rmax, vz=np.full(n, 1e8),
          Q=np.full(n, -1e-15), particleID=np.arange(1, n + 1), status=np.ones(n, np.uint64))
    b.npActive, b.nextParticleID, b.QoMC = n, n + 1, QoMC
    g = gpu.GpuInstance(f, capacity=n)
    g.upload_beam(b)
    g.zero_currents()
    g.deposit()
    plain = g.fields(f)["Jz"].copy()
    # all but 48 MB of the device taken: the ordered form's 400 MB do not fit (nor
    # with the 256 MB at most that closed instances leave)
    fill, step = [], 1 << 34
    while step >= 1 << 20:
        if torch.cuda.mem_get_info()[0] > step + (48 << 20):
            fill.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
        else:
            step >>= 1
    with pytest.raises(gpu.SpiffeGpuError):
        g.set_deposit_order(1)
    del fill
    torch.cuda.empty_cache()

    def deposited():
        g.zero_currents()
        g.deposit()
        return g.fields(f)["Jz"].copy()

    # n additions in another order: within n eps of their sum (all of one sign)
    assert np.all(np.abs(deposited() - plain) <= n * 2.3e-16 * np.abs(plain))
    g.set_deposit_order(1)
    one = deposited()
    assert np.all(np.abs(one - plain) <= n * 2.3e-16 * np.abs(plain))
    assert np.array_equal(one, deposited())
    g.close()
