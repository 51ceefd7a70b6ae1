"""Device memory kept from closed instances: new ones get it zeroed where
they promise zeros, instances of several threads do not share a block, and
what is kept is bounded."""
import threading

import numpy as np
import pytest

from spiffe_b200 import abi, geometry, gpu, workloads
from helpers import MODES, QoMC

pytestmark = pytest.mark.gpu


def instance(nz, nr, precision, seed):
    cfg = workloads.PillboxConfig(nz=nz, nr=nr)
    f = geometry.fields_for(nz, nr, cfg.zmin, cfg.zmax, cfg.rmax, cfg.geo_text(), modes=MODES)
    f.mesh.dt = cfg.dt
    f["Ez"] = cfg.initial_ez()
    rng = np.random.default_rng(seed)
    n = 3000
    b = abi.Beam(n)
    b.set(n, z=rng.uniform(0.2, 0.8, n) * cfg.zmax, r=rng.uniform(0, 0.5, n) * cfg.rmax, pz=rng.normal(size=n),
          vz=np.zeros(n), Q=np.full(n, -1e-14), particleID=np.arange(1, n + 1), status=np.ones(n, np.uint64))
    b.npActive, b.nextParticleID, b.QoMC = n, n + 1, QoMC
    g = gpu.GpuInstance(f, capacity=n, precision=precision)
    g.set_deposit_order(1)
    g.configure_run(space_charge=1, push=abi.push_options(abi.COMPACT_SWAP, abi.SCREEN_PARTICLE))
    g.upload_beam(b)
    return g, f, b


def result(nz, nr, precision, seed, steps=20):
    g, f, b = instance(nz, nr, precision, seed)
    g.run_steps(steps)
    out = g.fields(f)
    g.download_beam(b)
    g.close()
    at = np.argsort(b["particleID"][: b.np])
    return [out[n].copy() for n in ("Ez", "Er", "Bphi")] + [b[k][: b.np][at] for k in ("z", "r", "pz", "pr")]


def test_instances_of_many_threads_and_sizes_give_what_one_alone_gives():
    jobs = [(60 + 7 * k, 50 + 5 * (k % 3), p, k) for k in range(6) for p in (gpu.PRECISION_F64, gpu.PRECISION_SPLIT32)]
    alone = [result(*j) for j in jobs]
    again = [[None] * 3 for _ in jobs]

    def work(t):
        for k in range(t, len(jobs), 4):
            for rep in range(3):
                again[k][rep] = result(*jobs[k])

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, rows in zip(alone, again):
        for row in rows:
            assert all(np.array_equal(x, y) for x, y in zip(a, row))


def test_what_is_kept_is_bounded():
    import torch

    torch.cuda.init()
    instance(60, 50, gpu.PRECISION_F64, 0)[0].close()
    free0, _ = torch.cuda.mem_get_info()
    for nz in (200, 400, 600, 800, 1000, 1200):  # 10 to 60 MB of fields each
        for nr in (300, 301):
            instance(nz, nr, gpu.PRECISION_F64, 1)[0].close()
    free1, _ = torch.cuda.mem_get_info()
    # 256 MB, and what the driver keeps of its own (2 MB pages of small blocks)
    assert free0 - free1 <= (256 << 20) + (64 << 20)


def test_what_is_kept_is_given_back_on_request():
    import torch

    instance(200, 300, gpu.PRECISION_F64, 1)[0].close()
    torch.cuda.synchronize()
    kept = gpu.idle_memory()
    assert 0 < kept <= 256 << 20
    free0, _ = torch.cuda.mem_get_info()
    assert gpu.idle_memory(release=True) == kept
    free1, _ = torch.cuda.mem_get_info()
    assert free1 - free0 >= 0.9 * kept - (2 << 20)  # the driver's pages of small blocks may be shared
    assert gpu.idle_memory() == 0
    a = result(60, 50, gpu.PRECISION_SPLIT32, 2)
    assert all(np.array_equal(x, y) for x, y in zip(a, result(60, 50, gpu.PRECISION_SPLIT32, 2)))


RESET = """
import ctypes, glob, sys
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import numpy as np
from spiffe_b200 import gpu
from test_devmem import result
jobs = [(60, 50, p, 3) for p in (gpu.PRECISION_F64, gpu.PRECISION_SPLIT32)]
before = [result(*j) for j in jobs]
assert gpu.idle_memory() > 0
rt = ctypes.CDLL(glob.glob("/usr/local/cuda/lib64/libcudart.so*")[0])
assert rt.cudaDeviceReset() == 0
assert gpu.idle_memory() == 0
after = [result(*j) for j in jobs + jobs]
for a, b in zip(before + before, after):
    assert all(np.array_equal(x, y) for x, y in zip(a, b))
print("same")
"""


def test_a_program_may_reset_its_device_between_instances():
    """The reset ends the context and the memory kept in it: new instances must
    not be given its addresses."""
    import glob
    import os
    import subprocess
    import sys

    if not glob.glob("/usr/local/cuda/lib64/libcudart.so*"):
        pytest.skip("no CUDA runtime library to reset the device with")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", RESET.format(root=root)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "same", out.stdout + out.stderr
