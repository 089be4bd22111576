"""Fields and distributions large enough to cross to the host in pinned pieces, of a
size that is no multiple of a piece."""

import ctypes
import subprocess
import sys
import threading

import numpy as np
import pytest
import torch

from conftest import ROOT
from hemepure_b200 import lbm, vessels

pytestmark = pytest.mark.gpu

C = np.array([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
              (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1),
              (0, -1, 1)], float)


@pytest.mark.parametrize("precision,eps", [("fp64", 2.0 ** -53), ("fp32", 2.0 ** -24)])
# u below and above the size that goes in pieces, and f above it in both directions (75 MB up)
@pytest.mark.parametrize("radius,length", [(6.0, 31), (20.0, 151), (22.3, 317)])
def test_fields_arrive_in_reference_order(tmp_path, precision, eps, radius, length):
    v = vessels.Pipe(radius, length)
    vessels.voxelise(v, str(tmp_path / "c.gmy"))
    vessels.write_case_xml(str(tmp_path / "c.xml"), "c.gmy", v, vessels.CaseUnits(tau=0.8), 10, [vessels.VelocityBC(0.01)],
                           [vessels.PressureBC(1.0)])
    sim = lbm.LBM(str(tmp_path / "c.xml"), wall="BFL", precision=precision)
    rng = np.random.default_rng(3)
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
    f = w * (1.0 + 1e-3 * rng.standard_normal((sim.n, 19)))
    assert f.nbytes % (512 << 10) and (length < 300 or f.nbytes > 64 << 20)
    sim.SetFs(f)
    got = sim.GetFOld()
    # FP64 storage is exact; FP32 rounds the deviation from w, at most 5e-3 w.
    assert np.abs(got - f).max() <= (0.0 if precision == "fp64" else 5e-3 / 3 * eps)
    sim.step(1, macro=True, stress=True)
    rho, u, wss = sim.GetPropertyCache()
    # Sums of 19 rounded values of order 1 and below.
    assert np.abs(rho - got.sum(1)).max() <= 19 * eps
    assert np.abs(u - (got @ C) / got.sum(1)[:, None]).max() <= 40 * eps
    wall = sim.tables()["wall_mask"] != 0
    assert np.array_equal(wss < 1e300, wall)
    traction = sim.GetStress("traction")
    assert np.array_equal((traction != 0).any(1), wall)


def test_callers_pinned_array(tmp_path):
    v = vessels.Pipe(20.0, 151)
    vessels.voxelise(v, str(tmp_path / "c.gmy"))
    vessels.write_case_xml(str(tmp_path / "c.xml"), "c.gmy", v, vessels.CaseUnits(tau=0.8), 10, [vessels.VelocityBC(0.01)],
                           [vessels.PressureBC(1.0)])
    sim = lbm.LBM(str(tmp_path / "c.xml"), wall="BFL")
    sim.step(3)
    pinned = torch.zeros((sim.n, 19), dtype=torch.float64, pin_memory=True)
    assert lbm.library().hb_get_fs(sim._h, ctypes.cast(pinned.data_ptr(), ctypes.POINTER(ctypes.c_double))) == 0
    assert np.array_equal(pinned.numpy(), sim.GetFOld())


def test_two_handles_read_side_by_side(tmp_path):
    v = vessels.Pipe(20.0, 151)
    vessels.voxelise(v, str(tmp_path / "c.gmy"))
    vessels.write_case_xml(str(tmp_path / "c.xml"), "c.gmy", v, vessels.CaseUnits(tau=0.8), 10, [vessels.VelocityBC(0.01)],
                           [vessels.PressureBC(1.0)])
    sims = [lbm.LBM(str(tmp_path / "c.xml"), wall="BFL") for _ in range(2)]
    for k, sim in enumerate(sims):
        sim.step(3 + k, macro=True)
    ref = [(*sim.GetPropertyCache(), sim.GetFOld()) for sim in sims]
    same = [[], []]

    def read(k):
        for _ in range(4):
            got = (*sims[k].GetPropertyCache(), sims[k].GetFOld())
            same[k].append(all(np.array_equal(a, b) for a, b in zip(got, ref[k])))

    threads = [threading.Thread(target=read, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert same == [[True] * 4] * 2


SCRATCH = """
import sys
import torch
from hemepure_b200 import lbm
small, large = (lbm.LBM(x, wall="BFL", precision="fp32", geometry_reader="host") for x in sys.argv[1:3])
small.SetFs(small.GetFOld())  # the kernels are loaded
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
large.SetFs(large.GetFOld())
print(large.n, before - torch.cuda.mem_get_info()[0])
"""


def test_scratch_of_large_distributions_is_given_back(tmp_path):
    """Distributions of 186 MB go through device scratch of that size, of which the
    process keeps 128 MB at most (in a process of its own: a set-up on the device
    leaves the pool larger)."""
    for name, v in (("s", vessels.Pipe(6.0, 31)), ("l", vessels.Pipe(31.2, 400))):
        vessels.voxelise(v, str(tmp_path / (name + ".gmy")))
        vessels.write_case_xml(str(tmp_path / (name + ".xml")), name + ".gmy", v, vessels.CaseUnits(tau=0.8), 10,
                               [vessels.VelocityBC(0.01)], [vessels.PressureBC(1.0)])
    r = subprocess.run([sys.executable, "-c", SCRATCH, str(tmp_path / "s.xml"), str(tmp_path / "l.xml")], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    n, kept = map(int, r.stdout.split())
    assert n * 19 * 8 > 180e6 and kept <= 136 << 20
