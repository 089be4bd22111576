"""The walk of a bulk block over several tiles of sites in the one-launch step, which
lattices take from about 0.3M sites (FP64) or 0.6M (shifted forms) on: at two, three and
four tiles a block, with a last tile that ends raggedly and a last block whose later
tiles lie past the lattice."""

import numpy as np
import pytest

from hemepure_b200 import lbm, vessels
from oracle import oracle as O

pytestmark = pytest.mark.gpu

STEPS = 10
BLOCK, SMS, WAVES, MOST = 128, 148, 2, 4  # step_tiles.cuh
RESIDENT = {"fp64": 4, "fp32": 8, "fp16": 8}


@pytest.fixture(scope="module")
def pipes(tmp_path_factory):
    made = {}

    def get(radius, length):
        if (radius, length) not in made:
            d = tmp_path_factory.mktemp("pipe")
            v = vessels.Pipe(radius, length)
            vessels.voxelise(v, str(d / "c.gmy"))
            vessels.write_case_xml(str(d / "c.xml"), "c.gmy", v, vessels.CaseUnits(tau=0.8), 100, [vessels.VelocityBC(0.01)],
                                   [vessels.PressureBC(0.9995)], relaxation_parameter=3.0 / 16.0)
            made[radius, length] = str(d / "c.xml")
        return made[radius, length]
    return get


@pytest.mark.parametrize("precision,radius,length,tiles,kernel,wall",
                         [("fp64", 22.3, 204, 2, "LBGK", "BFL"), ("fp64", 22.3, 305, 3, "TRT", "GZS"),
                          ("fp64", 22.3, 407, 4, "TRT", "SBB"), ("fp32", 22.3, 407, 2, "TRT", "GZS"),
                          ("fp32", 31.2, 305, 3, "LBGK", "SBB"), ("fp32", 31.2, 401, 4, "TRT", "BFL"),
                          ("fp16", 31.2, 401, 4, "LBGK", "BFL")])
def test_several_tiles_a_block(pipes, precision, radius, length, tiles, kernel, wall):
    """Steps in one launch against steps with outputs, which take a thread per site in
    kernels of their own: the same bits, as a site's arithmetic is rounded as written
    whichever kernel steps it.  FP64 also against the oracle."""
    xml = pipes(radius, length)
    sims = [lbm.LBM(xml, kernel=kernel, wall=wall, precision=precision) for _ in range(2)]
    blocks = -(-sims[0].n // BLOCK)
    assert min(MOST, blocks // (SMS * RESIDENT[precision] * WAVES)) == tiles
    assert sims[0].n % BLOCK and blocks % tiles
    sims[0].step(STEPS)
    for _ in range(STEPS):
        sims[1].step(1, macro=True)
    f = [s.GetFOld() for s in sims]
    assert np.array_equal(f[0], f[1])
    if precision == "fp64":
        orc = O.Simulation(xml, kernel, wall)
        assert orc.run(STEPS) == 0
        assert np.array_equal(f[0], orc.f())
