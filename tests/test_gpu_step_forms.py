"""The GZS link list and the one-launch time step at sizes where their blocks end
raggedly: FP64 against the CPU oracle bit for bit, the shifted forms within their
rounding."""

import numpy as np
import pytest

from hemepure_b200 import lbm, vessels
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# FP32: each step rounds a deviation of order 1e-2 to 2^-24 of itself and 40 steps add
# at most linearly, against a velocity of order 1e-3; FP16 storage likewise with 2^-11.
U_TOL = {"fp32": 40 * 2.0 ** -24 * 1e-2 / 1e-3 * 4, "fp16": 40 * 2.0 ** -11 * 1e-2 / 1e-3 * 4}


def pipe_case(tmp, radius, length, velocity, trt):
    v = vessels.Pipe(radius, length)
    xml, gmy = str(tmp / "c.xml"), str(tmp / "c.gmy")
    vessels.voxelise(v, gmy)
    inlet = vessels.VelocityBC(0.01) if velocity else vessels.PressureBC(1.0005)
    vessels.write_case_xml(xml, "c.gmy", v, vessels.CaseUnits(tau=0.8), 100, [inlet], [vessels.PressureBC(0.9995)],
                           relaxation_parameter=3.0 / 16.0 if trt else None)
    return xml


@pytest.mark.parametrize("radius,length", [(2.3, 5), (4.1, 9), (7.6, 33)])
@pytest.mark.parametrize("kernel", ["LBGK", "TRT"])
@pytest.mark.parametrize("wall", ["GZS", "BFL", "SBB"])
@pytest.mark.parametrize("velocity", [False, True])
def test_step_forms_bit_exact(tmp_path, radius, length, kernel, wall, velocity):
    """First step (no gather), steady-state steps, an output step, and on from it."""
    xml = pipe_case(tmp_path, radius, length, velocity, kernel == "TRT")
    gpu, orc = lbm.LBM(xml, kernel=kernel, wall=wall), O.Simulation(xml, kernel, wall)
    for n in (1, 6, 13):
        gpu.step(n, macro=True)
        assert orc.run(n, macro=True) == 0
        np.testing.assert_array_equal(gpu.GetFOld(), orc.f())
        for a, b in zip(gpu.GetPropertyCache(), orc.macro()):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("wall", ["GZS", "BFL", "SBB"])
@pytest.mark.parametrize("radius,length", [(2.3, 5), (7.6, 33), (6.2, 70)])
def test_shifted_forms_follow_the_oracle(tmp_path, precision, wall, radius, length):
    """Pairs of sites across run ends, partial tiles and boundary records."""
    xml = pipe_case(tmp_path, radius, length, True, True)
    gpu, orc = lbm.LBM(xml, kernel="TRT", wall=wall, precision=precision), O.Simulation(xml, "TRT", wall)
    gpu.step(40, macro=True)
    assert orc.run(40, macro=True) == 0
    u, ref = gpu.GetPropertyCache()[1], orc.macro()[1]
    assert np.abs(u - ref).max() <= U_TOL[precision] * np.abs(ref).max()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("wall", ["GZS", "BFL"])
def test_first_and_output_steps_take_two_kernels(tmp_path, precision, wall):
    """One for the plain bulk sites and one for the boundary, which run side by side
    (a kernel for each kind of boundary work one after the other made an output step a
    quarter longer than before them); a step in between is one launch."""
    sim = lbm.LBM(pipe_case(tmp_path, 7.6, 33, True, True), kernel="TRT", wall=wall, precision=precision)
    for macro, launches in ((False, 2), (False, 1), (True, 2), (False, 1)):
        sim.step(1, macro=macro)
        assert sim.last_step_timing()[1] == launches
