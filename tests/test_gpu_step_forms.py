"""The GZS link list and the one-launch time step at sizes where their blocks end
raggedly: FP64 against the CPU oracle bit for bit, the shifted forms within their
rounding."""

import numpy as np
import pytest

from hemepure_b200 import lbm, vessels
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# Largest difference over the field's largest value.  Storing a deviation rounds it to
# 2^-24 (FP32) or 2^-11 (FP16) of itself at most, every step; such errors are unbiased and
# add like a random walk.  Twice that: the collision rounds too, and wall shear stress is
# a difference of such values.  (Seen: 0.66 and 0.16 of it.  Bounce-back in place of a BFL
# or GZS wall moves wall velocities by 0.16 and more, BFL in place of GZS by 0.008.)
TOL = {"fp32": 2 * np.sqrt(40) * 2.0 ** -24, "fp16": 2 * np.sqrt(40) * 2.0 ** -11}


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
    """Velocity everywhere, and wall shear stress at the wall records on its own, so
    that a fault of the boundary links alone shows."""
    xml = pipe_case(tmp_path, radius, length, True, True)
    gpu, orc = lbm.LBM(xml, kernel="TRT", wall=wall, precision=precision), O.Simulation(xml, "TRT", wall)
    gpu.step(40, macro=True)
    assert orc.run(40, macro=True) == 0
    (_, u, w), (_, u_ref, w_ref) = gpu.GetPropertyCache(), orc.macro()
    at = w_ref < 1e300
    assert at.any() and np.array_equal(at, w < 1e300)
    err = {"u": np.abs(u - u_ref).max() / np.abs(u_ref).max(), "u_wall": np.abs(u - u_ref)[at].max() / np.abs(u_ref[at]).max(),
           "wss": np.abs(w - w_ref)[at].max() / w_ref[at].max()}
    print(f"{precision} {wall} radius {radius}: {err}")
    assert max(err.values()) <= TOL[precision], err


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
