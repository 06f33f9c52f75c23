"""The mixed solver's forms for few particles: lists and sweeps shared by lanes (dam break),
and the sub-steps of a step enqueued by plan.  Both give the bits of the one-thread,
step-by-step forms: the cell sweeps of strategy 1 run one thread a particle, and profiling
takes the host through every sub-step.
"""
import numpy as np
import pytest

from sphinxsys_gb300 import cases
from sphinxsys_gb300 import native as N
from sphinxsys_gb300.dambreak import MixedPrecisionDamBreak
from sphinxsys_gb300.taylor_green import MixedPrecisionTaylorGreen

pytestmark = pytest.mark.gpu
FIELDS = ("Position", "Velocity", "Density", "Pressure")


def advance(sim, steps, profiled):
    if profiled:
        sim.set_profiling(True)
    subs = [sim.advection_step() for _ in range(steps)]
    if hasattr(sim, "fp64"):
        sim.sync_fp64()
        body = sim.fp64.water_block
    else:
        sim.download()
        body = sim.water_block
    return subs, sim.physical_time, [body.download(k) for k in FIELDS]


def same(a, b):
    assert a[0] == b[0] and a[1] == b[1]
    for x, y, k in zip(a[2], b[2], FIELDS):
        assert np.array_equal(x, y), k


# either side of 100, 200 particles per SM (152 SMs) and a handful of particles
@pytest.mark.parametrize("case", [cases.dambreak_2d(0.1), cases.dambreak_2d(0.0085), cases.dambreak_2d(0.008),
                                  cases.dambreak_3d(0.12), cases.dambreak_3d(0.037), cases.dambreak_3d(0.0355),
                                  cases.dambreak_3d(0.0295), cases.dambreak_3d(0.028)], ids=lambda c: c.name)
def test_lanes_and_plan_match_one_thread(case):
    same(advance(MixedPrecisionDamBreak(case), 4, False), advance(MixedPrecisionDamBreak(case, strategy=1), 4, True))


@pytest.mark.parametrize("case", [cases.dambreak_2d(), cases.dambreak_3d_reference(0.06), cases.dambreak_2d(0.002)],
                         ids=lambda c: c.name)  # both loop styles
def test_plan_matches_step_by_step(case):
    same(advance(MixedPrecisionDamBreak(case), 6, False), advance(MixedPrecisionDamBreak(case), 6, True))


@pytest.mark.parametrize("case", [cases.taylor_green_2d(50), cases.taylor_green_3d(24)], ids=lambda c: c.name)
def test_periodic_plan_matches_step_by_step(case):
    same(advance(MixedPrecisionTaylorGreen(case), 6, False), advance(MixedPrecisionTaylorGreen(case), 6, True))


@pytest.mark.parametrize("case", [cases.dambreak_2d(0.1), cases.dambreak_3d(0.12)], ids=lambda c: c.name)
def test_download_widens_every_float_exactly(case):
    """The download converts by integer instructions: zeros, subnormals and the limits too."""
    sim = MixedPrecisionDamBreak(case)
    body = sim.fp64.water_block
    special = np.array([0.0, -0.0, 1e-45, -1e-45, 1.1754942e-38, 1.17549435e-38, -5e-39, 3.4028235e38, -1.0, 0.1, 7e-30],
                       np.float32)
    values = np.resize(special, (body.n, case.dim)).astype(np.float64)
    for k in ("Velocity", "Force"):
        body.upload(k, values)
    N.call("sphx_mp_upload", sim.handle, body.handle)
    for k in ("Velocity", "Force"):
        body.upload(k, np.ones_like(values))
    sim.sync_fp64()
    for k in ("Velocity", "Force"):
        got = np.asarray(body.download(k)).reshape(values.shape)
        assert np.array_equal(got, values) and np.array_equal(np.signbit(got), np.signbit(values)), k
