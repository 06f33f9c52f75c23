"""The CK half steps' fixed-point sums against their general path.  The pair geometry is kept
between relation updates and used while the positions are those it was made from; moving one
particle by a rounding unit after that sends the same half steps through FP64 sums from the
current positions.  So does a value outside the fixed-point range.

Tolerance: both paths round each of at most 130 terms of a sum to 2^-52 or better; with the
terms' absolute sum at most 1000 times the largest result, 130 x 2^-52 x 1000 = 3e-11 of it.
"""
import numpy as np
import pytest

from sphinxsys_gb300 import cases
from sphinxsys_gb300.dambreak import DamBreakCKNested

pytestmark = pytest.mark.gpu
TOL = 3e-11
OUT = ("Velocity", "Force", "Pressure", "Density", "Compression", "CompressionRate", "Displacement")


def half_steps(case, speed, rate, nudge):
    sim = DamBreakCKNested(case)
    b, rng = sim.water_block, np.random.default_rng(3)
    n, d = b.n, case.dim
    x = b.download("Position").reshape(n, d) + rng.uniform(-0.2, 0.2, (n, d)) * case.dp
    v = speed * case.c0 * rng.uniform(-1, 1, (n, d))
    dt = 0.1 * case.dp / case.c0

    def load():
        sim.setup.exec()
        b.upload("Velocity", v)
        b.upload("Force", np.zeros((n, d)))
        b.upload("CompressionRate", rate / dt * rng2.uniform(-1, 1, n))

    b.upload("Position", x)
    b.updateCellLinkedList()
    sim.fp64.water_block_inner.updateConfiguration()
    sim.fp64.water_wall_contact.updateConfiguration()
    sim.regularization.exec()
    comp, rho = b.download("Compression"), b.download("Density")
    sim.setup.exec()
    sim.correction.exec()
    rng2 = np.random.default_rng(4)
    load()
    sim.first_half.exec(dt)  # makes the pair geometry
    b.upload("Compression", comp)
    b.upload("Density", rho)
    if nudge:
        x[n // 2, 0] = np.nextafter(x[n // 2, 0], np.inf)
        b.upload("Position", x)
    rng2 = np.random.default_rng(5)
    load()
    sim.first_half.exec(dt)
    sim.second_half.exec(dt)
    return {k: b.download(k) for k in OUT}


# threads per particle 4, 2, 1 in 2D; 8, 4, 2, 1 in 3D
CASES = [cases.dambreak_2d(0.03), cases.dambreak_2d(0.0045), cases.dambreak_2d(0.0035), cases.dambreak_3d(0.06),
         cases.dambreak_3d(0.026), cases.dambreak_3d(0.02), cases.dambreak_3d(0.0165)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
@pytest.mark.parametrize("speed,rate", [(0.05, 1e-2), (1e-5, 1e-6), (0.2, 0.6)])
def test_fixed_point_matches_general_path(case, speed, rate):
    a, b = (half_steps(case, speed, rate, nudge) for nudge in (False, True))
    for k in OUT:
        assert np.max(np.abs(a[k] - b[k])) <= TOL * max(np.max(np.abs(b[k])), 1e-300), k


def once_per_step(case, nudge, uneven):
    """Compression sum with the pair geometry, then correction and indication from it."""
    sim = DamBreakCKNested(case)
    b, rng = sim.water_block, np.random.default_rng(6)
    n, d = b.n, case.dim
    x = b.download("Position").reshape(n, d) + rng.uniform(-0.2, 0.2, (n, d)) * case.dp
    b.upload("Position", x)
    b.updateCellLinkedList()
    sim.fp64.water_block_inner.updateConfiguration()
    sim.fp64.water_wall_contact.updateConfiguration()
    sim.regularization.exec()
    out = {"fused sum": b.download("CompressionSummation")}
    if nudge:
        x[n // 2, 0] = np.nextafter(x[n // 2, 0], np.inf)
        b.upload("Position", x)
    sim.setup.exec()
    if uneven:  # volumes of a factor of two around the first particle's
        b.upload("VolumetricMeasure", b.download("VolumetricMeasure") * rng.uniform(0.7, 1.4, n))
    sim.regularization.exec()
    sim.correction.exec()
    for k in ("first", "again"):
        sim.indication.exec()
        out[k] = b.download("PositionDivergence")
        out[k + " indicator"] = b.download("Indicator")
    out["sum"] = b.download("CompressionSummation")
    out["correction"] = b.download("LinearCorrectionMatrix")
    return out


@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
@pytest.mark.parametrize("uneven", [False, True])
def test_once_per_step_matches_general_path(case, uneven):
    """The same tolerance: 3e-14 for a sum, and a correction matrix (the regularised inverse of
    one) of a condition number squared below 1000."""
    a, b = (once_per_step(case, nudge, uneven) for nudge in (False, True))
    for k in a:
        assert np.max(np.abs(a[k] - b[k])) <= TOL * np.max(np.abs(b[k])), k
    assert np.max(np.abs(a["fused sum"] - a["sum"])) <= TOL * np.max(np.abs(a["sum"]))
