"""The FP64 sweeps' fixed-point pair sums against the oracle: every number of threads per
particle, values far below and beyond the range of the format (the general path), particles
of different volume, and terms of very different size in one sum.

Tolerance: both sides round each of at most 130 terms of a sum to 2^-52 of itself or better;
with the terms' absolute sum at most 1000 times the largest result, 130 x 2^-52 x 1000 =
3e-11 of that result.
"""
import numpy as np
import pytest

from oracle import oracle as O
from sphinxsys_gb300 import cases
from sphinxsys_gb300.dambreak import DamBreak

pytestmark = pytest.mark.gpu
TOL = 3e-11

# threads per particle: 4, 2, 1 in 2D; 8, 4, 2, 1 in 3D
SIZES = {"2d-4": (2, 0.025), "2d-2": (2, 0.0055), "2d-1": (2, 0.0045), "3d-8": (3, 0.06), "3d-4": (3, 0.03),
         "3d-2": (3, 0.025), "3d-1": (3, 0.02)}


def state(case, n, speed, compression, spread, seed):
    rng = np.random.default_rng(seed)
    d = case.dim
    v = speed * case.c0 * rng.uniform(-1, 1, (n, d))
    rho = 1.0 + compression * rng.uniform(-1, 1, n)
    if spread:  # most terms 1e6 times smaller than a few
        small = rng.uniform(size=n) < 0.9
        v[small] *= 1e-6
        rho[small] = 1.0 + (rho[small] - 1.0) * 1e-6
    return {"Velocity": v, "Density": rho, "Force": np.zeros((n, d)), "DensityChangeRate": np.zeros(n)}


def compare(case, speed, compression, spread=False, volume=None):
    sim, oc = DamBreak(case), O.OracleCase(case)
    n = sim.water_block.n
    jitter = np.random.default_rng(1).uniform(-0.2, 0.2, (n, case.dim)) * case.dp
    st = state(case, n, speed, compression, spread, 2)
    st["Position"] = sim.water_block.download("Position").reshape(n, case.dim) + jitter
    if volume is not None:
        st["VolumetricMeasure"] = sim.water_block.download("VolumetricMeasure") * volume(n)
    for k, x in st.items():
        sim.water_block.upload(k, x)
        oc.set(k, x)
    sim.update_configuration()
    oc.update_cell_linked_list(O.FLUID)
    oc.update_configuration()
    dt = 0.1 * case.dp / case.c0
    sim.fluid_pressure_relaxation.exec(dt)
    oc.integration_1st_half(dt)
    names = ["Force", "Velocity", "Pressure", "DensityChangeRate"]
    got = {k + "/1st": (sim.water_block.download(k), oc.get(k)) for k in names}
    # the same velocities on both sides
    sim.water_block.upload("Velocity", st["Velocity"])
    oc.set("Velocity", st["Velocity"])
    for b in (sim.water_block.upload, oc.set):
        b("DensityChangeRate", np.zeros(n))
    sim.fluid_density_relaxation.exec(dt)
    oc.integration_2nd_half(dt)
    got.update({k + "/2nd": (sim.water_block.download(k), oc.get(k)) for k in ("Force", "Density", "DensityChangeRate")})
    for k, (a, b) in got.items():
        a, b = np.asarray(a).ravel(), np.asarray(b).ravel()
        assert np.max(np.abs(a - b)) <= TOL * np.max(np.abs(b)), (k, np.max(np.abs(a - b)) / np.max(np.abs(b)))


def build(name):
    dim, dp = SIZES[name]
    return cases.dambreak_2d(dp) if dim == 2 else cases.dambreak_3d(dp)


@pytest.mark.parametrize("name", list(SIZES))
def test_every_number_of_threads(name):
    compare(build(name), 0.05, 1e-2)


@pytest.mark.parametrize("name", ["2d-4", "3d-8", "3d-1"])
@pytest.mark.parametrize("speed,compression", [(1e-4, 1e-4), (0.3, 0.1), (0.05, 0.24), (1.5, 0.3)])
def test_small_values_and_the_general_path(name, speed, compression):
    compare(build(name), speed, compression)


@pytest.mark.parametrize("name", ["2d-1", "3d-4", "3d-1"])
def test_terms_of_different_size(name):
    compare(build(name), 0.2, 0.1, spread=True)


@pytest.mark.parametrize("name", ["2d-4", "3d-1"])
def test_particles_of_different_volume(name):
    compare(build(name), 0.05, 1e-2, volume=lambda n: 1.0 + 0.1 * (np.arange(n) % 3))
