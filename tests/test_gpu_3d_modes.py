"""Every solve variant in three dimensions, re-initialisation steps included: walls without
background pressure, walls with a velocity and background pressure, heat with thermostatic
walls.  FP64 against the oracle (a developed flow: no field is a small residual; 1e-12 after
three steps as in the tests of the gathers), the FP32-compensated form against FP64 within its
bar, 1e-4, in lanes and in threads.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 3


def box(mode, n, kernel="WendlandC2", seed=3):
    """A cube of n^3 particles between three layers of walls, every particle displaced and moving."""
    from ethersph_gb300 import _abi, scenes as sc
    from ethersph_gb300.types import (CommonLiquidParticles, CommonWeaklyCompressibleLiquidModel,
                                      CompulsiveWallParticles, DensityReinitializedFixedTimeIntervalForwardEuler,
                                      SmoothKernel, StaticVelocityWallParticles, ThermalLiquidParticles,
                                      ThermalWeaklyCompressibleLiquidModel, ThermostaticWallParticles)
    rng = np.random.default_rng(seed)
    dx = 1.0 / n
    rc = 3.0 * dx
    kern = SmoothKernel(rc, 3, kernel)
    c0, rho0, mu, g = 10.0, 1.0, 0.02, np.array([0.0, -1.0, 0.0])
    thermal = mode == "heat"
    if thermal:
        model = ThermalWeaklyCompressibleLiquidModel(rho0, c0, 0.02 * rho0 * c0 * c0, 7, mu, g, t_0_=0.5, kappa_0_=1.0,
                                                     cp_=30.0, beta_=1.0)
    else:
        model = CommonWeaklyCompressibleLiquidModel(rho0, c0, 0.001 * rho0 * c0 * c0, 7, mu, g)
    td = DensityReinitializedFixedTimeIntervalForwardEuler(0.05 * kern.h_ / c0, 100, 100, 100, 2)
    f = (ThermalLiquidParticles if thermal else CommonLiquidParticles)(n ** 3, 3)
    f.x_vec_[:] = sc.lattice_3d(0.0, 0.0, 0.0, n, n, n, dx) + rng.uniform(-0.08, 0.08, (n ** 3, 3)) * dx
    f.v_vec_[:] = rng.uniform(-0.05, 0.05, (n ** 3, 3)) * c0
    f.rho_[:] = rho0
    f.p_[:], f.c_[:] = sc._eos(f.rho_, model)
    f.mass_[:] = rho0 * dx ** 3
    f.gap_[:] = dx
    if thermal:
        f.t_[:] = rng.uniform(0.2, 0.8, n ** 3)
        f.kappa_[:] = rng.uniform(0.8, 1.2, n ** 3)
        f.cp_[:] = 30.0

    def side(cls, axis, far, t=3):
        lo, count = [0.0, 0.0, 0.0], [n, n, n]
        lo[axis], count[axis] = (1.0 if far else -t * dx), t
        normal = [0.0, 0.0, 0.0]
        normal[axis] = -1.0 if far else 1.0
        w = sc._walls(cls, sc.lattice_3d(*lo, *count, dx), normal, dx)
        if cls is ThermostaticWallParticles:
            w.t_[:] = 1.0 - far
            w.kappa_[:] = 1.0
        if cls is StaticVelocityWallParticles and axis == 1 and far:
            w.v_vec_[:] = [1.0, 0.0, 0.3]
        return w

    def sides(cls, axes):
        return cls.vcat(*[side(cls, a, far) for a in axes for far in (False, True)])

    if thermal:
        walls = [sides(CompulsiveWallParticles, (1, 2)), sides(ThermostaticWallParticles, (0,))]
        solve = _abi.SOLVE_FLUID_COMPULSIVE_THERMOSTATIC_WALL
    elif mode == "velocity":
        walls, solve = [sides(StaticVelocityWallParticles, (0, 1, 2))], _abi.SOLVE_FLUID_VELOCITY_WALL
    else:
        walls, solve = [sides(CompulsiveWallParticles, (0, 1, 2))], _abi.SOLVE_FLUID_WALL
    lo, hi = (-2 * rc,) * 3, (1.0 + 2 * rc,) * 3
    return sc.Scene("box_" + mode, f, walls, kern, model, td, solve, None, lo, hi, meta=dict(dx=dx))


def run(pkg, s, precision):
    with pkg.Simulation(s.params(precision=precision), s.n_fluid, s.n_wall) as sim:
        for w in s.walls:
            sim.upload_walls(w)
        sim.upload_fluid(s.fluid)
        sim.step(1, STEPS)
        return sim.download()


def close(got, ref, tol):
    for k in ("x", "v", "rho", "t"):
        if k in got:
            err = float(np.max(np.abs(got[k] - ref[k])) / np.max(np.abs(ref[k])))
            assert err <= tol, (k, err)


@pytest.mark.parametrize("kernel", ["CubicSpline", "Gaussian", "WendlandC2", "WendlandC4"])
@pytest.mark.parametrize("mode", ["walls", "velocity", "heat"])
def test_fp64_matches_oracle(pkg, orc, mode, kernel):
    s = box(mode, 9, kernel)
    fluid, walls = orc.scene_arrays(s)
    ref = orc.run(s.params(), fluid, walls, 1, STEPS, mode=orc.GATHER, threads=8)
    close(run(pkg, s, 0), ref, 1e-12)


@pytest.mark.parametrize("n", [9, 26, 37], ids=["lanes", "rows", "threads"])
@pytest.mark.parametrize("mode", ["walls", "velocity", "heat"])
def test_fp32_follows_fp64(pkg, mode, n):
    s = box(mode, n)
    close(run(pkg, s, 1), run(pkg, s, 0), 1e-4)
