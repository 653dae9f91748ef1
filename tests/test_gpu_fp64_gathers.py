"""The cooperative gathers of the plain FP64 form against the oracle, at the places where
they can go wrong: particle counts around a warp's and a block's share, neighbours beyond
the capacity of a particle's list (several passes), particles clamped into the edge cells
from near and from far outside the grid, periodic rows, non-uniform spacings, every kernel.

The flow is developed (particle disorder, velocities of a twentieth of the sound speed), so
fields are compared relative to magnitudes that do not cancel: an FP64 step rounds each term
to some 1e-16, sums of up to a few hundred terms over 3 steps stay below 1e-12.
"""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scenes_mod():
    from ethersph_gb300 import scenes
    return scenes


def developed(s, seed=3):
    rng = np.random.default_rng(seed)
    f = s.fluid
    f.x_vec_ += rng.uniform(-0.08, 0.08, f.x_vec_.shape) * s.meta["dx"]
    if s.periodic_x:
        f.x_vec_[:, 0] %= s.meta["L"]
    f.v_vec_[:] = rng.uniform(-0.05, 0.05, f.v_vec_.shape) * s.model.c_0_
    return dataclasses.replace(s, check=None, td=dataclasses.replace(s.td, density_reinitialized_interval_=3))


def subset(s, n):
    f = s.fluid
    g = type(f)(n, f.x_vec_.shape[1])
    for name in f._vector_fields + f._scalar_fields:
        getattr(g, name)[:] = getattr(f, name)[:n]
    return dataclasses.replace(s, fluid=g)


def squeezed(s, factor):
    # the same particles closer together: factor^dim times the neighbours within r_cut
    s.fluid.x_vec_ *= factor
    return s


def beyond(s, cells):
    # a grid that ends inside the fluid; some particles lie `cells` cells outside it
    f = s.fluid
    f.x_vec_[:, 1] += np.where(np.arange(len(f)) % 7 == 0, cells * s.kernel.influence_radius_ / 3.0, 0.0)
    hi = list(s.domain_hi)
    hi[1] = 0.4
    return dataclasses.replace(s, domain_hi=tuple(hi))


def make(name):
    sc = scenes_mod()
    d2 = lambda **k: sc.dam_break_2d(dx=0.05, **k)
    d3 = lambda: sc.dam_break_3d(dx=0.05, tank=(0.6, 0.3, 0.4), column=(0.25, 0.2, 0.3))
    if name.startswith("n"):
        return developed(subset(d2(), int(name[1:])))
    if name in ("CubicSpline", "Gaussian", "WendlandC2", "WendlandC4"):
        return developed(d2(kernel=name))
    if name == "gaps":
        s = developed(d2())
        s.fluid.gap_ *= np.random.default_rng(1).uniform(0.9, 1.1, s.n_fluid)
        return s
    return {"overflow_2d": lambda: squeezed(developed(d2()), 0.5), "overflow_3d": lambda: squeezed(developed(d3()), 0.7),
            "beyond_2d": lambda: beyond(developed(d2()), 5), "far_2d": lambda: beyond(developed(d2()), 200),
            "beyond_3d": lambda: beyond(developed(d3()), 4),
            "periodic": lambda: developed(sc.poiseuille_periodic_2d(n_across=8, length_factor=1.25)),
            "heat": lambda: developed(sc.natural_convection_2d(n=37)),
            "lid": lambda: developed(sc.lid_driven_cavity_2d(n=33))}[name]()


def rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


@pytest.mark.parametrize("name", ["n1", "n3", "n4", "n5", "n31", "n33", "n129", "n257", "overflow_2d", "overflow_3d",
                                  "beyond_2d", "far_2d", "beyond_3d", "periodic", "heat", "lid", "gaps", "CubicSpline",
                                  "Gaussian", "WendlandC2", "WendlandC4"])
@pytest.mark.parametrize("sub", [0, 1])
def test_fp64_gathers_match_oracle(pkg, orc, name, sub):
    s = make(name)
    prm = s.params(cell_subdivision=sub)
    with pkg.Simulation(prm, s.n_fluid, s.n_wall) as sim:
        for w in s.walls:
            sim.upload_walls(w)
        sim.upload_fluid(s.fluid)
        sim.step(1, 3)
        got = sim.download()
    fluid, walls = orc.scene_arrays(s)
    ref = orc.run(prm, fluid, walls, 1, 3, mode=orc.GATHER, threads=8)
    for k in ("x", "v", "rho") + (("t",) if "t" in got else ()):
        assert rel(got[k], ref[k]) <= 1e-12, (k, rel(got[k], ref[k]))


@pytest.mark.parametrize("n", [1, 9, 800, 5000])
def test_fp64_scene_is_the_same_alone_and_beside_others(pkg, n):
    # bitwise: a particle's sums do not depend on the block size or on its warp's other particles
    from ethersph_gb300 import batch
    sc = scenes_mod()
    a = developed(subset(sc.dam_break_2d(dx=0.02), n))
    b = squeezed(developed(sc.dam_break_2d(dx=0.03), 5), 0.5)
    with pkg.Simulation(a.params(), a.n_fluid, a.n_wall) as sim:
        for w in a.walls:
            sim.upload_walls(w)
        sim.upload_fluid(a.fluid)
        sim.step(1, 4)
        alone = sim.download()
    with batch.Batch(a.params(), 60_000, 400_000, 60_000, 8) as bt:
        bt.add_scene(b, 1, 4)
        k = bt.add_scene(a, 1, 4)
        bt.add_scene(b, 1, 4)
        bt.step(4)
        bt.synchronize()
        beside = bt.download(k)
    for f in alone:
        assert np.array_equal(alone[f], beside[f]), f
