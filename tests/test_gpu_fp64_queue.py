"""The work queue of the plain FP64 gathers: momentum draws its particles before it has waited
for the gather in front of it, so each gather of a step draws from a word of its own.

A batch whose scenes re-initialise at different steps launches momentum twice in a row, and
the stage timing repeats one gather; a draw counter left over from the launch in front would
skip or repeat particles.  Both are compared bit for bit with runs that launch it once.
"""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 24


def scenes_mod():
    from ethersph_gb300 import scenes
    return scenes


def developed(s, seed, reinit):
    rng = np.random.default_rng(seed)
    f = s.fluid
    f.x_vec_ += rng.uniform(-0.08, 0.08, f.x_vec_.shape) * s.meta["dx"]
    f.v_vec_[:] = rng.uniform(-0.05, 0.05, f.v_vec_.shape) * s.model.c_0_
    return dataclasses.replace(s, check=None, td=dataclasses.replace(s.td, density_reinitialized_interval_=reinit))


def alone(pkg, s, stages_after=None):
    with pkg.Simulation(s.params(), s.n_fluid, s.n_wall) as sim:
        for w in s.walls:
            sim.upload_walls(w)
        sim.upload_fluid(s.fluid)
        if stages_after:
            sim.step(1, stages_after)
            sim.time_stages(4)
            sim.step(1 + stages_after, STEPS - stages_after)
        else:
            sim.step(1, STEPS)
        return sim.download()


# launches of some 1,900 (a draw a warp), 10,600 (a block of six warps an SM) and 42,000
# particles (many draws a warp)
@pytest.mark.parametrize("dx", [0.05, 0.02, 0.01])
def test_scenes_that_reinitialise_apart_equal_themselves_alone(pkg, dx):
    from ethersph_gb300 import batch
    sc = scenes_mod()
    made = [developed(sc.dam_break_2d(dx=dx), 1, 2), developed(sc.dam_break_2d(dx=1.1 * dx), 2, 3),
            developed(sc.dam_break_2d(dx=1.7 * dx), 3, 5), developed(sc.dam_break_2d(dx=2 * dx), 4, 0)]
    need = [batch.footprint(s) for s in made]
    with batch.Batch(made[0].params(), *[sum(n[k] for n in need) + 8 for k in range(3)], len(made)) as bt:
        ids = [bt.add_scene(s, 1, STEPS) for s in made]
        bt.step(STEPS)
        bt.synchronize()
        got = [bt.download(k) for k in ids]
    for s, g in zip(made, got):
        ref = alone(pkg, s)
        for k in ref:
            assert np.array_equal(ref[k], g[k]), (s.meta["dx"], k)


@pytest.mark.parametrize("dx", [0.05, 0.013])
def test_timing_the_stages_leaves_the_run_as_it_is(pkg, dx):
    s = developed(scenes_mod().dam_break_2d(dx=dx), 5, 3)
    plain, timed = alone(pkg, s), alone(pkg, s, stages_after=10)
    for k in plain:
        assert np.array_equal(plain[k], timed[k]), k
