"""The FP32-compensated gathers run with lanes sharing a particle on small launches and with a
thread a particle on large ones; both form the same sums in the same order.  A scene alone
(lanes) and beside a scene of 45,000 or more particles (threads) is the same, bit for bit:
lists of every length modulo eight, lists that do not fit (rows of more than 16 neighbours,
more neighbours than the list holds), walls, heat, periodic rows, three dimensions.
"""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scenes_mod():
    from ethersph_gb300 import scenes
    return scenes


def developed(s, seed=3, squeeze=1.0):
    rng = np.random.default_rng(seed)
    f = s.fluid
    f.x_vec_ += rng.uniform(-0.08, 0.08, f.x_vec_.shape) * s.meta["dx"]
    f.x_vec_ *= squeeze
    if s.periodic_x:
        f.x_vec_[:, 0] %= s.meta["L"]
    f.v_vec_[:] = rng.uniform(-0.05, 0.05, f.v_vec_.shape) * s.model.c_0_
    return dataclasses.replace(s, check=None, td=dataclasses.replace(s.td, density_reinitialized_interval_=3))


def pair(name):
    sc = scenes_mod()
    d3 = lambda dx: sc.dam_break_3d(dx=dx, tank=(0.6, 0.3, 0.4), column=(0.25, 0.2, 0.3))
    return {"dam": lambda: (developed(sc.dam_break_2d(dx=0.03)), developed(sc.dam_break_2d(dx=0.0066))),
            "squeezed": lambda: (developed(sc.dam_break_2d(dx=0.03), squeeze=0.3),
                                 developed(sc.dam_break_2d(dx=0.0066), squeeze=0.98)),
            "heat": lambda: (developed(sc.natural_convection_2d(n=41)), developed(sc.natural_convection_2d(n=213))),
            "lid": lambda: (developed(sc.lid_driven_cavity_2d(n=37)), developed(sc.lid_driven_cavity_2d(n=213))),
            "periodic": lambda: (developed(sc.poiseuille_periodic_2d(n_across=10)),
                                 developed(sc.poiseuille_periodic_2d(n_across=107))),
            "dam_3d": lambda: (developed(d3(0.02)), developed(d3(0.0068))),
            "squeezed_3d": lambda: (developed(d3(0.02), squeeze=0.6), developed(d3(0.0068)))}[name]()


@pytest.mark.parametrize("name", ["dam", "squeezed", "heat", "lid", "periodic", "dam_3d", "squeezed_3d"])
def test_lanes_and_threads_give_the_same_bits(pkg, name):
    from ethersph_gb300 import batch
    a, big = pair(name)
    assert a.n_fluid < 40_000 < 45_000 <= big.n_fluid
    with pkg.Simulation(a.params(precision=1), a.n_fluid, a.n_wall) as sim:
        for w in a.walls:
            sim.upload_walls(w)
        sim.upload_fluid(a.fluid)
        sim.step(1, 5)
        alone = sim.download()
    need = [batch.footprint(s, 1) for s in (a, big)]
    with batch.Batch(a.params(precision=1), *[sum(n[k] for n in need) + 8 for k in range(3)], 4) as bt:
        bt.add_scene(big, 1, 5)
        k = bt.add_scene(a, 1, 5)
        bt.step(5)
        bt.synchronize()
        beside = bt.download(k)
    for f in alone:
        assert np.array_equal(alone[f], beside[f]), f


def beside_medium(name):
    sc = scenes_mod()
    d3 = lambda dx: sc.dam_break_3d(dx=dx, tank=(0.6, 0.3, 0.4), column=(0.25, 0.2, 0.3))
    big = {"dam": lambda: sc.dam_break_2d(dx=0.0085), "squeezed": lambda: sc.dam_break_2d(dx=0.0085),
           "heat": lambda: sc.natural_convection_2d(n=160), "lid": lambda: sc.lid_driven_cavity_2d(n=160),
           "periodic": lambda: sc.poiseuille_periodic_2d(n_across=80), "dam_3d": lambda: d3(0.0088),
           "squeezed_3d": lambda: d3(0.0088)}[name]()
    return pair(name)[0], developed(big)


@pytest.mark.parametrize("name", ["dam", "squeezed", "heat", "lid", "periodic", "dam_3d", "squeezed_3d"])
def test_rows_with_momentum_threads_give_the_same_bits(pkg, name):
    # launches of 19,457 (3D: 14,593) to 39,999 particles: continuity in lanes, which lists the
    # particles near walls and without a list for momentum's threads
    from ethersph_gb300 import batch
    a, big = beside_medium(name)
    assert 20_000 < big.n_fluid and a.n_fluid + big.n_fluid < 40_000
    with pkg.Simulation(a.params(precision=1), a.n_fluid, a.n_wall) as sim:
        for w in a.walls:
            sim.upload_walls(w)
        sim.upload_fluid(a.fluid)
        sim.step(1, 5)
        alone = sim.download()
    need = [batch.footprint(s, 1) for s in (a, big)]
    with batch.Batch(a.params(precision=1), *[sum(n[k] for n in need) + 8 for k in range(3)], 4) as bt:
        bt.add_scene(big, 1, 5)
        k = bt.add_scene(a, 1, 5)
        bt.step(5)
        bt.synchronize()
        beside = bt.download(k)
    for f in alone:
        assert np.array_equal(alone[f], beside[f]), f


@pytest.mark.parametrize("name", ["heat", "dam_3d"])
def test_packed_continuity_gives_the_same_bits(pkg, name):
    # 136,193 particles or more: continuity's thread kernel with fewer registers, which saves a
    # wave of blocks here (2D up to 175,104 particles, 3D up to 155,648)
    from ethersph_gb300 import batch
    a = pair(name)[0]
    sc = scenes_mod()
    big = developed(sc.natural_convection_2d(n=380) if name == "heat" else
                    sc.dam_break_3d(dx=0.0047, tank=(0.6, 0.3, 0.4), column=(0.25, 0.2, 0.3)))
    assert 136_193 <= big.n_fluid and a.n_fluid + big.n_fluid <= 155_648
    with pkg.Simulation(a.params(precision=1), a.n_fluid, a.n_wall) as sim:
        for w in a.walls:
            sim.upload_walls(w)
        sim.upload_fluid(a.fluid)
        sim.step(1, 5)
        alone = sim.download()
    need = [batch.footprint(s, 1) for s in (a, big)]
    with batch.Batch(a.params(precision=1), *[sum(n[k] for n in need) + 8 for k in range(3)], 4) as bt:
        bt.add_scene(big, 1, 5)
        k = bt.add_scene(a, 1, 5)
        bt.step(5)
        bt.synchronize()
        beside = bt.download(k)
    for f in alone:
        assert np.array_equal(alone[f], beside[f]), f
