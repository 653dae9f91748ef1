"""The FP32-compensated form where the neighbour list's memory is refused.

The library's host unit is built once more with cudaMalloc replaced by one that refuses
requests above a limit the test sets: no device memory is used up.  Without a list every
particle walks the cells, in lanes and in threads, re-initialisation steps included, and the
state follows the FP64 form within the form's bar, 1e-4; a list that could not grow deeper
keeps its depth; the next upload or scene gets its list, and the state is then that of a
run that was never refused, bit for bit.
"""
import ctypes as C
import dataclasses
import importlib
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 6  # re-initialisations at 3 and 6

FAKE = """
#include <cuda_runtime.h>
#include <stdint.h>
extern "C" {
size_t sph_test_malloc_limit = SIZE_MAX;
int sph_test_malloc_refused = 0;
}
template <typename T>
cudaError_t limited_malloc(T** p, size_t bytes) {
    if (bytes > sph_test_malloc_limit) {
        ++sph_test_malloc_refused;
        return cudaErrorMemoryAllocation;
    }
    return cudaMalloc(p, bytes);
}
#define cudaMalloc limited_malloc
"""


@pytest.fixture(scope="module")
def limited(pkg, tmp_path_factory):
    from ethersph_gb300 import _abi
    recipe = importlib.import_module(pkg.__name__ + ".build")
    tmp = tmp_path_factory.mktemp("limited")
    (tmp / "fake.h").write_text(FAKE)
    api, obj, so = recipe.CSRC / "sph_api.cu", tmp / "sph_api.o", tmp / "liblimited.so"
    nvcc = [recipe.nvcc(), *recipe.ARCH]
    subprocess.run([*nvcc, *recipe.COMMON, *recipe.UNIT_FLAGS["sph_api.cu"], "-include", str(tmp / "fake.h"), "-c",
                    str(api), "-o", str(obj)], check=True, capture_output=True)
    others = [str(recipe.BUILD / (p.stem + ".o")) for p in sorted(recipe.CSRC.glob("*.cu")) if p != api]
    subprocess.run([*nvcc, "-shared", "-o", str(so), str(obj), *others], check=True, capture_output=True)
    lib = _abi.load_library(so)
    lib.limit = C.c_size_t.in_dll(lib, "sph_test_malloc_limit")
    lib.refused = C.c_int.in_dll(lib, "sph_test_malloc_refused")
    return lib


NO_LIMIT = C.c_size_t(-1).value


def developed(s):
    rng = np.random.default_rng(3)
    f = s.fluid
    f.x_vec_ += rng.uniform(-0.08, 0.08, f.x_vec_.shape) * s.meta["dx"]
    f.v_vec_[:] = rng.uniform(-0.05, 0.05, f.v_vec_.shape) * s.model.c_0_
    return dataclasses.replace(s, check=None, td=dataclasses.replace(s.td, density_reinitialized_interval_=3))


def make(name):
    from ethersph_gb300 import scenes as sc
    d3 = lambda dx: sc.dam_break_3d(dx=dx, tank=(0.6, 0.3, 0.4), column=(0.25, 0.2, 0.3))
    return developed({"dam": lambda: sc.dam_break_2d(dx=0.03), "heat": lambda: sc.natural_convection_2d(n=41),
                      "heat_25k": lambda: sc.natural_convection_2d(n=160), "dam_46k": lambda: sc.dam_break_2d(dx=0.0066),
                      "heat_45k": lambda: sc.natural_convection_2d(n=213), "dam_3d": lambda: d3(0.02),
                      "dam_3d_47k": lambda: d3(0.0068), "lid": lambda: sc.lid_driven_cavity_2d(n=37)}[name]())


def upload(sim, s):
    for w in s.walls:
        sim.upload_walls(w)
    sim.upload_fluid(s.fluid)


def plain(pkg, s, precision=1):
    with pkg.Simulation(s.params(precision=precision), s.n_fluid, s.n_wall) as sim:
        upload(sim, s)
        sim.step(1, STEPS)
        return sim.download()


def follows(got, ref):
    for k in ("x", "v", "rho", "t"):
        if k in ref:
            err = float(np.max(np.abs(got[k] - ref[k])) / np.max(np.abs(ref[k])))
            assert err <= 1e-4, (k, err)
    assert np.array_equal(got["mass"], ref["mass"])


@pytest.mark.parametrize("name", ["dam", "heat", "lid", "dam_3d", "heat_25k", "dam_46k", "heat_45k", "dam_3d_47k"])
def test_without_a_list_the_cells_are_walked(pkg, limited, name):
    s = make(name)
    with pkg.Simulation(s.params(precision=1), s.n_fluid, s.n_wall, lib=limited) as sim:
        upload(sim, s)
        limited.limit.value = 0
        limited.refused.value = 0
        try:
            sim.step(1, STEPS)
        finally:
            limited.limit.value = NO_LIMIT
        assert limited.refused.value > 0
        assert b"no device memory for the neighbour list" in limited.sph_last_error(sim.h)
        got = sim.download()
        tried = limited.refused.value
        sim.upload_fluid(s.fluid)  # and again, with memory
        sim.step(1, STEPS)
        again = sim.download()
        assert limited.refused.value == tried
    follows(got, plain(pkg, s, 0))
    ref = plain(pkg, s)
    for k in ref:
        assert np.array_equal(ref[k], again[k]), k


def test_a_list_that_cannot_deepen_keeps_its_depth(pkg, limited):
    from ethersph_gb300 import batch
    a, b = make("dam"), make("dam")
    b.fluid.gap_[:] *= 0.5  # asks for lists of four times the depth, which it does not fill
    need = [batch.footprint(s, 1) for s in (a, b)]
    with batch.Batch(a.params(precision=1), *[sum(n[k] for n in need) + 8 for k in range(3)], 2, lib=limited) as bt:
        ia = bt.add_scene(a, 1, STEPS)
        bt.step(2)
        bt.synchronize()
        ib = bt.add_scene(b, 1, STEPS)
        limited.limit.value = 2 * a.n_fluid * 48 * 4
        limited.refused.value = 0
        try:
            bt.step(STEPS)
            bt.synchronize()
        finally:
            limited.limit.value = NO_LIMIT
        assert limited.refused.value > 0
        assert b"more than 48 neighbours" in limited.sph_last_error(bt.h)
        got_a, got_b = bt.download(ia), bt.download(ib)
    for s, got in ((a, got_a), (b, got_b)):
        ref = plain(pkg, s)
        for k in ref:
            assert np.array_equal(ref[k], got[k]), k
