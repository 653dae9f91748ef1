"""Downloads into arrays that touch but are page-locked one by one: each is copied alone (one
copy must not span two registrations)."""
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("locked", ["every array", "every other array", "every third array"])
def test_adjacent_registrations(pkg, locked):
    import torch
    from ethersph_gb300 import scenes
    s = scenes.natural_convection_2d(n=128)  # 16,384 particles: every array a multiple of 64 KiB
    n, every = s.n_fluid, {"every array": 1, "every other array": 2, "every third array": 3}[locked]
    names = {"x": 2, "v": 2, "rho": 1, "p": 1, "c": 1, "mass": 1, "gap": 1, "t": 1, "kappa": 1, "cp": 1}
    block = np.frombuffer(mmap.mmap(-1, 8 * n * sum(names.values())), dtype=np.float64)
    assert block.ctypes.data % mmap.PAGESIZE == 0 and 8 * n % mmap.PAGESIZE == 0
    block[:] = 0.0
    rt = torch.cuda.cudart()
    out, registered, at = {}, [], 0
    try:
        for q, (k, d) in enumerate(names.items()):
            a = block[at * n:(at + d) * n]
            out[k] = a.reshape(n, 2) if d == 2 else a
            if q % every == 0:
                assert int(rt.cudaHostRegister(a.ctypes.data, a.nbytes, 0)) == 0
                registered.append(a.ctypes.data)
            at += d
        with pkg.Simulation(s.params(), s.n_fluid, s.n_wall) as sim:
            for w in s.walls:
                sim.upload_walls(w)
            sim.upload_fluid(s.fluid)
            sim.step(1, 10)
            got, ref = sim.download(out=out), sim.download()
        for k in ref:
            assert np.array_equal(got[k], ref[k]), k
    finally:
        for p in registered:
            assert int(rt.cudaHostUnregister(p)) == 0
