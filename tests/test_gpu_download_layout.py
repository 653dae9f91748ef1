"""Downloads into caller arrays that lie apart, one behind the other (copied as one) and a
mixture of both give the same bytes and leave what lies behind them alone."""
import numpy as np
import pytest

import ethersph_gb300 as sph
from ethersph_gb300 import scenes

pytestmark = pytest.mark.gpu

NAMES = ("rho", "p", "c", "mass", "gap")


def _layout(kind, n, dim):
    """Arrays of n rows and the block they were cut from; `mixed` leaves gaps after v and p."""
    widths = [("x", n * dim), ("v", n * dim)] + [(k, n) for k in NAMES]
    pad = {"apart": 3, "joined": 0, "mixed": 0}[kind]
    block = np.full(sum(w for _, w in widths) + 8 * 8, -7.0)
    out, at, used = {}, 0, np.zeros(block.size, bool)
    for k, w in widths:
        out[k] = block[at:at + w].reshape((n, dim) if k in "xv" else (n,))
        used[at:at + w] = True
        at += w + (5 if kind == "mixed" and k in ("v", "p") else pad)
    return out, block, used


@pytest.mark.parametrize("dim", (2, 3))
def test_download_layouts(dim):
    s = scenes.dam_break_2d(dx=0.05) if dim == 2 else scenes.dam_break_3d(dx=0.05)
    with sph.Simulation(s.params(), s.n_fluid, s.n_wall) as sim:
        for w in s.walls:
            sim.upload_walls(w)
        sim.upload_fluid(s.fluid)
        sim.step(1, 3)
        want = sim.download()
        for kind in ("apart", "joined", "mixed"):
            out, block, used = _layout(kind, s.n_fluid, dim)
            got = sim.download(s.n_fluid, out=out)
            for k in want:
                assert np.array_equal(got[k], want[k]), (kind, k)
            assert np.all(block[~used] == -7.0), kind
        for _ in range(10):  # past the use at which the handle pins its transfer words
            assert np.array_equal(sim.download()["x"], want["x"])
