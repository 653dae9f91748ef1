"""bench.py counts the kernels of a step by the library's own rule: the line beyond which the FP32
momentum gather takes a thread a particle, and the wall walks a kernel of their own."""
import re
from pathlib import Path
from types import SimpleNamespace

import pytest

import bench

CSRC = Path(bench.__file__).parent / "ethersphcpu.jl_gb300" / "csrc"


@pytest.mark.parametrize("dim", [2, 3])
def test_the_line_is_the_librarys(dim):
    text = (CSRC / "sph_fp32.cuh").read_text()
    rule = re.search(r"constexpr int64_t kMomentumLanesUpTo = ([^;]+);", text).group(1)
    m = re.fullmatch(r"(\d+) \* (\d+) \* \(DIM == 3 \? (\d+) : (\d+)\)", rule)
    assert m, rule
    sms, particles, blocks_3d, blocks_2d = map(int, m.groups())
    line = sms * particles * (blocks_3d if dim == 3 else blocks_2d)
    scene = lambda n: SimpleNamespace(n_fluid=n, params=lambda: SimpleNamespace(dim=dim))
    shape = (1, 1, 1, 128)
    assert bench.gather_launches(scene(line), 1, shape, False) == 2
    assert bench.gather_launches(scene(line + 1), 1, shape, False) == 3
    assert bench.gather_launches(scene(line + 1), 0, shape, False) == 2
