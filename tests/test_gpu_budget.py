"""A batch sized to a device memory budget stays within it when it is full and stepping (beside
the scratch of transfers: uploads of a 3D scene stage its positions and velocities, 48 bytes
a particle)."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BUDGET = 1 << 30


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dim", [2, 3])
def test_a_full_batch_stays_within_its_budget(pkg, dim, precision):
    import torch
    from ethersph_gb300 import batch, scenes

    def scene(dx):
        if dim == 2:
            return scenes.dam_break_2d(dx=dx, water_w=2.0, water_h=2.0, box_w=4.0, box_h=3.0)
        return scenes.dam_break_3d(dx=dx, tank=(0.6, 0.4, 0.4), column=(0.5, 0.4, 0.35))

    prm = scene(0.05).params(precision=precision)
    with batch.Batch(prm, 20_000, 200_000, 80_000, 2) as warm:  # what the device keeps once for all handles
        warm.add_scene(scene(0.05), 1, 20)
        warm.step(20)
        warm.synchronize()
    free, _ = torch.cuda.mem_get_info()
    with batch.Batch.for_budget(prm, BUDGET, scene_capacity=2, cells_per_particle=3.2, walls_per_particle=0.25) as bt:
        n = bt.capacity[0]
        s = scene((4.0 / n) ** 0.5 * 1.001 if dim == 2 else (0.5 * 0.4 * 0.35 / n) ** (1 / 3) * 1.01)
        assert 0.9 * n < s.n_fluid <= n
        bt.add_scene(dataclasses.replace(s, check=None), 1, 20)
        bt.step(20)
        bt.synchronize()
        used = free - torch.cuda.mem_get_info()[0] - (48 * s.n_fluid if dim == 3 else 0)
        assert np.isfinite(bt.download(0)["rho"]).all()
    assert used <= 1.01 * BUDGET, used / BUDGET  # rounding of allocations, step graphs
