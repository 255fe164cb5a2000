"""The drowned basins' outlets where the outlet reach is wider than the map, so that a walk may take every cell
of it (a planet of a kilometre): the scratch stays bounded, and the cut is the oracle's with however many basins
at a time that leaves."""
import numpy as np
import pytest
import torch

import oracle
from cartogenesis_gb300 import Context, ErosionConfig, SeaLevelStage, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,seed", [(64, 32, 2), (1024, 512, 1), (2048, 1024, 5)])
def test_drained_cut_of_a_small_planet(W, H, seed):
    scale = dict(sea_level=0.70, world_width_km=1.0)
    h = synthetic.heights_field(W, H, seed)
    ctx = Context()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    s1, l1, r1, n1, p1 = SeaLevelStage.drained_cut(ErosionConfig(W, H, seed, **scale), h, ctx=ctx)
    used = free - torch.cuda.mem_get_info()[0]
    ctx.close()
    s0, l0, r0, n0, p0 = oracle.sea_level_drained_cut(oracle.default_params(W, H, seed, **scale), h)
    assert p1 > 0
    assert np.float32(s0).view(np.uint32) == np.float32(s1).view(np.uint32)
    assert (n0, p0) == (n1, p1)
    assert np.array_equal(l0, l1) and np.array_equal(r0.view(np.uint32), r1.view(np.uint32))
    assert used < (640 << 20) + 256 * W * H   # the lists' bound and the rest of the context's buffers
