"""A cell whose costs are all infinite or NaN: its minimum counts as FLT_MAX, so every
value of what it sends is capped there before the (infinite) mean is subtracted: -inf
in all four directions, at every hypothesis count (with and without padding lanes),
from the per-half-sweep kernel and the cluster launch, in both arithmetics.  All other
cells of its colour send what they send with finite costs in its place."""
import numpy as np
import pytest
import torch

from open_quadtree_mapping_b200.params import ARITH_IEEE, ARITH_REFERENCE, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [32, 48, 64, 96, 128])
@pytest.mark.parametrize("arith", [ARITH_IEEE, ARITH_REFERENCE])
@pytest.mark.parametrize("iters", [1, 2])  # one half-sweep: a launch each; two: the cluster
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_cell_without_finite_costs(D, arith, iters, bad, gpu):
    from open_quadtree_mapping_b200 import stages
    W, H = 52, 36
    rng = np.random.default_rng(D)
    p = Params.for_range(D, 0.5, 50.0, arith=arith, bp_levels=1, bp_iters=(iters,))
    cost = rng.uniform(0.0, 0.05, (H // 4, W // 4, D)).astype(np.float32)
    levels = torch.full((H, W), 2, dtype=torch.uint8, device=gpu)

    def messages(c):
        return stages.bp_extract(torch.from_numpy(c).to(gpu), W, H, levels, p,
                                 want_messages=True)[2].cpu().numpy()

    want = messages(cost)
    y, x = 4, 6  # swept by half-sweep 0
    cost[y, x] = bad
    got = messages(cost)
    assert np.all(got[:, y, x] == -np.inf)
    even = (np.add.outer(np.arange(H // 4), np.arange(W // 4)) % 2) == 0
    even[y, x] = False
    assert np.array_equal(got[:, even], want[:, even])
