"""The cost pyramid, three levels per launch: the coarse levels' messages (they
follow from the data terms alone) bit-identical to the oracle in IEEE arithmetic
for every number of levels that ends inside, at and beyond a launch's three,
with level sizes that are no multiple of a tile, down to one cell."""
import numpy as np
import pytest
import torch

from open_quadtree_mapping_b200.params import ARITH_IEEE, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [2, 3, 4, 5, 7, 8])
@pytest.mark.parametrize("cw,ch,D", [(4, 4, 32), (9, 7, 48), (17, 33, 64), (31, 8, 96),
                                     (66, 35, 128)])
def test_messages_vs_oracle(cw, ch, D, levels, oracle_mod, gpu):
    from open_quadtree_mapping_b200 import stages
    W, H = 4 * cw, 4 * ch
    rng = np.random.default_rng(100 * cw + levels)
    p = Params.for_range(D, 0.5, 50.0, arith=ARITH_IEEE, bp_levels=levels,
                         bp_iters=(2,) * levels)
    cost = rng.uniform(0.0, 1.0, (ch, cw, D)).astype(np.float32)
    lv = np.full((H, W), 2, np.uint8)
    sparse, labels, msgs = stages.bp_extract(torch.from_numpy(cost).to(gpu), W, H,
                                             torch.from_numpy(lv).to(gpu), p, want_messages=True)
    lo, so, mo = oracle_mod.bp_extract(cost, W, H, lv, p, want_messages=True)
    assert np.array_equal(msgs.cpu().numpy(), mo)
    assert np.array_equal(labels.cpu().numpy(), lo)
    assert np.array_equal(sparse.cpu().numpy(), so)
