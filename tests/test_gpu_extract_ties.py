"""The extraction's argmin over lanes that hold four hypotheses each: labels and
depths bit-identical to the oracle (IEEE arithmetic, no half-sweeps, so the data
term alone decides) where many hypotheses tie, all are equal, and where some or
all are infinite or NaN, for every count, on images that are not a whole number
of warps."""
import numpy as np
import pytest
import torch

from open_quadtree_mapping_b200.params import ARITH_IEEE, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [32, 48, 64, 96, 128])
@pytest.mark.parametrize("kind", ["two values", "three values", "constant", "inf", "nan"])
def test_labels_vs_oracle(D, kind, oracle_mod, gpu):
    from open_quadtree_mapping_b200 import stages
    W, H = 132, 76
    rng = np.random.default_rng(D)
    p = Params.for_range(D, 0.5, 50.0, arith=ARITH_IEEE, bp_levels=1, bp_iters=(0,))
    n = {"two values": 2, "constant": 1}.get(kind, 3)
    cost = rng.integers(0, n, (H // 4, W // 4, D)).astype(np.float32) * 0.25
    if kind in ("inf", "nan"):
        bad = np.float32(np.inf if kind == "inf" else np.nan)
        cost[rng.random(cost.shape) < 0.5] = bad
        cost[::5, ::3] = bad
    levels = np.full((H, W), 2, np.uint8)
    sparse, labels = stages.bp_extract(torch.from_numpy(cost).to(gpu), W, H,
                                       torch.from_numpy(levels).to(gpu), p)[:2]
    lo, so = oracle_mod.bp_extract(cost, W, H, levels, p)[:2]
    assert np.array_equal(labels.cpu().numpy(), lo)
    assert np.array_equal(sparse.cpu().numpy(), so, equal_nan=True)
