"""The top BP levels in one cluster launch: messages bit-identical to the oracle
(IEEE arithmetic) where a level has fewer cells than blocks, odd sizes, blocks
whose cells span several rows or less than one, cells the quadtree test skips,
levels that no longer fit a cluster's shared memory, and hypothesis counts with
padding lanes; and batches above the job count that takes narrower clusters
equal to the launch-per-half-sweep results bit for bit."""
import numpy as np
import pytest
import torch

from conftest import sequence
from open_quadtree_mapping_b200.params import ARITH_IEEE, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,D,iters", [
    (16, 16, 64, (4, 10, 10, 10)), (8, 40, 32, (2, 3, 2, 5)), (100, 52, 48, (4, 10, 10, 10)),
    (132, 20, 96, (3, 2, 2, 4)), (20, 132, 128, (4, 3, 2)), (256, 248, 64, (4, 3, 4, 2)),
    (256, 248, 128, (4, 3, 4, 2)), (500, 124, 32, (5, 2, 3, 2)), (4, 4, 64, (2,)),
    (60, 60, 64, (2, 2, 2, 2, 2, 2, 2, 2))])
def test_messages_vs_oracle(W, H, D, iters, oracle_mod, gpu):
    from open_quadtree_mapping_b200 import stages
    W, H = max(W, 8), max(H, 8)
    rng = np.random.default_rng(W + 1000 * H + D)
    p = Params.for_range(D, 0.5, 50.0, arith=ARITH_IEEE, bp_levels=len(iters), bp_iters=iters)
    img = rng.integers(0, 256, (H, W)).astype(np.uint8)
    img[: H // 2, W // 3:] = 77  # large blocks
    levels = stages.quadtree(torch.from_numpy(img).to(gpu), p)
    cost = rng.uniform(0.0, 0.05, (H // 4, W // 4, D)).astype(np.float32)
    sparse, labels, msgs = stages.bp_extract(torch.from_numpy(cost).to(gpu), W, H, levels, p,
                                             want_messages=True)
    lo, so, mo = oracle_mod.bp_extract(cost, W, H, levels.cpu().numpy(), p, want_messages=True)
    assert np.array_equal(msgs.cpu().numpy(), mo)
    assert np.array_equal(labels.cpu().numpy(), lo)
    assert np.array_equal(sparse.cpu().numpy(), so)


@pytest.mark.parametrize("W,H,D,n", [(160, 128, 64, 10), (320, 240, 48, 9), (160, 128, 128, 3)])
def test_batch_equals_single_launches(W, H, D, n, gpu):
    from open_quadtree_mapping_b200.depthmap import BatchDepthmap
    imgs, poses, _ = sequence(9, 15, W, H)
    desc = dict(width=W, height=H, fx=460.0 * W / 752, fy=460.0 * W / 752, cx=W / 2.0, cy=H / 2.0,
                num_hyp=D, num_slots=3)
    got = []
    for cells in (0, 4096, 1 << 20):
        b = BatchDepthmap([desc] * n, params=Params.for_range(D, 0.5, 50.0))
        b.set_branches(1)
        b.set_coarse_bp(cells)
        for i in range(15):
            has = b.add_frames([imgs[(i + k) % 15] for k in range(n)],
                               [poses[(i + k) % 15] for k in range(n)])
        assert all(has)
        got.append([(b.get_debug(k), b.get_variance(k)) for k in range(n)])
        b.close()
    for other in got[1:]:
        for (d0, v0), (d1, v1) in zip(got[0], other):
            assert np.array_equal(d0, d1)
            assert np.array_equal(v0, v1, equal_nan=True)
