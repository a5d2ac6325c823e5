"""Which BP levels the cluster launch takes by default: levels just below and above one
round of a cluster's lane groups (one keyframe: 1024, 2048 and 4096 cells at 128, 64 and
32 hypotheses), messages bit-identical to the oracle (IEEE arithmetic); and a few
streams, at both sides of two rounds, equal to the launch-per-half-sweep results."""
import numpy as np
import pytest
import torch

from conftest import sequence
from open_quadtree_mapping_b200.params import ARITH_IEEE, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cw,ch,D", [(32, 32, 128), (41, 25, 96), (45, 45, 64), (46, 45, 48),
                                     (64, 64, 32), (65, 64, 32)])
def test_messages_vs_oracle(cw, ch, D, oracle_mod, gpu):
    from open_quadtree_mapping_b200 import stages
    W, H = 4 * cw, 4 * ch
    rng = np.random.default_rng(cw + D)
    p = Params.for_range(D, 0.5, 50.0, arith=ARITH_IEEE, bp_iters=(3, 2, 3, 2))
    img = rng.integers(0, 256, (H, W)).astype(np.uint8)
    img[: H // 2, W // 3:] = 77  # large blocks
    levels = stages.quadtree(torch.from_numpy(img).to(gpu), p)
    cost = rng.uniform(0.0, 0.05, (ch, cw, D)).astype(np.float32)
    sparse, labels, msgs = stages.bp_extract(torch.from_numpy(cost).to(gpu), W, H, levels, p,
                                             want_messages=True)
    lo, so, mo = oracle_mod.bp_extract(cost, W, H, levels.cpu().numpy(), p, want_messages=True)
    assert np.array_equal(msgs.cpu().numpy(), mo)
    assert np.array_equal(labels.cpu().numpy(), lo)
    assert np.array_equal(sparse.cpu().numpy(), so)


@pytest.mark.parametrize("W,H,D,n", [(240, 136, 128, 2), (256, 128, 128, 2), (256, 136, 128, 3),
                                     (160, 128, 128, 16)])
def test_streams_equal_single_launches(W, H, D, n, gpu):
    from open_quadtree_mapping_b200.depthmap import BatchDepthmap
    f = 460.0 * W / 752.0
    imgs, poses, _ = sequence(9, 14, W, H)
    got = []
    for cells in (0, None):
        b = BatchDepthmap([dict(width=W, height=H, fx=f, fy=f, cx=W / 2.0, cy=H / 2.0,
                                num_hyp=D, num_slots=3)] * n, params=Params.for_range(D, 0.5, 50.0))
        if cells is not None:
            b.set_coarse_bp(cells)
        for i in range(14):
            has = b.add_frames([imgs[(i + k) % 14] for k in range(n)],
                               [poses[(i + k) % 14] for k in range(n)])
        assert all(has)
        got.append([(b.get_debug(k), b.get_variance(k)) for k in range(n)])
        b.close()
    for (d0, v0), (d1, v1) in zip(*got):
        assert np.array_equal(d0, d1)
        assert np.array_equal(v0, v1, equal_nan=True)
