"""The BP cluster launch's width follows the jobs of all branches that run at once:
batches at both sides of every step of that rule (7 clusters of 16 full blocks on a
B200, 14 of half ones) equal the launch-per-half-sweep results bit for bit, with the
default branches and with one, streams of two hypothesis counts among them."""
import numpy as np
import pytest

from conftest import sequence
from open_quadtree_mapping_b200.params import Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,counts", [(7, (64,)), (8, (64,)), (8, (96, 32)), (14, (128,)),
                                      (15, (64,)), (15, (48, 64))])
def test_widths_equal_single_launches(n, counts, gpu):
    from open_quadtree_mapping_b200.depthmap import BatchDepthmap
    W, H = 160, 128
    f = 460.0 * W / 752.0
    imgs, poses, _ = sequence(9, 15, W, H)
    descs = [dict(width=W, height=H, fx=f, fy=f, cx=W / 2.0, cy=H / 2.0,
                  num_hyp=counts[k % len(counts)], num_slots=3) for k in range(n)]
    got = []
    for cells, branches in ((0, 1), (4096, 3), (4096, 1)):
        b = BatchDepthmap(descs, params=Params.for_range(64, 0.5, 50.0))
        b.set_branches(branches)
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
