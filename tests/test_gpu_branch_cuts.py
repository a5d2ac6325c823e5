"""Branches by hypothesis count: streams given in any order of counts (more
counts than branches, one count with nearly all streams, one stream per count)
give the depth maps, debug maps and variances of the one-sequence run bit for
bit, each at its own stream."""
import numpy as np
import pytest

from conftest import sequence
from open_quadtree_mapping_b200.params import Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [
    (64, 48, 64, 48, 96), (128, 32, 48, 64, 96, 32, 128), (64,) * 6 + (32,), (96, 64), (48,) * 3])
def test_any_order(counts, gpu):
    from open_quadtree_mapping_b200.depthmap import BatchDepthmap
    sizes = [(160, 128), (208, 120), (96, 72)]
    shape = [sizes[i % 3] for i in range(len(counts))]
    seq = {s: sequence(11, 15, *s) for s in set(shape)}
    desc = [dict(width=w, height=h, fx=460.0 * w / 752, fy=460.0 * w / 752, cx=w / 2.0, cy=h / 2.0,
                 num_hyp=d, num_slots=2 + i % 3) for i, ((w, h), d) in enumerate(zip(shape, counts))]
    got = []
    for k in (1, 2, 4):
        b = BatchDepthmap(desc, params=Params.for_range(64, 0.5, 50.0))
        b.set_branches(k)
        for i in range(15):
            has = b.add_frames([seq[s][0][(i + j) % 15] for j, s in enumerate(shape)],
                               [seq[s][1][(i + j) % 15] for j, s in enumerate(shape)])
        assert all(has)
        got.append([(b.get_depth(j), b.get_debug(j), b.get_variance(j))
                    for j in range(len(counts))])
        b.close()
    for other in got[1:]:
        for one, two in zip(got[0], other):
            assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(one, two))
