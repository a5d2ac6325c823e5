"""A resident run after frames without a dense pass (semi2dense_ratio) repeats the
last dense pass: depth, debug map and variance equal those of a resident run right
after that pass, for one and several streams, at ratios whose results fall on one
step parity (2) and on both (3)."""
import numpy as np
import pytest

from conftest import sequence
from open_quadtree_mapping_b200.params import Params

pytestmark = pytest.mark.gpu

W, H = 160, 128


def _resident(ratio, n, skipped):
    from open_quadtree_mapping_b200.depthmap import BatchDepthmap
    f = 460.0 * W / 752.0
    imgs, poses, _ = sequence(5, 20, W, H)
    b = BatchDepthmap([dict(width=W, height=H, fx=f, fy=f, cx=W / 2.0, cy=H / 2.0, num_hyp=64,
                            num_slots=5, semi2dense_ratio=ratio)] * n,
                      params=Params.for_range(64, 0.5, 50.0))
    i = results = since = 0
    # the ring fills with one frame in `ratio`: the sequence is walked there and back
    while results < 3 or since < skipped:
        k = i % 38
        k = min(k, 38 - k)
        since += 1
        if all(b.add_frames([imgs[k]] * n, [poses[k]] * n)) and i > 0:
            results, since = results + 1, 0
        i += 1
    b.run_resident()
    got = [(b.get_depth(j), b.get_debug(j), b.get_variance(j)) for j in range(n)]
    b.close()
    return got


@pytest.mark.parametrize("ratio,n", [(2, 1), (3, 1), (2, 4)])
def test_resident_run_after_skipped_frames(ratio, n, gpu):
    want = _resident(ratio, n, 0)
    assert (want[0][1] > 0.0).any()
    for skipped in range(1, ratio):
        for a, b in zip(_resident(ratio, n, skipped), want):
            for x, y in zip(a, b):
                assert np.array_equal(x, y, equal_nan=True)
