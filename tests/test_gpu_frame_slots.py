"""Frame slots: the image of the last result stays in the slot it came in with.
170 frames (the ring of 60 fills and overflows; every third frame stands still
and does not join the ring), ratio 1 and 2: after every result the reference
image is that frame's, and the pipelined batch (two steps in flight) gives the
facade's depth bit for bit."""
import numpy as np
import pytest
import torch

from open_quadtree_mapping_b200.params import Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ratio", [1, 2])
def test_long_sequence(ratio, gpu):
    from open_quadtree_mapping_b200.depthmap import BatchDepthmap, Depthmap
    W, H, f = 96, 72, 60.0
    p = Params.for_range(32, 0.5, 50.0)
    dm = Depthmap(W, H, f, W / 2, f, H / 2, semi2dense_ratio=ratio, params=p)
    b = BatchDepthmap([dict(width=W, height=H, fx=f, fy=f, cx=W / 2, cy=H / 2, num_hyp=32,
                            num_slots=5, semi2dense_ratio=ratio)] * 2, params=p)
    rng = np.random.default_rng(1)
    base = rng.integers(0, 256, (H + 40, W + 400)).astype(np.uint8)
    outs = [[torch.empty((H, W), dtype=torch.float32, pin_memory=True).numpy() for _ in range(2)]
            for _ in range(3)]
    want, x = {}, 0
    for i in range(170):
        x += 0 if i % 3 == 2 else 1
        img = np.ascontiguousarray(base[x % 40:x % 40 + H, x:x + W])
        T = np.eye(3, 4, dtype=np.float32)
        T[0, 3] = -0.05 * x
        if dm.add_frames(img, T):
            assert np.array_equal(dm.getReferenceImage(), img)
            want[i] = dm.getDepthmap()
        b.submit([img, img], [T, T], outs=outs[i % 3])
        if i - 2 in want:  # that step has retired: two are in flight
            assert np.array_equal(outs[(i - 2) % 3][0], want[i - 2], equal_nan=True)
            assert np.array_equal(outs[(i - 2) % 3][1], want[i - 2], equal_nan=True)
        if i % 7 == 0:
            b.wait()
    b.wait()
    assert len(want) > 60
    last = max(want)
    assert np.array_equal(outs[last % 3][0], want[last], equal_nan=True)
    b.close()
    dm.close()
