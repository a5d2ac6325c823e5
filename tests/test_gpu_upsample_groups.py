"""The line solves' four-sample groups: an image that starts on no group's
boundary takes the passes sample by sample, and both give the same bits, from
one group of columns to the longest rows, with partial stripes and rounds."""
import numpy as np
import pytest
import torch

from open_quadtree_mapping_b200.params import ARITH_IEEE, ARITH_REFERENCE, Params

pytestmark = pytest.mark.gpu

SIZES = [(16, 8), (48, 24), (144, 136), (752, 480), (1008, 520), (1040, 1032), (1920, 1080)]


@pytest.mark.parametrize("arith", [ARITH_IEEE, ARITH_REFERENCE])
@pytest.mark.parametrize("W,H", SIZES)
def test_groups_equal_single_samples(W, H, arith, gpu):
    from open_quadtree_mapping_b200 import stages
    rng = np.random.default_rng(W + H)
    img = torch.from_numpy(rng.integers(0, 256, (H, W), dtype=np.uint8)).to(gpu)
    img[: H // 2] //= 16
    sparse = np.where(rng.random((H, W)) < 0.1, rng.uniform(0.5, 50.0, (H, W)), 0.0)
    sparse[0, 0] = 2.0
    sparse = torch.from_numpy(sparse.astype(np.float32)).to(gpu)
    off = torch.empty(H * W + 1, dtype=torch.uint8, device=gpu)[1:].view(H, W)
    off.copy_(img)
    p = Params.for_range(64, 0.5, 50.0, arith=arith)
    a, b = stages.upsample(sparse, img, p), stages.upsample(sparse, off, p)
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
