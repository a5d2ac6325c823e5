"""Kernels whose shape follows the image size, at both sides of every rule: the
fusion's pixels per thread (160 000, 1.2 M and 2.1 M pixels) and the five-level
quadtree's 32 x 32 tiles (ragged and missing quadrants).

Fusion in IEEE arithmetic against the FP64 oracle: the source table bit-exact;
fused depth, mean and variance within 1e-6 (FP64 update, float results).
Quadtree levels bit-exact."""
import numpy as np
import pytest
import torch

from open_quadtree_mapping_b200.params import ARITH_IEEE, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(16, 8), (400, 400), (401, 400), (1200, 1000), (1208, 1000),
                                 (2100, 1000), (2104, 1000)])
def test_fuse_pixels_per_thread(W, H, oracle_mod, gpu):
    from open_quadtree_mapping_b200 import stages
    rng = np.random.default_rng(W + H)
    cam = (0.7 * W, 0.7 * W, W / 2.0, H / 2.0)
    depth = rng.uniform(2.0, 4.0, (H, W)).astype(np.float32)
    depth[rng.random((H, W)) < 0.02] = 0.0
    seeds = np.stack([rng.uniform(0, 40, (H, W)), rng.uniform(3, 12, (H, W)),
                      rng.uniform(1.8, 4.2, (H, W)), rng.uniform(0.05, 5, (H, W))],
                     -1).astype(np.float32)
    T = np.eye(3, 4, dtype=np.float32)
    T[:, 3] = (0.05, -0.02, 0.03)
    T = T.reshape(12)
    p = Params.for_range(64, 0.5, 50.0, arith=ARITH_IEEE)
    gd, _, gs, gt = stages.fuse(torch.from_numpy(depth).to(gpu), torch.from_numpy(seeds).to(gpu), T,
                                cam, p)
    od, os_, ot, _ = oracle_mod.fuse(depth.astype(np.float64), seeds, T, cam)
    assert np.array_equal(gt.cpu().numpy(), ot)
    assert np.allclose(gd.cpu().numpy(), od, rtol=1e-6, atol=0)
    assert np.allclose(gs.cpu().numpy()[..., 2:], os_[..., 2:], rtol=1e-6, atol=0)


@pytest.mark.parametrize("W,H", [(32, 32), (33, 31), (64, 40), (31, 65), (16, 16), (97, 80),
                                 (48, 33)])
def test_five_level_tiles(W, H, oracle_mod, gpu):
    from open_quadtree_mapping_b200 import stages
    rng = np.random.default_rng(W * H)
    img = np.full((H, W), 100, np.uint8)
    img[rng.random((H, W)) < 3.0 / (W * H) + 0.001] = 240
    for p in (Params(qt_max_level=5), Params(qt_max_level=5, qt_min_level=0, qt_threshold=3.0)):
        lv = stages.quadtree(torch.from_numpy(img).to(gpu), p).cpu().numpy()
        assert np.array_equal(lv, oracle_mod.quadtree(img, p))
