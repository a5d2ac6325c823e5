"""Hypotheses out of a slot's view with cameras of either sign of the focal lengths
(mirrored images): the view bounds are widened by the size of the terms, whatever
their signs.  A telephoto camera whose slots leave the image by fractions of a pixel
per hypothesis, each at other hypotheses and many never seen by a tile: cost volumes
bit-identical to the oracle's, which projects every node at every hypothesis."""
import numpy as np
import pytest
import torch

from open_quadtree_mapping_b200.params import ARITH_IEEE, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sx,sy", [(1, 1), (-1, 1), (1, -1), (-1, -1)])
def test_focal_signs(sx, sy, oracle_mod, gpu):
    from open_quadtree_mapping_b200 import stages
    W, H, D, F = 128, 96, 128, 32
    f = 20000.0
    rng = np.random.default_rng(7)
    cam = (sx * f, sy * f, W / 2.0, H / 2.0)
    p = Params.for_range(D, 0.5, 50.0, arith=ARITH_IEEE)
    ref = rng.integers(0, 256, (H, W)).astype(np.uint8)
    slots = [rng.integers(0, 256, (H, W)).astype(np.uint8) for _ in range(F)]
    T = np.zeros((F, 3, 4), np.float32)
    for k in range(F):
        # a shift of up to 1.3 image sizes by turning, and 0.3 pixels a hypothesis
        a = 1.3 * (k - F / 2) / (F / 2) * np.array([W, H]) / f
        cx, cy = (0.0, a[1]) if k % 2 else (a[0], 0.0)
        R = np.array([[np.cos(cx), 0, np.sin(cx)], [0, 1, 0], [-np.sin(cx), 0, np.cos(cx)]])
        R = R @ np.array([[1, 0, 0], [0, np.cos(cy), -np.sin(cy)], [0, np.sin(cy), np.cos(cy)]])
        T[k, :, :3] = R
        T[k, :, 3] = 0.3 / (f * p.inv_depth_step) * np.array([k % 2 == 0, k % 2, 0.0])
    T = T.reshape(F, 12)
    levels = torch.full((H, W), 2, dtype=torch.uint8, device=gpu)
    got = stages.cost_volume(torch.from_numpy(ref).to(gpu), levels,
                             [torch.from_numpy(s).to(gpu) for s in slots], T, cam,
                             p).cpu().numpy()
    want, _ = oracle_mod.cost_volume(ref, levels.cpu().numpy(), slots, T, cam, p)
    assert np.array_equal(got, want)
