"""View ranges in reference arithmetic, where the oracle only comes close: one slot
among 31 that never are in view (which makes enough hypotheses x slots for the ranges
to be looked up) against the same slot alone, below that line: the same bits.  The 31
by themselves: the cost of an unseen hypothesis everywhere.  Motions: along the axis,
sideways, turned half out of the image, behind, and mirrored behind."""
import numpy as np
import pytest
import torch

from open_quadtree_mapping_b200.params import ARITH_IEEE, ARITH_REFERENCE, Params

pytestmark = pytest.mark.gpu


def _pose(yaw, pitch, t):
    c, s, d, e = np.cos(yaw), np.sin(yaw), np.cos(pitch), np.sin(pitch)
    R = (np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]])
         @ np.array([[1, 0, 0], [0, d, -e], [0, e, d]]))
    return np.concatenate([R, np.reshape(t, (3, 1))], 1).reshape(12)


@pytest.mark.parametrize("arith", [ARITH_REFERENCE, ARITH_IEEE])
@pytest.mark.parametrize("W,H,D", [(320, 240, 128), (640, 480, 64)])
def test_slot_among_unseen_ones(W, H, D, arith, gpu):
    from open_quadtree_mapping_b200 import stages
    rng = np.random.default_rng(W)
    p = Params.for_range(D, 0.5, 50.0, arith=arith)
    cam = (0.9 * W, 0.9 * W, 0.5 * W, 0.5 * H)  # rays within 0.56 of the axis
    image = lambda: torch.from_numpy(rng.integers(0, 256, (H, W)).astype(np.uint8)).to(gpu)  # noqa: E731
    ref = image()
    levels = torch.full((H, W), 2, dtype=torch.uint8, device=gpu)
    # turned a quarter, with centres so near that no point comes into view
    away = [_pose((1 if k % 2 else -1) * (np.pi / 2 + 0.004 * (k - 15)), 0.002 * k,
                  0.001 * rng.standard_normal(3)) for k in range(31)]
    away_img = [image() for _ in away]

    def cost(imgs, T):
        return stages.cost_volume(ref, levels, imgs, np.float32(T), cam, p)

    unseen = cost(away_img, away)
    assert torch.equal(unseen, cost(away_img[:1], away[:1]))
    assert torch.unique(unseen[1:-1, 1:-1]).numel() == 1
    seen = 0
    for T in (_pose(0, 0, (0, 0, 0.4)), _pose(0, 0, (0, 0, -0.4)), _pose(0.01, 0, (0.3, 0, 0)),
              _pose(0.55, 0.0, (0.1, 0, 0)), _pose(0.0, -0.5, (0, 0.2, 0)),
              _pose(np.pi, 0.0, (0.2, 0.1, 2.0)), _pose(0.0, 0.0, (0.0, 0.0, -5.0))):
        img = image()
        k = int(rng.integers(32))
        alone = cost([img], [T])
        assert torch.equal(cost(away_img[:k] + [img] + away_img[k:], away[:k] + [T] + away[k:]),
                           alone)
        seen += int((alone != unseen).any())
    assert seen == 7
