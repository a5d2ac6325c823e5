"""Slots whose hypotheses are skipped because no node of a tile can be in view
there: cost volumes bit-identical to the oracle (which projects every node at
every hypothesis, IEEE arithmetic) for sideways, forward and backward motion, a
slot behind the keyframe, turned away from or looking back at it, camera centres
on a node's ray at a hypothesis, equal poses, far translations, and inverse-depth
ranges that cross many or no view bounds."""
import numpy as np
import pytest
import torch

from open_quadtree_mapping_b200.params import ARITH_IEEE, Params

pytestmark = pytest.mark.gpu


def _turn(axis, a):
    c, s = np.cos(a), np.sin(a)
    R = np.eye(3)
    i, j = [(1, 2), (0, 2), (0, 1)][axis]
    R[i, i], R[i, j], R[j, i], R[j, j] = c, -s, s, c
    return R


@pytest.mark.parametrize("W,H,D,near,far", [(320, 96, 128, 0.02, 2000.0), (320, 240, 96, 0.5, 50.0),
                                            (1001, 401, 48, 1.0, 1.5), (752, 480, 64, 0.5, 50.0),
                                            (752, 480, 32, 0.3, 20.0)])
def test_every_motion(W, H, D, near, far, oracle_mod, gpu):
    from open_quadtree_mapping_b200 import stages
    rng = np.random.default_rng(W + D)
    cam = (0.7 * W, 0.75 * W, 0.47 * W, 0.55 * H)
    p = Params.for_range(D, near, far, arith=ARITH_IEEE)
    base = rng.integers(0, 256, (H, W)).astype(np.uint8)
    base[: H // 2, W // 2:] = 90
    ray = np.array([(4 * (W // 12) - cam[0 + 2]) / cam[0], (4 * (H // 9) - cam[3]) / cam[1], 1.0])
    ray /= np.linalg.norm(ray)
    on_ray = -ray / (p.min_inv_depth + p.inv_depth_step * (D // 3))
    motions = [(np.eye(3), (0.3, 0, 0)), (np.eye(3), (0, 0, 1.0)), (np.eye(3), (0, 0, -1.0)),
               (np.eye(3), (0, 0, 0)), (np.eye(3), on_ray), (_turn(1, 0.01), on_ray * 1.0001),
               (_turn(1, 0.5), (0.1, 0, 0)), (_turn(1, -1.2), (0, 0.2, 0)),
               (_turn(1, np.pi), (0.2, 0.1, 2.0)), (_turn(0, 1.5), (0, 0, 0.5)),
               (_turn(2, 0.4), (0, 0.05, 0)), (np.eye(3), (0, -40.0, 0)),
               (_turn(0, 0.03), (5.0, 0, 30.0)), (_turn(1, np.pi / 2), (0.0, 0, 0))]
    motions += [(_turn(i % 3, 0.04 * (i - 9)), 0.4 * rng.standard_normal(3)) for i in range(18)]
    T = np.stack([np.concatenate([R, np.asarray(t, float).reshape(3, 1)], 1).reshape(12)
                  for R, t in motions]).astype(np.float32)
    slots = [np.ascontiguousarray(np.roll(base, (i, -3 * i), (0, 1))) for i in range(len(T))]
    ref = torch.from_numpy(base).to(gpu)
    levels = stages.quadtree(ref, p)
    dev = [torch.from_numpy(s).to(gpu) for s in slots]
    assert len(T) == 32
    for pick in (range(32), (4,), (6, 8), (11,)):
        pick = list(pick)
        got = stages.cost_volume(ref, levels, [dev[i] for i in pick], T[pick], cam, p).cpu().numpy()
        want, _ = oracle_mod.cost_volume(base, levels.cpu().numpy(), [slots[i] for i in pick],
                                         T[pick], cam, p)
        assert np.array_equal(got, want)
