"""Cost volume over the ways a patch is taken: aligned, deferred and pixel by
pixel, in one call (slots turned by different angles), with word-aligned and
odd rows and image pointers, tiles shared by 1, 2 and 4 blocks, few nodes per
tile, one and many slots, duplicates.  IEEE arithmetic: bit-identical to the
oracle; reference arithmetic: within its tolerance for all but the projections
that its rounding moves across a pixel edge (one in a thousand)."""
import numpy as np
import pytest
import torch

from open_quadtree_mapping_b200.params import ARITH_IEEE, ARITH_REFERENCE, Params

pytestmark = pytest.mark.gpu

ROLLS = (0.0, 0.004, 0.03, 0.049, 0.052, 0.07, 0.3, -0.02, 3.1)


def _pose(rng, roll):
    a, b = 0.02 * rng.standard_normal(2)
    c, s = np.cos(roll), np.sin(roll)
    R = (np.array([[c, -s, 0], [s, c, 0], [0, 0, 1]])
         @ np.array([[1, 0, a], [0, 1, b], [-a, -b, 1]]))
    q, r = np.linalg.qr(R)
    q = q * np.sign(np.diag(r))
    return np.concatenate([q, 0.15 * rng.standard_normal((3, 1))], 1).astype(np.float32).reshape(12)


def _at(img, gpu, shift):
    """The image on the GPU, `shift` bytes past an aligned address."""
    buf = torch.empty(img.size + 16, dtype=torch.uint8, device=gpu)
    t = buf[shift:shift + img.size].view(img.shape)
    t.copy_(torch.from_numpy(img))
    return t


@pytest.mark.parametrize("W,H,D,F,shift", [
    (160, 128, 64, 5, 0), (160, 128, 48, 9, 1), (97, 61, 32, 6, 0), (98, 60, 96, 4, 2),
    (321, 203, 64, 9, 3), (320, 240, 128, 3, 0), (752, 480, 64, 6, 0), (755, 320, 96, 9, 0),
    (8, 8, 32, 1, 0), (36, 20, 64, 32, 0), (1280, 176, 48, 7, 4)])
def test_paths(W, H, D, F, shift, oracle_mod, gpu):
    from open_quadtree_mapping_b200 import stages
    rng = np.random.default_rng(W * 1000 + H + D)
    smooth = rng.integers(0, 256, (H // 7 + 2, W // 7 + 2)).astype(np.uint8)
    base = np.kron(smooth, np.ones((7, 7), np.uint8))[:H, :W].copy()
    base[: H // 3] = rng.integers(0, 256, (H // 3, W))
    slots = [np.ascontiguousarray(np.roll(base, (i, -2 * i), (0, 1))) for i in range(F)]
    T = np.stack([_pose(rng, ROLLS[i % len(ROLLS)]) for i in range(F)])
    if F > 4:
        slots[3], T[3] = slots[1], T[1]
    cam = (0.6 * W, 0.6 * W, W / 2.0, H / 2.0)
    ref = torch.from_numpy(base).to(gpu)
    dev = [_at(s, gpu, shift) for s in slots]
    if F > 4:
        dev[3] = dev[1]
    for arith in (ARITH_IEEE, ARITH_REFERENCE):
        p = Params.for_range(D, 0.5, 50.0, arith=arith)
        levels = stages.quadtree(ref, p)
        got = stages.cost_volume(ref, levels, dev, T, cam, p).cpu().numpy()
        want, _ = oracle_mod.cost_volume(base, levels.cpu().numpy(), slots, T, cam, p)
        if arith == ARITH_IEEE:
            assert np.array_equal(got, want)
        else:
            assert np.isclose(got, want, rtol=1e-6, atol=1e-9).mean() > 0.999
