"""Weighted upsampling (qm_upsample_w_*) at the edges of its line layouts:
one sample per segment, ragged last segments, lines whose column stripe is
narrower, and lines longer than shared memory holds (one thread per line).

Forward against the FP64 oracle: the solves are FP64, so the output differs
by its own rounding (2^-24) and is held to 1e-6 of the largest depth.  With a
fixed indicator the map sparse -> dense is linear, so sum(g * dense) =
sum(g_sparse * sparse) up to the float rounding of both (4e-7 of the sums of
magnitudes).  The weight factors' gradient against central differences of the
FP64 oracle (h = 1e-6) within 1e-4 of its largest component."""
import numpy as np
import pytest
import torch

from open_quadtree_mapping_b200.params import Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(16, 8), (32, 16), (48, 40), (528, 64), (1056, 24), (4096, 8),
                                 (16, 1160), (48, 2320), (7216, 8), (16, 7208)])
def test_line_layouts(W, H, oracle_mod, gpu):
    from open_quadtree_mapping_b200.diff import UpsampleW
    rng = np.random.default_rng(W * 10000 + H)
    p = Params()
    img = rng.integers(0, 60, (H, W)).astype(np.uint8)
    sparse = np.zeros((H, W), np.float32)
    sparse[::4, ::4] = rng.uniform(0.5, 8.0, sparse[::4, ::4].shape)
    omega = rng.uniform(0.0, 2.0, (H, W)).astype(np.float32)
    g = rng.standard_normal((H, W)).astype(np.float32)
    sp = torch.from_numpy(sparse).to(gpu).requires_grad_(True)
    om = torch.from_numpy(omega).to(gpu).requires_grad_(True)
    dense = UpsampleW.apply(sp, om, torch.from_numpy(img).to(gpu), p)
    dense.backward(torch.from_numpy(g).to(gpu))
    d = dense.detach().cpu().numpy().astype(np.float64)
    ref = oracle_mod.upsample_w(sparse.astype(np.float64), img, p, omega.astype(np.float64))
    assert np.abs(d - ref).max() <= 1e-6 * np.abs(ref).max()
    g_sp = sp.grad.cpu().numpy().astype(np.float64)
    left, right = g * ref, g_sp * sparse
    assert abs(left.sum() - right.sum()) <= 4e-7 * (np.abs(left).sum() + np.abs(right).sum())
    g_om = om.grad.cpu().numpy()
    picks = [(int(rng.integers(1, H)), int(rng.integers(1, W))) for _ in range(6)]
    fd = []
    for y, x in picks:
        v = []
        for sgn in (1, -1):
            o = omega.astype(np.float64)
            o[y, x] += sgn * 1e-6
            v.append((oracle_mod.upsample_w(sparse.astype(np.float64), img, p, o) * g).sum())
        fd.append((v[0] - v[1]) / 2e-6)
    got = np.array([g_om[y, x] for y, x in picks])
    assert np.abs(got - fd).max() <= 1e-4 * max(np.abs(fd).max(), np.abs(g_om).max())
