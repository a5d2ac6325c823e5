"""Gradients of the soft BP over the message states its forward keeps, against
FP64 torch autograd of the same forward (bp_torch_ref): odd, even, one and no
half-sweeps per level (shared states, inherited messages), cells the quadtree
test skips, odd cell counts, and levels inside and outside the coarse cluster
launch (4800 cells).

The FP64 mode follows the same selections as the reference and is held to
1e-6 of the largest component; the FP32 path's messages carry 1e-7 rounding
that the readout divides by tau, 1e-3 as in the end-to-end tests.  A second
backward over the same states gives the same gradient (up to the order of the
FP64 sums: 1e-12)."""
import numpy as np
import pytest
import torch

from conftest import cam_of, keyframe
from open_quadtree_mapping_b200.params import ARITH_IEEE, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,D,iters", [
    (64, 48, 64, (4, 10, 10, 10)), (64, 48, 64, (3, 5, 2, 7)), (100, 52, 48, (1, 2, 3, 1)),
    (100, 52, 32, (2, 0, 4, 1)), (68, 44, 96, (5,)), (100, 52, 128, (0, 3)),
    (320, 240, 32, (3, 2, 4, 2)), (320, 240, 32, (1, 4, 3, 0))])
def test_gradients(W, H, D, iters, gpu):
    from bp_torch_ref import soft_bp
    from open_quadtree_mapping_b200 import stages
    from open_quadtree_mapping_b200.diff import SoftBP
    kf = keyframe(3, 320, 240, 3)
    img = np.ascontiguousarray(kf.ref[:H, :W]).copy()
    img[: H // 2, : W // 2] = 90  # large quadtree blocks: cells the BP skips
    p = Params.for_range(D, 0.5, 50.0, arith=ARITH_IEEE, bp_levels=len(iters), bp_iters=iters)
    ref = torch.from_numpy(img).to(gpu)
    levels = stages.quadtree(ref, p)
    slots = [torch.from_numpy(np.ascontiguousarray(m[:H, :W])).to(gpu) for m in kf.meas]
    cost = stages.cost_volume(ref, levels, slots, kf.T_meas_ref, cam_of(kf), p)
    lv = levels.cpu().numpy().astype(np.int64)
    assert lv.max() > 2
    R = torch.from_numpy(np.random.default_rng(5).standard_normal((H, W)))
    P = [torch.tensor(float(np.float32(v)), dtype=torch.float64, requires_grad=True)
         for v in (p.P1, p.P2)]
    out = soft_bp(cost.cpu().double(), lv, p, P[0], P[1], 0.05)
    (out * R).sum().backward()
    want = np.array([0.0 if v.grad is None else v.grad.item() for v in P])
    scale = max(np.abs(want).max(), 1e-9)
    for fp64, rtol in ((True, 1e-6), (False, 1e-3)):
        pen = torch.tensor([float(np.float32(p.P1)), float(np.float32(p.P2))],
                           dtype=torch.float64, requires_grad=True)
        sparse = SoftBP.apply(pen, cost, levels, p, 0.05, fp64)
        loss = (sparse.double() * R.to(gpu)).sum()
        loss.backward(retain_graph=True)
        got = pen.grad.numpy().copy()
        assert np.abs(got - want).max() <= rtol * scale, (fp64, got, want)
        pen.grad = None
        loss.backward()
        assert np.abs(pen.grad.numpy() - got).max() <= 1e-12 * scale
