"""The tracker's stereo update at both of its tile sizes (256 pixels a block, 1024 from
1.21 M pixels a step): seeds and projected depths bit-identical to the oracle (IEEE
arithmetic) on images that are no whole number of tiles, and a batch whose streams make
large tiles together equal to the same streams one by one, in either arithmetic."""
import numpy as np
import pytest

from conftest import sequence
from open_quadtree_mapping_b200.params import ARITH_IEEE, ARITH_REFERENCE, Params
from test_gpu_semidense import _replay, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,n", [(24, 16, 5), (97, 65, 12), (1399, 866, 3), (1401, 867, 3)])
def test_tiles_vs_oracle(W, H, n, oracle_mod, gpu):
    steps = _replay(W, H, n, 4, ARITH_IEEE, oracle_mod, gpu)
    for i, (mode, dg, tg, pg, do, to, po, gt) in enumerate(steps):
        assert _same(tg, to), ("seeds (trk)", i, mode)
        assert _same(pg, po), ("seeds (dep)", i, mode)
        assert _same(dg, do), ("debug", i, mode)


@pytest.mark.parametrize("arith", [ARITH_IEEE, ARITH_REFERENCE])
def test_batch_of_large_tiles(arith, gpu):
    from open_quadtree_mapping_b200.depthmap import BatchDepthmap
    shapes = [(640, 480), (752, 480), (624, 408), (656, 488)]  # 1.24 M pixels
    seqs = [sequence(20 + k, 14, w, h) for k, (w, h) in enumerate(shapes)]
    descs = [dict(width=w, height=h, fx=460.0 * w / 752, fy=460.0 * w / 752, cx=w / 2.0,
                  cy=h / 2.0, num_hyp=32, num_slots=2) for w, h in shapes]
    p = Params.for_range(32, 0.5, 50.0, arith=arith)
    both = BatchDepthmap(descs, params=p)
    ones = [BatchDepthmap([d], params=p) for d in descs]
    for b in [both] + ones:
        b.set_semidense(True)
    for i in range(14):
        both.add_frames([s[0][i] for s in seqs], [s[1][i] for s in seqs])
        for s, b in zip(seqs, ones):
            b.add_frames([s[0][i]], [s[1][i]])
    for k, b in enumerate(ones):
        got, want = both.get_debug(k), b.get_debug(0)
        assert (want > 0).mean() > 0.05
        assert _same(got, want)
        b.close()
    both.close()
