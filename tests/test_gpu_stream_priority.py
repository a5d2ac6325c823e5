"""A batch of one stream runs at the default priority, beside the caller's own work;
only the branches of several streams are raised (the order among them matters)."""
import pytest
import torch

from open_quadtree_mapping_b200.params import Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3])
def test_priority_of_the_batch_stream(n, gpu):
    from open_quadtree_mapping_b200.depthmap import BatchDepthmap
    b = BatchDepthmap([dict(width=64, height=48, fx=40.0, fy=40.0, cx=32.0, cy=24.0)] * n,
                      params=Params())
    priority = torch.cuda.ExternalStream(b.stream_ptr()).priority
    default = torch.cuda.Stream().priority
    assert priority == default if n == 1 else priority < default
    b.close()
