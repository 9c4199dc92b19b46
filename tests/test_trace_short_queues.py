"""Queues shorter than the resident warps can fill are spread over all warps, each taking its share
of lanes: sizes on both sides of a share of one, of the largest share that is spread and of a full
warp, on single-mesh (flat) and instanced scenes, against the oracle."""
import numpy as np
import pytest

from imbatracer_b200 import scene as S
from oracle import oracle as O
from tests import helpers as H
from tests.test_traversal_gpu import run_gpu


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["config1", "config2"])
def test_short_queues_are_exact(cuda, name):
    import torch
    td = H.traversal_data(name)
    ds = S.DeviceScene(td)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    warps = [sms * w for w in (24, 28, 32)]          # resident warps of the launch shapes
    counts = {1, 2, 31, 32, 33, 257}
    for w in warps:
        counts |= {w - 1, w + 1, 8 * w - 1, 8 * w, 8 * w + 1}
    rays = H.ray_set(name, max(counts), seed=21)
    want = O.trace_node2(td, rays)
    occ = O.trace_node2(td, rays, any_hit=True)["tri_id"] >= 0
    for n in sorted(counts):
        hits, _, _ = run_gpu(ds, rays[:n])
        assert H.hits_equal(want[:n], hits).all(), n
        hits, _, _ = run_gpu(ds, rays[:n], any_hit=True)
        assert np.array_equal(occ[:n], hits["tri_id"] >= 0), n
    ds.close()
