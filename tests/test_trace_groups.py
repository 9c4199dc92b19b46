"""Short launches of several callers at once share the resident warps: ray batches, recorded ones and
frames on one stream and on many, each with the answers that a lone caller gets."""
import numpy as np
import pytest

from imbatracer_b200 import scene as S
from oracle import oracle as O
from tests import helpers as H
from tests.test_pt import small_mixed_scene


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["config1", "config2"])
@pytest.mark.parametrize("streams", [1, 2, 5, 40])       # one caller, a few, more than are told apart
def test_batches_of_many_callers(cuda, name, streams):
    import torch
    td = H.traversal_data(name)
    ds = S.DeviceScene(td)
    sizes = [1, 33, 700, 2049, 9001]
    rays = H.ray_set(name, max(sizes), seed=31)
    want = O.trace_node2(td, rays)
    occ = O.trace_node2(td, rays, any_hit=True)["tri_id"] >= 0
    d_rays = torch.from_numpy(rays.view(np.float32).reshape(-1, 8).copy()).cuda()
    st = [torch.cuda.Stream() for _ in range(streams)]
    torch.cuda.synchronize()
    out = []
    for rnd in range(3):
        for k, s in enumerate(st):
            n = sizes[(k + rnd) % len(sizes)]
            hits = [torch.full((n, 4), 7, dtype=torch.int32, device="cuda") for _ in range(2)]
            s.wait_stream(torch.cuda.current_stream())
            ds.trace(d_rays, hits[0], n, stream=s)
            ds.trace(d_rays, hits[1], n, any_hit=True, stream=s)
            out.append((n, hits))
    torch.cuda.synchronize()
    for n, (closest, any_hit) in out:
        assert np.array_equal(closest.cpu().numpy(), want[:n].view(np.int32).reshape(-1, 4))
        assert np.array_equal(any_hit[:, 0].cpu().numpy() >= 0, occ[:n])
    # Recorded, with other callers and without.
    hits = torch.zeros((2049, 4), dtype=torch.int32, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st[0]):
        ds.trace(d_rays, hits, 2049, stream=st[0])
    for _ in range(2):
        hits.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(hits.cpu().numpy(), want[:2049].view(np.int32).reshape(-1, 4))
    ds.close()


@pytest.mark.gpu
def test_frames_of_many_callers(cuda):
    """Frames of several contexts on streams of their own, before and after frames alone: the graph is
    sized for the company it has, the image is the lone one's up to the order of its sums."""
    import time
    import torch
    from imbatracer_b200.integrators import GpuScene, PathTracer
    gs = GpuScene(small_mixed_scene())
    pts = [PathTracer(gs, max_path_len=5) for _ in range(6)]
    st = [torch.cuda.Stream() for _ in pts]
    w, h = 48, 36

    def images(which):
        img = [torch.zeros((h, w, 3), device="cuda") for _ in which]
        torch.cuda.synchronize()
        for k, i in zip(which, img):
            pts[k].render(2, 11, w, h, image=i, stream=st[k], stats=False)
        torch.cuda.synchronize()
        return [i.cpu().numpy().astype(np.float64) for i in img]
    time.sleep(0.06)                                  # no other caller in the last 50 ms
    lone = images([0])[0]
    assert lone.sum() > 0
    for rnd in range(3):
        for img in images(range(6)):
            # At most 2 samples * 5 bounces * 2 float32 terms a pixel, in another order.
            assert (np.abs(img - lone) <= 20 * 2.0 ** -23 * np.maximum(img, lone)).all()
    time.sleep(0.06)
    again = images([3])[0]
    assert (np.abs(again - lone) <= 20 * 2.0 ** -23 * np.maximum(again, lone)).all()
    for pt in pts:
        pt.close()
