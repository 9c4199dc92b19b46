"""Handles made by one thread while another records a CUDA graph (thread-local capture): nothing on
the way waits for the whole device, which would end the capture."""
import threading

import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["hashgrid", "vcm", "pt"])
def test_create_beside_a_capture(cuda, kind):
    import torch
    from imbatracer_b200 import native as N
    lib = N.load()
    create, destroy = {"hashgrid": (lib.imbart_hashgrid_create, lib.imbart_hashgrid_destroy),
                       "vcm": (lib.imbart_vcm_create, lib.imbart_vcm_destroy),
                       "pt": (lib.imbart_pt_create, lib.imbart_pt_destroy)}[kind]
    destroy(create(0))                       # the library and its first-use state are loaded
    x = torch.arange(1000, dtype=torch.float32, device="cuda")
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    made = []
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        t = threading.Thread(target=lambda: made.append((create(0), N.last_error())))
        t.start()
        t.join()
        y.copy_(x).mul_(2.0)
    assert made[0][0], made
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, 2.0 * x)
    destroy(made[0][0])


@pytest.mark.gpu
def test_recorded_grid_builds(cuda):
    """A build and a query recorded after a first build grew the buffers, replayed, and builds after
    that: each finds the running state as it has to be."""
    import numpy as np
    import torch
    from imbatracer_b200.hashgrid import HashGrid
    from tests.test_hashgrid import photon_cloud
    p = torch.from_numpy(photon_cloud(5000, 3)).cuda()
    q = p[:700].contiguous()
    grid = HashGrid(0)
    grid.build(p, 0.5)
    want = [t.clone() for t in grid.query(q, 8, with_d2=True)]
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        grid.build(p, 0.5, stream=s)
        got = grid.query(q, 8, with_d2=True, stream=s)
    for _ in range(3):
        for t in got:
            t.zero_()
        g.replay()
        torch.cuda.synchronize()
        for a, b in zip(want, got):
            assert torch.equal(a, b)
    grid.build(p[:3000].contiguous(), 0.5)
    again = HashGrid(0)
    again.build(p[:3000].contiguous(), 0.5)
    for a, b in zip(grid.query(q, 8, with_d2=True), again.query(q, 8, with_d2=True)):
        assert np.array_equal(a.cpu().numpy(), b.cpu().numpy())
