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
