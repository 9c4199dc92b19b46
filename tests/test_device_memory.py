"""Device memory that calls take: what fits without the second copy of a buffer that only makes a
call faster still fits, and algorithms hold no buffers they never fill."""
import gc

import numpy as np
import pytest

from imbatracer_b200 import native as N
from imbatracer_b200 import scene as S
from imbatracer_b200 import scenegen as G
from tests.test_pt import small_mixed_scene

MB = 1 << 20


class Filled:
    """All device memory taken but `left` bytes."""

    def __init__(self, left):
        import torch
        gc.collect()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        N.load().imbart_invalidate_scenes()
        N.load().imbart_clear_error()
        free = torch.cuda.mem_get_info()[0]
        self.block = torch.empty(max(free - left, 0), dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        import torch
        del self.block
        torch.cuda.empty_cache()
        N.load().imbart_invalidate_scenes()
        N.load().imbart_clear_error()


def held_by(run):
    """Device bytes that stay taken after run() (whose result is kept until they are read)."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    kept = run()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    used = before - torch.cuda.mem_get_info()[0]
    del kept
    return used


@pytest.mark.gpu
def test_light_tracing_holds_no_vertices(cuda):
    """276 B a path, two shadow queues of 68 B, 6 B for the grouping by material, no vertex cache."""
    from imbatracer_b200.integrators import GpuScene, VcmIntegrator
    gs = GpuScene(small_mixed_scene())
    paths = 400000

    def run():
        vi = VcmIntegrator(gs, "lt", 64, 48, light_path_count=paths)
        vi.begin_iteration(1)
        vi.light_pass(3)
        assert len(vi.light_vertices()) == 0
        return vi
    run().close()
    assert held_by(run) <= (276 + 2 * 68 + 6) * paths + 8 * MB


@pytest.mark.gpu
def test_photon_mapping_holds_no_shadow_rays(cuda):
    """PPM queues no shadow rays, however many connections the settings ask for."""
    from imbatracer_b200.integrators import GpuScene, VcmIntegrator
    gs = GpuScene(small_mixed_scene())
    w, h = 256, 192

    def run():
        vi = VcmIntegrator(gs, "ppm", w, h, light_path_count=1000, num_connections=100)
        vi.render(1, 3, 4)
        return vi
    run().close()
    # 292 B a camera path, 1,000 light paths and 2,000 vertices; a shadow queue would be 6.9 KB a path.
    assert held_by(run) <= 292 * w * h + 12 * MB


@pytest.mark.gpu
def test_second_queue_of_the_forked_graph_is_as_large_as_its_frames(cuda):
    """The forked graph's second shadow queue follows the frames that use it, not the largest frame
    the context has seen."""
    from imbatracer_b200.integrators import GpuScene, PathTracer
    gs = GpuScene(small_mixed_scene())
    pt = PathTracer(gs, max_path_len=3)
    lib = N.load()

    def frame(w, h, graphs):
        N.check(lib.imbart_pt_set_graphs(pt.ctx, graphs), "imbart_pt_set_graphs")
        pt.render(1, 5, w, h)
    frame(1024, 1024, 0)
    frame(16, 16, 1)
    assert held_by(lambda: frame(32, 32, 2)) <= 16 * MB       # 68 B a path; 71 MB for the large frame's
    frame(1024, 1024, 2)                                      # and it grows when a larger frame needs it
    a = pt.render(1, 5, 1024, 1024).cpu().numpy().astype(np.float64)
    N.check(lib.imbart_pt_set_graphs(pt.ctx, 0), "imbart_pt_set_graphs")
    b = pt.render(1, 5, 1024, 1024).cpu().numpy().astype(np.float64)
    # At most 3 bounces * 2 float32 terms a pixel, in another order: 2^-24 of the pixel each.
    assert (np.abs(a - b) <= 6 * 2.0 ** -23 * np.maximum(a, b)).all()
    pt.close()


@pytest.mark.gpu
def test_connections_fit_with_one_shadow_queue(cuda):
    """A camera pass whose shadow rays fit once but not twice."""
    from imbatracer_b200.integrators import GpuScene, VcmIntegrator
    gs = GpuScene(small_mixed_scene())
    w, h, conn = 512, 384, 127

    def image(left=None):
        vi = VcmIntegrator(gs, "bpt", w, h, max_path_len=3, light_path_count=500, num_connections=conn)
        vi.begin_iteration(1)
        vi.light_pass(3)
        img = vi._image(None)
        vi._image(None)                                        # memory for the test's own tensors
        if left is None:
            vi.camera_pass(4, img)
        else:
            with Filled(left):
                vi.camera_pass(4, img)
                assert N.last_error()[0] == 0
        out = img.cpu().numpy().astype(np.float64)
        vi.close()
        return out
    ref = image()
    queue = 68 * (1 + conn) * w * h                            # 1.7 GB
    got = image(queue + 512 * MB)
    # At most 3 * (conn + 2) float32 terms a pixel, in another order: 2^-24 of the pixel each.
    assert (np.abs(got - ref) <= 3 * (conn + 2) * 2.0 ** -23 * np.maximum(got, ref)).all()


def mirrors():
    """A mirror ball over a mirror ground: light paths that leave no vertices."""
    rng = np.random.default_rng(2)
    mirror = G.Material(G.MIRROR, color=(0.9, 0.9, 0.9), eta=0.2, kappa=3.0)
    parts = [(*G.displaced_sphere(rng, 2, (0, 0, 0), 1.0), 0),
             (*G.quad([-20, -1.6, -20], [-20, -1.6, 20], [20, -1.6, 20], [20, -1.6, -20]), 0),
             (np.array([[-3, 6, -2], [3, 6, 2], [3, 6, -2]], np.float32), np.array([[0, 1, 2]], np.int32), 1)]
    e = (30.0, 28.0, 24.0)
    light = tuple(np.array(p, np.float32) for p in ([-3, 6, -2], [3, 6, 2], [3, 6, -2], e))
    cam = G.Camera(pos=(0.0, 1.0, -8.0), dir=(0.0, -0.1, 1.0), up=(0.0, 1.0, 0.0), fov=60.0, width=64, height=48)
    return G.SceneDesc([G._merge(parts)], [G.Instance(0)], [mirror, G.Material(G.EMISSIVE, color=(0, 0, 0), emission=e)],
                       [light], cam, None, "mirrors")


@pytest.mark.gpu
def test_light_pass_fits_without_spare_room(cuda):
    """A first light pass that fits with one shadow queue and a cache for its paths alone."""
    from imbatracer_b200.integrators import GpuScene, VcmIntegrator
    gs = GpuScene(mirrors())
    paths = 4000000

    def counts(left=None):
        vi = VcmIntegrator(gs, "bpt", 64, 48, max_path_len=4, light_path_count=paths)
        vi.begin_iteration(1)
        img = vi._image(None)
        if left is None:
            vi.light_pass(3, image=img)
        else:
            with Filled(left):
                vi.light_pass(3, image=img)
                assert N.last_error()[0] == 0
        assert len(vi.light_vertices()) == 0
        vi.close()
        return vi.last_stats[:3].tolist()
    want = counts()
    # 276 B a path, one shadow queue of 68, room for a vertex of 112 each.
    assert counts((276 + 68 + 112) * paths + 64 * MB) == want


@pytest.mark.gpu
def test_scene_build_fits_mesh_by_mesh(cuda):
    """48 meshes of 328 k triangles: built together they need 540 B a triangle, one after another
    the records (128 B a triangle) and the scratch of one mesh."""
    rng = np.random.default_rng(3)
    v, f = G.displaced_sphere(rng, 7, (0, 0, 0), 1.0)
    mesh = S.Mesh(v, np.concatenate([f, np.zeros((len(f), 1), np.int32)], 1).astype(np.int32))
    meshes, insts = [mesh] * 48, []
    for k in range(48):
        m = np.eye(4, dtype=np.float32)
        m[:3, 3] = (3.0 * (k % 7), 3.0 * (k // 7), 0.0)
        insts.append(S.Instance(k, m))
    n = sum(m.triangle_count for m in meshes)
    rays = G.random_rays(rng, 4000, [-2] * 3, [20, 20, 2])
    from tests.test_gpu_build import trace

    def hits(left=None):
        if left is None:
            ds = S.DeviceScene.build_gpu(meshes, insts)
        else:
            with Filled(left):
                ds = S.DeviceScene.build_gpu(meshes, insts)
                assert N.last_error()[0] == 0
        assert ds.info.triangles == n
        out = trace(ds, rays)[0]
        ds.close()
        return out
    want = hits()
    assert (want["tri_id"] >= 0).sum() > 100
    assert np.array_equal(want, hits(int(200 * n)))
