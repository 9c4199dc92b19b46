"""The light pass's vertex append and path compaction at slot counts around a scan tile (1,024), and
shadow rays traced beside the next wavefront: one pass's cache is, bit for bit, the caches of
ranges of its paths put back in (wavefront, path) order, and an iteration equals its two passes cut
into ranges up to the order of the float sums."""
import numpy as np
import pytest

from imbatracer_b200 import distributed as D
from tests.test_pt import small_mixed_scene


@pytest.mark.gpu
@pytest.mark.parametrize("cuts", [(0, 1, 1024, 2049), (0, 1023, 2048, 3072, 3073), (0, 31, 63, 1088, 9001)])
def test_cache_of_path_ranges(cuda, cuts):
    from imbatracer_b200.integrators import GpuScene, VcmIntegrator
    gs = GpuScene(small_mixed_scene())
    kw = dict(max_path_len=6, light_path_count=cuts[-1])
    one = VcmIntegrator(gs, "vcm", 48, 32, **kw)
    one.begin_iteration(2)
    ref = one.light_pass(71, 5).cpu().numpy().astype(np.float64)
    cache = one.light_vertices()
    assert len(cache) > 0
    # One context for all ranges: its buffers shrink and grow with them.
    part = VcmIntegrator(gs, "vcm", 48, 32, **kw)
    part.begin_iteration(2)
    parts, waves, total = [], [], 0.0
    for a, b in zip(cuts[:-1], cuts[1:]):
        img, wv = part.light_pass_range(a, b - a, 71, 5)
        parts.append(part.light_vertices_device())
        waves.append(wv.tolist())
        total = total + img.cpu().numpy().astype(np.float64)
    glob = D.assemble_light_vertices(parts, waves).cpu().numpy()
    assert np.array_equal(glob.view(np.int32), cache.view(np.int32))
    # Sums of float32 terms in another order: n terms a pixel are off by at most n ulps (2^-24 each),
    # and no pixel takes more than the pass's vertices.
    assert np.abs(total - ref).max() <= len(cache) * 2.0 ** -23 * max(1.0, np.abs(ref).max())
    part.close()
    one.close()


@pytest.mark.gpu
@pytest.mark.parametrize("algo", ["vcm", "bpt", "pt"])
@pytest.mark.parametrize("max_paths", [257, 1536])
def test_camera_wavefronts_beside_shadow_rays(cuda, algo, max_paths):
    """Few paths in flight: many regenerating wavefronts, both shadow queues reused each time."""
    from imbatracer_b200.integrators import GpuScene, VcmIntegrator
    gs = GpuScene(small_mixed_scene())
    w, h = 48, 32
    kw = dict(max_path_len=6, light_path_count=1025)
    imgs = []
    for paths in (0, max_paths):
        vi = VcmIntegrator(gs, algo, w, h, max_paths_in_flight=paths, **kw)
        imgs.append(vi.render(1, 5, 6, 3).cpu().numpy().astype(np.float64))
        vi.close()
    vi = VcmIntegrator(gs, algo, w, h, **kw)
    vi.begin_iteration(1)
    img = vi.light_pass(5, 3) if algo != "pt" else None
    for a, n in ((0, 1), (1, 700), (701, w * h - 701)):
        img = vi.camera_pass_range(a, n, 6, image=img)
    imgs.append(img.cpu().numpy().astype(np.float64))
    vi.close()
    assert imgs[0].sum() > 0
    # One sample a pixel and the light splats: at most about 1,025 * 6 float32 terms a pixel, in
    # another order from image to image, 2^-24 of the sum each.
    scale = max(1.0, np.abs(imgs[0]).max())
    for other in imgs[1:]:
        assert np.abs(other - imgs[0]).max() <= 1025 * 6 * 2.0 ** -23 * scale
