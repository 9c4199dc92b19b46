"""The light pass's vertex append and path compaction at slot counts around a scan tile (1,024), and
shadow rays traced beside the next wavefront: one pass's cache is, bit for bit, the caches of
ranges of its paths put back in (wavefront, path) order, and an iteration equals its two passes cut
into ranges up to the order of the float sums."""
import numpy as np
import pytest

from imbatracer_b200 import distributed as D
from tests.test_pt import small_mixed_scene


def splats(vi, cache):
    """Per pixel, the light vertices of `cache` that can have been connected to it: those projecting
    there or to a neighbour (the projection here is in double)."""
    m = np.array(vi.camera.world_to_raster[:], np.float64).reshape(4, 4)
    t = np.concatenate([cache[:, :3], np.ones((len(cache), 1))], 1).astype(np.float64) @ m.T
    x, y = np.floor(t[:, 1] / t[:, 3]), np.floor(t[:, 0] / t[:, 3])
    n = np.zeros((vi.height + 2, vi.width + 2))
    seen = (x >= -1) & (x <= vi.width) & (y >= -1) & (y <= vi.height)
    np.add.at(n, (y[seen].astype(int) + 1, x[seen].astype(int) + 1), 1)
    return sum(n[dy:dy + vi.height, dx:dx + vi.width] for dy in range(3) for dx in range(3))


def assert_same_sums(a, b, terms):
    """Two float32 sums of the same `terms` nonnegative terms a pixel, in two orders: each is off by at
    most 2^-24 of the sum a term."""
    assert (np.abs(a - b) <= (terms * 2.0 ** -23)[..., None] * np.minimum(a, b) * (1 + 1e-3) + 1e-30).all()


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
    parts, waves, total, rays = [], [], 0.0, np.zeros(2, np.int64)
    for a, b in zip(cuts[:-1], cuts[1:]):
        img, wv = part.light_pass_range(a, b - a, 71, 5)
        parts.append(part.light_vertices_device())
        waves.append(wv.tolist())
        rays += part.last_stats[:2]
        total = total + img.cpu().numpy().astype(np.float64)
    glob = D.assemble_light_vertices(parts, waves).cpu().numpy()
    assert np.array_equal(glob.view(np.int32), cache.view(np.int32))
    assert np.array_equal(rays, one.last_stats[:2])              # closest-hit and shadow rays
    assert_same_sums(total, ref, splats(one, cache))
    part.close()
    one.close()


@pytest.mark.gpu
@pytest.mark.parametrize("algo", ["vcm", "bpt", "ppm", "lt", "pt"])
@pytest.mark.parametrize("max_paths", [257, 1536])
def test_camera_wavefronts_beside_shadow_rays(cuda, algo, max_paths):
    """Few paths in flight: many regenerating wavefronts, both shadow queues reused each time."""
    from imbatracer_b200.integrators import GpuScene, VcmIntegrator
    gs = GpuScene(small_mixed_scene())
    w, h = 48, 32
    kw = dict(max_path_len=6, light_path_count=1025)
    # The same seeds trace the same light paths whichever algorithm keeps their vertices.
    vi = VcmIntegrator(gs, "vcm", w, h, **kw)
    vi.begin_iteration(1)
    vi.light_pass(5, 3)
    # A camera path adds an emission, a shadow ray, a connection and a merge for each of 6 vertices.
    terms = 6 * 4 + splats(vi, vi.light_vertices())
    vi.close()
    imgs, rays = [], []
    for paths in (0, max_paths):
        vi = VcmIntegrator(gs, algo, w, h, max_paths_in_flight=paths, **kw)
        imgs.append(vi.render(1, 5, 6, 3).cpu().numpy().astype(np.float64))
        rays.append(vi.last_stats[:2].copy())
        vi.close()
    vi = VcmIntegrator(gs, algo, w, h, **kw)
    vi.begin_iteration(1)
    img = vi.light_pass(5, 3)
    assert algo in ("lt", "pt") or len(vi.light_vertices()) > 0
    rays.append(vi.last_stats[:2].copy())
    for a, n in ((0, 1), (1, 700), (701, w * h - 701)):
        img = vi.camera_pass_range(a, n, 6, image=img)
        rays[-1] += vi.last_stats[3:5]
    imgs.append(img.cpu().numpy().astype(np.float64))
    vi.close()
    assert imgs[0].sum() > 0
    for k in (1, 2):
        assert np.array_equal(rays[k], rays[0])
        assert_same_sums(imgs[k], imgs[0], terms)
