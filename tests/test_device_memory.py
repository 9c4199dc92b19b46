"""Device memory that calls take: algorithms hold no buffers they never fill."""
import pytest

from tests.test_pt import small_mixed_scene

MB = 1 << 20


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
