"""A path tracer's context that outlives a scene: the next scene may stand at the same device
addresses (the allocator hands a freed block out again), and the recorded frame graph must not be
replayed with what belonged to the old one: the start in the single instance's tree, its id."""
import numpy as np
import pytest

from imbatracer_b200 import scene as S
from imbatracer_b200 import scenegen as G


@pytest.mark.gpu
@pytest.mark.parametrize("graphs", [1, 2])
@pytest.mark.parametrize("built", ["gpu", "host"])
def test_frame_follows_a_replaced_scene(cuda, built, graphs):
    import torch
    from imbatracer_b200.integrators import GpuScene, PathTracer
    desc = G._sphere_field(3, 3, 2, 64, 48, "field")
    moved = np.eye(4, dtype=np.float32)
    moved[:3, 3] = (6.0, 2.0, 1.0)

    def traversal(inst):
        if built == "gpu":
            return S.DeviceScene.build_gpu(desc.meshes, [inst])
        return S.DeviceScene(S.build_traversal_data(desc.meshes, [inst]))

    # The shading data stays: it holds the instance's inverse linear part, which a translation keeps.
    gs = GpuScene(desc, gpu_build=True)
    image = torch.zeros((48, 64, 3), dtype=torch.float32, device="cuda")
    kept = PathTracer(gs, max_path_len=4, graphs=graphs)

    def frame(pt):
        image.zero_()
        pt.render(1, 9, 64, 48, image=image)
        return image.cpu().numpy().astype(np.float64)

    # A translation by nothing (identity), then a real one, then none again.
    for inst in (S.Instance(0), S.Instance(0, moved), S.Instance(0)):
        gs.trace_scene.close()
        gs.trace_scene = traversal(inst)
        got = frame(kept)
        new = PathTracer(gs, max_path_len=4, graphs=0)
        ref = frame(new)
        assert np.array_equal(kept.last_stats[:2], new.last_stats[:2])
        # At most 4 bounces * 2 float32 terms a pixel, in another order: 2^-24 of the pixel each.
        assert (np.abs(got - ref) <= 8 * 2.0 ** -23 * np.maximum(got, ref)).all()
        new.close()
    kept.close()
    gs.close()
