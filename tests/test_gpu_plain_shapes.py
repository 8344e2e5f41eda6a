"""The plain form around the launch sizes where its shapes meet: as many paths as
the small shape takes, and some more (two launch shapes, the same frame bit for
bit), for shallow and deep paths, with and without the extended lobes, in small
and large scenes."""
import numpy as np
import pytest

from test_gpu_ext_shade import request, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,depth,halves", [("lean", 4, 5), ("lean", 5, 6), ("ext", 4, 3), ("ext", 7, 4), ("large", 3, 6),
                                               ("lean", 2, 2), ("field", 6, 4), ("field", 7, 6)])
def test_frames_on_both_sides_of_the_small_shape(kind, depth, halves):
    torch = pytest.importorskip("torch")
    from shiro_gb300 import GpuBackend, scenes

    if kind in ("large", "field"):  # 82 thousand triangles with an emitter; 307 thousand reflecting ones
        sc = scenes.field_scene(instances=16 if kind == "large" else 60, env_width=64, env_height=32)
    if kind == "large":
        sc.materials[3].emission_strength, sc.materials[3].emission_color = 2.0, (1.0, 0.9, 0.8)
    elif kind != "field":
        sc = scene()
        if kind == "lean":
            sc.materials[:] = [sc.materials[-1]] * len(sc.materials)
    lanes = torch.cuda.get_device_properties(0).multi_processor_count * 4 * 128
    frames = []
    with GpuBackend(0) as gpu:
        for height in (lanes * halves // 2 // 256, lanes * halves // 2 // 256 + 1):
            cam, st = request(256, height, 1, 1, depth)
            fb = gpu.render(sc, cam, st)
            (ref,) = gpu.render_batch(sc, [(cam, st)])
            for name in ("beauty", "albedo", "normal", "depth"):
                a, b = (np.ascontiguousarray(getattr(f, name)).view(np.uint32) for f in (fb, ref))
                assert np.array_equal(a, b), (height, name)
            frames.append(fb.beauty)
    assert all(np.isfinite(f).all() and f[..., :3].any() for f in frames)
