"""The plain form, whose lanes trace their rays warp by warp and take new paths
from a queue: frames of one path, part of a warp, a launch small enough for one
path per lane, just past what is resident, and several times that, bit for bit
the sums of the one-thread diagnostic's paths, on both trees."""
import numpy as np
import pytest

from test_gpu_ext_shade import request, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [0, 8])
@pytest.mark.parametrize("ext", [False, True])
@pytest.mark.parametrize("size", [(1, 1, 1, 1, 7), (7, 5, 1, 2, 3), (97, 61, 3, 1, 7), (611, 383, 1, 2, 2),
                                  (433, 300, 4, 1, 7)])
def test_frames_are_the_paths(size, ext, width):
    from shiro_gb300 import GpuBackend

    sc = scene()
    if not ext:
        lean = sc.materials[-1]
        sc.materials[:] = [lean] * len(sc.materials)
    cam, st = request(*size)
    with GpuBackend(0) as gpu:
        gpu.set_bvh_width(width)
        fb = gpu.render(sc, cam, st)
        n, spp = st.width * st.height, st.samples_per_pixel
        pixels = np.arange(n, dtype=np.uint32)
        rgb, alb, nrm = (np.zeros((n, 3), np.float32) for _ in range(3))
        hit, depth = np.zeros(n, np.float32), np.full(n, np.inf, np.float32)
        for k in range(spp):
            p = gpu.render_paths(sc, cam, st, pixels, np.full(n, k, np.uint32))
            rgb += p[:, 0:3]
            alb += p[:, 3:6]
            nrm += p[:, 6:9]
            hit += np.isfinite(p[:, 9])
            depth = np.minimum(depth, p[:, 9])
    beauty = np.concatenate([rgb, hit[:, None]], 1) / np.float32(spp)
    inv = np.float32(1.0) / np.float32(spp)
    for name, want in (("beauty", beauty), ("albedo", alb * inv), ("normal", nrm * inv), ("depth", depth)):
        got = np.ascontiguousarray(getattr(fb, name), np.float32).reshape(want.shape)
        assert np.array_equal(got.view(np.uint32), np.ascontiguousarray(want).view(np.uint32)), name
