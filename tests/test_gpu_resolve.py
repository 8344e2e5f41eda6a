"""Averaging of path records into the planes: batches whose frames begin and end
inside a warp, sample counts around the batch of loads, one pixel and whole
warps, bit for bit the sums of the listed paths in sample order."""
import numpy as np
import pytest

from test_gpu_ext_shade import request, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [[(1, 1, 1, 1, 3)], [(32, 1, 4, 1, 3), (64, 3, 5, 1, 3)],
                                   [(5, 3, 3, 1, 3), (33, 1, 8, 1, 3), (1, 1, 9, 1, 3), (31, 7, 1, 1, 3), (96, 5, 2, 1, 3)]])
def test_batch_planes_are_the_sums(batch):
    from shiro_gb300 import GpuBackend

    sc = scene()
    reqs = [request(*b) for b in batch]
    with GpuBackend(0) as gpu:
        for fb, (cam, st) in zip(gpu.render_batch(sc, reqs), reqs):
            n, spp = st.width * st.height, st.samples_per_pixel
            sums = np.zeros((n, 9), np.float32)
            hit, depth = np.zeros((n, 1), np.float32), np.full(n, np.inf, np.float32)
            for k in range(spp):
                p = gpu.render_paths(sc, cam, st, np.arange(n, dtype=np.uint32), np.full(n, k, np.uint32))
                sums += p[:, :9]
                hit[:, 0] += np.isfinite(p[:, 9])
                depth = np.minimum(depth, p[:, 9])
            cnt = np.float32(spp)
            inv = np.float32(1.0) / cnt
            for name, want in (("beauty", np.concatenate([sums[:, :3], hit], 1) / cnt), ("albedo", sums[:, 3:6] * inv),
                               ("normal", sums[:, 6:9] * inv), ("depth", depth)):
                got = np.ascontiguousarray(getattr(fb, name), np.float32).reshape(want.shape)
                assert np.array_equal(got.view(np.uint32), np.ascontiguousarray(want).view(np.uint32)), name
