"""Memory kept between uploads: counted, returned on request, and the resident
scene renders as before and after."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_trim_returns_memory_and_keeps_the_scene():
    torch = pytest.importorskip("torch")
    from shiro_gb300 import GpuBackend, scenes

    w = scenes.field_workload(64, 40, 2, 4, instances=16, env_width=512, env_height=256)
    with GpuBackend(0) as gpu:
        before = gpu.render(w.scene, w.camera, w.settings)
        torch.cuda.synchronize()
        held, free = gpu.last_stats()["device_bytes"], torch.cuda.mem_get_info()[0]
        gpu.trim()
        kept = gpu.last_stats()["device_bytes"]
        assert kept < held
        assert torch.cuda.mem_get_info()[0] > free
        after = gpu.render(w.scene, w.camera, w.settings)
        gpu.upload_scene(w.scene, force=True)
        again = gpu.render(w.scene, w.camera, w.settings)
    for fb in (after, again):
        assert np.array_equal(fb.beauty, before.beauty) and np.array_equal(fb.depth, before.depth)
