"""Autotuning on a scene with the extended lobes leaves the block size of the
reflecting scenes' shade stage, which such a scene does not use, as it was set."""
import pytest

from test_gpu_ext_shade import request, scene

pytestmark = pytest.mark.gpu


def test_shade_block_is_not_tuned_where_it_has_no_effect():
    from shiro_gb300 import GpuBackend

    sc = scene()
    cam, st = request(128, 96, 4, 1)
    with GpuBackend(0) as gpu:
        gpu.upload_scene(sc)
        base = gpu.wavefront_config()
        for _ in range(20):  # a trial of an identical launch wins by noise alone, now and then
            gpu.set_wavefront_config(**{**base, "use_graph": 1, "shade_block": 192})
            assert gpu.autotune(sc, cam, st)["shade_block"] == 192
        sc.materials[:] = [sc.materials[-1]] * len(sc.materials)
        assert gpu.autotune(sc, cam, st)["shade_block"] in (64, 128, 192, 256)
