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
        gpu.set_wavefront_config(use_graph=1, shade_block=192)
        tuned = gpu.autotune(sc, cam, st)
        assert tuned["shade_block"] == 192
        assert gpu.wavefront_config()["shade_block"] == 192
        sc.materials[:] = [sc.materials[-1]] * len(sc.materials)
        assert gpu.autotune(sc, cam, st)["shade_block"] in (64, 128, 192, 256)
