"""The dome tables at row widths and heights around a warp's 32, with rows and
texels without weight, bit for bit the reference's CDFs and masses and the
sequential alias sweep."""
import numpy as np
import pytest

from test_gpu_env_alias import _reference_mass

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (31, 3), (32, 33), (33, 32), (97, 1), (2, 1025), (640, 65)])
def test_tables_at_edge_sizes(w, h):
    import oracle
    from oracle import api
    from shiro_gb300 import GpuBackend, scenes
    from shiro_gb300.abi import DomeLight, Scene

    rng = np.random.default_rng(1000 * w + h)
    env = np.ascontiguousarray(rng.exponential(1.0, (h, w, 3)).astype(np.float32) ** 3)
    env[rng.random((h, w)) < 0.1] = 0.0
    if h > 2:
        env[h // 2] = 0.0
    base = scenes.sphere_scene(env_width=16, env_height=8)
    with GpuBackend(0) as gpu:
        gpu.upload_scene(Scene(materials=base.materials, meshes=base.meshes, dome_lights=[DomeLight(env=env)]))
        tab = gpu.env_tables(0)
    row, cond, mass = _reference_mass(env)
    for name, want in (("row_cdf", row), ("cond_cdf", cond), ("mass", mass)):
        assert np.array_equal(tab[name].view(np.uint32).ravel(), want.view(np.uint32).ravel()), name
    thr, alias = api.env_alias(oracle.port_checker(), env)
    assert np.array_equal(tab["alias_threshold_bits"], thr)
    assert np.array_equal(tab["alias_index"], alias)
