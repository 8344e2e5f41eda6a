"""Replay stages at the edges of their queues and light samples: one path, a
partial warp, several dome samples, no importance table (angular map), a
distant light, both clamps; gradients against the one-thread-per-path replay,
which sums the same terms in another order (float atomics: 1e-3 of each
gradient, 1e-5 of the largest)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, 2])
@pytest.mark.parametrize("width,height,spp,dome,angular", [(1, 1, 1, 1, False), (9, 5, 1, 1, False), (33, 17, 2, 3, False),
                                                           (40, 30, 2, 1, True), (64, 64, 8, 1, False)])
def test_wavefront_replay_matches_one_thread(width, height, spp, dome, angular, flags):
    import torch

    from shiro_gb300 import DistantLight, GpuBackend, RenderSettings, scenes
    from shiro_gb300.abi import ENV_ANGULAR

    scene = scenes.split_sphere_scene(parts=12, env_width=32, env_height=16, seed=5)
    scene.distant_lights = [DistantLight(direction=(-0.4, -1.0, -0.3), radiance=(1.5, 1.4, 1.2))]
    if angular:
        scene.dome_lights[0].layout = ENV_ANGULAR
    st = RenderSettings(width=width, height=height, samples_per_pixel=spp, max_depth=5, diffuse_depth=5, specular_depth=5,
                        dome_light_samples=dome, backend=1)
    cam = scenes.sphere_camera(width / height)
    g = torch.Generator(device="cuda").manual_seed(width)
    d = torch.rand((height, width, 4), generator=g, device="cuda")
    grads = []
    with GpuBackend(0) as gpu:
        gpu.upload_scene(scene)
        for wavefront in (True, False):
            gpu.set_adjoint_form(wavefront)
            out = {"base_color": torch.zeros((12, 3), device="cuda"), "roughness": torch.zeros(12, device="cuda"),
                   "metallic": torch.zeros(12, device="cuda"), "env": torch.zeros((16, 32, 3), device="cuda")}
            gpu.adjoint(cam, st, d, out, flags=flags)
            grads.append(out)
    for k, a in grads[0].items():
        b = grads[1][k]
        assert torch.isfinite(a).all()
        torch.testing.assert_close(a, b, rtol=1e-3, atol=1e-5 * float(b.abs().max()) + 1e-12, msg=k)
