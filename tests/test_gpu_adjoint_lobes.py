"""Material gradients of the lobes few materials have, each by itself and all
together, against finite differences of the frozen estimator; and the extended
replay stages at the edges of their queues against the one-thread replay.

The quotient is extrapolated from steps h and h / 2 (truncation O(h^4)); base
colour and metalness enter a BSDF at most quadratically, so 1e-2 is as good a
step as any, and the roughnesses of 0.4 to 0.55 move by 0.4 %.  A frame's 2 304
pixels each carry 2^-24 of rounding, which over a step of 2e-3 is 3e-5 of the
radiance in every one of them and averages out over the frame; the tolerance is
the 1e-2 of the other finite-difference tests."""
import numpy as np
import pytest

from test_gpu_adjoint import _loss, _step

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

NO_CLAMP = 2
LOBES = {
    "sheen": dict(sheen=0.8, sheen_color=(0.9, 0.5, 0.2), sheen_roughness=0.4),
    "subsurface": dict(subsurface=0.6, subsurface_radius=(0.5, 0.9, 0.3), subsurface_color=(0.9, 0.4, 0.3),
                       subsurface_scale=1.2, subsurface_anisotropy=0.3),
    "diffuse roughness": dict(diffuse_roughness=0.7),
    "anisotropy": dict(specular_anisotropy=0.7, specular_rotation=0.15),
    "tangent": dict(specular_anisotropy=-0.6, has_tangent_override=True, tangent_override=(0.1, 0.3, 1.0)),
    "thin film": dict(thin_film_thickness=480.0, thin_film_ior=1.4),
    "coat": dict(coat_weight=0.8, coat_roughness=0.2, coat_color=(0.8, 0.6, 0.9), coat_affect_color=0.6,
                 coat_affect_roughness=0.4, coat_anisotropy=0.5, coat_rotation=0.3),
    "coat normal": dict(coat_weight=0.6, coat_roughness=0.3, has_coat_normal_override=True,
                        coat_normal_override=(0.2, 1.0, 0.1)),
    "cut-out": dict(opacity=0.6, sheen=0.5),
}
LOBES["all"] = {k: v for name, kw in LOBES.items() if name not in ("tangent", "coat normal", "cut-out") for k, v in kw.items()}


def _parameters(scene):
    t = lambda v: torch.tensor(v, dtype=torch.float32, device="cuda")  # noqa: E731
    return dict(base_color=t([m.base_color for m in scene.materials]), roughness=t([m.roughness for m in scene.materials]),
                metallic=t([m.metallic for m in scene.materials]), env=t(scene.dome_lights[0].env))


@pytest.mark.parametrize("lobe", list(LOBES))
def test_finite_differences(lobe):
    from shiro_gb300 import DistantLight, GpuBackend, RenderSettings, scenes, standard_surface

    scene = scenes.sphere_scene(64, 32)
    scene.dome_lights[0].env = np.minimum(scene.dome_lights[0].env, np.float32(4.0))
    scene.distant_lights = [DistantLight(direction=(-0.4, -1.0, -0.3), radiance=(1.5, 1.4, 1.2))]
    scene.materials[0] = standard_surface((0.7, 0.5, 0.3), 0.45, 0.3, 1.5, **LOBES[lobe])
    scene.materials[1] = standard_surface((0.4, 0.6, 0.5), 0.55, 0.2, 1.5, **LOBES[lobe])
    st = RenderSettings(width=48, height=48, samples_per_pixel=8, max_depth=3, diffuse_depth=3, specular_depth=3, backend=1)
    cam = scenes.look_at((0.0, 1.6, 4.5), (0.0, 0.9, 0.0), 45.0, 1.0)
    gen = torch.Generator(device="cpu").manual_seed(7)
    d = torch.rand((48, 48, 4), generator=gen)
    d[..., 3] = 0.0
    d = d.cuda()
    p = _parameters(scene)
    with GpuBackend(0) as gpu:
        gpu.upload_scene(scene)
        grads = {}
        for form in (True, False):
            gpu.set_adjoint_form(form)
            grads[form] = {k: torch.zeros_like(v) for k, v in p.items()}
            gpu.adjoint(cam, st, d, grads[form], flags=NO_CLAMP)

        def quotient(name, i, h):
            out = []
            for s in (h, -h):
                q = {k: v.clone() for k, v in p.items()}
                q[name].view(-1)[i] += s
                out.append(_loss(d, gpu.render_frozen(cam, st, q["base_color"], q["roughness"], q["metallic"], q["env"],
                                                      flags=NO_CLAMP)))
            return (out[0] - out[1]) / (2.0 * h)

        errs = []
        for name, scale in (("base_color", 10.0), ("roughness", 4.0), ("metallic", 10.0)):
            g = grads[True][name].flatten()
            for i in range(g.numel()):
                h = scale * _step(name, float(p[name].flatten()[i]))
                fd = (4.0 * quotient(name, i, 0.5 * h) - quotient(name, i, h)) / 3.0
                errs.append((abs(float(g[i]) - fd) / max(abs(fd), 1e-3 * float(g.abs().max())), name, i, float(g[i]), fd))
        errs.sort(reverse=True)
        print("worst relative errors:", errs[:4])
        assert errs[0][0] <= 1e-2, errs[:4]
        for k, a in grads[True].items():
            b = grads[False][k]
            torch.testing.assert_close(a, b, rtol=1e-3, atol=1e-5 * float(b.abs().max()), msg=k)


@pytest.mark.parametrize("flags", [0, 2])
@pytest.mark.parametrize("width,height,spp,dome", [(1, 1, 1, 1), (9, 5, 1, 1), (33, 17, 2, 3), (40, 30, 2, 1), (64, 64, 8, 1)])
def test_extended_replay_matches_one_thread(width, height, spp, dome, flags):
    from shiro_gb300 import DistantLight, GpuBackend, RenderSettings, scenes

    scene = scenes.split_sphere_scene(parts=12, env_width=32, env_height=16, seed=5)
    scene.distant_lights = [DistantLight(direction=(-0.4, -1.0, -0.3), radiance=(1.5, 1.4, 1.2))]
    for k in (2, 9):
        scene.materials[k].emission_strength, scene.materials[k].emission_color = 4.0, (1.0, 0.8, 0.6)
    for k in (4, 7, 10):
        scene.materials[k].opacity = 0.4
    st = RenderSettings(width=width, height=height, samples_per_pixel=spp, max_depth=5, diffuse_depth=5, specular_depth=5,
                        dome_light_samples=dome, backend=1)
    cam = scenes.sphere_camera(width / height)
    g = torch.Generator(device="cuda").manual_seed(width)
    d = torch.rand((height, width, 4), generator=g, device="cuda")
    p = _parameters(scene)
    grads = []
    with GpuBackend(0) as gpu:
        gpu.upload_scene(scene)
        for wavefront in (True, False):
            gpu.set_adjoint_form(wavefront)
            out = {k: torch.zeros_like(v) for k, v in p.items()}
            gpu.adjoint(cam, st, d, out, flags=flags)
            grads.append(out)
    for k, a in grads[0].items():
        b = grads[1][k]
        assert torch.isfinite(a).all()
        torch.testing.assert_close(a, b, rtol=1e-3, atol=1e-5 * float(b.abs().max()) + 1e-12, msg=k)
