"""The extended shade stage (glass, media, emitters, cut-outs), whose blocks go
through its phases together: queues shorter than a block, of one entry, past
several blocks' shares, requests with fewer light samples than the wave's, and
every register cap, bit for bit the one-thread-per-path form's frames."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scene():
    from shiro_gb300 import (DistantLight, DomeLight, Material, Mesh, Scene, lambert, scenes, standard_surface,
                             usd_preview_surface)

    p, n, i = scenes.uv_sphere((0.0, 0.0, 0.0), 1.0, 16, 8)
    gp, gn, gi = scenes.ground_quad(8.0)
    mats = [standard_surface((1.0, 1.0, 1.0), 0.0, 0.0, 1.5, transmission=1.0),
            standard_surface((1.0, 1.0, 1.0), 0.2, 0.0, 1.4, transmission=0.8, transmission_depth=0.7,
                             transmission_color=(0.6, 0.8, 0.9), transmission_scatter=(0.2, 0.1, 0.1)),
            usd_preview_surface((0.7, 0.3, 0.2), 0.4, opacity=0.5),
            Material(emission_color=(1.0, 0.8, 0.6), emission_strength=4.0, base_color=(0.1, 0.1, 0.1)),
            standard_surface((0.6, 0.5, 0.2), 0.3, 0.0, 1.5, coat_weight=0.8, sheen=0.5, specular_anisotropy=0.5),
            lambert((0.5, 0.5, 0.5))]
    meshes = [Mesh(p * np.float32(0.5) + np.array([(k - 2) * 1.1, 0.5, 0.2 * k], np.float32), i, n, k) for k in range(5)]
    meshes.append(Mesh(gp, gi, gn, 5))
    return Scene(materials=mats, meshes=meshes, dome_lights=[DomeLight(env=scenes.procedural_hdri(64, 32, 3))],
                 distant_lights=[DistantLight(direction=(-0.3, -1.0, -0.2), radiance=(1.0, 1.0, 1.0))])


def request(width, height, spp, dome, depth=7):
    from shiro_gb300 import RenderSettings, scenes

    cam = scenes.look_at((0.4, 1.6, 4.5), (0.0, 0.5, 0.0), 50.0, width / height)
    return cam, RenderSettings(width=width, height=height, samples_per_pixel=spp, max_depth=depth, diffuse_depth=depth,
                               specular_depth=depth, dome_light_samples=dome, backend=1)


@pytest.mark.parametrize("regs", [80, 96, 128])
@pytest.mark.parametrize("sizes", [[(1, 1, 1, 1)], [(5, 3, 2, 1)], [(97, 61, 3, 1)], [(400, 300, 8, 1)],
                                   [(31, 17, 2, 1), (64, 40, 1, 4), (9, 9, 5, 2)]])
def test_frames_match_plain(sizes, regs):
    from shiro_gb300 import GpuBackend

    sc = scene()
    reqs = [request(*s) for s in sizes]
    with GpuBackend(0) as gpu:
        gpu.set_wavefront_config(use_graph=1, shade_regs=regs)
        fbs = gpu.render_batch(sc, reqs)
        for fb, (cam, st) in zip(fbs, reqs):
            ref = gpu.render(sc, cam, st)
            for k in ("beauty", "albedo", "normal", "depth"):
                assert np.array_equal(getattr(fb, k).view(np.uint32), getattr(ref, k).view(np.uint32)), k
