"""The compressed wide BVH and its stages where they can go wrong: large
triangles kept out of the Morton tree (each a leaf of its own under the root,
up to the limit of 8 and past it), trees smaller than one wide node, equal
distances, and queues shorter and longer than a warp's chunk.  Hits, distances
and occlusion are compared bit for bit with the CPU oracle (the same
Moller-Trumbore arithmetic); the wavefront stages' frames with the plain
form's."""
import numpy as np
import pytest

import oracle
from oracle import api

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def port():
    oracle.build_port()
    return oracle.port_checker()


def soup(small, large, seed, repeat=1):
    """`small` little triangles in a box, `large` ones spanning it; the small mesh `repeat` times over (ties)."""
    from shiro_gb300 import DomeLight, Mesh, Scene, lambert, scenes

    rng = np.random.default_rng(seed)
    meshes = []
    if small:
        c = rng.uniform(-1, 1, (small, 1, 3))
        p = (c + rng.normal(0, 0.08, (small, 3, 3))).astype(np.float32).reshape(-1, 3)
        for _ in range(repeat):
            meshes.append(Mesh(p, np.arange(3 * small, dtype=np.uint32), None, 0))
    if large:
        p = rng.uniform(-1.5, 1.5, (large, 3, 3)).astype(np.float32)
        p[:, 1] += 3.0
        p[:, 2, 2] -= 3.0
        meshes.append(Mesh(p.reshape(-1, 3), np.arange(3 * large, dtype=np.uint32), None, 1))
    return Scene(materials=[lambert((0.7, 0.5, 0.3)), lambert((0.2, 0.6, 0.4))], meshes=meshes,
                 dome_lights=[DomeLight(env=scenes.procedural_hdri(32, 16, seed))])


@pytest.mark.parametrize("small,large,repeat", [(1, 0, 1), (2, 0, 1), (9, 0, 1), (20, 1, 1), (20, 2, 1), (40, 5, 1),
                                                (300, 8, 1), (300, 11, 1), (33, 3, 2), (2000, 2, 1)])
def test_wide_hits_match_oracle(port, small, large, repeat):
    from shiro_gb300 import GpuBackend

    scene = soup(small, large, 31 * small + large, repeat)
    rng = np.random.default_rng(small)
    n = 4099
    o = rng.uniform(-3, 3, (n, 3)).astype(np.float32)
    d = (rng.uniform(-1, 1, (n, 3)) - o).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[:6] = np.array([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1]], np.float32)
    tmax = rng.uniform(0.5, 6.0, n).astype(np.float32)
    want = api.trace_rays(port, scene, o, d, tmax)
    with GpuBackend(0) as gpu:
        for width in (8, 2):
            gpu.set_bvh_width(width)
            got = gpu.trace_rays(scene, o, d, tmax)
            for g, w, what in zip(got, want, ("triangle", "distance", "occlusion")):
                assert np.array_equal(g, w), f"{what} on the {width}-wide BVH"


@pytest.mark.parametrize("width,height,spp", [(1, 1, 1), (7, 5, 1), (33, 1, 2), (64, 48, 3)])
@pytest.mark.parametrize("small,large", [(2, 0), (40, 5), (600, 2)])
def test_stages_match_plain(small, large, width, height, spp):
    from shiro_gb300 import GpuBackend, RenderSettings, scenes

    scene = soup(small, large, 7 * small + large)
    cam = scenes.look_at((0.5, 1.0, 4.0), (0.0, 0.0, 0.0), 50.0, width / height)
    st = RenderSettings(width=width, height=height, samples_per_pixel=spp, max_depth=6, diffuse_depth=6,
                        specular_depth=6, backend=1)
    with GpuBackend(0) as gpu:
        ref = gpu.render(scene, cam, st)
        for coop in (2, 1):
            gpu.set_wavefront_config(use_graph=1, coop_extend=coop, coop_occlude=coop)
            (fb,) = gpu.render_batch(scene, [(cam, st)])
            for k in ("beauty", "albedo", "normal", "depth"):
                assert np.array_equal(getattr(fb, k).view(np.uint32), getattr(ref, k).view(np.uint32)), (k, coop)
