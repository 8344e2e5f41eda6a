"""Listed rays, spread over warps by their number: one, around a warp, fewer than
the chip's warps, several a warp and whole warps give each ray the same answer,
on both trees, and the answers of the brute-force double-precision test where
a ray is not at an edge."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rays(n):
    rng = np.random.default_rng(5)
    o = rng.normal(size=(n, 3)) * 2.0 + np.array([0.0, 0.5, 0.0])
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return o.astype(np.float32), d.astype(np.float32), rng.uniform(0.1, 6.0, n).astype(np.float32)


@pytest.fixture(scope="module")
def answers():
    """Every ray through a large launch."""
    from shiro_gb300 import GpuBackend
    from test_gpu_ext_shade import scene

    sc, r = scene(), rays(100003)
    with GpuBackend(0) as gpu:
        return sc, r, [np.array(x) for x in gpu.trace_rays(sc, *r)]


@pytest.mark.parametrize("width", [0, 8])
@pytest.mark.parametrize("n", [1, 31, 33, 1003, 2433, 40007, 100003])
def test_answers_do_not_depend_on_the_number(answers, n, width):
    from shiro_gb300 import GpuBackend

    sc, (o, d, tmax), want = answers
    with GpuBackend(0) as gpu:
        gpu.set_bvh_width(width)
        got = gpu.trace_rays(sc, o[:n], d[:n], tmax[:n])
    for g, w in zip(got, want):
        assert np.array_equal(np.asarray(g), w[:n])


def test_answers_are_the_triangles(answers):
    sc, (o, d, tmax), (prim, t, occ) = answers
    tri = np.concatenate([np.asarray(m.positions, np.float64)[np.asarray(m.indices).reshape(-1, 3)] for m in sc.meshes])
    for k in range(0, 100003, 997):
        p0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
        pv = np.cross(d[k].astype(np.float64), e2)
        det = np.einsum("ij,ij->i", e1, pv)
        with np.errstate(divide="ignore", invalid="ignore"):
            tv = o[k].astype(np.float64) - p0
            u = np.einsum("ij,ij->i", tv, pv) / det
            qv = np.cross(tv, e1)
            v = qv @ d[k].astype(np.float64) / det
            tt = np.einsum("ij,ij->i", e2, qv) / det
        edge = 1.0e-4
        sure = (abs(det) > 1e-7) & (u > edge) & (v > edge) & (u + v < 1 - edge) & (tt > 2e-4)
        near = (abs(det) > 1e-9) & (u > -edge) & (v > -edge) & (u + v < 1 + edge) & (tt > 5e-5)
        if (sure != near).any():
            continue
        best = tt[sure].min() if sure.any() else np.inf
        assert (prim[k] == 0xFFFFFFFF) == (not sure.any())
        if sure.any():
            assert abs(t[k] - best) <= 1e-4 * max(1.0, best)
        if abs(best - tmax[k]) > 1e-3:
            assert bool(occ[k]) == bool(best <= tmax[k])
