"""Device memory of scene uploads, over a CUDA runtime without a device
(tests/cpp/fake_cuda.cpp): any allocation may fail, and a call that fails leaves
nothing queued behind it."""
import ctypes as C
import glob
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def lib():
    from shiro_gb300 import build

    build.build()
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    out = os.path.join(HERE, "cpp", "_build", "libshiro_gpu_fake.so")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    objs = sorted(glob.glob(os.path.join(build.BUILD, "*.o")))
    r = subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", cuda,
                        "-o", out, os.path.join(HERE, "cpp", "fake_cuda.cpp")] + objs + ["-pthread", "-ldl"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    so = C.CDLL(out)
    p, u = C.c_void_p, C.c_size_t
    for name, args, res in (("fake_reset", [C.c_long, u], None), ("fake_mallocs", [], C.c_long),
                            ("fake_live_bytes", [], u), ("fake_busy_streams", [], C.c_int), ("fake_pool_new", [], p),
                            ("fake_pool_delete", [p], None), ("fake_pool_get", [p, u], p), ("fake_pool_put", [p, p], None),
                            ("shiro_gpu_create", [C.c_int, p], C.c_int), ("shiro_gpu_destroy", [p], None),
                            ("shiro_gpu_upload_scene", [p, p], C.c_int), ("shiro_gpu_set_bvh_build", [p, C.c_uint32], C.c_int),
                            ("shiro_gpu_set_params", [p] * 5, C.c_int), ("shiro_gpu_last_error", [p], C.c_char_p),
                            ("shiro_gpu_last_stats", [p, p], C.c_int), ("shiro_gpu_trim", [p], C.c_int)):
        f = getattr(so, name)
        f.argtypes, f.restype = args, res
    return so


ANY = (1 << 64) - 1


@pytest.fixture
def context(lib):
    lib.fake_reset(-1, ANY)
    ctx = C.c_void_p()
    assert lib.shiro_gpu_create(0, C.byref(ctx)) == 0
    assert lib.shiro_gpu_set_bvh_build(ctx, 0) == 0
    yield ctx
    lib.fake_reset(-1, ANY)
    lib.shiro_gpu_destroy(ctx)
    assert lib.fake_live_bytes() == 0


def scene():
    from shiro_gb300 import scenes
    from shiro_gb300.abi import MarshalledScene

    sc = scenes.sphere_scene(16, 8, segments=8, rings=6)
    sc.materials[1].emission_strength, sc.materials[1].emission_color = 2.0, (1.0, 1.0, 1.0)
    return MarshalledScene(sc)


def test_an_upload_succeeds_after_one_that_ran_out_of_memory(lib):
    from shiro_gb300.abi import SHIRO_ERR_OUT_OF_MEMORY as OUT_OF_MEMORY

    ms = scene()
    total, failed = 1, 0
    k = 1
    while k <= total:
        lib.fake_reset(-1, ANY)
        ctx = C.c_void_p()
        assert lib.shiro_gpu_create(0, C.byref(ctx)) == 0
        lib.shiro_gpu_set_bvh_build(ctx, 0)
        lib.fake_reset(k, ANY)
        rc = lib.shiro_gpu_upload_scene(ctx, ms.ref())
        if rc != 0:
            failed += 1
            total = k + 1
            assert rc == OUT_OF_MEMORY, (k, rc, lib.shiro_gpu_last_error(ctx))
        assert lib.fake_busy_streams() == 0, (k, rc)
        lib.fake_reset(-1, ANY)
        assert lib.shiro_gpu_upload_scene(ctx, ms.ref()) == 0, (k, lib.shiro_gpu_last_error(ctx))
        lib.shiro_gpu_destroy(ctx)
        assert lib.fake_live_bytes() == 0
        k += 1
    assert failed > 40


def test_a_refused_parameter_update_leaves_nothing_queued(lib, context):
    """The materials are written before the missing texture is noticed."""
    ms = scene()
    ms.desc.dome_light_count = 0
    assert lib.shiro_gpu_upload_scene(context, ms.ref()) == 0
    rough, env = np.full(2, 0.5, np.float32), np.ones((8, 16, 3), np.float32)
    assert lib.shiro_gpu_set_params(context, None, rough.ctypes.data, None, env.ctypes.data) == -1
    assert b"no environment texture" in lib.shiro_gpu_last_error(context)
    assert lib.fake_busy_streams() == 0


def test_pool_takes_no_more_than_asked_where_that_decides(lib):
    """Blocks of common sizes are up to an eighth larger than asked; not those
    too large to be kept, nor where only the size asked for is left."""
    pool = lib.fake_pool_new()
    lib.fake_reset(-1, ANY)
    large = (5 << 30) + 512  # past the pool's bound of idle bytes
    p = lib.fake_pool_get(pool, large)
    assert p and lib.fake_live_bytes() == large
    lib.fake_pool_put(pool, p)
    assert lib.fake_live_bytes() == 0
    asked = (64 << 20) + 512
    lib.fake_reset(-1, asked)
    p = lib.fake_pool_get(pool, asked)
    assert p and lib.fake_live_bytes() == asked
    lib.fake_pool_put(pool, p)
    lib.fake_reset(-1, ANY)
    lib.fake_pool_delete(pool)
    assert lib.fake_live_bytes() == 0


def test_pool_reuses_bounds_and_retries(lib):
    pool = lib.fake_pool_new()
    lib.fake_reset(-1, ANY)
    a = lib.fake_pool_get(pool, 1000)
    lib.fake_pool_put(pool, a)
    assert lib.fake_pool_get(pool, 900) == a and lib.fake_mallocs() == 1  # the same block for a similar size
    b = lib.fake_pool_get(pool, 1000)
    assert b != a  # the first is in use
    lib.fake_pool_put(pool, b)
    c = lib.fake_pool_get(pool, 100)
    assert c != b  # the idle one is too large for this
    lib.fake_pool_put(pool, a)
    lib.fake_pool_put(pool, c)
    big = [lib.fake_pool_get(pool, 400 << 20) for _ in range(3)]
    for p in big:
        lib.fake_pool_put(pool, p)
    assert lib.fake_live_bytes() <= 1 << 30  # 1.2 GB given back: the bound's worth is kept
    lib.fake_reset(-1, 900 << 20)
    p = lib.fake_pool_get(pool, 850 << 20)  # fits only once the idle ones are gone
    assert p and lib.fake_live_bytes() <= 900 << 20
    lib.fake_pool_put(pool, p)
    lib.fake_reset(-1, ANY)
    lib.fake_pool_delete(pool)
    assert lib.fake_live_bytes() == 0


def test_device_bytes_and_trim(lib, context):
    """What a context says it holds is what is allocated; trimming gives back
    what its scene does not need, and the next upload takes it again."""
    from shiro_gb300.abi import RenderStats

    ms, st = scene(), RenderStats()

    def held():
        assert lib.shiro_gpu_last_stats(context, C.byref(st)) == 0
        assert st.device_bytes == lib.fake_live_bytes()
        return st.device_bytes

    assert lib.shiro_gpu_upload_scene(context, ms.ref()) == 0
    whole = held()
    assert lib.shiro_gpu_trim(context) == 0
    assert held() < whole
    assert lib.shiro_gpu_upload_scene(context, ms.ref()) == 0  # the geometry stays: shading blocks alone
    held()
    lib.fake_reset(1, ANY)  # no new memory: the idle blocks serve
    assert lib.shiro_gpu_upload_scene(context, ms.ref()) == 0
    assert lib.shiro_gpu_trim(None) == -1
