"""The device sampler where its table of radical inverses ends (4 096 indices
per base): bit for bit the oracle's values on both sides of the edge, at index
0, and far past it, in every base."""
import numpy as np
import pytest

import oracle
from oracle import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("index", [0, 1, 63, 4093, 4094, 4095, 4096, 4097, 1 << 20, 0xfffffffe])
def test_sampler_matches_oracle(index):
    from shiro_gb300 import GpuBackend

    oracle.build_port()
    branch = np.arange(0, 64, dtype=np.uint32)  # dimensions 0 .. 127: every base several times
    px = (branch * 37 % 1920).astype(np.uint32)
    py = (branch * 91 % 1080).astype(np.uint32)
    idx = np.full(branch.size, index, np.uint32)
    with GpuBackend(0) as gpu:
        got = gpu.sample(px, py, idx, branch)
    want = api.sampler(oracle.port_checker(), px, py, idx, branch)
    assert np.array_equal(got.view(np.uint32), np.asarray(want, np.float32).reshape(got.shape).view(np.uint32))
