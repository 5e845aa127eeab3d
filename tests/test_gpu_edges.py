"""Kernels at the sizes where a branch of their dispatch or an edge of their
tiles could go wrong, against the oracle.  Whole numbers and moved values are
compared bit for bit."""
import numpy as np
import pytest

from neslgpu_gb300 import ops, workloads as W

pytestmark = pytest.mark.gpu


def _group(gpu):
    """Draws that one pass of RAND's largest grid makes (16 CTAs of 1024 draws per SM)."""
    return gpu.cvl.gcvl_sm_count() * 16 * 1024


@pytest.mark.parametrize("n", [1, 255, 256, 257, 1023, 1024, 1025, "g-1", "g", "g+1", "2g+777"])
def test_rand_group_edges(gpu, oracle, n):
    if isinstance(n, str):
        n = {"g-1": _group(gpu) - 1, "g": _group(gpu), "g+1": _group(gpu) + 1, "2g+777": 2 * _group(gpu) + 777}[n]
    r = W.rng(n % 9973)
    bounds = r.integers(1, 2 ** 31, size=n, dtype=np.int64).astype(np.int32)
    assert np.array_equal(ops.rand_u(gpu, bounds, seed=n + 5), ops.rand_u(oracle, bounds, seed=n + 5))
