"""Which kernel a product goes to, by the library's own rule (host code; no launch)."""
import pytest

from inference_b200._native import kernels


def _pairs(T, N, K, act=0, fp32=0, mode=-1, block_n=0, ctas=0):
    return bool(kernels().swb_gemm_takes_pairs(T, N, K, act, fp32, mode, block_n, ctas))


@pytest.mark.parametrize("T", [65, 200, 1000])
def test_a_forced_launch_shape_is_the_one_sm_kernels(T):
    assert _pairs(T, 4096, 4096)
    for kw in (dict(ctas=7), dict(ctas=148), dict(ctas=-1), dict(block_n=128), dict(mode=0), dict(mode=0, ctas=20)):
        assert not _pairs(T, 4096, 4096, **kw), kw
    assert _pairs(T, 4096, 4096, mode=3) and _pairs(T, 4096, 4096, mode=3, ctas=2)
    assert not _pairs(64, 4096, 4096) and not _pairs(T, 120, 4096) and not _pairs(T, 4100, 4096)
