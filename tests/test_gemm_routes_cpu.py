"""Which kernel a product goes to, by the library's own rule (host code; no launch)."""
import pytest
import torch

from inference_b200._native import kernels


def _pairs(T, N, K, act=0, fp32=0, mode=-1, block_n=0, ctas=0, bias=0, residual=0):
    return bool(kernels().swb_gemm_takes_pairs(T, N, K, bias, residual, act, fp32, mode, block_n, ctas))


@pytest.mark.parametrize("T", [65, 200, 1000])
def test_a_forced_launch_shape_is_the_one_sm_kernels(T):
    assert _pairs(T, 4096, 4096)
    for kw in (dict(ctas=7), dict(ctas=148), dict(ctas=-1), dict(block_n=128), dict(mode=0), dict(mode=0, ctas=20)):
        assert not _pairs(T, 4096, 4096, **kw), kw
    assert _pairs(T, 4096, 4096, mode=3) and _pairs(T, 4096, 4096, mode=3, ctas=2)
    assert not _pairs(64, 4096, 4096) and not _pairs(T, 120, 4096) and not _pairs(T, 4100, 4096)


# (rows, outputs, reduction): measured faster on one SM per tile / on pairs of SMs, by 2 % or more
ONE_SM = [(257, 12288, 3072), (384, 12288, 3072), (300, 11008, 4096), (300, 10240, 2560), (300, 21504, 3072), (300, 28672, 4096), (600, 28672, 4096),
          (300, 24576, 2048), (300, 36864, 3072), (1100, 2048, 512)]
PAIRS = [(256, 12288, 3072), (400, 12288, 3072), (900, 12288, 3072), (3000, 12288, 3072), (257, 9216, 3072), (300, 6144, 4096), (300, 4096, 14336),
         (300, 16384, 4096), (300, 13824, 5120), (300, 3072, 12288), (513, 9216, 3072), (700, 28672, 4096), (8000, 28672, 4096), (300, 1024, 1024),
         (1231, 12288, 3072), (4608, 9216, 3072), (300, 18432, 3072), (300, 8192, 2048)]


def test_products_take_the_faster_of_both_kernels():
    for T, N, K in ONE_SM:
        assert not _pairs(T, N, K) and not _pairs(T, N, K, mode=-2), (T, N, K)
        assert _pairs(T, N, K, bias=1, act=2) and _pairs(T, N, K, fp32=1)       # the epilogue's share is smaller on pairs
        assert _pairs(T, N, K, act=3)                                   # a gated pair has the two-SM kernel alone
    for T, N, K in PAIRS:
        assert _pairs(T, N, K) and _pairs(T, N, K, bias=1, residual=1, act=1), (T, N, K)
    for kw in ({}, dict(bias=1, residual=1), dict(bias=1, act=1)):
        assert not _pairs(1100, 4096, 14336, **kw), kw


def test_gated_projections_pay_for_a_pass_only_where_that_is_faster():
    fused = kernels().swb_gemm_gated_in_pairs
    assert not any(fused(T, 2 * F, K) for T, F, K in [(257, 5632, 2048), (384, 5632, 2048), (257, 11008, 4096), (384, 11008, 4096), (64, 1024, 4096)])
    assert all(fused(T, 2 * F, K) for T, F, K in [(65, 14336, 4096), (256, 5632, 2048), (400, 5632, 2048), (900, 11008, 4096), (900, 14336, 4096),
                                                  (300, 8192, 2048), (300, 1024, 2048), (8000, 14336, 4096), (300, 64, 512)])


def test_convolutions_of_few_pixels_go_through_a_patch_matrix():
    from inference_b200 import ops

    def implicit(n, h, w, c, cout):
        return ops.conv3x3_implicit(torch.empty(n, h, w, c, device="meta"), cout)
    assert not any(implicit(*s) for s in [(1, 8, 8, 512, 512), (1, 1, 1, 64, 64), (4, 4, 4, 128, 128), (1, 9, 9, 32, 64), (1, 9, 9, 64, 4)])
    assert all(implicit(*s) for s in [(1, 5, 13, 512, 512), (1, 6, 12, 64, 8), (2, 6, 6, 64, 72), (1, 8, 16, 64, 3), (1, 152, 104, 512, 512)])
