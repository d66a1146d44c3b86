"""Wrappers for the media kernels: sampler axpy, GroupNorm(+SiLU), nearest upsample, row softmax, RGB8."""
from __future__ import annotations

import os

import torch

from .._native import kernels
from .runtime import check, ptr, require_cuda, stream_ptr


def axpy(a: float, x: torch.Tensor, b: float, y: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    """out = a * x + b * y (the flow-matching Euler update is axpy(1, x, dt, v))."""
    require_cuda(x, y)
    assert x.shape == y.shape and x.dtype == y.dtype and x.is_contiguous() and y.is_contiguous()
    if out is None:
        out = torch.empty_like(x)
    rc = kernels().swb_axpy(x.data_ptr(), y.data_ptr(), out.data_ptr(), x.numel(), a, b,
                            1 if x.dtype == torch.float32 else 0, stream_ptr())
    check(rc, "swb_axpy")
    return out


def groupnorm_nhwc(x: torch.Tensor, gamma: torch.Tensor, beta: torch.Tensor, groups: int = 32, eps: float = 1e-6,
                   silu: bool = False, out: torch.Tensor | None = None, sums: torch.Tensor | None = None) -> torch.Tensor:
    """x: [N, H, W, C] bf16 channels-last. GroupNorm with optional fused SiLU. sums fp32 [N, groups, 2]: each group's sum and sum of squares, where
    the kernel that made x has them (see conv3x3_sums); x is then read once."""
    require_cuda(x)
    N, H, W, C = x.shape
    assert x.is_contiguous() and x.dtype == torch.bfloat16
    if out is None:
        out = torch.empty_like(x)
    if sums is not None:
        assert sums.shape == (N, groups, 2) and sums.dtype == torch.float32 and sums.is_contiguous()
        rc = kernels().swb_groupnorm_apply(x.data_ptr(), sums.data_ptr(), gamma.data_ptr(), beta.data_ptr(), out.data_ptr(), N, H * W, C, groups,
                                           eps, 1 if silu else 0, stream_ptr())
        check(rc, "swb_groupnorm_apply")
        return out
    stats = torch.empty((N, groups, 2), dtype=torch.float32, device=x.device)
    rc = kernels().swb_groupnorm(x.data_ptr(), stats.data_ptr(), gamma.data_ptr(), beta.data_ptr(), out.data_ptr(), N,
                                 H * W, C, groups, eps, 1 if silu else 0, stream_ptr())
    check(rc, "swb_groupnorm")
    return out


def upsample2x_nhwc(x: torch.Tensor) -> torch.Tensor:
    require_cuda(x)
    N, H, W, C = x.shape
    out = torch.empty((N, 2 * H, 2 * W, C), dtype=x.dtype, device=x.device)
    check(kernels().swb_upsample2x(x.data_ptr(), out.data_ptr(), N, H, W, C, stream_ptr()), "swb_upsample2x")
    return out


def softmax_rows(scores: torch.Tensor, scale: float = 1.0) -> torch.Tensor:
    """fp32 [R, C] -> bf16 probabilities softmax(scale * scores)."""
    require_cuda(scores)
    assert scores.dtype == torch.float32 and scores.stride(1) == 1
    out = torch.empty(scores.shape, dtype=torch.bfloat16, device=scores.device)
    check(kernels().swb_softmax_rows(scores.data_ptr(), out.data_ptr(), scores.shape[0], scores.shape[1],
                                     scores.stride(0), out.stride(0), scale, stream_ptr()), "swb_softmax_rows")
    return out


def rgb8_nhwc(x: torch.Tensor) -> torch.Tensor:
    """[N, H, W, C>=3] bf16 in [-1, 1] -> uint8 [N, H, W, 3] (round half to even)."""
    require_cuda(x)
    N, H, W, C = x.shape
    out = torch.empty((N, H, W, 3), dtype=torch.uint8, device=x.device)
    check(kernels().swb_rgb8(x.data_ptr(), out.data_ptr(), N * H * W, C, stream_ptr()), "swb_rgb8")
    return out


def conv3x3_supported(x: torch.Tensor, cout: int = 8) -> bool:
    """Shapes the implicit-GEMM convolution takes: 64-channel slabs, and 16-byte rows of the output (any image size) or whole
    128-pixel tiles that are a run of one image row or a stack of whole rows."""
    N, H, W, C = x.shape
    return C % 64 == 0 and (cout % 8 == 0 or ((H * W) % 128 == 0 and (W % 128 == 0 or 128 % W == 0)))


def conv3x3_implicit(x: torch.Tensor, cout: int = 8) -> bool:
    """True when conv3x3_nhwc writes no patch matrix. Up to 64 pixels it does: the matrix is small, and its product runs on the decode kernel,
    which splits the reduction over the chip. 8 x 8 pixels, 512 -> 512 channels take 7.9 us so and 24.9 as one row of implicit
    tiles; 6 x 12 pixels 45 and 25."""
    return x.shape[0] * x.shape[1] * x.shape[2] > 64 and conv3x3_supported(x, cout)


def _rows_of_16_bytes(bias: torch.Tensor | None, res2: torch.Tensor | None) -> bool:
    return (bias is None or bias.data_ptr() % 16 == 0) and (res2 is None or (res2.data_ptr() % 16 == 0 and res2.stride(0) % 8 == 0))


def conv3x3_sums(x: torch.Tensor, w: torch.Tensor, bias: torch.Tensor | None, residual: torch.Tensor | None, groups: int) -> bool:
    """Whether conv3x3_nhwc of these operands can add up the sums of its output for a norm over `groups` groups of channels."""
    cout = w.shape[0]
    res2 = residual.reshape(-1, cout) if residual is not None else None
    return (cout % 8 == 0 and cout % groups == 0 and cout // groups in (4, 8, 16, 32) and _rows_of_16_bytes(bias, res2) and
            conv3x3_implicit(x, cout) and os.environ.get("SWB_CONV3X3", "implicit") != "im2col")


def conv3x3_nhwc(x: torch.Tensor, w: torch.Tensor, bias: torch.Tensor | None = None, residual: torch.Tensor | None = None,
                 act: str | None = None, sums: torch.Tensor | None = None) -> torch.Tensor:
    """3x3 convolution (stride 1, zero padding 1) of x [N, H, W, C] bf16 with w [Cout, 9 * C] (columns ordered ky, kx,
    c) -> [N, H, W, Cout], bias / activation / residual [N, H, W, Cout] in the epilogue. Implicit GEMM on the tcgen05
    kernel: the nine shifted views of x are fetched by TMA, no patch matrix is materialised. Shapes outside
    `conv3x3_implicit` take the patch-gather + GEMM path. sums fp32 [N, groups, 2] (where conv3x3_sums says so): the sum and the sum of squares of
    each group of neighbouring output channels are added to it."""
    from .gemm import ACT, gemm_bf16

    require_cuda(x, w)
    N, H, W, C = x.shape
    Cout = w.shape[0]
    assert x.is_contiguous() and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and w.shape[1] == 9 * C and w.stride(1) == 1
    res2 = residual.reshape(N * H * W, Cout) if residual is not None else None
    rows_ok = _rows_of_16_bytes(bias, res2)
    assert sums is None or (sums.dtype == torch.float32 and sums.is_contiguous() and sums.shape[::2] == (N, 2) and conv3x3_sums(x, w, bias, residual, sums.shape[1]))
    if not conv3x3_implicit(x, Cout if rows_ok else 1) or os.environ.get("SWB_CONV3X3", "implicit") == "im2col":
        return gemm_bf16(im2col3x3_nhwc(x), w, bias=bias, residual=res2, act=act).view(N, H, W, Cout)
    out = torch.empty((N * H * W, Cout), dtype=torch.bfloat16, device=x.device)
    if res2 is not None:
        assert res2.dtype == torch.bfloat16 and res2.stride(1) == 1
    rc = kernels().swb_conv3x3_nhwc_stats(x.data_ptr(), N, H, W, C, w.data_ptr(), w.stride(0), Cout, out.data_ptr(), out.stride(0),
                                          ptr(bias), ptr(res2), res2.stride(0) if res2 is not None else 0, ACT[act], ptr(sums),
                                          sums.shape[1] if sums is not None else 0, stream_ptr())
    check(rc, "swb_conv3x3_nhwc_stats")
    return out.view(N, H, W, Cout)


def conv3x3_of_norm(x: torch.Tensor, sums: torch.Tensor, gamma: torch.Tensor, beta: torch.Tensor, eps: float, w: torch.Tensor,
                    bias: torch.Tensor) -> torch.Tensor | None:
    """conv3x3_nhwc(groupnorm_nhwc(x, gamma, beta, groups, eps, silu=True, sums=sums), w, bias) for the eight output channels in which a decoder
    ends, in one pass over x that stores no normed copy of it. None where the kernel is not made for these operands (64 or 128 channels in, eight out, a bias)."""
    require_cuda(x)
    N, H, W, C = x.shape
    if C not in (64, 128) or w.shape != (8, 9 * C) or os.environ.get("SWB_CONV3X3", "implicit") == "im2col":
        return None
    if any(t.dtype != torch.bfloat16 or not t.is_contiguous() or t.data_ptr() % 16 for t in (x, gamma, beta, w, bias)) or sums.data_ptr() % 16:
        return None
    assert sums.shape[::2] == (N, 2) and sums.dtype == torch.float32 and sums.is_contiguous() and C % sums.shape[1] == 0
    assert gamma.numel() == beta.numel() == C and bias.numel() == 8
    out = torch.empty((N, H, W, 8), dtype=torch.bfloat16, device=x.device)
    check(kernels().swb_norm_silu_conv3x3_few(x.data_ptr(), N, H, W, C, sums.data_ptr(), sums.shape[1], gamma.data_ptr(), beta.data_ptr(), eps,
                                              w.data_ptr(), bias.data_ptr(), out.data_ptr(), stream_ptr()), "swb_norm_silu_conv3x3_few")
    return out


def im2col3x3_nhwc(x: torch.Tensor) -> torch.Tensor:
    """[N, H, W, C] bf16 -> [N*H*W, 9*C] patches (stride 1, zero padding 1), column order (kh, kw, c)."""
    require_cuda(x)
    N, H, W, C = x.shape
    assert x.is_contiguous() and x.dtype == torch.bfloat16
    out = torch.empty((N * H * W, 9 * C), dtype=x.dtype, device=x.device)
    check(kernels().swb_im2col3x3(x.data_ptr(), out.data_ptr(), N, H, W, C, stream_ptr()), "swb_im2col3x3")
    return out
