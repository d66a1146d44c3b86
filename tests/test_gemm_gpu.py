"""tcgen05 GEMM against a plain PyTorch fp32 reference of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, w, bias, residual, act):
    y = a.float() @ w.float().t()
    if bias is not None:
        y = y + bias.float()
    if act == "silu":
        y = torch.nn.functional.silu(y)
    elif act == "gelu_tanh":
        y = torch.nn.functional.gelu(y, approximate="tanh")
    if residual is not None:
        y = y + residual.float()
    return y


def _check(T, N, K, *, mode=-1, block_n=0, ctas=0, bias=False, residual=False, act=None, out_dtype=torch.bfloat16):
    from inference_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T * 7919 + N * 31 + K)
    a = (torch.randn(T, K, device="cuda", generator=g) * 0.5).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).bfloat16()
    b = (torch.randn(N, device="cuda", generator=g) * 0.1).bfloat16() if bias else None
    r = (torch.randn(T, N, device="cuda", generator=g) * 0.5).bfloat16() if residual else None
    y = ops.gemm_bf16(a, w, bias=b, residual=r, act=act, mode=mode, block_n=block_n, ctas=ctas,
                      out_dtype=out_dtype)
    ops.check_status()
    ref = _ref(a, w, b, r, act)
    err = (y.float() - ref).abs().max().item()
    scale = ref.abs().max().item() + 1e-6
    tol = 2e-2 if out_dtype == torch.bfloat16 else 2e-3
    assert err / scale < tol, f"T={T} N={N} K={K} mode={mode} bn={block_n} ctas={ctas}: err {err} scale {scale}"
    return y


@pytest.mark.parametrize("T", [1, 5, 16, 33, 64, 128, 200, 256])
def test_swapped_small_tokens(T):
    _check(T, 512, 256)
    _check(T, 384, 1024, bias=True, residual=True)


@pytest.mark.parametrize("T", [65, 128, 129, 200, 256])
def test_swapped_kernel_of_many_tokens(T):
    """The 128- and 256-wide tiles of the weights-as-M kernel and their stream-K sums: asked for, with a number of CTAs, and
    taken for an odd or a small number of outputs."""
    _check(T, 512, 256, mode=1)
    _check(T, 384, 1024, mode=1, bias=True, residual=True)
    _check(T, 1024, 2048, mode=1, ctas=20, act="silu")
    _check(T, 384, 1024, ctas=7, bias=True)
    _check(T, 777, 1032, bias=True, residual=True, act="gelu_tanh")
    _check(T, 96, 4096, out_dtype=torch.float32)


@pytest.mark.parametrize("ctas", [-1, 3, 7, 20, 148])
def test_stream_k_deterministic(ctas):
    y0 = _check(8, 1024, 2048, mode=1, ctas=ctas, bias=True, act="silu")
    y1 = _check(8, 1024, 2048, mode=1, ctas=ctas, bias=True, act="silu")
    assert torch.equal(y0, y1)
    _check(300, 640, 1024, mode=0, ctas=ctas, residual=True)


@pytest.mark.parametrize("shape", [(300, 256, 128), (512, 1024, 512), (1000, 776, 328), (129, 4096, 4096)])
@pytest.mark.parametrize("block_n", [0, 64, 128])
def test_tokens_as_m(shape, block_n):
    T, N, K = shape
    _check(T, N, K, mode=0, block_n=block_n)
    _check(T, N, K, mode=0, block_n=block_n, bias=True, residual=True, act="gelu_tanh")


def test_fp32_out_and_ragged_edges():
    _check(77, 1000, 264, mode=0, out_dtype=torch.float32)
    _check(7, 1000, 264, mode=1, out_dtype=torch.float32, bias=True)
    _check(40, 136, 72, mode=1)
    _check(260, 136, 72)


def test_llama_shapes():
    for T in (1, 8, 64):
        _check(T, 6144, 4096)
        _check(T, 4096, 14336, residual=True)
    _check(1024, 6144, 4096)
    _check(1024, 4096, 14336, residual=True)


def test_strided_views():
    from inference_b200 import ops

    a = (torch.randn(48, 1024, device="cuda") * 0.5).bfloat16()
    w = (torch.randn(256, 512, device="cuda") * 0.05).bfloat16()
    y = ops.gemm_bf16(a[:, 512:], w)
    ref = a[:, 512:].float() @ w.float().t()
    assert (y.float() - ref).abs().max().item() < 0.05 * ref.abs().max().item()


@pytest.mark.parametrize("cluster", [1, 2, 3, 5, 6, 8])
@pytest.mark.parametrize("T", [1, 7, 16, 31, 64])
def test_cluster_split_k_decode(T, cluster):
    y0 = _check(T, 1024, 2048, mode=2, ctas=cluster, bias=True, residual=True, act="silu")
    y1 = _check(T, 1024, 2048, mode=2, ctas=cluster, bias=True, residual=True, act="silu")
    assert torch.equal(y0, y1)
    _check(T, 1000, 1096, mode=2, ctas=cluster, out_dtype=torch.float32)


@pytest.mark.parametrize("N,K", [(512, 256), (2816, 2048), (200, 320)])
def test_grouped_gemm_matches_per_group_matmul(N, K):
    """Each 128-row tile multiplies the weight group its table entry names; skipped tiles stay untouched."""
    from inference_b200 import ops

    G = 5
    g = torch.Generator(device="cuda").manual_seed(0)
    w = (torch.randn(G, N, K, device="cuda", generator=g) * 0.05).bfloat16()
    table = torch.tensor([3, 0, -1, 4, 4, 1, -1, 2], dtype=torch.int32, device="cuda")
    R = table.numel() * 128
    a = torch.randn(R, K, device="cuda", generator=g).bfloat16()
    out = torch.full((R, N), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.gemm_bf16_grouped(a, w, table, out=out)
    ops.check_status()
    for i, e in enumerate(table.tolist()):
        rows = slice(i * 128, (i + 1) * 128)
        if e < 0:
            assert torch.all(out[rows] == 7.0)
            continue
        ref = a[rows].float() @ w[e].float().t()
        torch.testing.assert_close(out[rows].float(), ref, rtol=2e-2, atol=2e-2)
    act = ops.gemm_bf16_grouped(a, w, table, act="silu")
    ref = torch.nn.functional.silu(a[:128].float() @ w[3].float().t())
    torch.testing.assert_close(act[:128].float(), ref, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("T,F,K,act", [(1, 256, 1024, "silu"), (64, 14336, 4096, "silu"), (17, 1000, 768, "gelu_tanh"),
                                       (200, 512, 1024, "silu")])
def test_gated_projection_pairs(T, F, K, act):
    """Gate-up projection with interleaved (gate, up) rows: fused epilogue (decode sizes) and GEMM + paired
    activation kernel (larger) both equal act(x Wg^T) * (x Wu^T)."""
    from inference_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T + F)
    wg = (torch.randn(F, K, device="cuda", generator=g) * 0.03).bfloat16()
    wu = (torch.randn(F, K, device="cuda", generator=g) * 0.03).bfloat16()
    x = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    pairs = torch.stack([wg, wu], dim=1).reshape(2 * F, K).contiguous()
    y = ops.linear_gated(x, pairs, act)
    ops.check_status()
    gate, up = x.float() @ wg.float().t(), x.float() @ wu.float().t()
    fn = torch.nn.functional.silu if act == "silu" else (lambda t: torch.nn.functional.gelu(t, approximate="tanh"))
    torch.testing.assert_close(y.float(), fn(gate) * up, rtol=3e-2, atol=3e-2)
    assert ops.gated_fused(T, 2 * F, K) == (T <= 64)


@pytest.mark.parametrize("block_n,splits", [(0, 0), (256, 1), (192, 2), (128, 1), (128, 3), (64, 2)])
@pytest.mark.parametrize("T,N,K", [(65, 128, 64), (255, 136, 584), (257, 520, 1096), (1000, 776, 2048)])
def test_pairs_of_sms(T, N, K, block_n, splits):
    """The two-SM kernel at the edges of its 256-row tiles, with columns and reduction blocks left over, every tile width and
    k-splits: bias, activation and residual, gates per group of rows, and gated pairs. One rounding to bf16 of an fp32 sum: at most half of the
    last of 8 bits, 2^-8 of the value; the sum itself is off by less than 1e-4 (terms of size 1, fast exponentials)."""
    from inference_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T + N)
    a = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    b = torch.randn(N, device="cuda", generator=g).bfloat16()
    r = torch.randn(T, N, device="cuda", generator=g).bfloat16()

    def close(y, want):
        ops.check_status()
        assert ((y.float() - want).abs() <= 2 ** -8 * want.abs() + 1e-4).all()

    kw = dict(mode=3, block_n=block_n, ctas=splits) if block_n else {}
    z = a.float() @ w.float().t()
    y = ops.gemm_bf16(a, w, bias=b, residual=r, act="silu", **kw)
    close(y, torch.nn.functional.silu(z + b.float()) + r.float())
    assert torch.equal(y, ops.gemm_bf16(a, w, bias=b, residual=r, act="silu", **kw))       # split order, not arrival order
    out = r.clone()
    ops.gemm_bf16(a, w, residual=out, out=out, **kw)
    close(out, z + r.float())
    torch.testing.assert_close(ops.gemm_bf16(a, w, out_dtype=torch.float32, **kw), z, rtol=1e-5, atol=1e-5)
    y = ops.gemm_bf16(a, w, bias=b, residual=r, act="silu", out_dtype=torch.float32, **kw)
    torch.testing.assert_close(y, torch.nn.functional.silu(z + b.float()) + r.float(), rtol=1e-5, atol=1e-4)
    if N % 16 == 0:
        close(ops.gemm_bf16(a, w, act="swiglu_pairs", **kw), torch.nn.functional.silu(z[:, 0::2]) * z[:, 1::2])
    if not block_n:
        gate = torch.randn(2, 2 * N, device="cuda", generator=g).bfloat16()[:, N:]
        rows = (T + 1) // 2
        y = ops.gemm_bf16(a, w, bias=b, residual=r, gate=gate, rows_per_gate=rows)
        close(y, (z + b.float()) * gate.float()[torch.arange(T, device="cuda") // rows] + r.float())


@pytest.mark.parametrize("splits", [1, 2])
@pytest.mark.parametrize("T,N,K", [(65, 128, 64), (255, 232, 584), (257, 352, 1096), (1000, 784, 2048), (300, 4480, 1024)])
def test_pairs_of_sms_with_tiles_of_224_columns(T, N, K, splits):
    """One half of the warps has 128 columns of a tile, the other 96; the same cases and tolerances as the other widths."""
    test_pairs_of_sms(T, N, K, 224, splits)


@pytest.mark.parametrize("T,N,K", [(65, 64, 2048), (256, 120, 520), (257, 96, 2048), (3863, 64, 2048), (1000, 72, 64)])
def test_few_columns_of_fp32(T, N, K):
    """Routers above 64 rows: k-splits on pairs of SMs, in the workspace or on scratch of the call's own. fp32 sums of K terms of size K^-0.5."""
    from inference_b200 import ops
    from inference_b200._native import kernels

    assert kernels().swb_gemm_takes_pairs(T, N, K, 0, 0, 0, 1, -1, 0, 0) and not kernels().swb_gemm_takes_pairs(T, N, K, 0, 0, 0, 1, -2, 0, 0)
    g = torch.Generator(device="cuda").manual_seed(T + N)
    a = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    y = ops.gemm_bf16(a, w, out_dtype=torch.float32)
    ops.check_status()
    torch.testing.assert_close(y.double(), a.double() @ w.double().t(), rtol=1e-5, atol=1e-5)
    assert torch.equal(y, ops.gemm_bf16(a, w, out_dtype=torch.float32))


@pytest.mark.parametrize("T,N,K,pairs", [(3072, 72, 64, 1), (3073, 72, 760, 0), (3073, 72, 768, 1), (3073, 64, 376, 0), (3073, 64, 384, 1), (4001, 120, 64, 0)])
def test_few_columns_of_many_rows(T, N, K, pairs):
    """On both sides of the lines up to which a short reduction of many rows goes to one SM a tile."""
    from inference_b200 import ops
    from inference_b200._native import kernels

    assert kernels().swb_gemm_takes_pairs(T, N, K, 0, 0, 0, 1, -1, 0, 0) == pairs
    g = torch.Generator(device="cuda").manual_seed(T + N)
    a = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    y = ops.gemm_bf16(a, w, out_dtype=torch.float32)
    ops.check_status()
    torch.testing.assert_close(y.double(), a.double() @ w.double().t(), rtol=1e-5, atol=1e-5)



@pytest.mark.parametrize("T,N,K", [(1100, 2048, 512), (300, 12288, 3072)])
def test_residual_in_place_above_256_rows(T, N, K):
    """The same product in place on the kernel of its choice (one SM a tile here) and on pairs of SMs: one rounding of fp32 sums each."""
    from inference_b200 import ops
    from inference_b200._native import kernels

    assert not kernels().swb_gemm_takes_pairs(T, N, K, 0, 1, 0, 0, -1, 0, 0)
    g = torch.Generator(device="cuda").manual_seed(T)
    a, r = torch.randn(T, K, device="cuda", generator=g).bfloat16(), torch.randn(T, N, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    want = a.float() @ w.float().t() + r.float()
    for kw in ({}, dict(mode=3)):
        out = r.clone()
        ops.gemm_bf16(a, w, residual=out, out=out, **kw)
        ops.check_status()
        assert ((out.float() - want).abs() <= 2 ** -8 * want.abs() + 1e-4).all(), kw


@pytest.mark.parametrize("T,N,K", [(1, 128, 512), (16, 776, 1096), (63, 3072, 4096), (64, 520, 584), (64, 512, 128)])
def test_gates_of_few_rows(T, N, K):
    """Gate and residual behind the decode kernel's fp32 sums (and, below its smallest reduction, in the two-SM kernel): one rounding to bf16.
    Rows that are not aligned are refused by either."""
    from inference_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T + N)
    a = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    b, r = torch.randn(N, device="cuda", generator=g).bfloat16(), torch.randn(T, N, device="cuda", generator=g).bfloat16()
    gate = torch.randn(2, 2 * N, device="cuda", generator=g).bfloat16()[:, N:]
    rows = (T + 1) // 2
    want = (a.double() @ w.double().t() + b.double()) * gate.double()[torch.arange(T, device="cuda") // rows] + r.double()
    y, out = ops.gemm_bf16(a, w, bias=b, residual=r, gate=gate, rows_per_gate=rows), r.clone()
    ops.gemm_bf16(a, w, bias=b, residual=out, gate=gate, rows_per_gate=rows, out=out)
    ops.check_status()
    assert ((y.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-4).all() and torch.equal(y, out)
    odd = torch.empty(T * N + 1, device="cuda", dtype=torch.bfloat16)[1:].view(T, N)
    for kw in (dict(residual=odd), dict(residual=r, out=odd)):
        with pytest.raises(ops.KernelError):
            ops.gemm_bf16(a, w, gate=gate, rows_per_gate=rows, **kw)
    with pytest.raises(ops.KernelError):
        ops.gemm_bf16(a, w, residual=r, gate=torch.zeros(2 * N + 1, device="cuda", dtype=torch.bfloat16)[1:].view(2, N), rows_per_gate=rows)


@pytest.mark.parametrize("T,N,K", [(300, 1024, 8192), (700, 512, 4096)])
def test_products_split_along_k_run_beside_each_other(T, N, K):
    """Products with k-splits on several streams at once, launched one by one and replayed from graphs: each gives the bits it gives
    alone. Streams and captures have counters of their own, which are zero afterwards."""
    from inference_b200 import ops
    from inference_b200._native import kernels
    from inference_b200.ops import gemm

    assert kernels().swb_gemm_split_bytes(T, N, K, 0, 0) > 0
    g = torch.Generator(device="cuda").manual_seed(T)
    streams = [torch.cuda.Stream() for _ in range(4)]
    data = [(torch.randn(T, K, device="cuda", generator=g).bfloat16(), torch.randn(N, K, device="cuda", generator=g).bfloat16()) for _ in streams]
    want = [ops.gemm_bf16(a, w) for a, w in data]
    torch.cuda.synchronize()
    graphs, outs = [], []
    for a, w in data:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs.append(ops.gemm_bf16(a, w))
        graphs.append(graph)
    for _ in range(20):
        got = []
        for s, (a, w) in zip(streams, data):
            with torch.cuda.stream(s):
                got.append([ops.gemm_bf16(a, w) for _ in range(3)])
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for xs, y in zip(got, want) for x in xs)
        for o in outs:
            o.zero_()
        torch.cuda.synchronize()
        for s, graph in zip(streams, graphs):
            with torch.cuda.stream(s):
                graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for x, y in zip(outs, want))
    ops.check_status()
    used = {k: t for k, t in gemm._SPLIT_COUNTERS.items() if k[1] in {s.cuda_stream for s in streams} and k[2] == 0}
    assert len({t.data_ptr() for t in used.values()}) == len(streams) and not any(t.any() for t in used.values())
    assert len({k[2] for k in gemm._SPLIT_COUNTERS}) > len(graphs)


@pytest.mark.parametrize("T,E,top,H,f,renorm", [(1, 4, 2, 64, 24, True), (33, 8, 8, 128, 72, False), (700, 5, 3, 200, 136, True),
                                                (2100, 64, 8, 256, 128, False), (300, 4, 2, 24, 8, True), (150, 3, 2, 72, 16, False),
                                                (40, 5003, 2, 64, 8, True), (20100, 5003, 2, 64, 8, False)])
@pytest.mark.parametrize("shared", [False, True])
def test_routed_segments_in_row_tiles(T, E, top, H, f, renorm, shared):
    """Dense expert segments in tiles of 256 rows (none, one row, remainders, several tiles an expert), gated pairs in the epilogue, and
    the weighted sum per token with a gated extra branch. Rounding: inputs are exact, u and y are bf16 (2^-9 each), the result too."""
    from inference_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T + E)

    def rnd(*shape, std=1.0):
        return (torch.randn(*shape, device="cuda", generator=g) * std).bfloat16()
    h, up, down, z = rnd(T, H), rnd(E, 2 * f, H, std=H ** -0.5), rnd(E, H, f, std=f ** -0.5), torch.randn(T, E, device="cuda", generator=g)
    z[:, 0] += 3.0          # a popular expert
    counters = ops.routing_counters(E, h.device)
    plan, rows = ops.logits_routing(z, E, top, rows=h, renorm=renorm, counters=counters, tiles256=True)
    y = ops.routed_gated_ffn(rows, up, down, plan, "silu")
    extra, gate = (rnd(T, H), torch.randn(T, 3, device="cuda", generator=g)[:, 1]) if shared else (None, None)
    got = ops.combine_routed(y, plan, 1.5, extra, gate)
    ops.check_status()
    assert not counters.any()
    share, which = z.double().softmax(-1).topk(top, -1)
    if renorm:
        share = share / share.sum(-1, keepdim=True)
    want = torch.zeros(T, H, dtype=torch.float64, device="cuda")
    for e in range(E):
        u = h.double() @ up[e].double().T
        o = (torch.nn.functional.silu(u[:, 0::2]) * u[:, 1::2]) @ down[e].double().T
        want += 1.5 * o * (share * (which == e)).sum(-1, keepdim=True)
    if shared:
        want += extra.double() * torch.sigmoid(gate.double())[:, None]
    assert (got.double() - want).norm() < 2.0 ** -8 * want.norm()


def test_pairs_of_sms_give_up_a_wait_together():
    """The epilogue's wait for one very long reduction (milliseconds) with a limit of a nanosecond: the launch ends by itself, its warps
    leave together, the status says where, and the next product is right."""
    from inference_b200 import ops
    from inference_b200._native import kernels

    L = kernels()
    K = 1 << 20
    a, w = (torch.full((n, K), 0.5, dtype=torch.bfloat16, device="cuda") for n in (300, 256))
    ops.check_status()
    L.swb_set_wait_limit_ns(1)
    try:
        ops.gemm_bf16(a, w, mode=3, block_n=256, ctas=1)
        st = ops.device_status()
    finally:
        L.swb_set_wait_limit_ns(2_000_000_000)
        L.swb_status_clear()
    assert st[0] == 1, st      # whichever role noticed first
    y = ops.gemm_bf16(a[:, :512], w[:, :512], mode=3, block_n=256, ctas=1)
    ops.check_status()
    assert (y == 128.0).all()


def test_counters_are_zero_again_after_a_wait_ran_out():
    """A launch that gives up may leave its k-splits partly counted (here: counters set by hand beside one such launch). Reading its
    status clears them, and the next split products are right."""
    from inference_b200 import ops
    from inference_b200._native import kernels
    from inference_b200.ops import gemm

    L = kernels()
    K = 1 << 20
    a, w = (torch.full((n, K), 0.5, dtype=torch.bfloat16, device="cuda") for n in (300, 256))
    dev = a.device
    ops.gemm_bf16(a[:, :4096], w[:, :4096])
    ops.check_status()
    L.swb_set_wait_limit_ns(1)
    try:
        ops.gemm_bf16(a, w, mode=3, block_n=256, ctas=2)
        gemm.split_counters(dev).fill_(1)
        ops.gemm_workspace(dev)[:L.swb_gemm_counter_bytes()].fill_(1)
        with pytest.raises(ops.KernelError):
            ops.check_status()
    finally:
        L.swb_set_wait_limit_ns(2_000_000_000)
        L.swb_status_clear()
    assert not gemm.split_counters(dev).any() and not ops.gemm_workspace(dev)[:L.swb_gemm_counter_bytes()].any()
    for T in (300, 200, 64):
        y = ops.gemm_bf16(a[:T, :8192], w[:, :8192], mode=3 if T > 64 else 1, block_n=128, ctas=2 if T > 64 else 20)
        ops.check_status()
        assert (y == 2048.0).all()


# widths that 256, 192 and 64 divide; a last tile of rows that is not full; columns that end inside a tile
@pytest.mark.parametrize("T,n1,n2,K", [(300, 768, 1024, 256), (513, 576, 400, 512), (1000, 64, 72, 128), (257, 9216, 12288, 192)])
@pytest.mark.parametrize("acts", [(None, "gelu_tanh"), ("silu", None)])
def test_one_product_into_two_outputs(T, n1, n2, K, acts):
    """The same bits as two products on the same kernel."""
    from inference_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T)
    a = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(n1 + n2, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    bias = torch.randn(n1 + n2, device="cuda", generator=g).bfloat16()
    first = torch.full((T, n1 + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    second = torch.full((T, n2 + 24), 7.0, device="cuda", dtype=torch.bfloat16)
    assert ops.gemm_bf16_two(a, w, first[:, :n1], second[:, 16:16 + n2], bias=bias, act=acts)
    ops.check_status()
    for got, rows, act in ((first[:, :n1], slice(0, n1), acts[0]), (second[:, 16:16 + n2], slice(n1, None), acts[1])):
        assert torch.equal(got, ops.gemm_bf16(a, w[rows], bias=bias[rows].contiguous(), act=act, mode=3, ctas=1))
    assert (first[:, n1:] == 7.0).all() and (second[:, :16] == 7.0).all() and (second[:, 16 + n2:] == 7.0).all()
    assert not ops.gemm_bf16_two(a, w, torch.empty(T, n1 + 8, device="cuda", dtype=torch.bfloat16)[:, 4:n1 + 4], second[:, 16:16 + n2], act=acts)
