"""Weight-only quantised GEMM kernels against CPU dequantisation + fp32 matmul."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["Q4_K", "Q8_0", "AFFINE4", "AFFINE8"])
@pytest.mark.parametrize("T,N,K,splits", [(1, 256, 512, 0), (8, 1000, 1024, 0), (64, 384, 2048, 3), (33, 128, 256, 1)])
def test_gemm_quant_matches_reference(fmt, T, N, K, splits):
    from inference_b200 import ops
    from inference_b200.ops import quant

    g = torch.Generator().manual_seed(T * 131 + N)
    w = torch.randn(N, K, generator=g) * 0.05
    qw = quant.quantize_weight(w, fmt).to("cuda")
    wref = quant.dequantize_reference(qw)                       # fp32 [N, K] from plain CPU math
    dense = quant.dequantize(qw)
    assert (dense.float().cpu() - wref).abs().max().item() <= 4e-3 * max(1.0, wref.abs().max().item())
    a = (torch.randn(T, K, generator=g) * 0.5).bfloat16().cuda()
    bias = (torch.randn(N, generator=g) * 0.1).bfloat16().cuda()
    for rep in range(2):                                         # second call reuses the workspace counters
        out = quant.linear_quant(a, qw, bias=bias, splits=splits)
        ops.check_status()
        ref = a.float().cpu() @ wref.t() + bias.float().cpu()
        err = (out.float().cpu() - ref).abs().max().item()
        assert err < 2e-2 * max(1.0, ref.abs().max().item()), (fmt, rep, err)


@pytest.mark.parametrize("T,N,K", [(1, 200, 256), (3, 512, 4096), (5, 300, 14336), (8, 130, 7168), (2, 33, 1024)])
def test_q4k_matvec_kernel_matches_reference_and_the_tensor_core_path(T, N, K):
    """Up to 8 tokens of Q4_K run the integer matrix-vector kernel (int8 activations per 32-block); splits = -1 keeps
    the dequantising tensor-core kernel. Both against CPU dequantisation + fp32 matmul."""
    from inference_b200 import ops
    from inference_b200.ops import quant

    g = torch.Generator().manual_seed(T * 7 + K)
    w = torch.randn(N, K, generator=g) * 0.05
    qw = quant.quantize_weight(w, "Q4_K").to("cuda")
    wref = quant.dequantize_reference(qw)
    a = (torch.randn(T, K, generator=g) * 0.5).bfloat16().cuda()
    bias = (torch.randn(N, generator=g) * 0.1).bfloat16().cuda()
    ref = a.float().cpu() @ wref.t() + bias.float().cpu()
    tol = 2e-2 * max(1.0, ref.abs().max().item())
    mv = quant.linear_quant(a, qw, bias=bias)
    tc = quant.linear_quant(a, qw, bias=bias, splits=-1)
    ops.check_status()
    assert (mv.float().cpu() - ref).abs().max().item() < tol
    assert (tc.float().cpu() - ref).abs().max().item() < tol
    assert not torch.equal(mv, tc) or T * N < 64          # two different kernels produced the two results
    # activations with a zero block and a large outlier block keep their per-block scales
    a2 = a.clone()
    a2[:, :32] = 0
    a2[:, 32:64] *= 40
    ref2 = a2.float().cpu() @ wref.t()
    out2 = quant.linear_quant(a2, qw)
    assert (out2.float().cpu() - ref2).abs().max().item() < 2e-2 * max(1.0, ref2.abs().max().item())


@pytest.mark.parametrize("T,N,K", [(8, 37, 18432), (4, 4801, 2304), (1, 9473, 512), (6, 2369, 256), (5, 2368, 768), (3, 1, 4352), (8, 130, 256)])
def test_q4k_matvec_pairs_of_rows(T, N, K):
    """A last pair of one row, slices that end inside a row, several pairs per warp, a row per warp and its limit, the largest activations. Against 64 bits with the
    activations rounded as the kernel rounds them (int8 per block of 32), so what is left are fp32 sums and the rounding to bf16."""
    from inference_b200 import ops
    from inference_b200.ops import quant

    g = torch.Generator(device="cuda").manual_seed(T * 7 + K)
    qw = quant.quantize_on_device((torch.randn(N, K, device="cuda", generator=g) * 0.05).bfloat16(), "Q4_K")
    a = (torch.randn(T, K, device="cuda", generator=g) * 0.5).bfloat16()
    blocks = a.float().reshape(T, K // 32, 32)
    top = blocks.abs().amax(-1, keepdim=True)
    seen = (blocks * (127.0 / top)).round().double() * (top * (1.0 / 127.0)).double()
    ref = seen.reshape(T, K) @ quant.dequantize_reference(qw).double().cuda().T
    got = quant.linear_quant(a, qw)
    ops.check_status()
    assert (got.double() - ref).abs().max().item() < 2.0 ** -8 * ref.abs().max().item()


# a tile of one row; more than 16 tiles of a CTA; one, two and four passes over the reduction index; activations far apart in size
@pytest.mark.parametrize("T,N,K", [(1, 1, 256), (4, 16 * 148 * 16 + 18, 256), (7, 2390, 4096), (8, 98, 14336), (8, 34, 28416), (5, 64, 1536), (3, 4096, 512)])
def test_q4k_matvec_chain_links(T, N, K):
    """Both links of a folded-norm chain and gated pairs, against 64 bits. Operands are exact, so what is left are fp32 sums (K of them at 2^-24) and
    the rounding to bf16; activations that are 10^5 times smaller than others of their super-block count as much as the rest."""
    from inference_b200 import ops
    from inference_b200.ops import quant

    g = torch.Generator(device="cuda").manual_seed(T + N)
    qw = quant.quantize_on_device((torch.randn(N, K, device="cuda", generator=g) * 0.05).bfloat16(), "Q4_K")
    w = quant.dequantize_reference(qw).double().cuda()
    assert ops.normed_supported(T, qw)
    a = torch.randn(T, K, device="cuda", generator=g)
    a[:, : K // 2] *= 1e-5
    a[:, 32:64] = 0
    a[T - 1] *= 1e2
    a = a.bfloat16()
    bias = (torch.randn(N, generator=g, device="cuda") * 0.1).bfloat16()
    res = torch.randn(T, N, device="cuda", generator=g).bfloat16()

    def product(x):
        return x.double() @ w.T, x.double().abs() @ w.abs().T * (2.0 ** -22 + K * 2.0 ** -26)

    out, zero = ops.ssq_buffer(a.device), torch.ones(64, dtype=torch.int64, device="cuda")
    y = res.clone()
    ops.linear_normed(a, qw, out=y, bias=bias, residual=y, ssq_out=out, ssq_zero=zero)
    ops.check_status()
    exact, near = product(a)
    exact += bias.double()
    want = exact + res.double()
    assert ((y.double() - want).abs() - near - 2.0 ** -8 * (exact.abs() + want.abs())).max().item() <= 0
    assert not zero.any() and not out[T:].any()
    torch.testing.assert_close(ops.ssq_values(out)[:T], y.float().pow(2).sum(1), rtol=1e-5, atol=1e-5)

    y32 = ops.linear_normed(a.float(), qw, out=res.float(), bias=bias, residual=res.float())      # bf16 values in fp32: the same operands
    assert ((y32.double() - want).abs() - near - 2.0 ** -22 * want.abs()).max().item() <= 0

    ssq = ops.ssq_buffer(a.device)
    ssq[:T] = (a.double().pow(2).sum(1) * 2.0 ** 24).round().long()
    rms = (a.double().pow(2).mean(1, keepdim=True) + 1e-5).rsqrt()
    exact, near = (t * rms for t in product(a))
    z = ops.linear_normed(a, qw, ssq_in=ssq, norm_dim=K, eps=1e-5)
    assert ((z.double() - exact).abs() - near - 2.0 ** -8 * exact.abs()).max().item() <= 0
    if N % 2 == 0:
        for act, f in (("swiglu_pairs", torch.nn.functional.silu), ("geglu_pairs", lambda t: torch.nn.functional.gelu(t, approximate="tanh"))):
            u = ops.linear_normed(a, qw, act=act, ssq_in=ssq, norm_dim=K, eps=1e-5)
            gate, up = exact[:, 0::2], exact[:, 1::2]
            e_gate, e_up = (near + 2.0 ** -8 * exact.abs())[:, 0::2], (near + 2.0 ** -8 * exact.abs())[:, 1::2]
            bound = 1.2 * e_gate * (up.abs() + e_up) + f(gate).abs() * e_up      # slopes of both functions stay below 1.2
            assert ((u.double() - f(gate) * up).abs() - bound - 2.0 ** -8 * (f(gate) * up).abs()).max().item() <= 1e-6


@pytest.mark.parametrize("T,N,K", [(1, 2, 256), (4, 98, 1536), (8, 2390, 4096)])
@pytest.mark.parametrize("act", [None, "swiglu_pairs", "geglu_pairs"])
def test_q4k_matvec_chain_adds_the_bias_behind_the_norm(T, N, K, act):
    """D = act(rms * A W^T + bias): the projections of a decoder with biases, whose stream is far from unit size (1 / rms is 2^-6, 1 and 2^6 of a row)."""
    from inference_b200 import ops
    from inference_b200.ops import quant

    g = torch.Generator(device="cuda").manual_seed(T + N)
    qw = quant.quantize_on_device((torch.randn(N, K, device="cuda", generator=g) * 0.05).bfloat16(), "Q4_K")
    w = quant.dequantize_reference(qw).double().cuda()
    a = (torch.randn(T, K, device="cuda", generator=g) * 64.0 ** (torch.arange(T, device="cuda") % 3 - 1)[:, None]).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g).bfloat16()
    ssq = ops.ssq_buffer(a.device)
    ssq[:T] = (a.double().pow(2).sum(1) * 2.0 ** 24).round().long()
    got = ops.linear_normed(a, qw, bias=bias, act=act, ssq_in=ssq, norm_dim=K, eps=1e-5).double()
    ops.check_status()
    rms = (a.double().pow(2).mean(1, keepdim=True) + 1e-5).rsqrt()
    want = a.double() @ w.T * rms + bias.double()
    # fp32 sums of K terms and a square root; the sum with the bias
    near = (a.double().abs() @ w.abs().T * rms) * (2.0 ** -22 + K * 2.0 ** -26) + 2.0 ** -23 * want.abs()
    if act is None:
        assert ((got - want).abs() - near - 2.0 ** -8 * want.abs()).max().item() <= 0
        return
    f = torch.nn.functional.silu if act == "swiglu_pairs" else lambda t: torch.nn.functional.gelu(t, approximate="tanh")  # noqa: E731
    gate, up, e_gate, e_up = want[:, 0::2], want[:, 1::2], near[:, 0::2], near[:, 1::2]
    want = f(gate) * up
    # slopes of both functions stay below 1.2; the functions' own exponentials and quotients are good to 2^-20 of the gate
    bound = (1.2 * e_gate + 2.0 ** -20 * gate.abs()) * (up.abs() + e_up) + f(gate).abs() * e_up
    assert ((got - want).abs() - bound - 2.0 ** -8 * want.abs()).max().item() <= 0


@pytest.mark.parametrize("T,most", [(8, 28672), (7, 32768)])
def test_q4k_matvec_chain_takes_reductions_up_to_four_passes(T, most):
    """The longest reduction of whole super-blocks that it takes, and no longer one."""
    from inference_b200 import ops
    from inference_b200._native import kernels
    from inference_b200.ops import quant

    assert all(kernels().swb_gemv_q4k_supported(T, k) for k in range(256, most + 1, 256)) and not kernels().swb_gemv_q4k_supported(T, most + 256)
    g = torch.Generator(device="cuda").manual_seed(T)
    qw = quant.quantize_on_device((torch.randn(18, most, device="cuda", generator=g) * 0.05).bfloat16(), "Q4_K")
    a = torch.randn(T, most, device="cuda", generator=g).bfloat16()
    w = quant.dequantize_reference(qw).double().cuda()
    got, want = ops.linear_normed(a, qw).double(), a.double() @ w.T
    ops.check_status()
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + (2.0 ** -22 + most * 2.0 ** -26) * (a.double().abs() @ w.abs().T)).all()


def test_q4k_matvec_chain_sees_small_activations():
    """Tokens and super-blocks of any size: what one holds is not measured by another's largest."""
    from inference_b200 import ops
    from inference_b200.ops import quant

    g = torch.Generator(device="cuda").manual_seed(1)
    qw = quant.quantize_on_device((torch.randn(64, 768, device="cuda", generator=g) * 0.05).bfloat16(), "Q4_K")
    w = quant.dequantize_reference(qw).double().cuda()
    a = torch.randn(6, 768, device="cuda", generator=g)
    a *= torch.tensor([1e-30, 1e-12, 0.0, 1.0, 1e9, 1e30], device="cuda")[:, None]
    a = a.bfloat16()
    got, want = ops.linear_normed(a, qw).double(), a.double() @ w.T
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * (a.double().abs() @ w.abs().T)).all()


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_q4k_matvec_chain_keeps_what_is_no_number_in_its_token(value):
    from inference_b200 import ops
    from inference_b200.ops import quant

    g = torch.Generator(device="cuda").manual_seed(3)
    qw = quant.quantize_on_device((torch.randn(48, 512, device="cuda", generator=g) * 0.05).bfloat16(), "Q4_K")
    a = torch.randn(3, 512, device="cuda", generator=g).bfloat16()
    want = ops.linear_normed(a, qw)
    a[1, 300] = value
    got = ops.linear_normed(a, qw)
    assert torch.equal(got[0], want[0]) and torch.equal(got[2], want[2]) and not got[1].isfinite().any()


def test_a_q4k_decoder_chains_its_products_in_decode():
    """Steps of up to eight rows join the stream and apply its norm inside the products: six launches a layer. The same logits as with the
    kernels in between, within the rounding of what those store in bf16."""
    import os

    from inference_b200.engine.llm_engine import EngineConfig, LlmEngine
    from inference_b200.models import ModelConfig
    from inference_b200.models.llama import LlamaGpu

    cfg = ModelConfig.from_json({"hidden_size": 512, "intermediate_size": 1024, "num_hidden_layers": 3, "num_attention_heads": 4,
                                 "num_key_value_heads": 2, "head_dim": 128, "vocab_size": 1024, "rope_theta": 10000.0})
    model = LlamaGpu(cfg).init_random(seed=1).quantize_("Q4_K")
    logits, launches = {}, {}
    for chain in ("1", "0"):
        os.environ["SWB_NORM_CHAIN"] = chain
        try:
            eng = LlmEngine(model, EngineConfig(max_batch=8, max_seq_len=64))
            seqs = [eng.new_sequence() for _ in range(3)]
            eng.runner.prefill(seqs, [[1, 2, 3], [4, 5], [6, 7, 8, 9]])
            for _ in range(2):
                logits[chain] = eng.runner.decode(seqs, [3, 4, 5], want_logits=True).clone()
            launches[chain] = eng.runner.launches_last
        finally:
            del os.environ["SWB_NORM_CHAIN"]
    assert launches["1"] == launches["0"] - 3 * 3 + 3        # the first norm stays, the stream is converted to 32 bits and back
    assert (logits["1"] - logits["0"]).norm() < 0.03 * logits["0"].norm()


def test_a_q4k_decoder_with_biases_matches_the_oracle():
    """Query, key and value biases of the size of their projections, norm weights away from one, several layers: decode and a prompt of a few tokens, on the
    chain and with the kernels in between, against 32 bits on the weights that the packed blocks stand for."""
    import os

    from inference_b200.engine.kv_pool import PagedKvPool, PagedSequence
    from inference_b200.engine.runner import ModelRunner
    from inference_b200.models import ModelConfig
    from inference_b200.models.llama import LlamaGpu
    from inference_b200.models.oracle import OracleLlama, random_llama_weights
    from inference_b200.ops import quant

    cfg = ModelConfig.from_json({"model_type": "qwen2", "hidden_size": 512, "intermediate_size": 1024, "num_hidden_layers": 4, "num_attention_heads": 4,
                                 "num_key_value_heads": 2, "head_dim": 128, "vocab_size": 1024, "rms_norm_eps": 1e-5, "rope_theta": 10000.0})
    g = torch.Generator().manual_seed(11)
    w = {k: v.bfloat16().float() for k, v in random_llama_weights(cfg, seed=4, std=0.05, bias=True).items()}
    for k in w:
        if k.endswith("layernorm.weight"):
            w[k] = (torch.rand(w[k].shape, generator=g) + 0.5).bfloat16().float()
        elif k.endswith("proj.bias"):
            w[k] = torch.randn(w[k].shape, generator=g).bfloat16().float()
    model = LlamaGpu(cfg, device=torch.device("cuda")).load_state_dict(w).quantize_("Q4_K")
    seen = dict(w)          # the norm weights are part of the projections before these are packed
    for i in range(cfg.num_layers):
        p = f"model.layers.{i}."
        for norm, names in (("input_layernorm", ("self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj")),
                            ("post_attention_layernorm", ("mlp.gate_proj", "mlp.up_proj")), (None, ("self_attn.o_proj", "mlp.down_proj"))):
            by = w[f"{p}{norm}.weight"] if norm else 1.0
            for n in names:
                folded = (w[f"{p}{n}.weight"] * by).bfloat16().float()
                seen[f"{p}{n}.weight"] = quant.dequantize_reference(quant.quantize_on_device(folded, "Q4_K"))
            if norm:
                seen[f"{p}{norm}.weight"] = torch.ones_like(w[f"{p}{norm}.weight"])
    oracle = OracleLlama(cfg, seen, dtype=torch.float32, device="cuda")
    prompts, steps = [[5, 6, 7], [40, 41], [900]], ([3, 4, 5], [600, 2, 77])
    want = [[], [], []]
    for i, p in enumerate(prompts):
        cache = oracle.make_cache()
        for toks in (p, [steps[0][i]], [steps[1][i]]):
            want[i].append(oracle.decode_logits(torch.tensor([toks], device="cuda"), cache, cache.offset)[0])
    for chain in ("1", "0"):
        os.environ["SWB_NORM_CHAIN"] = chain
        try:
            pool = PagedKvPool(cfg.num_layers, 64, model.hkv, cfg.head_dim, 16, device="cuda")
            runner = ModelRunner(model, pool, max_batch=8, max_seq_len=64)
            seqs = [PagedSequence(pool) for _ in prompts]
            got = [runner.prefill(seqs, prompts, want_logits=True).clone()] + [runner.decode(seqs, list(t), want_logits=True).clone() for t in steps]
        finally:
            del os.environ["SWB_NORM_CHAIN"]
        for i in range(3):
            for step in range(3):
                # bf16 between the kernels of four layers, int8 activations in the products of a step without the chain
                err = (got[step][i] - want[i][step]).norm() / want[i][step].norm()
                assert err < 0.05, (chain, i, step, err.item())


@pytest.mark.parametrize("T", [65, 130, 256])
def test_expanded_weights_are_complete_before_they_are_multiplied(T):
    """Token counts above the fused kernel's expand the weight and multiply it right behind: the product must not start from
    what the buffer held before. Two weights take turns in the same reused buffer."""
    from inference_b200.ops import quant

    g = torch.Generator(device="cuda").manual_seed(T)
    N, K = 14336, 4096
    qws = [quant.quantize_on_device(torch.randn(N, K, generator=g, device="cuda") * s, "Q4_K") for s in (0.05, 5.0)]
    a = (torch.randn(T, K, generator=g, device="cuda") * 0.5).bfloat16()
    wants = [a.float() @ quant.dequantize(q).float().t() for q in qws]
    for _ in range(6):
        outs = [quant.linear_quant(a, q) for q in qws]
        for out, want in zip(outs, wants):         # one rounding to bf16 of fp32 sums
            assert (out.float() - want).abs().max().item() < 2 ** -8 * want.abs().max().item()


@pytest.mark.parametrize("T,N,K", [(65, 3581, 4096), (200, 5117, 4096), (256, 96, 14336), (130, 120, 14336)])
def test_expanded_weights_are_complete_on_the_one_sm_kernels(T, N, K):
    """The same for shapes that the two-SM kernel does not take (odd or small output widths). Their kernel for so many tokens loads a
    weight ahead, so an expanded one goes to the kernel that waits."""
    from inference_b200._native import kernels
    from inference_b200.ops import quant

    assert not kernels().swb_gemm_takes_pairs(T, N, K, 0, 0, 0, 0, -2, 0, 0)
    g = torch.Generator(device="cuda").manual_seed(T + N)
    qws = [quant.quantize_on_device(torch.randn(N, K, generator=g, device="cuda") * s, "Q8_0") for s in (0.05, 5.0)]
    a = (torch.randn(T, K, generator=g, device="cuda") * 0.5).bfloat16()
    wants = [a.float() @ quant.dequantize(q).float().t() for q in qws]
    for _ in range(6):
        outs = [quant.linear_quant(a, q) for q in qws]
        for out, want in zip(outs, wants):         # one rounding to bf16 of fp32 sums
            assert (out.float() - want).abs().max().item() < 2 ** -8 * want.abs().max().item()


@pytest.mark.parametrize("first,then", [(100, 5), (100, 60), (200, 100)])
def test_a_kept_nvfp4_expansion_is_complete_before_it_is_read_ahead(first, then):
    """Products right behind the one that expanded the weight for good. An expansion inside a capture is not kept: its buffer is written
    by replays only."""
    from inference_b200.ops import nvfp4 as nv

    g = torch.Generator(device="cuda").manual_seed(first + then)
    N, K = 4099, 4096
    x = torch.randn(first, K, device="cuda", generator=g).bfloat16()
    for s in (0.02, 2.0, 0.02, 2.0):
        t = nv.Nvfp4Tensor.pack(torch.randn(N, K, device="cuda", generator=g) * s)
        want = x.float() @ t.dequantize().float().T
        torch.cuda.synchronize()
        lin = nv.Nvfp4Linear(t, keep_dense=True)
        whole, part = lin(x), lin(x[:then])
        assert (whole.float() - want).abs().max().item() < 2 ** -7 * want.abs().max().item()      # the weight and the result in bf16
        assert (part.float() - want[:then]).abs().max().item() < 2 ** -7 * want.abs().max().item()
        assert torch.equal(lin(x), whole) and lin.dense_bf16() is lin._dense
    lin = nv.Nvfp4Linear(t, keep_dense=True)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = lin(x)
    assert lin._dense is None
    graph.replay()
    torch.cuda.synchronize()
    assert (y.float() - want).abs().max().item() < 2 ** -7 * want.abs().max().item()


def test_large_token_count_uses_dense_path():
    from inference_b200.ops import quant

    w = torch.randn(512, 512) * 0.05
    qw = quant.quantize_weight(w, "Q8_0").to("cuda")
    a = (torch.randn(200, 512) * 0.5).bfloat16().cuda()
    out = quant.linear_quant(a, qw)
    ref = a.float().cpu() @ quant.dequantize_reference(qw).t()
    assert (out.float().cpu() - ref).abs().max().item() < 2e-2 * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("T,N,K", [(1, 256, 512), (16, 384, 1024), (64, 200, 256), (33, 3072, 3072)])
def test_nvfp4_gemm_and_dequant_match_cpu_container(T, N, K):
    """The device decode of E2M1 codes and swizzled E4M3 scales reproduces the container's dequantised values
    exactly (they are bf16-representable up to the scale product), and the fused GEMM matches fp32 matmul on them."""
    from inference_b200 import ops
    from inference_b200.ops import nvfp4 as nv

    g = torch.Generator().manual_seed(T + N)
    w = torch.randn(N, K, generator=g) * 0.05
    w[1, 3] = 1.5
    bias = (torch.randn(N, generator=g) * 0.1).bfloat16().cuda()
    lin = nv.Nvfp4Linear(nv.Nvfp4Tensor.pack(w).to("cuda"), bias)
    ref_w = lin.t.dequantize()                                     # fp32 on the device, torch ops
    dense = lin.dense_bf16()
    ops.check_status()
    torch.testing.assert_close(dense.float(), ref_w.bfloat16().float(), rtol=1e-2, atol=1e-6)
    x = torch.randn(T, K, generator=g).bfloat16().cuda()
    y = lin(x)
    ops.check_status()
    ref = x.float() @ dense.float().t() + bias.float()             # the kernel multiplies exactly these bf16 weights
    torch.testing.assert_close(y.float(), ref, rtol=2e-2, atol=2e-2)
    big = torch.randn(130, K, generator=g).bfloat16().cuda()       # more than 64 rows: expand + dense GEMM
    torch.testing.assert_close(lin(big).float(), big.float() @ dense.float().t() + bias.float(), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("rows,cols,dtype", [(130, 80, torch.float32), (64, 4096, torch.bfloat16), (1, 16, torch.float32),
                                            (257, 3072, torch.float32)])
def test_nvfp4_device_quantiser_is_bit_identical_to_the_host_packer(rows, cols, dtype):
    from inference_b200 import ops
    from inference_b200.ops import nvfp4 as nv

    g = torch.Generator().manual_seed(rows + cols)
    x = (torch.randn(rows, cols, generator=g) * 0.3).to(dtype)
    x[0, 0] = 7.0                                           # an outlier fixes the tensor scale
    x[rows // 2, : min(32, cols)] = 0.0                     # all-zero blocks: scale byte 0, codes 0
    if cols >= 32:
        x[rows - 1, 16:32] = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, -0.25] * 2).to(dtype) * 0.01
    host = nv.Nvfp4Tensor.pack(x)
    dev = nv.quantize_on_device(x.cuda())
    ops.check_status()
    assert dev.global_scale == host.global_scale
    assert torch.equal(dev.scales.cpu(), host.scales)
    assert torch.equal(dev.packed.cpu(), host.packed)
    torch.testing.assert_close(nv.quantize_activations(x.cuda()).cpu().float(), host.dequantize().to(dtype).float())


@pytest.mark.parametrize("T,N,K", [(128, 128, 256), (300, 400, 512), (1000, 272, 1024), (65, 4096, 3072)])
def test_nvfp4_w4a4_tensor_core_gemm_matches_the_dequantised_product(T, N, K):
    """Both operands 4-bit in the tensor core: the result equals the fp32 product of the two dequantised NVFP4
    tensors (every partial product is exact in fp32; only the accumulation order differs)."""
    from inference_b200 import ops
    from inference_b200.ops import nvfp4 as nv

    g = torch.Generator().manual_seed(T + N + K)
    w = torch.randn(N, K, generator=g) * 0.05
    x = (torch.randn(T, K, generator=g) * 0.7).bfloat16()
    x[:, :16] *= 6.0                                              # one loud block per row: block scales matter
    wq = nv.Nvfp4Tensor.pack(w).to("cuda")
    bias = (torch.randn(N, generator=g) * 0.1).bfloat16().cuda()
    out = nv.gemm_w4a4(x.cuda(), wq, bias)
    ops.check_status()
    xq = nv.Nvfp4Tensor.pack(x.float())
    ref = xq.dequantize() @ wq.to("cpu").dequantize().t() + bias.float().cpu()
    err = (out.float().cpu() - ref).abs().max().item()
    assert err < 1e-2 * max(1.0, ref.abs().max().item()), err
    lin = nv.Nvfp4Linear(wq, bias, act_precision=nv.ActPrecision.W4A4)
    assert torch.equal(lin(x.cuda()), out)                       # the layer takes the same path above 64 rows
