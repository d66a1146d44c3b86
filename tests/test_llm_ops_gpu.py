"""Fused LLM glue kernels and attention against plain PyTorch fp32 references."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rope_tables(max_pos, rot_dim, theta=10000.0):
    inv = 1.0 / (theta ** (torch.arange(0, rot_dim, 2, dtype=torch.float32) / rot_dim))
    ang = torch.arange(max_pos, dtype=torch.float32)[:, None] * inv[None, :]
    return ang.cos().cuda().contiguous(), ang.sin().cuda().contiguous()


def test_rmsnorm_and_residual():
    from inference_b200 import ops

    for T, H in ((1, 4096), (7, 256), (33, 8192), (5, 3072), (3, 1024)):
        x = torch.randn(T, H, device="cuda").bfloat16()
        r = torch.randn(T, H, device="cuda").bfloat16()
        w = (torch.randn(H, device="cuda") * 0.1 + 1).bfloat16()
        y = ops.rmsnorm(x, w, 1e-5)
        xf = x.float()
        ref = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * w.float()
        assert torch.allclose(y.float(), ref, atol=3e-2, rtol=2e-2)
        r2 = r.clone()
        y2 = ops.rmsnorm(x, w, 1e-5, residual=r2)
        s = (x.float() + r.float()).bfloat16()
        assert torch.equal(r2, s)
        sf = s.float()
        ref2 = sf * torch.rsqrt(sf.pow(2).mean(-1, keepdim=True) + 1e-5) * w.float()
        assert torch.allclose(y2.float(), ref2, atol=3e-2, rtol=2e-2)


def test_layernorm_mod_and_gated_residual():
    from inference_b200 import ops

    B, S, H = 2, 37, 3072
    x = torch.randn(B, S, H, device="cuda").bfloat16()
    sc = (torch.randn(B, H, device="cuda") * 0.2).bfloat16()
    sh = (torch.randn(B, H, device="cuda") * 0.2).bfloat16()
    y = ops.layernorm_mod(x, scale=sc, shift=sh, rows_per_batch=S, eps=1e-6)
    ref = torch.nn.functional.layer_norm(x.float(), (H,), eps=1e-6) * (1 + sc.float()[:, None]) + sh.float()[:, None]
    assert torch.allclose(y.float(), ref, atol=4e-2, rtol=2e-2)
    b = torch.randn(B, S, H, device="cuda").bfloat16()
    z = ops.gated_residual(x, b, sc, rows_per_batch=S)
    refz = x.float() + sc.float()[:, None] * b.float()
    assert torch.allclose(z.float(), refz, atol=3e-2, rtol=2e-2)


# one, two and three vectors of a thread, the last of them in part; rows further apart than they are long
@pytest.mark.parametrize("T,H,per,ld", [(1, 1024, 0, 1024), (5, 1032, 3, 1040), (7, 2048, 2, 2048), (9, 2056, 4, 2056), (6, 3072, 5, 3080), (3, 3080, 1, 3080)])
def test_layernorm_of_any_width(T, H, per, ld):
    from inference_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(H)
    x = (torch.randn(T, ld, device="cuda", generator=g) * 3 + 20).bfloat16()[:, :H]
    B = (T + per - 1) // per if per else 1
    mods = [(torch.randn(B, H, device="cuda", generator=g) * 0.3).bfloat16() for _ in range(2)]
    y = ops.layernorm_mod(x, scale=mods[0], shift=mods[1], rows_per_batch=per or T)
    rows = torch.arange(T, device="cuda") // (per or T)
    want = torch.nn.functional.layer_norm(x.double(), (H,), eps=1e-6) * (1 + mods[0].double()[rows]) + mods[1].double()[rows]
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()      # fp32 sums of values that are 7 times their spread


# both sides of every line between the forms by rows of an SM, and one vector of a row
@pytest.mark.parametrize("T,H", [(600, 8), (9, 512), (9, 520), (443, 1032), (444, 2048), (443, 2056), (591, 2056), (1183, 3072), (1184, 3072), (443, 3080), (444, 4096),
                                 (2071, 4104), (2072, 8192), (148, 8200), (149, 16384)])
def test_layernorm_of_many_rows(T, H):
    test_layernorm_of_any_width(T, H, 100, H + 8)


@pytest.mark.parametrize("H", [512, 1536, 2056, 3072, 3840, 6144, 16384])
def test_layernorm_of_a_row_whatever_comes_with_it(H):
    from inference_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(H)
    x = torch.randn(4608, H, device="cuda", generator=g).bfloat16()
    mods = [(torch.randn(1, H, device="cuda", generator=g) * 0.3).bfloat16() for _ in range(2)]
    whole = ops.layernorm_mod(x, scale=mods[0], shift=mods[1], rows_per_batch=4608)
    for T in (5, 256, 512, 1231):
        assert torch.equal(ops.layernorm_mod(x[:T], scale=mods[0], shift=mods[1], rows_per_batch=T), whole[:T])


@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("D,rot", [(128, 128), (64, 64), (128, 64), (96, 32)])
def test_rope_kv_write(interleaved, D, rot):
    from inference_b200 import ops

    T, Hq, Hkv, bs, nblk = 19, 4, 2, 16, 8
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device="cuda").bfloat16()
    pos = torch.randint(0, 500, (T,), device="cuda", dtype=torch.int32)
    slots = torch.randperm(nblk * bs, device="cuda")[:T].to(torch.int64)
    cos, sin = _rope_tables(512, rot)
    kc = torch.zeros(nblk, Hkv, bs, D, device="cuda", dtype=torch.bfloat16)
    vc = torch.zeros_like(kc)
    ref = qkv.float().reshape(T, Hq + 2 * Hkv, D).clone()
    c = cos[pos.long()][:, None, :]
    s = sin[pos.long()][:, None, :]
    qk = ref[:, : Hq + Hkv, :rot]
    if interleaved:
        x0, x1 = qk[..., 0::2], qk[..., 1::2]
        rot_out = torch.stack([x0 * c - x1 * s, x1 * c + x0 * s], dim=-1).flatten(-2)
    else:
        x0, x1 = qk[..., : rot // 2], qk[..., rot // 2:]
        rot_out = torch.cat([x0 * c - x1 * s, x1 * c + x0 * s], dim=-1)
    ref[:, : Hq + Hkv, :rot] = rot_out
    ops.rope_kv_write(qkv, pos, slots, cos, sin, kc, vc, Hq, Hkv, D, rot_dim=rot, interleaved=interleaved,
                      block_size=bs)
    got = qkv.float().reshape(T, Hq + 2 * Hkv, D)
    assert torch.allclose(got[:, :Hq], ref[:, :Hq], atol=3e-2, rtol=2e-2)
    blk, off = slots // bs, slots % bs
    kgot = kc[blk, :, off].float()
    vgot = vc[blk, :, off].float()
    assert torch.allclose(kgot, ref[:, Hq:Hq + Hkv], atol=3e-2, rtol=2e-2)
    assert torch.allclose(vgot, ref[:, Hq + Hkv:], atol=1e-6)


def test_qk_norm_rope():
    from inference_b200 import ops

    T, Hq, Hkv, D = 5, 4, 2, 128
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device="cuda").bfloat16()
    ref = qkv.float().reshape(T, -1, D).clone()
    pos = torch.arange(T, device="cuda", dtype=torch.int32)
    cos, sin = _rope_tables(64, D)
    qw = (torch.rand(D, device="cuda") + 0.5).bfloat16()
    kw = (torch.rand(D, device="cuda") + 0.5).bfloat16()
    ops.rope_kv_write(qkv, pos, None, cos, sin, None, None, Hq, Hkv, D, q_norm=qw, k_norm=kw, norm_eps=1e-6)

    def nrm(x, w):
        return (x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * w.float()).bfloat16().float()

    q = nrm(ref[:, :Hq], qw)
    c, s = cos[pos.long()][:, None], sin[pos.long()][:, None]
    q = torch.cat([q[..., :64] * c - q[..., 64:] * s, q[..., 64:] * c + q[..., :64] * s], -1)
    got = qkv.float().reshape(T, -1, D)[:, :Hq]
    assert torch.allclose(got, q, atol=4e-2, rtol=2e-2)


# a CTA per 32 (16) heads of a token below 296 tokens, all of a token's heads from there on; heads that fill the last round in part; rows 16 bytes apart
# from a whole vector go to the general kernel
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("T,Hq,Hkv,ld_extra", [(1, 1, 1, 0), (3, 40, 7, 8), (295, 5, 3, 0), (296, 33, 2, 0), (300, 7, 7, 0), (9, 3, 1, 2)])
def test_rope_of_whole_heads(interleaved, T, Hq, Hkv, ld_extra):
    from inference_b200 import ops

    D, bs = 128, 16
    g = torch.Generator(device="cuda").manual_seed(T + Hq)
    width = (Hq + 2 * Hkv) * D
    qkv = torch.randn(T, width + ld_extra, device="cuda", generator=g).bfloat16()[:, :width]
    pos = torch.randint(0, 500, (T,), device="cuda", dtype=torch.int32, generator=g)
    nblk = (T + bs - 1) // bs + 1
    slots = torch.randperm(nblk * bs, device="cuda", generator=g)[:T].to(torch.int64)
    slots[T // 2] = -1                      # this token's keys and values go to no cache
    cos, sin = _rope_tables(512, D)
    qw, kw = ((torch.rand(D, device="cuda", generator=g) + 0.5).bfloat16() for _ in range(2))
    kc, vc = (torch.full((nblk, Hkv, bs, D), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    x = qkv.double().reshape(T, Hq + 2 * Hkv, D)
    w = torch.cat([qw.double().expand(Hq, D), kw.double().expand(Hkv, D)])
    n = (x[:, :Hq + Hkv] * (x[:, :Hq + Hkv].pow(2).mean(-1, keepdim=True) + 1e-6).rsqrt() * w).bfloat16().double()
    c, s = cos[pos.long()].double()[:, None], sin[pos.long()].double()[:, None]
    a, b = (n[..., 0::2], n[..., 1::2]) if interleaved else (n[..., :64], n[..., 64:])
    ref = torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2) if interleaved else torch.cat([a * c - b * s, b * c + a * s], -1)
    values = qkv.reshape(T, -1, D)[:, Hq + Hkv:].clone()
    ops.rope_kv_write(qkv, pos, slots, cos, sin, kc, vc, Hq, Hkv, D, q_norm=qw, k_norm=kw, norm_eps=1e-6, interleaved=interleaved, block_size=bs)
    got = qkv.reshape(T, -1, D)
    bound = 2.0 ** -8 * 2 * n.abs().amax(-1, keepdim=True)      # a norm that falls to the other side of a rounding, and the rounding of the result
    assert ((got[:, :Hq + Hkv].double() - ref).abs() <= bound).all()
    blk, off = slots // bs, slots % bs
    kept = slots >= 0
    assert torch.equal(kc[blk, :, off][kept], got[:, Hq:Hq + Hkv][kept]) and torch.equal(vc[blk, :, off][kept], values[kept])
    rest = torch.ones(nblk * bs, dtype=torch.bool, device="cuda")
    rest[slots[kept]] = False
    assert (kc.transpose(1, 2).reshape(nblk * bs, -1)[rest] == 7.0).all() and (vc.transpose(1, 2).reshape(nblk * bs, -1)[rest] == 7.0).all()


# heads that fill half of a CTA and one more; several tokens to a CTA, the last CTA with fewer; 64 tokens of more heads than a CTA has, and 65
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("T,Hq,Hkv", [(1, 4, 1), (301, 4, 1), (67, 12, 2), (67, 13, 2), (66, 4, 2), (66, 5, 2), (64, 40, 7), (65, 40, 7)])
def test_rope_of_few_heads_or_tokens(interleaved, T, Hq, Hkv):
    test_rope_of_whole_heads(interleaved, T, Hq, Hkv, 0)


# sequences with fewer key tiles than parts, rows that see no key of the last part, one row, a last tile that ends inside a page
@pytest.mark.parametrize("splits", [2, 3, 8])
@pytest.mark.parametrize("news,olds,Hq,Hkv,bs", [([700], [1900], 4, 2, 16), ([130, 1, 300], [1000, 2500, 0], 2, 1, 32), ([5, 257], [3, 640], 3, 3, 64)])
def test_paged_prefill_with_split_keys(news, olds, Hq, Hkv, bs, splits):
    from inference_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(sum(news))
    T, lens = sum(news), [n + o for n, o in zip(news, olds)]
    need = [(x + bs - 1) // bs for x in lens]
    perm = torch.randperm(sum(need), device="cuda", generator=g).int()
    table = torch.zeros(len(news), max(need), dtype=torch.int32, device="cuda")
    for i, parts in enumerate(perm.split(need)):
        table[i, :need[i]] = parts
    kc, vc = (torch.randn(sum(need), Hkv, bs, 128, device="cuda", generator=g).bfloat16() for _ in range(2))
    q = torch.randn(T, Hq, 128, device="cuda", generator=g).bfloat16() * 2
    cu = torch.tensor([0, *torch.tensor(news).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    kvl = torch.tensor(lens, dtype=torch.int32, device="cuda")

    def run(n):
        return ops.paged_attention(q, kc, vc, table, kvl, cu_q=cu, max_q_len=max(news), scale=128 ** -0.5, prefill_splits=n).double()

    whole, split = run(1), run(splits)
    ops.check_status()
    want, at = torch.empty_like(whole), 0
    for i, (n, o) in enumerate(zip(news, olds)):
        rows = table[i, :need[i]].long()
        k, v = (c[rows].transpose(1, 2).reshape(-1, Hkv, 128)[:n + o].double().repeat_interleave(Hq // Hkv, 1) for c in (kc, vc))
        s = torch.einsum("qhd,khd->hqk", q[at:at + n].double(), k) * 128 ** -0.5
        seen = torch.arange(n + o, device="cuda")[None] <= torch.arange(o, o + n, device="cuda")[:, None]
        want[at:at + n] = torch.einsum("hqk,khd->qhd", s.masked_fill(~seen, -math.inf).softmax(-1), v).reshape(n, -1)
        at += n
    # probabilities in bf16 on both sides, rounded against different maxima
    assert (split - want).norm() <= 1.2 * (whole - want).norm() + 1e-4 * want.norm()
    assert (split - want).abs().max() <= 2.0 ** -6 * want.abs().max()


@pytest.mark.parametrize("splits", [1, 2, 5])
def test_paged_prefill_leaves_rows_of_no_sequence_alone(splits):
    """Rows before the first and behind the last sequence, of a sequence without context and behind the query tiles that max_q_len asks for: the keys may be
    split or not, such rows of the result stay as they are."""
    from inference_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(3)
    Hq, Hkv, bs, first, news, lens = 4, 2, 16, 3, [40, 9, 300], [900, 0, 1300]
    T = first + sum(news) + 70
    table = torch.randperm(3 * 82, device="cuda", generator=g).int().view(3, 82)
    kc, vc = (torch.randn(3 * 82, Hkv, bs, 128, device="cuda", generator=g).bfloat16() for _ in range(2))
    q = torch.randn(T, Hq, 128, device="cuda", generator=g).bfloat16()
    cu = torch.tensor([first, first + 40, first + 49, first + 349], dtype=torch.int32, device="cuda")
    kvl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    junk = torch.full((splits * Hq * T * 130,), math.nan, device="cuda")      # what the allocator hands out next
    del junk
    out = torch.full((T, Hq * 128), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.paged_attention(q, kc, vc, table, kvl, cu_q=cu, max_q_len=200, scale=128 ** -0.5, prefill_splits=splits, out=out)
    ops.check_status()
    rows = torch.zeros(T, dtype=torch.bool, device="cuda")
    rows[first:first + 40] = True
    rows[first + 49:first + 49 + 256] = True              # 200 rows asked for are one tile of 256
    assert (out[~rows] == 7.0).all()
    assert out[rows].isfinite().all() and not (out[rows] == 7.0).all(1).any()


@pytest.mark.parametrize("T", [5, 150])
@pytest.mark.parametrize("E,top", [(1, 1), (32, 32), (33, 4), (64, 8), (100, 7), (128, 3), (200, 40), (256, 6), (257, 5)])
def test_routing_chooses_in_order(E, top, T):
    """The largest logits, ties (and the two zeros) by number of the expert, at every number of registers per lane."""
    from inference_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(E)
    z = (torch.randn(T, E, device="cuda", generator=g) * 4).round() / 2
    z[0] = 0.0
    z[0, ::3] = -0.0
    z[1, : E // 2] = -math.inf
    z[2] = z[2].abs() * -1e30
    plan, _ = ops.logits_routing(z, E, top)
    ops.check_status()
    order = torch.sort(z, dim=-1, descending=True, stable=True).indices[:, :top]
    expert = torch.repeat_interleave(torch.arange(E, device="cuda"), plan.offsets.long().diff())[plan.dest.long()]
    assert torch.equal(expert, order)
    want = torch.softmax(z.double(), -1).gather(1, order)
    assert torch.allclose(plan.weights.double(), want, rtol=1e-5, atol=1e-30)
    assert torch.equal(plan.src.long()[plan.dest.long()], torch.arange(T, device="cuda")[:, None].expand(T, top))


# 16 and 32 weight rows to a CTA; two and three CTAs to an SM on both sides of the lines (CTAs, length of the reduction); segments of one row to three passes
@pytest.mark.parametrize("E,top,N,K,T", [(4, 2, 72, 520, 3), (8, 1, 1176, 64, 9), (8, 1, 1192, 2568, 200), (16, 2, 1800, 2560, 40), (16, 2, 1800, 2568, 40), (64, 2, 1576, 2568, 90)])
@pytest.mark.parametrize("pairs", [False, True])
def test_rows_of_experts_at_every_split(E, top, N, K, T, pairs):
    from inference_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    w = torch.empty(E, N, K, device="cuda", dtype=torch.bfloat16).normal_(0.0, K ** -0.5, generator=g)
    z = torch.randn(T, E, device="cuda", generator=g)
    z[:, 0] += 2                            # one expert has most rows
    plan, _ = ops.logits_routing(z, E, top)
    got = ops.gemm_grouped_rows(x, w, plan, gather=True, act="swiglu_pairs" if pairs else None).double()
    ops.check_status()
    for e, (lo, hi) in enumerate(zip(plan.offsets.tolist(), plan.offsets.tolist()[1:])):
        if lo == hi:
            continue
        want = x[plan.src[lo:hi].long()].double() @ w[e].double().T
        if pairs:
            want = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
        # one rounding of fp32 sums of K terms of size K^-0.5
        assert ((got[lo:hi] - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5).all()


@pytest.mark.parametrize("value", [math.nan, math.inf, -math.inf])
def test_routing_of_what_is_no_number_names_experts(value):
    from inference_b200 import ops

    z = torch.full((4, 40), value, device="cuda")
    z[1:, :3] = torch.tensor([1.0, 2.0, 3.0], device="cuda")
    plan, _ = ops.logits_routing(z, 40, 6)
    ops.check_status()
    expert = torch.repeat_interleave(torch.arange(40, device="cuda"), plan.offsets.long().diff())[plan.dest.long()]
    assert all(len(set(row)) == 6 for row in expert.tolist())


def test_gated_act_embedding_argmax():
    from inference_b200 import ops

    gu = torch.randn(9, 2 * 1376, device="cuda").bfloat16()
    y = ops.gated_act_mul(gu)
    ref = torch.nn.functional.silu(gu[:, :1376].float()) * gu[:, 1376:].float()
    assert torch.allclose(y.float(), ref, atol=3e-2, rtol=2e-2)
    table = torch.randn(1000, 256, device="cuda").bfloat16()
    ids = torch.randint(0, 1000, (4, 7), device="cuda")
    e = ops.embedding(ids, table)
    assert torch.equal(e, table[ids.reshape(-1)])
    logits = torch.randn(6, 128256, device="cuda")
    logits[2, 77] = 50.0
    logits[2, 99000] = 50.0
    am = ops.argmax(logits)
    assert torch.equal(am, logits.argmax(-1)) or am[2].item() == 77
    assert am[2].item() == 77
    allow = torch.zeros(128256, dtype=torch.uint8, device="cuda")
    allow[1000:2000] = 1
    am2 = ops.argmax(logits.bfloat16(), allow)
    assert torch.equal(am2, logits.bfloat16()[:, 1000:2000].float().argmax(-1) + 1000)
    t = torch.tensor([[5, 6, 7, 8, 9], [5, 1, 7, 8, 9]], device="cuda")
    d = torch.tensor([[5, 6, 7, 0], [5, 6, 7, 8]], device="cuda")
    n, nxt = ops.spec_verify_greedy(t, d)
    assert n.tolist() == [3, 1] and nxt.tolist() == [8, 1]


def _ref_attn(q, k, v, scale, causal):
    # q [Sq, Hq, D], k/v [Skv, Hkv, D]
    Sq, Hq, D = q.shape
    Skv, Hkv, _ = k.shape
    G = Hq // Hkv
    kf = k.float().repeat_interleave(G, dim=1)
    vf = v.float().repeat_interleave(G, dim=1)
    s = torch.einsum("qhd,khd->hqk", q.float(), kf) * scale
    if causal:
        i = torch.arange(Sq, device=q.device)[:, None]
        j = torch.arange(Skv, device=q.device)[None, :]
        s = s.masked_fill(j > i + (Skv - Sq), float("-inf"))
    p = torch.softmax(s, dim=-1)
    return torch.einsum("hqk,khd->qhd", p, vf).reshape(Sq, Hq * D)


def _build_paged(kv_lens, Hkv, D, bs=16, extra=3):
    nblk_per = [(n + bs - 1) // bs for n in kv_lens]
    total = sum(nblk_per) + extra
    perm = torch.randperm(total).tolist()
    kc = torch.randn(total, Hkv, bs, D, device="cuda").bfloat16()
    vc = torch.randn(total, Hkv, bs, D, device="cuda").bfloat16()
    maxb = max(nblk_per)
    table = torch.zeros(len(kv_lens), maxb, dtype=torch.int32)
    ks, vs = [], []
    it = iter(perm)
    for i, n in enumerate(kv_lens):
        ids = [next(it) for _ in range(nblk_per[i])]
        table[i, : len(ids)] = torch.tensor(ids, dtype=torch.int32)
        kk = kc[ids].permute(0, 2, 1, 3).reshape(-1, Hkv, D)[:n]
        vv = vc[ids].permute(0, 2, 1, 3).reshape(-1, Hkv, D)[:n]
        ks.append(kk)
        vs.append(vv)
    return kc, vc, table.cuda(), ks, vs


@pytest.mark.parametrize("Hq,Hkv", [(8, 2), (4, 4)])
def test_paged_prefill(Hq, Hkv):
    from inference_b200 import ops

    D = 128
    q_lens = [70, 1, 129, 64]
    kv_lens = [70, 40, 200, 64]
    kc, vc, table, ks, vs = _build_paged(kv_lens, Hkv, D)
    T = sum(q_lens)
    q = torch.randn(T, Hq, D, device="cuda").bfloat16()
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device="cuda")
    kvl = torch.tensor(kv_lens, dtype=torch.int32, device="cuda")
    scale = 1 / math.sqrt(D)
    out = ops.paged_attention(q, kc, vc, table, kvl, cu_q=cu, max_q_len=max(q_lens), scale=scale, causal=True)
    o = 0
    for i, n in enumerate(q_lens):
        ref = _ref_attn(q[o:o + n], ks[i], vs[i], scale, True)
        err = (out[o:o + n].float() - ref).abs().max().item()
        assert err < 3e-2, (i, err)
        o += n


@pytest.mark.parametrize("bs", [8, 16, 32, 128])
def test_paged_prefill_tcgen05_against_reference_and_mma_sync(bs, monkeypatch):
    """Prefill on top of earlier context, pages read through TMA: several page sizes, contexts that end mid page and
    mid tile, one sequence with no earlier context, uniform query lengths without cu_q, and the non-causal form."""
    from inference_b200 import ops

    D, Hq, Hkv = 128, 8, 2
    q_lens = [300, 17, 128, 256]
    kv_lens = [1500, 401, 128, 257]
    kc, vc, table, ks, vs = _build_paged(kv_lens, Hkv, D, bs=bs)
    T = sum(q_lens)
    q = torch.randn(T, Hq, D, device="cuda").bfloat16()
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device="cuda")
    kvl = torch.tensor(kv_lens, dtype=torch.int32, device="cuda")
    scale = 1 / math.sqrt(D)
    for causal in (True, False):
        out = ops.paged_attention(q, kc, vc, table, kvl, cu_q=cu, max_q_len=max(q_lens), scale=scale, causal=causal)
        o = 0
        for i, n in enumerate(q_lens):
            ref = _ref_attn(q[o:o + n], ks[i], vs[i], scale, causal)
            err = (out[o:o + n].float() - ref).abs().max().item()
            assert err < 3e-2, (causal, i, err)
            o += n
    if bs == 16:
        monkeypatch.setenv("SWB_PAGED_PREFILL", "legacy")
        old = ops.paged_attention(q, kc, vc, table, kvl, cu_q=cu, max_q_len=max(q_lens), scale=scale, causal=True)
        monkeypatch.setenv("SWB_PAGED_PREFILL", "tcgen05")
        new = ops.paged_attention(q, kc, vc, table, kvl, cu_q=cu, max_q_len=max(q_lens), scale=scale, causal=True)
        assert (old.float() - new.float()).abs().max().item() < 3e-2
    # uniform query lengths, no cu_q
    kv2 = [200, 136, 264]
    kc, vc, table, ks, vs = _build_paged(kv2, Hkv, D, bs=bs)
    q = torch.randn(3 * 136, Hq, D, device="cuda").bfloat16()
    out = ops.paged_attention(q, kc, vc, table, torch.tensor(kv2, dtype=torch.int32, device="cuda"), cu_q=None, max_q_len=136,
                              scale=scale, causal=True)
    for i in range(3):
        ref = _ref_attn(q[i * 136:(i + 1) * 136], ks[i], vs[i], scale, True)
        assert (out[i * 136:(i + 1) * 136].float() - ref).abs().max().item() < 3e-2, i


@pytest.mark.parametrize("use_tma", [True, False])
@pytest.mark.parametrize("splits", [1, 3, 8])
@pytest.mark.parametrize("q_len", [1, 3])
def test_paged_decode(splits, q_len, use_tma):
    from inference_b200 import ops

    D, Hq, Hkv = 128, 16, 4
    kv_lens = [1 + q_len, 63, 64, 65, 500, 1300]
    kc, vc, table, ks, vs = _build_paged(kv_lens, Hkv, D)
    B = len(kv_lens)
    q = torch.randn(B * q_len, Hq, D, device="cuda").bfloat16()
    kvl = torch.tensor(kv_lens, dtype=torch.int32, device="cuda")
    scale = 1 / math.sqrt(D)
    out = ops.paged_attention(q, kc, vc, table, kvl, cu_q=None, max_q_len=q_len, scale=scale, causal=True,
                              decode=True, num_splits=splits, use_tma=use_tma)
    ops.check_status()
    for i in range(B):
        ref = _ref_attn(q[i * q_len:(i + 1) * q_len], ks[i], vs[i], scale, True)
        err = (out[i * q_len:(i + 1) * q_len].float() - ref).abs().max().item()
        assert err < 3e-2, (i, err)


def test_dense_attention_noncausal():
    from inference_b200 import ops

    B, S, H, D = 2, 333, 6, 128
    qkv = torch.randn(B, S, 3, H, D, device="cuda").bfloat16()
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    scale = 1 / math.sqrt(D)
    out = ops.dense_attention(q, k, v, scale=scale)
    for b in range(B):
        ref = _ref_attn(q[b], k[b], v[b], scale, False)
        assert (out[b].float() - ref).abs().max().item() < 3e-2


@pytest.mark.parametrize("B,Sq,Skv,Hq,Hkv,qmul", [(1, 4608, 4608, 4, 4, 1.0), (2, 300, 1000, 8, 2, 1.0),
                                                   (1, 1024, 2048, 2, 1, 6.0), (1, 129, 257, 2, 2, 1.0),
                                                   (1, 256, 128, 1, 1, 12.0)])
def test_dense_attention_tcgen05(B, Sq, Skv, Hq, Hkv, qmul):
    """tcgen05 kernel against fp32 math and against the mma.sync kernel; qmul > 1 spreads the logits so that the
    running maximum keeps growing and the lazy accumulator rescale is exercised."""
    from inference_b200 import ops
    from inference_b200.ops.attention import set_dense_impl

    g = torch.Generator(device="cuda").manual_seed(Sq * 31 + Skv)
    q = (torch.randn(B, Sq, Hq, 128, device="cuda", generator=g) * qmul).bfloat16()
    k = torch.randn(B, Skv, Hkv, 128, device="cuda", generator=g).bfloat16()
    v = torch.randn(B, Skv, Hkv, 128, device="cuda", generator=g).bfloat16()
    if qmul > 1:   # keys later in the sequence score higher on average
        k = (k.float() + q.float().mean(1, keepdim=True)[:, :, :Hkv] * torch.linspace(
            0, 0.05, Skv, device="cuda")[None, :, None, None]).bfloat16()
    scale = 1 / math.sqrt(128)
    out = ops.dense_attention(q, k, v, scale=scale)
    ops.check_status()
    set_dense_impl(True)
    try:
        legacy = ops.dense_attention(q, k, v, scale=scale)
    finally:
        set_dense_impl(False)
    from inference_b200._native import kernels

    forced = []
    try:
        for tiles in (1, 2):          # both schedules: one query tile per CTA, two with softmax / MMA overlap
            kernels().swb_attn_dense_set_tiles(tiles)
            forced.append(ops.dense_attention(q, k, v, scale=scale))
            ops.check_status()
    finally:
        kernels().swb_attn_dense_set_tiles(0)
    for b in range(B):
        ref = _ref_attn(q[b], k[b], v[b], scale, False)
        err = (out[b].float() - ref).abs().max().item()
        assert err < 3e-2, (b, err)
        assert (out[b].float() - legacy[b].float()).abs().max().item() < 3e-2
        for f in forced:
            assert (f[b].float() - ref).abs().max().item() < 3e-2


@pytest.mark.parametrize("lens,Hq,Hkv", [([300, 17, 1024, 129], 8, 2), ([64], 4, 4), ([1000, 1000], 2, 1)])
def test_varlen_causal_attention_tcgen05(lens, Hq, Hkv):
    """Packed fresh-prefill attention straight from a QKV buffer (strided views) against fp32 causal attention."""
    from inference_b200 import ops

    T = sum(lens)
    g = torch.Generator(device="cuda").manual_seed(T)
    qkv = torch.randn(T, (Hq + 2 * Hkv) * 128, device="cuda", generator=g).bfloat16()
    q = qkv[:, : Hq * 128].view(T, Hq, 128)
    k = qkv[:, Hq * 128:(Hq + Hkv) * 128].view(T, Hkv, 128)
    v = qkv[:, (Hq + Hkv) * 128:].view(T, Hkv, 128)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device="cuda")
    scale = 1 / math.sqrt(128)
    out = ops.varlen_causal_attention(q, k, v, cu, max(lens), scale=scale)
    ops.check_status()
    lo = 0
    for n in lens:
        ref = _ref_attn(q[lo:lo + n], k[lo:lo + n], v[lo:lo + n], scale, True)
        err = (out[lo:lo + n].float() - ref).abs().max().item()
        assert err < 3e-2, (n, err)
        lo += n


def _one_by_one(a, b, D, causal=False):
    """softmax of the scores a_i b_j (exact products of bf16 numbers), probability by probability: the values are rows of the unit
    matrix for D keys at a time. a [queries], b [keys] -> [queries, keys], bf16 as the kernel stores it."""
    from inference_b200 import ops

    n, m = a.numel(), b.numel()
    q, k = torch.zeros(1, n, 1, D, device="cuda", dtype=torch.bfloat16), torch.zeros(1, m, 1, D, device="cuda", dtype=torch.bfloat16)
    q[0, :, 0, 0], k[0, :, 0, 0] = a, b
    got = torch.empty(n, m, device="cuda", dtype=torch.bfloat16)
    for j in range(0, m, D):
        v = torch.zeros_like(k)
        w = min(D, m - j)
        v[0, j:j + w, 0, :w] = torch.eye(w, device="cuda")
        if causal:
            cu = torch.tensor([0, n], dtype=torch.int32, device="cuda")
            out = ops.varlen_causal_attention(q[0], k[0], v[0], cu, n, scale=1.0)
        else:
            out = ops.dense_attention(q, k, v, scale=1.0)[0]
        got[:, j:j + w] = out[:, :w]
    ops.check_status()
    return got


@pytest.mark.parametrize("D,keys,causal", [(128, 300, False), (64, 300, False), (128, 300, True), (64, 129, False), (128, 1100, True)])
def test_dense_attention_probabilities_one_by_one(D, keys, causal):
    """Scores from 0 down to -140, in an order whose maximum grows by little and by much from tile to tile. Two roundings to bf16 (the weight
    and the result, 2^-8 each: half of the last of 8 bits) and 1e-4 for the exponent in fp32. What is masked or far below stays under 2^-120."""
    g = torch.Generator(device="cuda").manual_seed(keys + D)
    b = (-140 * torch.rand(keys, device="cuda", generator=g) ** 2).bfloat16()
    b[:128] -= 60
    b[keys // 2] = 0
    a = torch.tensor([1.0, 0.5, 0.75, 0.0078125, 1.25, 0.0], device="cuda").bfloat16().repeat(keys // 6 + 1)[:keys]
    got = _one_by_one(a, b, D, causal).double()
    scores = a.double()[:, None] * b.double()[None, :]
    if causal:
        scores = scores.masked_fill(torch.arange(keys, device="cuda")[None, :] > torch.arange(keys, device="cuda")[:, None], -torch.inf)
    want = scores.softmax(-1)
    assert ((got - want).abs() <= (2.0 ** -7 + 1e-4) * want + 2.0 ** -120).all()


@pytest.mark.parametrize("D", [64, 128])
def test_dense_attention_numbers_that_are_none(D):
    """A query that is not a number and one whose score overflows give rows that are none; a key at minus infinity has no weight; the
    other rows are as they are without them."""
    a = torch.linspace(0.5, 1.0, 200, device="cuda").bfloat16()
    b = torch.linspace(-20.0, -1.0, 333, device="cuda").bfloat16()
    clean = _one_by_one(a, b, D)
    a2 = a.clone()
    a2[7], a2[150] = torch.nan, -3e38
    got = _one_by_one(a2, b, D)
    rows = torch.ones(200, dtype=torch.bool, device="cuda")
    rows[7] = rows[150] = False
    assert got[~rows].isnan().all() and torch.equal(got[rows], clean[rows])
    b2 = b.clone()
    b2[40], b2[332] = -torch.inf, -torch.inf
    got = _one_by_one(a, b2, D).double()
    want = (a.double()[:, None] * b2.double()[None, :]).softmax(-1)
    assert ((got - want).abs() <= (2.0 ** -7 + 1e-4) * want + 2.0 ** -120).all()
