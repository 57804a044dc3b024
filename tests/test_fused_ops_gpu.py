"""The projections either side of GCA with their small operations fused in (inference path):
``gca_row_rms`` + ``gca_linear`` through the C ABI, against plain float32 PyTorch on the same bf16
inputs, and ``TritonGroupCrossAttention.forward_fused`` against the fixture produced by the
REFERENCE's module class (``tests/golden/module_ref.npz``, ``model/DRT.py:345-398``) and against
this repository's unfused ``forward_indexed``.  bf16 data, float32 accumulation: per element
|a - b| <= 1e-2 * scale + 2e-2 * |b| with scale = max |b|.
"""
import os

import numpy as np
import pytest
import torch

import make_golden as MG

pytestmark = pytest.mark.gpu


def close(a, b, what=""):
    a, b = a.detach().float().cpu(), torch.as_tensor(b).float().cpu()
    scale = b.abs().max().item() + 1e-12
    bad = (a - b).abs() > 1e-2 * scale + 2e-2 * b.abs()
    assert not bad.any(), (what, int(bad.sum()), ((a - b).abs().max() / scale).item())


def need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


@pytest.mark.parametrize("m,d", [(1, 768), (37, 128), (4100, 768)])
def test_row_rms(m, d):
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    x = (torch.randn(m, d, generator=torch.Generator().manual_seed(m)) * 3).bfloat16().cuda()
    got = F.row_rms(x, 1e-5)
    ref = torch.rsqrt(x.float().pow(2).mean(-1) + 1e-5)
    assert torch.allclose(got, ref, rtol=1e-5, atol=0)


@pytest.mark.parametrize("m,n,k", [(1, 768, 768), (300, 768, 768), (129, 48, 128), (1000, 1024, 3072), (64, 272, 64)])
@pytest.mark.parametrize("with_scale,with_res", [(False, False), (True, False), (False, True), (True, True)])
def test_linear_against_float32(m, n, k, with_scale, with_res):
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    import long_context_modeling_b200 as lcm
    g = torch.Generator().manual_seed(m * 7 + n)
    x = torch.randn(m, k, generator=g).bfloat16().cuda()
    w = (torch.randn(n, k, generator=g) / k ** 0.5).bfloat16().cuda()
    sc = (torch.rand(m, generator=g) + 0.5).cuda() if with_scale else None
    res = torch.randn(m, n, generator=g).bfloat16().cuda() if with_res else None
    out = torch.full((m, n), 7.0, dtype=torch.bfloat16, device="cuda")
    F.linear(x, w, row_scale=sc, residual=res, out=out)
    ref = x.float() @ w.float().T
    if with_scale:
        ref = ref * sc[:, None]
    if with_res:
        ref = ref + res.float()
    close(out, ref, (m, n, k))
    assert lcm.read_status() == 0


def test_linear_writes_only_its_rows_and_columns():
    """Strided output (a column block of a wider matrix, a row block of a taller one): nothing outside
    the (M, N) window changes."""
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    g = torch.Generator().manual_seed(3)
    x = torch.randn(200, 128, generator=g).bfloat16().cuda()
    w = (torch.randn(64, 128, generator=g) / 11).bfloat16().cuda()
    big = torch.full((260, 256), -5.0, dtype=torch.bfloat16, device="cuda")
    F.linear(x, w, out=big[30:230, 64:128])
    close(big[30:230, 64:128], x.float() @ w.float().T)
    mask = torch.ones_like(big, dtype=torch.bool)
    mask[30:230, 64:128] = False
    assert (big[mask] == -5.0).all()


def test_linear_rejects_bad_arguments():
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    x = torch.zeros(8, 96, dtype=torch.bfloat16, device="cuda")            # K not a multiple of 64
    w = torch.zeros(64, 96, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(ValueError):
        F.linear(x, w)
    with pytest.raises(ValueError):
        F.linear(torch.zeros(8, 128, device="cuda"), torch.zeros(64, 128, dtype=torch.bfloat16, device="cuda"))
    with pytest.raises(RuntimeError):
        F.linear(torch.zeros(8, 128, dtype=torch.bfloat16), torch.zeros(64, 128, dtype=torch.bfloat16))


def test_rmsnorm_linear_matches_norm_then_projection():
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    g = torch.Generator().manual_seed(9)
    x = (torch.randn(2, 5, 64, 768, generator=g) * 2).bfloat16().cuda()
    gain = (1 + 0.2 * torch.randn(768, generator=g)).cuda()
    w = (torch.randn(768, 768, generator=g) / 28).bfloat16().cuda()
    got = F.rmsnorm_linear(x, F.fold_gain(w, gain), 1e-5)
    xf = x.float()
    normed = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * gain
    close(got, normed @ w.float().T)
    assert got.shape == (2, 5, 64, 768)


def _fixture_module(golden_dir):
    import long_context_modeling_b200 as lcm
    g = np.load(os.path.join(golden_dir, "module_ref.npz"))
    cfg = MG.ModuleConfig()
    n, c, k = 1, 3, cfg.chunk_topk
    hidden, gk, gv, w, dout, params = MG.module_case(51, n, c, cfg.num_attention_heads, k, cfg.hidden_size)
    mod = lcm.TritonGroupCrossAttention(cfg).cuda()
    mod.load_state_dict({k_: v_.cuda() for k_, v_ in params.items()})
    return g, cfg, mod.bfloat16().eval(), hidden, gk, gv, w


def test_fused_module_path_matches_reference_class(golden_dir):
    """forward_fused (RMSNorm folded into q_proj's GEMM, o_proj with residual epilogue) in bf16 against
    the reference class's float32 output for the same parameters and inputs; the gathered chunks of
    the fixture serve as the cache, read through an identity index."""
    need_gpu()
    g, cfg, mod, hidden, gk, gv, w = _fixture_module(golden_dir)
    k = cfg.chunk_topk
    n, dk = gk.shape[:2]
    idx = torch.arange(dk, dtype=torch.int32).view(1, dk // k, k).expand(n, -1, -1).contiguous().cuda()
    hs = hidden.bfloat16().cuda()
    kc, vc = gk.bfloat16().cuda(), gv.bfloat16().cuda()
    with torch.no_grad():
        o = mod.forward_fused(hs, kc, vc, idx, w.cuda())
        close(o, g["triton_eval_o"], "no residual")
        assert o[:, :64].abs().max().item() == 0            # the first chunk retrieves nothing
        res = torch.randn(o.shape, generator=torch.Generator().manual_seed(1)).bfloat16().cuda()
        o2 = mod.forward_fused(hs, kc, vc, idx, w.cuda(), residual=res)
        close(o2, torch.as_tensor(g["triton_eval_o"]) + res.float().cpu(), "with residual")
        assert torch.equal(o2[:, :64], res[:, :64])
        # and against the unfused path of this repository
        close(o2, (mod.forward_indexed(hs, kc, vc, idx, w.cuda()).float() + res.float()), "vs forward_indexed")
        # one-row decode step (chunk_size == 1: nothing is skipped)
        o1 = mod.forward_fused(hs[:, 1:2, :1], kc[:, :k], vc[:, :k], idx[:, :1], w[:, :1].cuda())
        close(o1, g["triton_decode_o"], "decode")


@pytest.mark.parametrize("n,heads,rows,k,chunks", [(1, 12, 1, 8, 64), (3, 4, 2, 1, 5), (7, 8, 1, 5, 9), (2, 16, 2, 12, 40), (1, 12, 2, 16, 30),
                                                   (5, 16, 1, 3, 7), (9, 12, 1, 8, 20), (1, 16, 1, 13, 20)])
def test_one_launch_decode_step(n, heads, rows, k, chunks):
    """The whole sub-layer of a decode step as one launch -- (head, slot) tiles that do not divide evenly among the cluster's CTAs,
    padding slots, a sequence without any, with and without residual -- against the unfused path; the last two are outside its
    range and take the three launches."""
    need_gpu()
    import long_context_modeling_b200 as lcm
    g = torch.Generator().manual_seed(7)
    dim = heads * 64
    mod = lcm.TritonGroupCrossAttention(dim, heads, chunk_topk=k).to("cuda", torch.bfloat16).eval()
    hs = torch.randn(n, 1, rows, dim, generator=g).bfloat16().cuda()
    kc, vc = (torch.randn(n, chunks, 64, dim, generator=g).bfloat16().cuda() for _ in range(2))
    idx = torch.stack([torch.randperm(max(chunks, k), generator=g)[:k] for _ in range(n)]).view(n, 1, k).to(torch.int32)
    idx[idx >= chunks] = -1
    idx[0, 0, k // 2:] = -1
    if n > 2:
        idx[2] = -1
    w = torch.softmax(torch.randn(n, 1, k, generator=g), -1).masked_fill(idx < 0, 0.0).cuda()
    idx = idx.cuda()
    res = torch.randn(n, rows, dim, generator=g).bfloat16().cuda()
    with torch.no_grad():
        want = mod.forward_indexed(hs, kc, vc, idx, w).float()
        close(mod.forward_fused(hs, kc, vc, idx, w), want, "no residual")
        close(mod.forward_fused(hs, kc, vc, idx, w, residual=res), want + res.float(), "with residual")
    assert lcm.read_status() == 0


def _window_reference(q, k, v, window, slopes, scale):
    """float32: explicit scores, ALiBi bias, window + causal mask, softmax (model/llama.py:684-688 semantics)."""
    n, hq, sq, d = q.shape
    hkv, t = k.shape[1], k.shape[2]
    g = hq // hkv
    kf = k.float().repeat_interleave(g, 1)
    vf = v.float().repeat_interleave(g, 1)
    s = torch.einsum("nhid,nhjd->nhij", q.float(), kf) * scale
    pos = torch.arange(t - sq, t).view(sq, 1)
    j = torch.arange(t).view(1, t)
    dist = (pos - j).float()
    bias = torch.zeros(hq, sq, t) if slopes is None else -slopes.view(hq, 1, 1).cpu() * dist
    bias = bias.masked_fill((dist < 0) | (dist > window), float("-inf"))
    p = torch.softmax(s.cpu() + bias, -1)
    return torch.einsum("nhij,nhjd->nhid", p, vf.cpu())


@pytest.mark.parametrize("n,hq,hkv,sq,t,window,alibi", [
    (2, 12, 12, 1, 513, 512, True),       # the model's decode step: one new position, full window
    (3, 4, 4, 2, 300, 512, True),         # two new positions, fewer keys than the window
    (2, 8, 4, 2, 700, 128, True),         # grouped-query heads, keys older than the window are skipped
    (1, 2, 2, 1, 1, 16, False),           # a single key, no ALiBi
    (2, 4, 1, 1, 97, 40, True),           # four q heads on one kv head
    (1, 12, 12, 3, 1030, 512, True),      # three rows
])
def test_window_decode_against_float32(n, hq, hkv, sq, t, window, alibi):
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    g = torch.Generator().manual_seed(t + sq)
    q = torch.randn(n, hq, sq, 64, generator=g).bfloat16().cuda()
    k = torch.randn(n, hkv, t, 64, generator=g).bfloat16().cuda()
    v = torch.randn(n, hkv, t, 64, generator=g).bfloat16().cuda()
    slopes = torch.tensor([2.0 ** (-8.0 * (i + 1) / hq) for i in range(hq)]).cuda() if alibi else None
    got = F.window_decode(q, k, v, window, slopes, 0.125)
    ref = _window_reference(q, k, v, window, slopes, 0.125)
    close(got, ref, (n, hq, hkv, sq, t, window))


@pytest.mark.parametrize("items,g,sq,t,window", [
    (3, 1, 1, 1, 7), (2, 1, 1, 2, 7), (4, 1, 1, 17, 16), (4, 1, 1, 18, 40),      # one warp: a single key, the last row beside one and sixteen keys
    (5, 1, 1, 513, 512), (5, 2, 1, 641, 700), (12, 1, 1, 640, 639),              # clusters of CTAs
    (60, 1, 1, 350, 349), (60, 2, 1, 200, 300), (148, 1, 1, 513, 512),           # one round, two rounds
    (390, 1, 1, 200, 199), (150, 3, 1, 260, 300), (800, 2, 1, 66, 65),           # several rounds, a row pair that is half empty
    (700, 1, 1, 300, 299), (350, 4, 1, 330, 329), (1500, 2, 1, 50, 49),          # ... and waves, two pairs, a single warp a CTA
    (2, 1, 2, 40, 16), (150, 1, 2, 500, 300), (300, 2, 2, 300, 64),              # rows at two positions: each sees a key that the other does not
])
@pytest.mark.parametrize("poison", [False, True])
def test_window_decode_splits(items, g, sq, t, window, poison):
    """Every split of the keys over warps, CTAs and rounds, linear and (one position) ring; with `poison`, rows that no query may see
    hold NaN, and one visible value is infinite: only that output column is."""
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    gen = torch.Generator().manual_seed(items + t)
    h = 2 if items % 2 == 0 else 1
    n = items // h
    k, v = (torch.randn(n, h, t, 64, generator=gen).bfloat16().cuda() for _ in range(2))
    q = torch.randn(n, h * g, sq, 64, generator=gen).bfloat16().cuda()
    slopes = torch.linspace(0.02, 0.3, h * g).cuda()
    k_seen, v_seen = k.clone(), v.clone()
    if poison:
        v[0, 0, t - sq, 5] = v_seen[0, 0, t - sq, 5] = float("inf")        # the first position's own row: every position sees it
        if t - sq - window > 0:
            k[:, :, :t - sq - window], v[:, :, :t - sq - window] = float("nan"), float("nan")
    ref = _window_reference(q, k_seen, v_seen, window, slopes, 0.125)
    forms = [F.window_decode(q, k, v, window, slopes, 0.125)]
    if sq == 1 and t <= window + 1:
        turn = 2 * t // 3                                          # the ring starts there; its oldest row is about to be overwritten
        count = torch.full((1,), 5 * t + turn, dtype=torch.int64).cuda()
        kr, vr = (torch.roll(x, turn + 1, 2) for x in (k, v))
        if poison:
            kr[:, :, turn], vr[:, :, turn] = float("nan"), float("nan")
        forms.append(F.window_ring_decode(q, kr, vr, k[:, :, t - 1:].contiguous(), v[:, :, t - 1:].contiguous(), count, window, slopes, 0.125))
        assert torch.equal(kr.roll(-(turn + 1), 2), k) and torch.equal(vr.roll(-(turn + 1), 2), v)
    for got in forms:
        got = got.float().cpu()
        inf = torch.isinf(ref)
        assert torch.equal(torch.isinf(got), inf) and not torch.isnan(got).any()
        got, want = got.masked_fill(inf, 0.0), ref.masked_fill(inf, 0.0)
        # bf16: eight significant bits, the error half a unit of the last place, 2^-8 of the value; float32 sums (2^-18 of the largest)
        assert ((got - want).abs() <= want.abs() * 2.0 ** -8 + 2.0 ** -18 * want.abs().max()).all()


def test_window_decode_reads_strided_caches():
    """k / v as (N, T, H, 64) token-major storage viewed as (N, H, T, 64): the reference's cache layout."""
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    g = torch.Generator().manual_seed(5)
    q = torch.randn(2, 1, 6, 64, generator=g).bfloat16().cuda().transpose(1, 2)          # (N, H, 1, 64) view
    k = torch.randn(2, 200, 6, 64, generator=g).bfloat16().cuda().transpose(1, 2)
    v = torch.randn(2, 200, 6, 64, generator=g).bfloat16().cuda().transpose(1, 2)
    slopes = torch.full((6,), 0.05).cuda()
    close(F.window_decode(q, k, v, 64, slopes, 0.125), _window_reference(q, k, v, 64, slopes, 0.125))


@pytest.mark.parametrize("m,v,k", [(300, 50265, 768), (1, 1000, 64), (129, 257, 128), (2000, 4096, 768)])
def test_linear_cross_entropy_against_float32(m, v, k):
    """LM head + cross-entropy without logits in memory, against torch on float32 logits of the same
    bf16 inputs; ignored rows (target -100) give 0."""
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    import long_context_modeling_b200 as lcm
    g = torch.Generator().manual_seed(m + v)
    x = torch.randn(m, k, generator=g).bfloat16().cuda()
    w = (torch.randn(v, k, generator=g) * (3.0 / k ** 0.5)).bfloat16().cuda()
    t = torch.randint(0, v, (m,), generator=g).cuda()
    if m > 4:
        t[3] = -100
        t[m - 1] = v - 1
    loss, lse = F.linear_cross_entropy(x, w, t, return_lse=True)
    logits = x.float() @ w.float().T
    ref = torch.nn.functional.cross_entropy(logits, t, reduction="none", ignore_index=-100)
    assert torch.allclose(loss, ref, rtol=2e-4, atol=2e-4), (loss - ref).abs().max().item()
    assert torch.allclose(lse, torch.logsumexp(logits, -1), rtol=2e-5, atol=2e-4)
    if m > 4:
        assert loss[3].item() == 0.0
    assert lcm.read_status() == 0


def test_linear_cross_entropy_with_rmsnorm_scale_and_bad_target():
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    g = torch.Generator().manual_seed(11)
    x = (torch.randn(2, 70, 128, generator=g) * 2).bfloat16().cuda()
    w = (torch.randn(513, 128, generator=g) / 4).bfloat16().cuda()
    t = torch.randint(0, 513, (2, 70), generator=g).cuda()
    sc = F.row_rms(x, 1e-5)
    loss = F.linear_cross_entropy(x, w, t, row_scale=sc)
    xf = x.float()
    logits = (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5)) @ w.float().T
    ref = torch.nn.functional.cross_entropy(logits.view(-1, 513), t.view(-1), reduction="none").view(2, 70)
    assert loss.shape == (2, 70)
    assert torch.allclose(loss, ref, rtol=3e-4, atol=3e-4)
    t[0, 0] = 513                                   # outside the vocabulary: the loss says so
    assert torch.isnan(F.linear_cross_entropy(x, w, t)[0, 0])


@pytest.mark.parametrize("n,h,t", [(2, 3, 513), (1, 1, 1), (3, 2, 41), (2, 12, 640)])
def test_window_shift_append_in_place(n, h, t):
    """Oldest row out, new row in, in place, against torch.cat + slice; batch-strided windows and new rows that
    are views of a wider projection output."""
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    g = torch.Generator().manual_seed(t)
    big_k = torch.randn(n + 1, h, t, 64, generator=g).bfloat16().cuda()
    big_v = torch.randn(n + 1, h, t, 64, generator=g).bfloat16().cuda()
    kw, vw = big_k[1:], big_v[1:]                                   # views with an offset
    qkv = torch.randn(n, 3 * h * 64, generator=g).bfloat16().cuda()
    kn = qkv[:, h * 64:2 * h * 64].view(n, 1, h, 64).transpose(1, 2)  # (N, H, 1, 64) strided views
    vn = qkv[:, 2 * h * 64:].view(n, 1, h, 64).transpose(1, 2)
    ref_k, ref_v = torch.cat([kw, kn], 2)[:, :, 1:].clone(), torch.cat([vw, vn], 2)[:, :, 1:].clone()
    guard = big_k[0].clone()
    F.window_shift_append(kw, vw, kn, vn)
    assert torch.equal(kw, ref_k) and torch.equal(vw, ref_v)
    assert torch.equal(big_k[0], guard)                              # nothing outside the windows moved


@pytest.mark.gpu
@pytest.mark.parametrize("n,hq,hkv,t,steps", [(3, 2, 2, 41, 5), (2, 4, 2, 64, 70), (32, 12, 12, 513, 3)])
def test_window_ring_decode_equals_shift_then_decode(n, hq, hkv, t, steps):
    """The ring form (new row replaces the oldest inside the attention kernel, a device counter gives the
    phase) against moving the window and attending to it, step by step: outputs equal within bf16 rounding
    (the keys reach the online softmax in another order), and the ring rolled back by the phase IS the moved
    window -- also after the counter has wrapped around the ring."""
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    g = torch.Generator().manual_seed(t + steps)
    ring_k = torch.randn(n, hkv, t, 64, generator=g).bfloat16().cuda()
    ring_v = torch.randn(n, hkv, t, 64, generator=g).bfloat16().cuda()
    lin_k, lin_v = ring_k.clone(), ring_v.clone()
    slopes = (2.0 ** -torch.arange(1, hq + 1).float()).cuda()
    written = torch.zeros(1, dtype=torch.int64, device="cuda")
    for s in range(steps):
        qkv = torch.randn(n, (hq + 2 * hkv) * 64, generator=g).bfloat16().cuda()
        q = qkv[:, :hq * 64].view(n, 1, hq, 64).transpose(1, 2)
        kn = qkv[:, hq * 64:(hq + hkv) * 64].view(n, 1, hkv, 64).transpose(1, 2)
        vn = qkv[:, (hq + hkv) * 64:].view(n, 1, hkv, 64).transpose(1, 2)
        F.window_shift_append(lin_k, lin_v, kn, vn)
        want = F.window_decode(q, lin_k, lin_v, t - 1, slopes, 0.125)
        got = F.window_ring_decode(q, ring_k, ring_v, kn, vn, written, t - 1, slopes, 0.125)
        written += 1
        assert (got.float() - want.float()).abs().max().item() <= 1e-2 * want.float().abs().max().item(), s
    assert torch.equal(torch.roll(ring_k, -(steps % t), 2), lin_k)
    assert torch.equal(torch.roll(ring_v, -(steps % t), 2), lin_v)


@pytest.mark.gpu
def test_window_ring_decode_rejects_bad_arguments():
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    q = torch.zeros(1, 1, 1, 64, dtype=torch.bfloat16, device="cuda")
    ring = torch.zeros(1, 1, 8, 64, dtype=torch.bfloat16, device="cuda")
    new = torch.zeros(1, 1, 64, dtype=torch.bfloat16, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
    with pytest.raises(ValueError):
        F.window_ring_decode(q, ring, ring, new, new, cnt.int(), 7)                    # counter must be int64
    with pytest.raises(ValueError):
        F.window_ring_decode(q, ring, ring, new, new, cnt, 3)                          # rows of the ring outside the window
    with pytest.raises(ValueError):
        F.window_ring_decode(q.expand(1, 1, 2, 64).contiguous(), ring, ring, new, new, cnt, 7)      # one new position only


@pytest.mark.gpu
@pytest.mark.parametrize("m,inter", [(1, 8), (32, 2048), (257, 1536)])
def test_silu_mul_against_float32(m, inter):
    """silu(gate) * up over the output of one stacked gate|up projection, against float32 (one bf16 rounding),
    from a row-strided input; argument checks."""
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    g = torch.Generator().manual_seed(m + inter)
    wide = (torch.randn(m, 2 * inter + 16, generator=g) * 3).bfloat16().cuda()
    gu = wide[:, :2 * inter]                                        # row stride wider than the row
    want = torch.nn.functional.silu(gu[:, :inter].float()) * gu[:, inter:].float()
    got = F.silu_mul(gu)
    assert got.shape == (m, inter) and got.dtype == torch.bfloat16
    assert (got.float() - want).abs().max().item() <= 1e-2 * want.abs().max().item()
    assert torch.equal(F.silu_mul(gu.view(1, m, 2 * inter).contiguous()).view(m, inter), got)
    with pytest.raises(ValueError):
        F.silu_mul(gu[:, :2 * inter - 8].contiguous()[:, :2 * inter - 12])   # halves not a multiple of 8 wide


@pytest.mark.parametrize("m,n,k", [(1, 16, 64), (16, 768, 768), (17, 48, 2080), (33, 512, 96 * 2), (65, 768, 768), (128, 1024, 1024)])
@pytest.mark.parametrize("with_res", [False, True])
def test_few_row_linear_and_fused_norm_against_float32(m, n, k, with_res):
    """The latency-bound form (up to 128 rows): every number of 16-row tiles, contractions that do not split evenly over the
    warps, and RMSNorm fused into the projection."""
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    k = k // 64 * 64
    g = torch.Generator().manual_seed(m + n)
    x, w, r = ((torch.randn(*s, generator=g) * c).bfloat16().cuda() for s, c in (((m, k), 1.0), ((n, k), k ** -0.5), ((m, n), 1.0)))
    y = F.linear(x, w, residual=r if with_res else None)
    ref = x.float() @ w.float().t() + (r.float() if with_res else 0)
    assert (y.float() - ref).abs().max() <= 2e-2 * ref.abs().max()
    z = F.rmsnorm_linear(x * 3, w, 1e-5)
    xf = (x * 3).float()
    ref = (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5)) @ w.float().t()
    assert (z.float() - ref).abs().max() <= 2e-2 * ref.abs().max()


@pytest.mark.parametrize("m,n,k", [(200, 768, 768), (3000, 272, 128), (6912, 768, 768), (20011, 784, 192), (40000, 768, 768)])
def test_linear_tile_widths_against_float32(m, n, k):
    """Every tile the GEMM chooses from (64 to 256 columns, pairs of CTAs on 256 x 256), ragged in rows and columns, with the
    row scale and the residual."""
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    g = torch.Generator(device="cuda").manual_seed(m)
    x, w, r = ((torch.randn(*s, generator=g, device="cuda") * c).bfloat16() for s, c in (((m, k), 1.0), ((n, k), k ** -0.5), ((m, n), 1.0)))
    sc = torch.rand(m, generator=g, device="cuda") + 0.5
    y = F.linear(x, w, row_scale=sc, residual=r)
    ref = (x.float() @ w.float().t()) * sc[:, None] + r.float()
    assert (y.float() - ref).abs().max() <= 2e-2 * ref.abs().max()
    assert torch.equal(y, F.linear(x, w, row_scale=sc, residual=r))


@pytest.mark.parametrize("m,n,k", [(129, 64, 64), (200, 768, 768), (1000, 1008, 192), (2333, 512, 512), (7105, 768, 768),     # 64 .. 192 columns
                                   (5100, 768, 64), (20001, 256, 128), (25000, 768, 768)])      # fewer K steps than stages, 256 columns, pairs
def test_norm_from_the_tiles_of_x(m, n, k):
    """RMSNorm + projection whose row factors are summed up beside the MMAs (or by a launch before, for pairs), against 64 bits; rows
    of very different sizes, several tiles per CTA."""
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    import long_context_modeling_b200 as lcm
    g = torch.Generator(device="cuda").manual_seed(m)
    x = (torch.randn(m, k, generator=g, device="cuda") * torch.exp2(torch.randint(-20, 20, (m, 1), generator=g, device="cuda").float())).bfloat16()
    w = (torch.randn(n, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    got = F.rmsnorm_linear(x, w, 1e-5).double()
    xd = x.double()
    ref = (xd @ w.double().t()) * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5)
    # the rounding to bf16, 2^-8 of the value, and float32: k terms of 2^-24 of the row's largest, the factor's 2^-22
    assert ((got - ref).abs() <= ref.abs() * (2.0 ** -8 + 2.0 ** -22) + k * 2.0 ** -24 * ref.abs().amax(-1, keepdim=True)).all()
    assert torch.equal(got, F.rmsnorm_linear(x, w, 1e-5).double()) and lcm.read_status() == 0


@pytest.mark.parametrize("m,n,k", [(130, 80, 64), (2333, 512, 512), (7105, 784, 192), (12400, 768, 512), (25000, 1024, 1024)])
def test_residual_read_ahead_and_norm_tiles(m, n, k):
    """The residual is read two passes ahead of the stores: adding onto it in place gives what a residual of its own gives, in 1 to 4 passes of a thread's
    columns, a last one of 16.  The same sizes with the norm: 64 to 256 columns in up to six waves, and pairs behind a launch for the factors."""
    need_gpu()
    from long_context_modeling_b200 import fused_ops as F
    g = torch.Generator(device="cuda").manual_seed(m)
    x, w, r = ((torch.randn(*s, generator=g, device="cuda") * c).bfloat16() for s, c in (((m, k), 1.0), ((n, k), k ** -0.5), ((m, n), 1.0)))
    y = F.linear(x, w, residual=r)
    close(y, x.float() @ w.float().t() + r.float())
    there = r.clone()
    F.linear(x, w, residual=there, out=there)
    assert torch.equal(there, y)
    xf = x.float()
    close(F.rmsnorm_linear(x, w, 1e-5), (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5)) @ w.float().t())


def exactly(got, ref, k):
    """Against 64 bits: the rounding to bf16, 2^-8 of the value, and float32: k terms of 2^-24 of the row's largest, the factor's 2^-22."""
    bound = ref.abs() * (2.0 ** -8 + 2.0 ** -22) + k * 2.0 ** -24 * ref.abs().amax(-1, keepdim=True)
    assert ((got.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("m,n,k", [(9100, 1808, 2048), (4100, 4112, 1024), (49153, 528, 4096), (24580, 1040, 2048)])
def test_pairs_of_ctas_in_linear_products(m, n, k):
    """Sizes whose tiles are shared by two CTAs, ragged in rows and in columns: row scale, residual in a place of its own and in the output's, and the norm
    whose factors a launch before sums up, rows of very different sizes."""
    need_gpu()
    import long_context_modeling_b200 as lcm
    from long_context_modeling_b200 import fused_ops as F
    g = torch.Generator(device="cuda").manual_seed(m)
    x = (torch.randn(m, k, generator=g, device="cuda") * torch.exp2(torch.randint(-20, 20, (m, 1), generator=g, device="cuda").float())).bfloat16()
    w = (torch.randn(n, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    r = torch.randn(m, n, generator=g, device="cuda").bfloat16()
    sc = torch.rand(m, generator=g, device="cuda") + 0.5
    product, factor = x.double() @ w.double().t(), torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5)
    exactly(F.linear(x, w), product, k)
    exactly(F.linear(x, w, row_scale=sc), product * sc.double()[:, None], k)
    exactly(F.rmsnorm_linear(x, w, 1e-5), product * factor, k)
    y = F.linear(x, w, row_scale=sc, residual=r)
    # a sum that cancels keeps the error of its terms
    ref, terms = product * sc.double()[:, None] + r.double(), (product * sc.double()[:, None]).abs() + r.double().abs()
    assert ((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + (k * 2.0 ** -24) * terms.amax(-1, keepdim=True)).all()
    there = r.clone()
    F.linear(x, w, row_scale=sc, residual=there, out=there)
    assert torch.equal(there, y) and lcm.read_status() == 0


@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("residual", [None, "own", "in place"])
def test_pairs_of_ctas_over_batches(norm, residual):
    """The C entries over blocks of rows with a gap between them, whose 256-row tiles hold rows of two blocks; lead rows get the residual alone, or zeros."""
    need_gpu()
    import ctypes as C
    from long_context_modeling_b200 import _lib
    b, m, n, k, lead = 3, 3033, 1808, 2048, 0 if norm else 64
    g = torch.Generator(device="cuda").manual_seed(7)
    x, w, r = ((torch.randn(*s, generator=g, device="cuda") * c).bfloat16() for s, c in (((b, m + 64, k), 3.0), ((n, k), k ** -0.5), ((b, m + 64, n), 1.0)))
    out = r.clone() if residual == "in place" else torch.full_like(r, 7.0)
    res = out if residual == "in place" else r if residual else None
    a = _lib.LinearBatchedArgs()
    o, esize = a.one, 2
    o.x, o.w, o.out = x.data_ptr() + 64 * k * esize, w.data_ptr(), out.data_ptr() + 64 * n * esize
    if res is not None:
        o.residual, o.residual_stride, a.residual_batch_stride = res.data_ptr() + 64 * n * esize, n, (m + 64) * n
    o.M, o.N, o.K, o.x_stride, o.w_stride, o.out_stride = m, n, k, k, k, n
    a.x_batch_stride, a.out_batch_stride, a.batches, a.lead_rows = (m + 64) * k, (m + 64) * n, b, lead
    stream = torch.cuda.current_stream().cuda_stream
    if norm:
        a.rms_eps = 1e-5
        scratch = torch.empty(b * m, device="cuda")
        _lib.call("gca_rms_linear_batched", C.byref(a), scratch.data_ptr(), stream)
    else:
        _lib.call("gca_linear_batched", C.byref(a), stream)
    xd = x[:, 64:].double()
    ref = xd @ w.double().t()
    if norm:
        ref = ref * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5)
    terms = ref.abs()
    if residual:
        ref, terms = ref + r[:, 64:].double(), terms + r[:, 64:].double().abs()
    assert ((out[:, 64:].double() - ref).abs() <= ref.abs() * (2.0 ** -8 + 2.0 ** -22) + k * 2.0 ** -24 * terms.amax(-1, keepdim=True)).all()
    untouched = r if residual == "in place" else torch.full_like(r, 7.0)
    if lead:
        assert torch.equal(out[:, :64], r[:, :64] if residual else torch.zeros_like(r[:, :64]))
    else:
        assert torch.equal(out[:, :64], untouched[:, :64])


@pytest.mark.parametrize("n,c,dim", [(1, 1, 256), (3, 5, 512), (5, 61, 768), (2, 300, 1024)])
def test_projection_append_tile_widths(n, c, dim):
    """K, V and landmark rows of an append at a position behind earlier chunks, against float32, small and large products."""
    need_gpu()
    import long_context_modeling_b200 as lcm
    g = torch.Generator(device="cuda").manual_seed(c)
    x = torch.randn(n, c, 64, dim, generator=g, device="cuda").bfloat16()
    wk, wv = ((torch.randn(dim, dim, generator=g, device="cuda") * dim ** -0.5).bfloat16() for _ in range(2))
    cache = lcm.ChunkKVManager(zero_landmark=True, capacity=c + 3)
    with torch.no_grad():
        cache.append_projected(x[:, :1], wk, wv)
        cache.append_projected(x, wk, wv)
    for got, w in ((cache.chunk_k, wk), (cache.chunk_v, wv)):
        ref = x.float() @ w.float().t()
        ref[:, :, -1] = 0
        ref = torch.cat([ref[:, :1], ref], 1)
        assert (got.float() - ref).abs().max() <= 2e-2 * ref.abs().max()
    assert torch.equal(cache.past_lmk_embeds, torch.cat([x[:, :1, -1], x[:, :, -1]], 1))


@pytest.mark.parametrize("n,c,dim", [(1, 40, 512), (3, 32, 512), (2, 12, 1024), (1, 45, 1024), (1, 17, 1280), (5, 61, 768), (1, 2, 256)])
def test_projection_append_stays_in_its_rows_and_chunks(n, c, dim):
    """Widths that the column tile does not divide: the last tile must not run on into the next row (the tile that has those
    columns writes them at the same time) or past the appended chunks.  Chunks before and behind keep their contents; launches that
    follow each other into the same cache leave the bits of the last one."""
    need_gpu()
    from long_context_modeling_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(dim + c)
    xs = [torch.randn(n, c, 64, dim, generator=g, device="cuda").bfloat16() for _ in range(2)]
    wk, wv = ((torch.randn(dim, dim, generator=g, device="cuda") * dim ** -0.5).bfloat16() for _ in range(2))
    k, v = (torch.full((n, c + 2, 64, dim), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    lmk = torch.full((n, c + 2, dim), 7.0, dtype=torch.bfloat16, device="cuda")
    refs = [[(x.float() @ w.float().t()) for w in (wk, wv)] for x in xs]
    bits = [None, None]
    for i in range(12):
        for _ in range(3):
            _lib.host().kv_project_append(xs[1 - i % 2], wk, wv, k, v, lmk, 1, c + 2, False)
        _lib.host().kv_project_append(xs[i % 2], wk, wv, k, v, lmk, 1, c + 2, False)
        for got, ref in zip((k, v), refs[i % 2]):
            assert (got[:, 1:c + 1].float() - ref).abs().max() <= 2e-2 * ref.abs().max()
            assert (got[:, 0] == 7).all() and (got[:, c + 1:] == 7).all()
        assert torch.equal(lmk[:, 1:c + 1], xs[i % 2][:, :, -1]) and (lmk[:, 0] == 7).all() and (lmk[:, c + 1:] == 7).all()
        now = [k.clone(), v.clone()]
        bits[i % 2] = bits[i % 2] or now
        assert all(torch.equal(a, b) for a, b in zip(now, bits[i % 2]))


@pytest.mark.parametrize("m,n,k,few", [(16, 16576, 64, True), (16, 16592, 64, False), (32, 9472, 64, True), (32, 9488, 64, False),
                                       (64, 3552, 128, True), (64, 3568, 128, False), (128, 2304, 768, False), (96, 3072, 1024, False)])
def test_few_row_form_on_both_sides_of_its_line(m, n, k, few):
    """Products on either side of the line between the latency-bound form and the tiles; RMSNorm + projection, whose line lies
    elsewhere, at the same sizes."""
    need_gpu()
    from long_context_modeling_b200 import _lib
    rows = _lib.lib().gca_linear_few_rows
    assert rows(m, n, k, 0) == int(few) and rows(129, n, k, 1) == 0 and rows(1, 768, 768, 1) == 1
    test_few_row_linear_and_fused_norm_against_float32(m, n, k, True)


def test_decode_step_too_wide_for_the_few_row_form():
    """64 sequences x 2 rows of a 2,048-wide sub-layer: row norms and tiled projections around the decode attention."""
    need_gpu()
    from long_context_modeling_b200 import _lib
    assert _lib.lib().gca_linear_few_rows(128, 2048, 2048, 1) == 0
    test_one_launch_decode_step(64, 32, 2, 2, 3)
