"""Landmark scoring / top-k / cache on the GPU against the canonical CPU oracle and the
golden vectors produced by the reference's own retrieval code.  Indices must match
BIT-EXACTLY (ties to the lower chunk id); weights and scores within float32 rounding.
"""
import math
import os

import numpy as np
import pytest
import torch

import cases
from oracle import retrieval_oracle as R

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lcm():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import long_context_modeling_b200 as m
    return m


def oracle_rows(lq, lk, topk, q_pos0=None, e_base=0, noise=None, head_dim=0, score_round="fp32"):
    """Per-sequence oracle over a batch: returns idx (N, Cq[, H], K), weights, scores, nvalid."""
    n, cq, d = lq.shape
    e = lk.shape[1]
    q_pos0 = (e - cq) if q_pos0 is None else q_pos0
    limit = q_pos0 + np.arange(cq)
    out = []
    for b in range(n):
        s = R.canonical_scores(lq[b].float().numpy(), lk[b].float().numpy(), head_dim=head_dim, score_round=score_round)
        if head_dim:
            per_head = [R.canonical_topk(s[:, hh, :], limit, topk, e_base=e_base) for hh in range(s.shape[1])]
            out.append(tuple(np.stack([ph[i] for ph in per_head], axis=1) for i in range(4)))
        else:
            nz = None if noise is None else noise[b].numpy()
            out.append(R.canonical_topk(s, limit, topk, noise=nz, e_base=e_base))
    return tuple(np.stack([o[i] for o in out]) for i in range(4))


def check(res, ref, exact_scores=True):
    idx, clean, w, nv = ref
    assert np.array_equal(res.indices.cpu().numpy(), idx), "indices must be bit-exact"
    assert np.array_equal(res.n_valid.cpu().numpy(), nv)
    got_s = res.scores.cpu().numpy()
    fin = np.isfinite(clean)
    if exact_scores:
        assert np.array_equal(got_s[fin].view(np.uint32), clean[fin].view(np.uint32)), "scores must be bit-exact"
    assert np.all(np.isneginf(got_s[~fin]))
    assert np.allclose(res.weights.cpu().numpy(), w, atol=2e-6)


@pytest.mark.parametrize("n,cq,e,d,k", [(2, 12, 12, 768, 8), (1, 260, 260, 768, 8), (3, 5, 37, 128, 4),
                                         (2, 1, 300, 768, 8), (1, 7, 7, 256, 32), (2, 3, 1000, 512, 16)])
def test_topk_bit_exact_vs_canonical_oracle(lcm, n, cq, e, d, k):
    lq, lk = cases.landmark_case(21, n, cq, e, d=d)
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), k)
    check(res, oracle_rows(lq, lk, k))


def test_topk_matches_reference_golden(lcm, golden_dir):
    """Indices / weights produced by the reference's ``_perform_batch_retrieval`` and its
    decode-time block, run from the reference source on CPU."""
    g = np.load(os.path.join(golden_dir, "retrieval_ref_batch.npz"))
    n, c, d, topk = 2, 12, 768, 8
    lq, lk = cases.landmark_case(3, n, c, c, d=d)
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), topk)
    idx = res.indices.cpu().numpy()
    w = res.weights.cpu().numpy()
    ref_w = g["weights"].reshape(n, c - 1, topk)
    for b in range(n):
        for i in range(c - 1):
            m = min(i, topk)
            assert np.array_equal(idx[b, i, :m], g["indices"][b, i, :m])
            assert np.allclose(w[b, i, :m], ref_w[b, i, :m], atol=1e-5)
            assert np.all(idx[b, i, m:] == -1) and np.all(w[b, i, m:] == 0)
    gd = np.load(os.path.join(golden_dir, "retrieval_ref_decode.npz"))
    hidden = torch.randn(n, 2, d, generator=torch.Generator().manual_seed(9)).bfloat16()
    res = lcm.lmk_score_topk(hidden[:, -1:].cuda(), lk.cuda(), topk)
    assert np.array_equal(res.indices.cpu().numpy()[:, 0], gd["indices"])
    assert np.allclose(res.weights.cpu().numpy(), gd["weights"], atol=1e-5)


def test_ties_masked_rows_and_all_masked(lcm):
    g = torch.Generator().manual_seed(2)
    lk = torch.randn(1, 50, 768, generator=g).bfloat16()
    lk[0, 31] = lk[0, 4]
    lk[0, 17] = lk[0, 4]                      # three identical landmarks: exact ties
    lq = (lk[:, 4:5] * 3).bfloat16()
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), 8, q_pos0=50)
    assert res.indices[0, 0, :3].tolist() == [4, 17, 31]
    check(res, oracle_rows(lq, lk, 8, q_pos0=50))
    # fewer visible chunks than K, and a row that sees nothing
    lq3 = torch.randn(1, 3, 768, generator=g).bfloat16()
    res = lcm.lmk_score_topk(lq3.cuda(), lk.cuda(), 8, q_pos0=0)    # rows see 0, 1, 2 chunks
    assert res.n_valid[0].tolist() == [0, 1, 2]
    assert torch.all(res.weights[0, 0] == 0) and torch.all(res.indices[0, 0] == -1)
    check(res, oracle_rows(lq3, lk, 8, q_pos0=0))


@pytest.mark.parametrize("splits", [1, 2, 7, 40])
def test_result_independent_of_split_count(lcm, splits):
    lq, lk = cases.landmark_case(22, 2, 2, 5000, d=768)
    base = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), 8, splits=1)
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), 8, splits=splits)
    assert torch.equal(res.keys, base.keys) and torch.equal(res.indices, base.indices)
    check(res, oracle_rows(lq, lk, 8))


def test_per_head_mode(lcm):
    lq, lk = cases.landmark_case(23, 2, 1, 3000, d=768, std=0.125)
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), 8, head_dim=64)
    assert res.indices.shape == (2, 1, 12, 8)
    check(res, oracle_rows(lq, lk, 8, head_dim=64))


@pytest.mark.parametrize("splits", [1, 3, 20, 40, 160, 161])
@pytest.mark.parametrize("d,head_dim", [(768, 0), (768, 64), (72, 0), (520, 0), (1024, 64), (1000, 0)])
def test_equal_scores_in_every_batch_and_list(lcm, d, head_dim, splits):
    """Five distinct landmarks over and over: every maximum of a batch, and of the lists that are merged, is held by many at once (a plain cache
    in front, so that lists are full of distinct scores before).  Also widths whose last piece not every lane has, and 0 landmarks in a block."""
    g = torch.Generator().manual_seed(d + splits)
    e, k = 161 * 9 + 4, 8 if splits != 20 else 21
    lq, lk = cases.landmark_case(d, 1, 1, e, d=d)
    lk[:, 700:] = lk[:, :5][:, torch.randint(0, 5, (e - 700,), generator=g)]
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), k, q_pos0=e - 2, head_dim=head_dim, splits=splits)
    check(res, oracle_rows(lq, lk, k, q_pos0=e - 2, head_dim=head_dim))


@pytest.mark.parametrize("head_dim", [0, 64])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 16, 31, 32])
def test_batches_that_change_a_list_by_any_number_of_entries(lcm, k, head_dim):
    """From batch to batch 0 to 128 scores beat all that the list holds, K - 1, K and K + 1 among them: inserted one by one or taken by maxima.  Scores are
    the sums of two products, so no two of them are equal; the last batch is a short one."""
    d, counts = 512, [5, 0, 1, 2, 3, k - 1, k, k + 1, 128, 1, 20]
    g = torch.Generator().manual_seed(k)
    lk = torch.zeros(1, 128 * len(counts), d)
    fine = torch.randperm(lk.shape[1], generator=g)
    for b, m in enumerate(counts):
        at = 128 * b + torch.randperm(128, generator=g)
        lk[0, at, 0] = torch.where(torch.arange(128) < m, 1.0 + b, -1.0 - b)
    lk[0, :, 1] = (fine % 128) / 128.0
    lk[0, :, 2] = (fine // 128) / 4096.0
    lk = lk[:, :-90].repeat_interleave(d // 64 if head_dim else 1, 0)
    lk = (torch.stack([torch.roll(lk[h], 64 * h, 1) for h in range(lk.shape[0])]).sum(0, keepdim=True) if head_dim else lk).bfloat16()
    lq = torch.ones(1, 1, d).bfloat16()
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), k, q_pos0=lk.shape[1], head_dim=head_dim, splits=1)
    check(res, oracle_rows(lq, lk, k, q_pos0=lk.shape[1], head_dim=head_dim))


@pytest.mark.parametrize("splits", [33, 64, 65, 148, 160, 161])
@pytest.mark.parametrize("k", [1, 10, 13, 27, 32])
def test_merge_of_many_lists(lcm, splits, k):
    """33 to 160 lists a row are merged by a warp, in one to four trips of its block; more are ranked by counting.  Full lists and lists that end before K,
    scores that all differ and scores that are each held by landmarks of many lists, one row and a row per head."""
    g = torch.Generator().manual_seed(splits + k)
    for rows, distinct, head_dim in [(40, 0, 0), (40, 6, 0), (9, 0, 64), (9, 40, 64), (2, 3, 0)]:
        e = rows * splits - 1
        lq, lk = cases.landmark_case(splits, 1, 1, e, d=256)
        if distinct:
            lk = lk[:, :distinct][:, torch.randint(0, distinct, (e,), generator=g)]
        res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), k, q_pos0=e, head_dim=head_dim, splits=splits)
        check(res, oracle_rows(lq, lk, k, q_pos0=e, head_dim=head_dim))


@pytest.mark.parametrize("d,head_dim", [(768, 0), (776, 0), (1024, 64)])
@pytest.mark.parametrize("n,e", [(1, 9473), (1, 19000), (4, 2369), (4, 4737), (9, 1025), (32, 257)])
def test_ranges_in_steps_of_the_rows_taken_at_once(lcm, n, e, d, head_dim):
    """Ranges as the library cuts them, just past one, two and four steps of a block (of 64 rows, of 32 beyond a width of 768), with as many lists as a warp
    merges and one more: the result does not depend on the cut."""
    lq, lk = cases.landmark_case(e, n, 1, e, d=d)
    lq, lk = lq.cuda(), lk.cuda()
    got = lcm.lmk_score_topk(lq, lk, 16, q_pos0=e, head_dim=head_dim)
    one = lcm.lmk_score_topk(lq, lk, 16, q_pos0=e, head_dim=head_dim, splits=1)
    assert torch.equal(got.indices, one.indices) and torch.equal(got.scores, one.scores) and torch.equal(got.weights, one.weights)
    check(lcm.Retrieval(*(t[:1] for t in got)), oracle_rows(lq[:1].cpu(), lk[:1].cpu(), 16, q_pos0=e, head_dim=head_dim))


@pytest.mark.parametrize("splits", [1, 7, 40, 160])
@pytest.mark.parametrize("head_dim", [0, 64])
@pytest.mark.parametrize("k", [1, 8, 17, 32])
def test_scores_rounded_to_16_bits_are_often_equal(lcm, k, head_dim, splits):
    """Equal scores within a batch, between a batch and the list, and between the lists that are merged: the lowest id each time."""
    e = 160 * 13 + 5
    lq, lk = cases.landmark_case(k, 1, 1, e, d=256)
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), k, q_pos0=e, head_dim=head_dim, splits=splits, score_round="bf16")
    check(res, oracle_rows(lq, lk, k, q_pos0=e, head_dim=head_dim, score_round="bf16"))


def test_noise_selects_but_weights_stay_noise_free(lcm):
    """Training: Gumbel noise perturbs the selection only (DRT.py:616-626)."""
    n, c, d, k = 2, 20, 768, 4
    lq, lk = cases.landmark_case(24, n, c, c, d=d)
    noise = -torch.empty(n, c, c).exponential_(generator=torch.Generator().manual_seed(3)).log()
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), k, noise=noise.cuda())
    check(res, oracle_rows(lq, lk, k, noise=noise))
    plain = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), k)
    assert not torch.equal(plain.indices, res.indices)


def test_bf16_score_rounding_mode(lcm):
    lq, lk = cases.landmark_case(25, 1, 2, 4000, d=768)
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), 8, score_round="bf16")
    check(res, oracle_rows(lq, lk, 8, score_round="bf16"))


def test_set_equality_with_torch_topk(lcm):
    lq, lk = cases.landmark_case(26, 2, 6, 500, d=768)
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), 8)
    ti, tw = R.torch_reference_retrieval(lq.float(), lk.float(), 8)
    for b in range(2):
        for i in range(6):
            assert set(res.indices[b, i].tolist()) == set(ti[b, i].tolist())
    assert np.allclose(np.sort(res.weights.cpu().numpy(), -1), np.sort(tw.numpy(), -1), atol=1e-5)


def test_merge_of_shards_equals_single_scan(lcm):
    """Chunk-range sharding: local top-k per shard (global ids) + merge == one scan."""
    lq, lk = cases.landmark_case(27, 1, 1, 8192, d=768)
    full = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), 8)
    for shards in (2, 4, 8):
        per = 8192 // shards
        parts = [lcm.lmk_score_topk(lq.cuda(), lk[:, r * per:(r + 1) * per].contiguous().cuda(), 8,
                                    q_pos0=8191, e_base=r * per).keys for r in range(shards)]
        merged = lcm.merge_topk(torch.cat(parts, dim=-1), 8)
        assert torch.equal(merged.keys, full.keys)
        assert torch.equal(merged.indices, full.indices)
        assert torch.allclose(merged.weights, full.weights, atol=1e-6)
        ref = R.merge_candidates(torch.cat(parts, -1).cpu().numpy().view(np.uint64).reshape(1, -1), 8)
        assert np.array_equal(merged.keys.cpu().numpy().view(np.uint64).reshape(1, -1), ref)


def test_full_size_16m_token_landmark_scan(lcm):
    """BASELINE retrieval config: 262,144 landmarks x 768 (bf16), one query, top-8 per head
    and per sequence.  Checked against the oracle on the winners' neighbourhood: every
    selected score must be the canonical score of that chunk, sorted, and no unselected
    chunk of a random sample may beat the 8th."""
    e, d = 262144, 768
    g = torch.Generator().manual_seed(0)
    lk = (torch.randn(e, d, generator=g) * 0.125).bfloat16()
    lq = (torch.randn(1, d, generator=g) * 0.125).bfloat16()
    for head_dim in (0, 64):
        res = lcm.lmk_score_topk(lq[None].cuda(), lk[None].cuda(), 8, head_dim=head_dim)
        idx = res.indices.cpu().numpy().reshape(-1, 8)
        sc = res.scores.cpu().numpy().reshape(-1, 8)
        sample = np.unique(np.concatenate([idx.reshape(-1), np.random.default_rng(0).integers(0, e - 1, 4096)]))
        s = R.canonical_scores(lq.float().numpy(), lk[sample].float().numpy(), head_dim=head_dim).reshape(-1, len(sample))
        pos = {int(v): i for i, v in enumerate(sample)}
        for r in range(idx.shape[0]):
            assert np.all(idx[r] < e - 1)                      # the newest chunk is never visible
            mine = np.array([s[r, pos[int(i)]] for i in idx[r]], dtype=np.float32)
            assert np.array_equal(mine.view(np.uint32), sc[r].view(np.uint32))
            assert np.all(np.diff(sc[r]) <= 0)
            others = np.delete(s[r], [pos[int(i)] for i in idx[r]])
            assert others.max() <= sc[r, -1]
    # whole-scan equality against float64 argsort on a tie-free instance
    full = (lk.double() @ lq[0].double()).numpy() / math.sqrt(d)
    full[-1] = -np.inf
    top = np.argsort(-full, kind="stable")[:8]
    res = lcm.lmk_score_topk(lq[None].cuda(), lk[None].cuda(), 8)
    assert set(res.indices.cpu().numpy().reshape(-1).tolist()) == set(top.tolist())


def test_chunk_cache_manager_and_drop_in_retrieval(lcm, golden_dir):
    """ChunkKVManager mirror + perform_batch_retrieval against the reference's own outputs."""
    g = np.load(os.path.join(golden_dir, "retrieval_ref_batch.npz"))
    n, c, dmodel, heads, topk = 2, 12, 768, 12, 8
    lq, lk = cases.landmark_case(3, n, c, c, d=dmodel)
    gen = torch.Generator().manual_seed(4)
    chunk_k = torch.randn(n, c, 64, dmodel, generator=gen)
    chunk_v = torch.randn(n, c, 64, dmodel, generator=gen)
    mgr = lcm.ChunkKVManager(False, 1)
    mgr.append(chunk_k[:, :5].cuda(), chunk_v[:, :5].cuda(), lk[:, :5].float().cuda())
    mgr.append(chunk_k[:, 5:].cuda(), chunk_v[:, 5:].cuda(), lk[:, 5:].float().cuda())   # growth
    assert len(mgr) == c and torch.equal(mgr.chunk_k.cpu(), chunk_k) and torch.equal(mgr.chunk_v.cpu(), chunk_v)
    assert torch.equal(mgr.past_lmk_embeds.cpu(), lk.float())
    ck, cv, cw, indices = lcm.perform_batch_retrieval(lq.float().cuda(), mgr, 0, num_heads=heads, chunk_topk=topk,
                                                      use_cache=True)
    assert tuple(ck.shape) == tuple(g["chunk_k_shape"]) and indices.dtype == torch.int64
    ref_w = g["weights"]
    assert np.allclose(cw.cpu().numpy(), ref_w, atol=1e-5)
    # gathered tensors: compare per-(row, head, slot) sums where the weight is non-zero
    live = (ref_w > 0)[:, None, :]
    ks = ck.double().sum(dim=(-1, -2)).cpu().numpy()
    vs = cv.double().sum(dim=(-1, -2)).cpu().numpy()
    assert np.allclose(np.where(live, ks, 0), np.where(live, g["chunk_k_sum"], 0), atol=1e-6)
    assert np.allclose(np.where(live, vs, 0), np.where(live, g["chunk_v_sum"], 0), atol=1e-6)
    cur_k, cur_v, cur_w = mgr.current_retrieved_chunk(0)
    assert np.allclose(cur_w.cpu().numpy(), g["cur_w"], atol=1e-5)
    assert np.allclose(cur_k.double().sum(dim=(-1, -2)).cpu().numpy(), g["cur_k_sum"], atol=1e-6)
    # zero-landmark append variant (DRT.py:771-781 folded into the append kernel)
    mgr2 = lcm.ChunkKVManager(zero_landmark=True, capacity=64)
    mgr2.append(chunk_k.cuda().bfloat16(), chunk_v.cuda().bfloat16(), lk.cuda())
    assert mgr2.chunk_k[:, :, -1].abs().max().item() == 0 and mgr2.chunk_v[:, :, -1].abs().max().item() == 0
    assert torch.equal(mgr2.chunk_k[:, :, :-1].cpu(), chunk_k.bfloat16()[:, :, :-1])


def test_differentiable_weights_match_reference_autograd(lcm):
    """Gradients of the retrieval weights w.r.t. the landmarks equal autograd through the
    reference sequence softmax(scores.gather(topk)) (DRT.py:612-626)."""
    n, c, d, k = 2, 9, 768, 4
    lq, lk = cases.landmark_case(28, n, c, c, d=d)
    lqg = lq.float().cuda().requires_grad_()
    lkg = lk.float().cuda().requires_grad_()
    res = lcm.lmk_score_topk(lqg, lkg, k)
    w = lcm.differentiable_weights(lqg, lkg, res.indices)
    probe = torch.randn(w.shape, generator=torch.Generator().manual_seed(1)).cuda()
    (w * probe).sum().backward()
    a = lq.float().requires_grad_()
    b = lk.float().requires_grad_()
    ti, tw = R.torch_reference_retrieval(a, b, k)
    # align slots: the reference orders by score too; padding differs only where weight is 0
    (tw * probe.cpu()).sum().backward()
    assert torch.allclose(w.detach().cpu(), tw.detach(), atol=1e-5)
    assert torch.allclose(lqg.grad.cpu(), a.grad, atol=1e-4)
    assert torch.allclose(lkg.grad.cpu(), b.grad, atol=1e-4)


def test_projection_with_append_epilogue_matches_reference_statements(lcm, golden_dir):
    """``ChunkKVManager.append_projected`` (one tensor-core GEMM whose epilogue writes K and V into the
    cache, landmark rows cleared, landmark embeddings extracted) against the reference's own statements
    ``model/DRT.py:766-784`` run on the reference's own manager, for an append that follows an earlier
    one (non-zero position, cache growth)."""
    import make_golden as MG
    g = np.load(os.path.join(golden_dir, "projection_ref.npz"))
    enc_prev, enc_new, wk, wv = MG.projection_case(61)
    assert abs(cases.checksum(enc_prev, enc_new, wk, wv) - float(g["in_checksum"])) < 1e-6
    mgr = lcm.ChunkKVManager(zero_landmark=True, capacity=2)          # capacity 2 < 3 chunks: the buffer also grows
    wk_d, wv_d = wk.cuda().bfloat16(), wv.cuda().bfloat16()
    with torch.no_grad():
        for enc in (enc_prev, enc_new):
            mgr.append_projected(enc.cuda().bfloat16(), wk_d, wv_d)
    torch.cuda.synchronize()
    assert lcm.read_status() == 0 and len(mgr) == 3 and not mgr.tracks_gradients
    for name, got in (("chunk_k", mgr.chunk_k), ("chunk_v", mgr.chunk_v), ("lmk", mgr.past_lmk_embeds)):
        ref = torch.from_numpy(g[name].astype(np.float32))
        assert got.shape == ref.shape, name
        err = (got.float().cpu() - ref).abs().max().item() / (ref.abs().max().item() + 1e-12)
        assert err <= 1e-2, (name, err)
    assert mgr.chunk_k[:, :, -1].abs().max().item() == 0 and mgr.chunk_v[:, :, -1].abs().max().item() == 0
    # more row tiles than CTAs, and a row count that is not a multiple of the 128-row tile
    gen = torch.Generator().manual_seed(62)
    enc = torch.randn(3, 101, 64, 256, generator=gen).bfloat16()
    big = lcm.ChunkKVManager(zero_landmark=False)
    with torch.no_grad():
        big.append_projected(enc.cuda(), wk_d, wv_d)
    want_k = (enc.float() @ wk.t())
    err = (big.chunk_k.float().cpu() - want_k).abs().max().item() / want_k.abs().max().item()
    assert err <= 1e-2, err
    assert lcm.read_status() == 0


def test_virtual_memory_cache_grows_in_place():
    """``ChunkKVManager(max_chunks=...)``: K and V sit in a virtual-address reservation, memory is mapped
    behind it as the cache fills.  Same contents as the doubling buffer after every append (plain and
    projected), addresses never change, the kernels read it like any cache, the reservation's limit is
    enforced, and the memory comes back on close()."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import long_context_modeling_b200 as lcm
    dev = torch.device("cuda", 0)
    g = torch.Generator().manual_seed(21)
    n, l, hd = 3, 64, 256                                    # 32 KB per chunk: a 2 MB page holds 64 of them
    virt = lcm.ChunkKVManager(zero_landmark=True, max_chunks=200, capacity=16)
    plain = lcm.ChunkKVManager(zero_landmark=True)
    free0 = torch.cuda.mem_get_info(dev)[0]
    ptr = None
    wk = (torch.randn(hd, hd, generator=g) / 16).bfloat16().to(dev)
    wv = (torch.randn(hd, hd, generator=g) / 16).bfloat16().to(dev)
    for step in range(7):
        count = 23 + step
        if step % 2 == 0:
            k = torch.randn(n, count, l, hd, generator=g).bfloat16().to(dev)
            v = torch.randn(n, count, l, hd, generator=g).bfloat16().to(dev)
            lm = torch.randn(n, count, hd, generator=g).bfloat16().to(dev)
            virt.append(k, v, lm)
            plain.append(k, v, lm)
        else:
            x = torch.randn(n, count, l, hd, generator=g).bfloat16().to(dev)
            virt.append_projected(x, wk, wv)
            plain.append_projected(x, wk, wv)
        assert len(virt) == len(plain)
        assert torch.equal(virt.chunk_k, plain.chunk_k) and torch.equal(virt.chunk_v, plain.chunk_v)
        assert torch.equal(virt.past_lmk_embeds, plain.past_lmk_embeds)
        if ptr is None:
            ptr = virt.chunk_k.data_ptr()
        assert virt.chunk_k.data_ptr() == ptr                # grown in place
    c = len(virt)
    assert c == sum(23 + s for s in range(7)) and c <= 200
    # the kernels read the virtual cache like any other: retrieval + indexed GCA
    q = torch.randn(n, 1, 4, 1, 64, generator=g).bfloat16().to(dev)
    lq = torch.randn(n, 1, hd, generator=g).bfloat16().to(dev)
    r = lcm.lmk_score_topk(lq, virt.past_lmk_embeds, 8)
    rp = lcm.lmk_score_topk(lq, plain.past_lmk_embeds, 8)
    assert torch.equal(r.indices, rp.indices)
    o = lcm.gca_indexed_nograd(q, virt.chunk_k, virt.chunk_v, r.indices, r.weights, 0.125)
    op = lcm.gca_indexed_nograd(q, plain.chunk_k, plain.chunk_v, rp.indices, rp.weights, 0.125)
    assert torch.equal(o, op)
    with pytest.raises(ValueError):                           # beyond the reservation
        virt.append(torch.zeros(n, 60, l, hd, dtype=torch.bfloat16, device=dev), torch.zeros(n, 60, l, hd, dtype=torch.bfloat16, device=dev),
                    torch.zeros(n, 60, hd, dtype=torch.bfloat16, device=dev))
    torch.cuda.synchronize()
    used = free0 - torch.cuda.mem_get_info(dev)[0]
    del o, r
    virt.close()
    assert len(virt) == 0
    assert torch.cuda.mem_get_info(dev)[0] > free0 - used + 2 * n * (1 << 21)        # the mapped pages were released


@pytest.mark.parametrize("n,cq,e,d,k,noisy", [(1, 64, 64, 768, 3, False), (2, 65, 129, 64, 28, True), (3, 64, 640, 256, 1, False),
                                              (1, 70, 2200, 768, 8, True), (2, 130, 130, 1024, 16, True), (9, 200, 191, 128, 5, False)])
def test_tensor_core_screening_bit_exact_vs_canonical_oracle(lcm, n, cq, e, d, k, noisy):
    """Many query rows: approximate scores choose the candidates, exact ones decide.  Ragged tiles in both axes,
    several tiles per candidate list, rows that see fewer chunks than K."""
    lq, lk = cases.landmark_case(31, n, cq, e, d=d)
    q_pos0 = max(0, e - cq)
    noise = -torch.empty(n, cq, e).exponential_(generator=torch.Generator().manual_seed(5)).log() if noisy else None
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), k, q_pos0=q_pos0, noise=None if noise is None else noise.cuda())
    check(res, oracle_rows(lq, lk, k, q_pos0=q_pos0, noise=noise))


@pytest.mark.parametrize("e,k,noisy", [(2101, 28, True), (4200, 12, False), (2240, 13, True)])
def test_tensor_core_screening_merges_tiles(lcm, e, k, noisy):
    """Several tiles per candidate list, lists of up to 16 and of up to 32 entries, noise rows aligned to 16 bytes and not."""
    test_tensor_core_screening_bit_exact_vs_canonical_oracle(lcm, 1, 66, e, 64, k, noisy)


@pytest.mark.parametrize("copies", [2, 40, 200])
def test_tensor_core_screening_with_copies_of_landmarks(lcm, copies):
    """Ties that the candidate lists cannot hold (copies of one landmark) and near ties: the exact scan takes over, ties go to
    the lower id."""
    lq, lk = cases.landmark_case(34, 2, 80, 300, d=192)
    lk[0, 3:3 + copies] = lq[0, 7]
    lk[1, ::2] = lk[1, 0]
    lk[1, 1::4, 5] += 0.015625
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), 8, q_pos0=260)
    check(res, oracle_rows(lq, lk, 8, q_pos0=260))


@pytest.mark.parametrize("n,cq,e,d,k,per_head,noisy", [
    (1, 1, 3, 768, 8, False, False), (1, 1, 64, 768, 1, True, False),       # one block, fewer landmarks than places
    (2, 3, 65, 512, 32, False, True), (3, 2, 449, 256, 7, True, False),     # two and eight blocks, a last one of a single landmark, hidden landmarks
    (5, 1, 512, 1024, 16, True, False), (12, 1, 500, 768, 8, False, True),  # clusters of eight
    (32, 1, 200, 768, 8, False, False), (40, 1, 512, 768, 8, False, False),     # clusters of four; too many rows for clusters
])
def test_scan_that_merges_for_itself(lcm, n, cq, e, d, k, per_head, noisy):
    lq, lk = cases.landmark_case(36, n, cq, e, d=d)
    head_dim = 64 if per_head else 0
    noise = -torch.empty(n, cq, e).exponential_(generator=torch.Generator().manual_seed(4)).log() if noisy else None
    lk[:, e // 2] = lk[:, 0]                                   # a tie between blocks
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), k, q_pos0=e - 1, noise=None if noise is None else noise.cuda(), head_dim=head_dim)
    check(res, oracle_rows(lq, lk, k, q_pos0=e - 1, noise=noise, head_dim=head_dim))
    apart = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), k, q_pos0=e - 1, noise=None if noise is None else noise.cuda(), head_dim=head_dim, splits=9)
    assert all(torch.equal(a, b) for a, b in zip(res, apart))


@pytest.mark.parametrize("e,k,splits", [(9000, 32, 33), (70001, 1, 0), (5000, 7, 1024), (3000, 8, 1500)])
def test_many_candidate_lists_per_row(lcm, e, k, splits):
    lq, lk = cases.landmark_case(32, 1, 1, e, d=128)
    res = lcm.lmk_score_topk(lq.cuda(), lk.cuda(), k, splits=splits)
    check(res, oracle_rows(lq, lk, k))


@pytest.mark.parametrize("n,c,d,k", [(1, 3, 64, 2), (2, 37, 768, 8), (1, 150, 1024, 32), (3, 65, 264, 5)])
def test_retrieval_weight_gradients_against_float32(lcm, n, c, d, k):
    """``retrieve`` on bf16 landmarks that require grad: weights and both gradients against float32 autograd over the
    same selection; both outputs (whole, without the last row) carry gradient."""
    lq, lk = cases.landmark_case(33, n, c, c, d=d, std=0.5)
    q, m = lq.cuda().requires_grad_(), lk.cuda().requires_grad_()
    chunks = type("Chunks", (), {"past_lmk_embeds": m})
    idx, w, full = lcm.retrieve(q, chunks, min(k, c))
    g = torch.Generator().manual_seed(2)
    probe, probe_all = (torch.randn(x.shape, generator=g).cuda() for x in (w, full.weights))
    dq, dm = torch.autograd.grad([w, full.weights], [q, m], [probe, probe_all])
    qf, mf = lq.cuda().float().requires_grad_(), lk.cuda().float().requires_grad_()
    ref = lcm.differentiable_weights(qf, mf, full.indices)
    rq, rm = torch.autograd.grad([ref[:, :-1], ref], [qf, mf], [probe, probe_all])
    assert torch.equal(idx, full.indices[:, :-1]) and torch.allclose(w, ref[:, :-1], atol=1e-5)
    for got, want in ((dq, rq), (dm, rm)):
        assert (got.float() - want).norm() <= 4e-3 * want.norm() + 1e-6


def _retrieve_with_float32_twin(lcm, n, c, d, k, seed):
    """(q, landmarks, ids, weights, whole result) of a bf16 retrieval that records gradients, and the same weights as float32
    torch operations over the same selection: (q, landmarks, weights, whole weights)."""
    lq, lk = cases.landmark_case(seed, n, c, c, d=d, std=0.5)
    q, m = lq.cuda().requires_grad_(), lk.cuda().requires_grad_()
    idx, w, full = lcm.retrieve(q, type("Chunks", (), {"past_lmk_embeds": m}), k)
    qf, mf = lq.cuda().float().requires_grad_(), lk.cuda().float().requires_grad_()
    ref = lcm.differentiable_weights(qf, mf, full.indices)
    return (q, m, idx, w, full), (qf, mf, ref[:, :-1], ref)


def test_in_place_changes_to_a_retrieval_and_its_gradients(lcm):
    """The returned selection belongs to the caller: changed ids and scores do not reach the backward pass, a change to the weights
    is recorded like that of any view (both results see it)."""
    (q, m, idx, w, full), (qf, mf, wf, ref) = _retrieve_with_float32_twin(lcm, 2, 37, 768, 8, 35)
    factor = torch.rand(w.shape, generator=torch.Generator().manual_seed(7)).cuda()
    idx.fill_(0)
    full.indices[:, -1] = 0
    full.scores.zero_()
    w.mul_(factor)
    wf.mul_(factor)
    full.weights.add_(w.sum())
    ref.add_(wf.sum())
    assert torch.allclose(full.weights, ref, atol=1e-4) and torch.equal(full.weights[:, :-1], w)
    g = torch.Generator().manual_seed(8)
    probe, probe_all = (torch.randn(x.shape, generator=g).cuda() for x in (w, full.weights))
    got = torch.autograd.grad([w, full.weights], [q, m], [probe, probe_all])
    want = torch.autograd.grad([wf, ref], [qf, mf], [probe, probe_all])
    for a, b in zip(got, want):                              # each gradient is a float32 sum rounded to bf16 once (2^-9)
        assert (a.float() - b).norm() <= 4e-3 * b.norm()


def test_gradients_of_retrieval_weights_can_be_differentiated_and_batched(lcm):
    """A gradient penalty (backward of the backward) and batched gradients (vmap), against float32 torch operations over the same
    selection; two outputs, rows with fewer chunks than slots."""
    (q, m, _, w, full), (qf, mf, wf, ref) = _retrieve_with_float32_twin(lcm, 2, 9, 64, 4, 36)
    g = torch.Generator().manual_seed(9)
    probe, probe_all = (torch.randn(x.shape, generator=g).cuda() for x in (w, full.weights))

    def penalty(outs, ins, probes):
        first = torch.autograd.grad(outs, ins, probes, create_graph=True)
        return first, torch.autograd.grad(sum(x.float().pow(2).sum() for x in first), (*ins, *probes))

    got = penalty([w, full.weights], [q, m], [probe.requires_grad_(), probe_all.requires_grad_()])
    want = penalty([wf, ref], [qf, mf], [probe, probe_all])
    # the first row sees no chunk: zeros here, where a softmax over nothing differentiated twice is NaN
    for a, b in zip(got[0] + got[1], want[0] + want[1]):       # bf16 results of float32 sums, the second ones of rounded first ones
        assert (a.float() - b.nan_to_num(0.0)).norm() <= 1e-2 * b.nan_to_num(0.0).norm() and torch.isfinite(a).all()
    once = torch.autograd.grad(w, [q, m], probe, retain_graph=True)
    several = torch.stack([probe, -2 * probe]).detach()
    for x, y in zip(torch.autograd.grad(w, [q, m], several, is_grads_batched=True), once):
        assert (x[0].float() - y.float()).norm() <= 8e-3 * y.float().norm()
        assert (x[1].float() + 2 * y.float()).norm() <= 16e-3 * y.float().norm()


def test_forward_mode_differentiation_is_followed_or_refused(lcm):
    """Tangents of the landmarks reach the retrieval weights (against the backward pass: <dw, J t> = <J^T dw, t>); GCA, which has
    no forward-mode derivative, refuses them instead of dropping them."""
    import torch.autograd.forward_ad as fwd
    (q, m, _, w, _), (qf, mf, wf, _) = _retrieve_with_float32_twin(lcm, 2, 9, 64, 4, 37)
    g = torch.Generator().manual_seed(10)
    tq, tm, probe = (torch.randn(x.shape, generator=g).cuda() for x in (q, m, w))
    dq, dm = torch.autograd.grad(wf, [qf, mf], probe)
    with fwd.dual_level():
        dual_q, dual_m = fwd.make_dual(q, tq.bfloat16()), fwd.make_dual(m, tm.bfloat16())
        _, dual_w, _ = lcm.retrieve(dual_q, type("Chunks", (), {"past_lmk_embeds": dual_m}), 4)
        tangent = fwd.unpack_dual(dual_w).tangent.clone()
        tangent[:, 0] = 0                                    # the first row sees no chunk: torch's tangent of a softmax over nothing is NaN
        got, want = (tangent * probe).sum(), (dq * tq.bfloat16()).sum() + (dm * tm.bfloat16()).sum()
        # bf16 scores on the way: 2^-9 of each of the tangent's contributions
        size = ((dq * tq.bfloat16()).abs().sum() + (dm * tm.bfloat16()).abs().sum())
        assert (got - want).abs() <= 2 ** -7 * size
        x = torch.randn(2, 3, 4, 64, 64, generator=g).bfloat16().cuda()
        kv = torch.randn(2, 5, 64, 256, generator=g).bfloat16().cuda()
        ids, wt = torch.zeros(2, 3, 2, dtype=torch.int32, device="cuda"), torch.ones(2, 3, 2, device="cuda")
        for args in ((fwd.make_dual(x, x), kv, kv, ids, wt), (x, kv, fwd.make_dual(kv, kv), ids, wt), (x, kv, kv, ids, fwd.make_dual(wt, wt))):
            with pytest.raises(NotImplementedError):
                lcm.gca_indexed(*args, 0.125)
        cr = kv.view(2, 5, 64, 4, 64).permute(0, 3, 1, 2, 4)
        with pytest.raises(NotImplementedError):
            lcm.attention(x[:, 0], fwd.make_dual(cr, cr), cr, torch.ones(2, 5, device="cuda"), 0.125)


@pytest.mark.parametrize("n,cq,e,d,k,noisy", [(1, 64, 700, 768, 8, False), (2, 65, 300, 1024, 28, False), (3, 200, 331, 64, 1, True),
                                              (9, 70, 64, 448, 5, False)])
def test_rows_that_the_block_scans(lcm, n, cq, e, d, k, noisy):
    """Rows whose candidate lists may hide a winner: all scores equal (a zero row), half of the landmarks one landmark; one row per
    block and several, rows that see fewer landmarks than a block has warps.  Bits of the row scan (``splits`` takes it)."""
    lq, lk = cases.landmark_case(38, n, cq, e, d=d)
    lq[:, ::3] = 0
    lk[:, 1::2] = lk[:, 1:2]
    noise = None
    if noisy:                                                # ties in the noisy scores too
        noise = torch.randint(0, 2, (n, cq, e), generator=torch.Generator().manual_seed(3)).float().cuda()
    for q_pos0 in (0, max(0, e - cq)):
        res, want = (lcm.lmk_score_topk(lq.cuda(), lk.cuda(), k, q_pos0=q_pos0, noise=noise, splits=s) for s in (0, 1))
        for a, b in zip(res, want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("where", ["landmark", "query", "noise"])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
def test_screening_with_values_that_are_not_finite(lcm, where, value):
    """NaN and infinities in a landmark (seen by some rows, and in the same tile as landmarks that others see), in a query row, in
    the noise: keys, ids and scores of the row scan (``splits`` takes it)."""
    lq, lk = cases.landmark_case(39, 2, 80, 300, d=128)
    noise = torch.zeros(2, 80, 300)
    lk[:, 200:240] *= 2.0 ** 12                              # the largest norms share the tile with the value
    lk[:, 205:240] = lk[:, 200:201]                          # and tie
    if where == "landmark":
        lk[0, 250, 5] = value
    elif where == "query":
        lq[1, 3, 7] = value
    else:
        noise[0, 5, 100] = noise[1, 60, 3] = value
    args = dict(q_pos0=205, noise=noise.cuda() if where == "noise" else None)
    res, want = (lcm.lmk_score_topk(lq.cuda(), lk.cuda(), 8, splits=s, **args) for s in (0, 1))
    assert torch.equal(res.keys, want.keys) and torch.equal(res.indices, want.indices) and torch.equal(res.n_valid, want.n_valid)
    for a, b in ((res.scores, want.scores), (res.weights, want.weights)):
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(7.0), b.nan_to_num(7.0))
