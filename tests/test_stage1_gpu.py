"""GPU: stage-1 scorer against the fp32 oracle and the golden vectors.
Tolerance: |got - ref| <= 2e-2, or within 2^-7 relative where a score is large (the output is
bf16 and a row's 16 units of probability can sit on a handful of keys: one bf16 step at 8..16
is 2^-4, already above 2e-2)."""
import os

import numpy as np
import pytest
import torch

import oracle
import infllm_v2
from helpers import det_tensor, cu
from inputs import det_array

pytestmark = pytest.mark.gpu
DEV = "cuda"
MAX_ABS, REL = 2e-2, 2.0 ** -7


def _within(got, ref):
    got, ref = torch.as_tensor(got).float(), torch.as_tensor(ref).float()
    diff = (got - ref).abs()
    ok = (diff <= MAX_ABS) | (diff <= REL * ref.abs())
    return bool(ok.all()), diff.max().item()


def _run(q, kc, cu_q, cu_k, max_q, max_k, causal):
    s = infllm_v2.infllmv2_attn_stage1(q.to(DEV), kc.to(DEV), kc.to(DEV), cu_q.to(DEV), cu_k.to(DEV),
                                       cu_k.to(DEV), max_q, max_k, causal=causal)
    infllm_v2.check_device_status()
    assert s.dtype == torch.bfloat16 and s.shape == (kc.shape[1], q.shape[0], max_k)
    return s.float().cpu()


def test_stage1_golden(golden_dir):
    g = np.load(os.path.join(golden_dir, "stage1.npz"))
    for key in [k for k in g.files if k.endswith("_shape")]:
        base = key[:-6]
        lq, lc, seed = (int(x) for x in g[key][:3])
        if len(g[key]) == 4:                 # "compressed LSE" case: row sums over coarser keys
            lcv = int(g[key][3])
            q = torch.from_numpy(det_array((lq, 32, 128), seed, 0.5)).to(torch.bfloat16)
            k = torch.from_numpy(det_array((lc, 2, 128), seed + 1000)).to(torch.bfloat16)
            kv = torch.from_numpy(det_array((lcv, 2, 128), seed + 2000)).to(torch.bfloat16)
            got = infllm_v2.infllmv2_attn_stage1(q.to(DEV), k.to(DEV), kv.to(DEV), cu([lq], DEV),
                                                 cu([lc], DEV), cu([lcv], DEV), lq, lc,
                                                 causal=bool(g[base + "_causal"])).float().cpu()
            infllm_v2.check_device_status()
            ok, err = _within(got, g[base + "_out"])
            assert ok, (base, err)
            continue
        q = torch.from_numpy(det_array((lq, 32, 128), seed)).to(torch.bfloat16)
        k = torch.from_numpy(det_array((lc, 2, 128), seed + 1000)).to(torch.bfloat16)
        got = _run(q, k, cu([lq]), cu([lc]), lq, lc, bool(g[base + "_causal"]))
        ok, err = _within(got, g[base + "_out"])
        assert ok, (base, err)
        assert not np.isnan(got.numpy()).any()


@pytest.mark.parametrize("lens_q,causal", [([4096], True), ([700, 33, 1500], True), ([513], False),
                                           ([40], True), ([4096 + 64], True)])
def test_stage1_vs_oracle(lens_q, causal):
    hq, hk, d = 32, 2, 128
    seed = sum(lens_q)
    q = det_tensor((sum(lens_q), hq, d), seed, 0.5)
    k = det_tensor((sum(lens_q), hk, d), seed + 1, 0.5)
    kc, cu_c = oracle.compress_keys(k, cu(lens_q))
    max_k = int(np.diff(cu_c).max())
    if max_k == 0:
        pytest.skip("no compressed key")
    cu_c_t = torch.tensor(cu_c, dtype=torch.int32)
    got = _run(q, kc, cu(lens_q), cu_c_t, max(lens_q), max_k, causal)
    ref = oracle.stage1_scores(q, kc, cu(lens_q), cu_c_t, max_k, causal)
    ok, err = _within(got, ref)
    assert ok, err
    rows = ref.sum(-1)
    assert ((got.sum(-1) - rows).abs() < 0.25).all()          # visible rows sum to 16, others to 0


def test_stage1_query_chunk_bottom_right_alignment():
    # a query chunk shorter than the span of the keys (context-parallel prefix scoring)
    hq, hk, d = 32, 2, 128
    full = 1024
    q = det_tensor((full, hq, d), 31, 0.5)
    k = det_tensor((full, hk, d), 32, 0.5)
    kc, cu_c = oracle.compress_keys(k, cu([full]))
    whole = _run(q, kc, cu([full]), torch.tensor(cu_c, dtype=torch.int32), full, cu_c[-1], True)
    tail = _run(q[512:], kc, cu([512]), torch.tensor(cu_c, dtype=torch.int32), 512, cu_c[-1], True)
    assert (whole[:, 512:] - tail).abs().max() <= 1e-2


@pytest.mark.parametrize("lens_q,cache,local,init", [([4096], 0, 2, 1), ([700, 33, 1500], 0, 32, 1),
                                                     ([513], 0, 1, 0), ([40], 0, 2, 1),
                                                     ([2048 + 64], 0, 32, 1)])
def test_fused_block_scores_equal_pool_of_scores(lens_q, cache, local, init):
    """The fused stage-1 + max-pool kernel against the two separate kernels: bit-exact."""
    hq, hk, d = 32, 2, 128
    seed = sum(lens_q) + 5
    q = det_tensor((sum(lens_q), hq, d), seed, 0.5).to(DEV)
    k = det_tensor((sum(lens_q), hk, d), seed + 1, 0.5)
    kc, cu_c = oracle.compress_keys(k, cu(lens_q))
    max_k = int(np.diff(cu_c).max())
    cu_q, cu_ct = cu(lens_q).to(DEV), torch.tensor(cu_c, dtype=torch.int32, device=DEV)
    kc = kc.to(DEV)
    pooled, scores = infllm_v2.infllmv2_stage1_block_scores(
        q, kc, cu_q, cu_ct, max(lens_q), max_k, local, init, cache_len=cache, return_scores=True)
    infllm_v2.check_device_status()
    plain = infllm_v2.infllmv2_attn_stage1(q, kc, kc, cu_q, cu_ct, cu_ct, max(lens_q), max_k, causal=True)
    assert torch.equal(scores, plain)
    if len(lens_q) == 1:
        ref = infllm_v2.max_pooling_1d(plain, cache, local, init)
    else:
        ref = infllm_v2.max_pooling_1d_varlen(plain, cu_q, cu_ct, torch.zeros(len(lens_q), dtype=torch.int32, device=DEV),
                                              max(lens_q), max_k, local, init)
    assert pooled.shape == ref.shape
    assert torch.equal(pooled, ref)
    only = infllm_v2.infllmv2_stage1_block_scores(q, kc, cu_q, cu_ct, max(lens_q), max_k, local, init,
                                                  cache_len=cache)
    assert torch.equal(only, ref)


def test_fused_block_scores_query_chunk_with_cache_len():
    hq, hk, d, full = 32, 2, 128, 2048
    q = det_tensor((full, hq, d), 41, 0.5).to(DEV)
    k = det_tensor((full, hk, d), 42, 0.5)
    kc, cu_c = oracle.compress_keys(k, cu([full]))
    kc = kc.to(DEV)
    cu_ct = torch.tensor(cu_c, dtype=torch.int32, device=DEV)
    start = 1024
    got = infllm_v2.infllmv2_stage1_block_scores(q[start:], kc, cu([full - start]).to(DEV), cu_ct, full - start,
                                                 cu_c[-1], 2, 1, cache_len=start)
    plain = infllm_v2.infllmv2_attn_stage1(q[start:], kc, kc, cu([full - start]).to(DEV), cu_ct, cu_ct,
                                           full - start, cu_c[-1], causal=True)
    assert torch.equal(got, infllm_v2.max_pooling_1d(plain, start, 2, 1))


@pytest.mark.parametrize("lens,causal", [([1000, 130, 64, 700], True), ([2048], True), ([300, 500], False)])
def test_stage1_compressed_lse_vs_oracle(lens, causal):
    """Row sums over a coarser compression of the same keys (kernel 128 / stride 64), packed
    ragged sequences including ones with no coarse key at all; scores and fused block scores."""
    hq, hk = 32, 2
    seed = sum(lens) + 5
    q = det_tensor((sum(lens), hq, 128), seed, 0.5)
    k = det_tensor((sum(lens), hk, 128), seed + 1, 0.5)
    kc, cu_c = oracle.compress_keys(k, cu(lens), 32, 16)
    kv, cu_v = oracle.compress_keys(k, cu(lens), 128, 64)
    max_k = int(np.diff(cu_c).max())
    exp = oracle.stage1_scores(q, kc, cu(lens).tolist(), cu_c, max_k, causal, lse_keys=kv, cu_seqlens_v=cu_v)
    cq = cu(lens, DEV)
    ck = torch.tensor(cu_c, dtype=torch.int32, device=DEV)
    cv = torch.tensor(cu_v, dtype=torch.int32, device=DEV)
    got = infllm_v2.infllmv2_attn_stage1(q.to(DEV), kc.to(DEV), kv.to(DEV), cq, ck, cv, max(lens), max_k,
                                         causal=causal)
    infllm_v2.check_device_status()
    ok, err = _within(got.float().cpu(), exp)
    assert ok, err
    if causal:
        pooled = infllm_v2.infllmv2_stage1_block_scores(q.to(DEV), kc.to(DEV), cq, ck, max(lens), max_k, 2, 1,
                                                        lse_keys=kv.to(DEV), cu_seqlens_v=cv)
        ref = infllm_v2.max_pooling_1d_varlen(got, cq, ck, torch.zeros(len(lens), dtype=torch.int32, device=DEV),
                                              max(lens), max_k, 2, 1)
        assert torch.equal(pooled, ref)


def test_stage1_compressed_lse_without_any_coarse_key():
    """Sequences all shorter than the coarse window: the row-sum tensor is empty (its pointer is
    null), cu_seqlens_v is all zeros and every score is 0, as in the oracle."""
    lens, hq, hk = [100, 40, 127], 32, 2
    q = det_tensor((sum(lens), hq, 128), 3, 0.5)
    k = det_tensor((sum(lens), hk, 128), 4, 0.5)
    kc, cu_c = oracle.compress_keys(k, cu(lens), 32, 16)
    kv, cu_v = oracle.compress_keys(k, cu(lens), 128, 64)
    assert kv.shape[0] == 0 and not any(cu_v)
    max_k = int(np.diff(cu_c).max())
    exp = oracle.stage1_scores(q, kc, cu(lens).tolist(), cu_c, max_k, True, lse_keys=kv, cu_seqlens_v=cu_v)
    assert not exp.any()
    got = infllm_v2.infllmv2_attn_stage1(q.to(DEV), kc.to(DEV), kv.to(DEV), cu(lens, DEV),
                                         torch.tensor(cu_c, dtype=torch.int32, device=DEV),
                                         torch.tensor(cu_v, dtype=torch.int32, device=DEV), max(lens), max_k,
                                         causal=True)
    infllm_v2.check_device_status()
    assert got.shape == exp.shape and not got.float().cpu().any()


@pytest.mark.parametrize("lens_c,hk,causal", [([700, 1, 512, 513, 33], 2, False), ([2047, 16], 8, False),
                                              ([40, 0, 1025], 2, False),
                                              ([300, 64, 5], 2, True)])
def test_stage1_decode_path(lens_c, hk, causal):
    """One query token per sequence takes the chunk-parallel kernel pair: same scores as the
    oracle, zeros past every sequence's keys, and as the general kernel (forced by giving one
    sequence two tokens, which leaves the rows of the single-token sequences unchanged)."""
    bsz = len(lens_c)
    seed = sum(lens_c) + hk
    q = det_tensor((bsz, hk * 16, 128), seed, 0.5)
    kc = det_tensor((sum(lens_c), hk, 128), seed + 1, 0.5)
    cu_q, cu_c = cu([1] * bsz), cu(lens_c)
    max_c = max(lens_c)
    exp = oracle.stage1_scores(q, kc, cu_q.tolist(), cu_c.tolist(), max_c, causal)
    got = infllm_v2.infllmv2_attn_stage1(q.to(DEV), kc.to(DEV), kc.to(DEV), cu_q.to(DEV), cu_c.to(DEV),
                                         cu_c.to(DEV), 1, max_c, causal=causal)
    infllm_v2.check_device_status()
    assert got.shape == (hk, bsz, max_c)
    ok, err = _within(got.float().cpu(), exp)
    assert ok, err
    for b, n in enumerate(lens_c):                       # nothing but zeros past a sequence's keys
        assert (got[:, b, n:] == 0).all()
    if not causal:
        # the general kernel on the same rows: append a second token to the last sequence
        q2 = torch.cat([q, q[-1:]], 0)
        cu_q2 = cu([1] * (bsz - 1) + [2])
        ref = infllm_v2.infllmv2_attn_stage1(q2.to(DEV), kc.to(DEV), kc.to(DEV), cu_q2.to(DEV), cu_c.to(DEV),
                                             cu_c.to(DEV), 2, max_c, causal=False)
        diff = (got.float() - ref[:, :bsz].float()).abs()
        assert (diff <= torch.maximum(torch.tensor(2e-2, device=DEV), ref[:, :bsz].float().abs() * 2.0 ** -7)).all()


@pytest.mark.parametrize("lens", [[40] * 130 + [1, 700, 15, 33, 2049], [9000]])
def test_items_taken_in_turn_match_one_item_per_cta(lens):
    # up to 2048 compressed keys CTAs stay and take several 16-token items (odd counts, items without a visible
    # key, one-tile items between long ones); above, each CTA has one: the same scores and block scores, bit for bit
    hk = 2
    n = sum(lens)
    q = det_tensor((n, hk * 16, 128), 21, 0.5).to(DEV)
    k = det_tensor((n, hk, 128), 22, 0.5).to(DEV)
    cu_q = cu(lens, DEV)
    kc, cu_c = infllm_v2.compress_keys(k, cu_q)
    most = int((cu_c[1:] - cu_c[:-1]).max())
    a = infllm_v2.infllmv2_attn_stage1(q, kc, kc, cu_q, cu_c, cu_c, max(lens), max(most, 1), causal=True)
    b = infllm_v2.infllmv2_attn_stage1(q, kc, kc, cu_q, cu_c, cu_c, max(lens), 2049, causal=True)
    infllm_v2.check_device_status()
    assert torch.equal(a[..., :most], b[..., :most]) and not b[..., most:].any()
    blocks = (max(lens) + 63) // 64
    pa = infllm_v2.infllmv2_stage1_block_scores(q, kc, cu_q, cu_c, max(lens), max(most, 1), 1, 1, causal=True)
    pb = infllm_v2.infllmv2_stage1_block_scores(q, kc, cu_q, cu_c, max(lens), 2049, 1, 1, causal=True)
    infllm_v2.check_device_status()
    shared = min(pa.shape[-1], pb.shape[-1], blocks)
    assert torch.equal(pa[..., :shared], pb[..., :shared])


def _many_items(layout, causal, hk=2, seed=3):
    """About 400 short sequences (more than 1000 items of 16 tokens and a KV head for 148 CTAs), some without scored
    or without row-sum keys, in the given layout: q, cu_q, keys, their arguments and the packed keys for the oracle."""
    rng = np.random.default_rng(seed)
    n = 400
    lens_q = rng.choice([1, 15, 16, 17, 33, 40, 100], n)
    lens_c = rng.choice([0, 0, 1, 5, 128, 129, 300], n)
    lens_v = rng.choice([0, 1, 7, 128, 129, 200], n) if layout.startswith("coarse") else lens_c
    q = det_tensor((int(lens_q.sum()), hk * 16, 128), seed, 0.5)
    kc = det_tensor((int(lens_c.sum()), hk, 128), seed + 1, 0.5)
    kv = det_tensor((int(lens_v.sum()), hk, 128), seed + 2, 0.5)
    kw = {}
    if layout == "paged":
        table = torch.zeros(n, 3, dtype=torch.int32)
        pages = det_tensor((int((-(-lens_c // 128)).sum()) + 1, 128, hk, 128), seed + 3, 3.0)   # unused rows: large keys
        free, at = list(rng.permutation(pages.shape[0])), 0
        for b, l in enumerate(lens_c):
            for j in range(-(-int(l) // 128)):
                table[b, j] = int(free.pop())
                m = min(128, int(l) - 128 * j)
                pages[table[b, j], :m] = kc[at:at + m]
                at += m
        k, kw["block_table"] = pages, table.to(DEV)
        cu_k = cu(lens_c)
    elif layout == "leftpad" or layout.startswith("coarse_used"):
        # extents longer than what is in use: five rows in front, or seven (in some sequences all rows) behind
        front, behind = (5, 0) if layout == "leftpad" else (0, 7)
        parts, at = [], 0
        for b, l in enumerate(lens_c):
            junk = det_tensor((front + behind, hk, 128), seed + 4, 3.0)
            parts += [junk[:front], kc[at:at + int(l)], junk[front:]]
            at += int(l)
        k, cu_k = torch.cat(parts), cu(lens_c + front + behind)
        if front:
            kw["leftpad_k"] = torch.full((n,), front, dtype=torch.int32, device=DEV)
        else:
            kw["seqused_k"] = torch.tensor(lens_c, dtype=torch.int32, device=DEV)
    else:
        k, cu_k = kc, cu(lens_c)
    vd, cu_v = None, cu_k
    if layout.startswith("coarse"):
        vd, cu_v = kv.to(DEV), cu(lens_v)
        if layout == "coarse_used_both":
            used = np.maximum(lens_v - 3, 0)                      # (the oracle gets these rows only)
            kw["seqused_v"] = torch.tensor(used, dtype=torch.int32, device=DEV)
            o = np.concatenate([[0], np.cumsum(lens_v)])
            kv = torch.cat([kv[o[b]:o[b] + int(u)] for b, u in enumerate(used)])
            lens_v = used
    k = k.to(DEV)
    args = dict(q=q.to(DEV), k=k, v=vd if vd is not None else k, cu_q=cu(lens_q, DEV), cu_k=cu_k.to(DEV),
                cu_v=cu_v.to(DEV), max_q=int(lens_q.max()), kw=kw)
    return args, oracle.stage1_scores(q, kc, cu(lens_q).tolist(), cu(lens_c).tolist(), 300, causal,
                                      lse_keys=kv if vd is not None else None, cu_seqlens_v=cu(lens_v).tolist())


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("layout", ["packed", "coarse", "coarse_used", "coarse_used_both", "paged", "leftpad"])
def test_items_taken_in_turn_in_every_key_layout(layout, causal):
    # passes of different lengths, and one or both of them empty, between each other on one CTA: an item that sees
    # row-sum keys but no scored key must not shift the row constants of the next one
    a, ref = _many_items(layout, causal)
    coarse = layout.startswith("coarse")

    def scores(max_k):
        return infllm_v2.infllmv2_attn_stage1(a["q"], a["k"], a["v"], a["cu_q"], a["cu_k"], a["cu_v"], a["max_q"], max_k,
                                              causal=causal, **a["kw"])

    def blocks(max_k):
        extra = dict(lse_keys=a["v"], cu_seqlens_v=a["cu_v"]) if coarse else {}
        return infllm_v2.infllmv2_stage1_block_scores(a["q"], a["k"], a["cu_q"], a["cu_k"], a["max_q"], max_k, 0, 0,
                                                      max_cache_len=0, cache_len=1100, causal=causal, **extra, **a["kw"])
    for _ in range(3):
        got = scores(300)
        infllm_v2.check_device_status()
        ok, err = _within(got.float().cpu(), ref)
        assert ok, err
    if layout != "paged":                      # (its three pages a sequence cover 384 keys)
        assert torch.equal(got, scores(2049)[..., :300])          # one item a CTA
        assert torch.equal(blocks(300), blocks(2049))
    if layout in ("packed", "coarse"):
        lens = torch.full((a["cu_q"].numel() - 1,), 1100, dtype=torch.int32, device=DEV)
        pooled = infllm_v2.max_pooling_1d_varlen(got, a["cu_q"], a["cu_k"], lens, a["max_q"], 300, 0, 0)
        mine = blocks(300)
        shared = min(pooled.shape[-1], mine.shape[-1])
        assert shared > 10 and torch.equal(mine[..., :shared], pooled[..., :shared])
    infllm_v2.check_device_status()


@pytest.mark.parametrize("lens", [[16] * 600, [0, 5] * 400 + [1, 0, 0],                       # so many numbers a sequence
                                  [3000, 0, 17, 1400, 0], [2399, 15], [0, 2385],             # added up
                                  [0] * 90 + [300] + [0] * 300 + [1, 33] * 90])               # searched for
def test_numbering_of_the_items(lens):
    # the three ways in which a staying CTA finds its items, with empty sequences between and at both ends: bit for bit
    # what one item a CTA gives; rows of q past the last sequence belong to nobody
    hk, n = 2, sum(lens)
    q = det_tensor((n + 21, hk * 16, 128), 31, 0.5).to(DEV)
    kc = det_tensor((3 * len(lens), hk, 128), 32, 0.5).to(DEV)
    cu_q, cu_k = cu(lens, DEV), cu([3] * len(lens), DEV)
    a, b = (infllm_v2.infllmv2_attn_stage1(q, kc, kc, cu_q, cu_k, cu_k, max(lens), m, causal=False) for m in (3, 2049))
    infllm_v2.check_device_status()
    assert torch.equal(a[:, :n], b[:, :n, :3]) and (a[:, :n].float().sum(-1) - 16).abs().max() < 0.25


@pytest.mark.parametrize("lens,keys,hk", [
    ([2048], 1088, 2), ([2048], 1089, 2), ([5008], 1692, 2), ([5008], 1693, 2), ([49152], 3071, 1),
    ([2400, 1, 1], 2123, 2), ([2400, 1, 1], 2124, 2),
])
def test_scores_on_both_sides_of_the_line_of_staying_ctas(lens, keys, hk):
    # whether CTAs stay follows from the mean walk (at most 1024 keys, with more than 4 items per SM 1536, 2048 where most
    # tiles would be empty) and never shows in the results: a loose max_seqlen_k takes one item a CTA
    q = det_tensor((sum(lens), hk * 16, 128), 41, 0.5).to(DEV)
    kc = det_tensor((keys * len(lens), hk, 128), 42, 0.5).to(DEV)
    cu_q, cu_k = cu(lens, DEV), cu([keys] * len(lens), DEV)
    cache = 16 * keys + 16 - max(lens)
    a, b = (infllm_v2.infllmv2_stage1_block_scores(q, kc, cu_q, cu_k, max(lens), m, 1, 1, cache_len=cache, max_cache_len=cache,
                                                   causal=True) for m in (keys, 5000))
    infllm_v2.check_device_status()
    assert torch.equal(a, b) and a.isfinite().any()
