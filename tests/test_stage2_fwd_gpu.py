"""GPU: stage-2 block-sparse attention forward against the fp32 dense-with-mask oracle.
Tolerance (bf16 outputs): max-abs <= 2e-2 and mean-rel <= 1e-2."""
import os

import numpy as np
import pytest
import torch

import oracle
import infllm_v2
from helpers import det_tensor, cu, local_topk, err_stats
from inputs import det_array, det_perm_rows

pytestmark = pytest.mark.gpu
DEV = "cuda"
MAX_ABS, MEAN_REL = 2e-2, 1e-2


def _run(q, k, v, cu_q, cu_k, idx, causal):
    out, lse, _ = infllm_v2.infllmv2_attn_varlen_func(
        q.to(DEV), k.to(DEV), v.to(DEV), cu_q.to(DEV), cu_k.to(DEV),
        int((cu_q[1:] - cu_q[:-1]).max()), int((cu_k[1:] - cu_k[:-1]).max()),
        causal=causal, topk_idx=None if idx is None else idx.to(DEV), return_attn_probs=True)
    infllm_v2.check_device_status()
    return out.cpu(), lse.cpu()


def _check(q, k, v, cu_q, cu_k, idx, causal):
    out, lse = _run(q, k, v, cu_q, cu_k, idx, causal)
    ref, ref_lse = oracle.sparse_attention_fwd(q, k, v, cu_q, cu_k, idx, causal=causal)
    assert not torch.isnan(out.float()).any()
    mx, mr = err_stats(out, ref)
    assert mx <= MAX_ABS and mr <= MEAN_REL, (mx, mr)
    empty = torch.isinf(ref_lse)
    assert torch.equal(torch.isinf(lse) & (lse > 0), empty)
    assert (lse[~empty] - ref_lse[~empty]).abs().max() < 2e-2
    return out


@pytest.mark.parametrize("lens_q,lens_k,k_sel,causal", [
    ([128], [128], 2, True), ([200, 136], [200, 136], 3, True), ([64, 192], [160, 300], 3, True),
    ([1000], [1000], 8, True), ([77, 5, 130], [77, 5, 130], 2, True), ([256], [256], 4, False),
    ([8], [8], 1, True), ([3], [700], 4, True),
])
def test_fwd_sparse(lens_q, lens_k, k_sel, causal):
    hq, hk, d = 32, 2, 128
    seed = sum(lens_q) + k_sel
    q = det_tensor((sum(lens_q), hq, d), seed, 0.25)
    k = det_tensor((sum(lens_k), hk, d), seed + 1, 0.25)
    v = det_tensor((sum(lens_k), hk, d), seed + 2)
    idx = local_topk(hk, lens_q, lens_k, k_sel, seed)
    _check(q, k, v, cu(lens_q), cu(lens_k), idx, causal)


def test_fwd_dense_and_large_scores():
    # dense (topk_idx=None) with scores large enough to force accumulator rescales
    hq, hk, d = 32, 2, 128
    q = det_tensor((300, hq, d), 1, 1.0)
    k = det_tensor((300, hk, d), 2, 1.0)
    v = det_tensor((300, hk, d), 3)
    _check(q, k, v, cu([300]), cu([300]), None, True)


def test_fwd_rows_without_keys_and_unselected_blocks():
    hq, hk, d = 32, 2, 128
    q = det_tensor((130, hq, d), 4, 0.25)
    k = det_tensor((130, hk, d), 5, 0.25)
    v = det_tensor((130, hk, d), 6)
    idx = torch.full((hk, 130, 2), -1, dtype=torch.int32)
    idx[:, 70:, 0] = 0                      # tokens < 70 select nothing at all
    idx[0, 100:, 1] = 1
    out = _check(q, k, v, cu([130]), cu([130]), idx, True)
    assert out[:70].abs().max() == 0


def test_fwd_golden_inputs(golden_dir):
    g = np.load(os.path.join(golden_dir, "stage2.npz"))
    step = int(g["out_row_step"])
    hq, hk, d = 32, 2, 128
    for name in ("a", "b", "c"):
        seed, k_sel = (int(x) for x in g[f"s2_{name}_seed"])
        cu_q, cu_k = torch.from_numpy(g[f"s2_{name}_cuq"]), torch.from_numpy(g[f"s2_{name}_cuk"])
        sk = int((cu_k[1:] - cu_k[:-1]).max())
        q = torch.from_numpy(det_array((int(cu_q[-1]), hq, d), seed, 0.25)).to(torch.bfloat16)
        k = torch.from_numpy(det_array((int(cu_k[-1]), hk, d), seed + 1000, 0.25)).to(torch.bfloat16)
        v = torch.from_numpy(det_array((int(cu_k[-1]), hk, d), seed + 2000)).to(torch.bfloat16)
        idx = torch.from_numpy(det_perm_rows(hk * int(cu_q[-1]), (sk + 63) // 64, k_sel, seed + 3000)
                               ).view(hk, -1, k_sel)
        for causal in (0, 1):
            key = f"s2_{name}_{causal}_out"
            if key not in g.files:
                continue
            out, _ = _run(q, k, v, cu_q, cu_k, idx, bool(causal))
            mx, mr = err_stats(out[::step], torch.from_numpy(g[key]))
            assert mx <= MAX_ABS and mr <= MEAN_REL, (key, mx, mr)


def test_fwd_multiword_mask_eight_kv_heads():
    # 8 KV heads, > 64 key blocks (two mask words), block lists shared per 64-token query block
    hq, hk, d = 128, 8, 128
    lens = [4500]
    q = det_tensor((lens[0], hq, d), 21, 0.25)
    k = det_tensor((lens[0], hk, d), 22, 0.25)
    v = det_tensor((lens[0], hk, d), 23)
    idx = local_topk(hk, lens, lens, 6, 24, shared_per_block=True)
    out, _ = _run(q, k, v, cu(lens), cu(lens), idx, True)
    sl = slice(4300, 4500)                     # check the tail rows (most blocks) on the CPU oracle
    ref, _ = oracle.sparse_attention_fwd(q, k, v, cu(lens), cu(lens), idx, causal=True)
    mx, mr = err_stats(out[sl], ref[sl])
    assert mx <= MAX_ABS and mr <= MEAN_REL, (mx, mr)


@pytest.mark.parametrize("n_sel", [1, 2, 3, 5])
@pytest.mark.parametrize("len_k", [320, 333, 384])
def test_fwd_odd_and_even_block_counts(n_sel, len_k):
    # scores and P have two buffers: a last block in the first and in the second of them, a ragged block in
    # either, and tokens of one tile that select different blocks
    hq, hk, d, lq = 32, 2, 128, 21
    q = det_tensor((lq, hq, d), 31, 0.25)
    k = det_tensor((len_k, hk, d), 32, 0.25)
    v = det_tensor((len_k, hk, d), 33)
    shared = local_topk(hk, [lq], [len_k], n_sel, 34 + n_sel)[:, -1:].expand(-1, lq, -1).contiguous()
    _check(q, k, v, cu([lq]), cu([len_k]), shared, True)
    _check(q, k, v, cu([lq]), cu([len_k]), local_topk(hk, [lq], [len_k], n_sel, 40 + n_sel), False)


@pytest.mark.parametrize("jump", [1, 2, 3, 4])
def test_fwd_reference_moves_at_any_block(jump):
    # the scores of block `jump` (counted in walking order, highest block first) exceed all before it
    # by ~60 (natural log units): the running reference has to move, in either buffer of scores and P
    hq, hk, d, n_blk = 32, 2, 128, 6
    q = torch.zeros(9, hq, d, dtype=torch.bfloat16)
    q[..., 0] = 1.0
    q[..., 1:9] = det_tensor((9, hq, 8), 51, 0.25)
    k = det_tensor((n_blk * 64, hk, d), 52, 0.25)
    k[..., 0] = 0.0
    first = (n_blk - 1 - jump) * 64
    k[first:first + 64, :, 0] = 680.0                      # 680 / sqrt(128) = 60
    v = det_tensor((n_blk * 64, hk, d), 53)
    _check(q, k, v, cu([9]), cu([n_blk * 64]), None, False)


@pytest.mark.parametrize("packed", [False, True])
def test_registered_operators_are_used_when_something_traces(packed):
    # a plain eager call runs the bodies directly; under a dispatch mode the registered operators are
    # what the mode sees, with the same results
    from torch.utils._python_dispatch import TorchDispatchMode
    seen = []

    class Recorder(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    hq, hk, d, n = 32, 2, 128, 200
    idx = local_topk(hk, [n], [n], 2, 77).to(DEV)
    sel = dict(block_mask=infllm_v2.topk_to_uint64(idx, n, 64)[0]) if packed else dict(topk_idx=idx)
    res = []
    for mode in (None, Recorder()):
        q, k, v = (det_tensor((n, h, d), 78 + i, 0.25, device=DEV).requires_grad_(True) for i, h in enumerate((hq, hk, hk)))
        def call():
            out = infllm_v2.infllmv2_attn_varlen_func(q, k, v, cu([n], DEV), cu([n], DEV), n, n, causal=True, **sel)
            return (out.detach(),) + torch.autograd.grad(out, (q, k, v), det_tensor((n, hq, d), 81, 0.5, device=DEV))
        if mode is None:
            res.append(call())
        else:
            with mode:
                res.append(call())
    assert all(torch.equal(a, b) for a, b in zip(*res))
    assert any("_infllmv2_attn_varlen_forward" in s for s in seen)
    # (the engine runs the backward in a thread of its own, which the mode does not cover; the next test
    # keeps it in this thread)


def test_registered_backward_is_used_under_a_dispatch_mode():
    from torch.utils._python_dispatch import TorchDispatchMode
    seen = []

    class Recorder(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    hq, hk, d, n = 32, 2, 128, 130
    q, k, v = (det_tensor((n, h, d), 84 + i, 0.25, device=DEV).requires_grad_(True) for i, h in enumerate((hq, hk, hk)))
    dout = det_tensor((n, hq, d), 87, 0.5, device=DEV)

    def grads():
        out = infllm_v2.infllmv2_attn_varlen_func(q, k, v, cu([n], DEV), cu([n], DEV), n, n, causal=True)
        return torch.autograd.grad(out, (q, k, v), dout)

    plain = grads()
    with torch.autograd.set_multithreading_enabled(False), Recorder():
        watched = grads()
    assert all(torch.equal(a, b) for a, b in zip(plain, watched))
    assert any("_infllmv2_attn_varlen_backward" in s for s in seen)


@pytest.mark.parametrize("rows", ["all", "some"])
@pytest.mark.parametrize("keys", [1, 64])
@pytest.mark.parametrize("bits", [7, 9, 13, 15])
def test_fwd_scores_rise_to_either_side_of_the_limit(bits, keys, rows):
    """One or all keys of a later block lie `bits` powers of two above every score before it, for all rows
    or for some rows of a warp only: the reference moves beyond 8, and the row maximum that decides it is
    taken when the exponentials of a block sum up to 2^7, which one key at 7 just does with the others."""
    hq, hk, d, n_blk, lq = 32, 2, 128, 5, 9
    q = torch.zeros(lq, hq, d, dtype=torch.bfloat16)
    q[..., 0] = 1.0
    if rows == "some":
        q[1::2, :, 0] = 0.0
        q[:, 1::3, 0] = 0.0
    q[..., 1:9] = det_tensor((lq, hq, 8), 61, 0.25)
    k = det_tensor((n_blk * 64, hk, d), 62, 0.25)
    k[..., 0] = 0.0
    first = (n_blk - 3) * 64                                # the third block of the walk (highest first)
    k[first + 64 - keys:first + 64, :, 0] = bits * np.log(2.0) * d ** 0.5
    v = det_tensor((n_blk * 64, hk, d), 63)
    _check(q, k, v, cu([lq]), cu([n_blk * 64]), None, False)


def test_fwd_weight_of_a_score_far_above_the_rest_is_exact():
    """A score more than 8 powers of two above everything before it becomes the reference of its row, so that
    its weight is 1 and takes no rounding to bf16.  Only that key has a value here: what is left is the
    rounding of the result, 2^-9 in [0.5, 1), and fp32 arithmetic; a rounded weight would add up to 2^-9."""
    hq, hk, d, n_blk, lq = 32, 2, 128, 5, 21
    q = torch.zeros(lq, hq, d)
    q[..., 0] = torch.linspace(0.7, 1.0, lq * hq).view(lq, hq)
    k, v = torch.zeros(n_blk * 64, hk, d), torch.zeros(n_blk * 64, hk, d)
    key = (n_blk - 3) * 64 + 17                             # in the third block of the walk (highest first)
    k[key, :, 0] = 13.5 * np.log(2.0) * d ** 0.5            # 9.4 .. 13.5 powers of two for the rows above
    v[key] = 1.0
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    out, _ = _run(q, k, v, cu([lq]), cu([n_blk * 64]), None, False)
    w = (q[..., 0].double() * k[key, 0, 0].double() * d ** -0.5).exp()
    ref = (w / (w + n_blk * 64 - 1))[..., None].expand(-1, -1, d)
    assert ref.min() > 0.5 and (out.double() - ref).abs().max() <= 2.0 ** -9 + 1e-5


@pytest.mark.parametrize("n_blk,picks", [(2049, "edges"), (2200, "edges"), (2200, "many"), (2200, None), (4200, "edges"), (4200, "many")])
def test_fwd_block_lists_of_several_chunks_of_words(n_blk, picks):
    """More than 32 mask words, so that the walk goes over two or three chunks of them: every token with
    blocks of its own on both sides of the borders, more than 32 visited blocks in `many`, all of them
    without a mask.  Against the fp32 result over the selected keys."""
    hk, d, lq, n = 1, 128, 11, n_blk * 64 - 7
    g = torch.Generator(device=DEV).manual_seed(n_blk)
    q = torch.randn(lq, 16 * hk, d, generator=g, device=DEV, dtype=torch.bfloat16)
    k, v = (torch.randn(n, hk, d, generator=g, device=DEV, dtype=torch.bfloat16).mul_(0.5) for _ in range(2))
    sel, kw = torch.ones(hk, lq, n_blk, dtype=torch.bool, device=DEV), {}
    if picks is not None:
        sel.zero_()
        edges = [b for b in (0, 63, 64, 1983, 1984, 2047, 2048, 2111, 2112, 4095, 4096, n_blk - 2, n_blk - 1) if b < n_blk]
        for t in range(lq):
            sel[:, t, [edges[(t + i) % len(edges)] for i in range(5)]] = True
        if picks == "many":
            sel |= torch.rand(hk, lq, n_blk, generator=g, device=DEV) < 60 / n_blk
        kw = dict(block_mask=infllm_v2.blockmask_to_uint64(sel)[0])
    out, lse, _ = infllm_v2.infllmv2_attn_varlen_func(q, k, v, cu([lq], DEV), cu([n], DEV), lq, n, causal=True,
                                                      return_attn_probs=True, **kw)
    infllm_v2.check_device_status()
    pos = torch.arange(n, device=DEV)
    seen = sel[:, :, pos // 64] & (pos <= torch.arange(n - lq, n, device=DEV)[:, None])            # (hk, lq, n)
    s = torch.einsum("thgd,nhd->htgn", q.view(lq, hk, 16, d).float(), k.float()) * d ** -0.5
    s = s.masked_fill(~seen[:, :, None, :], float("-inf"))
    ref = torch.einsum("htgn,nhd->thgd", s.softmax(-1), v.float()).reshape(lq, 16 * hk, d)
    mx, mr = err_stats(out, ref)
    assert mx <= MAX_ABS and mr <= MEAN_REL, (mx, mr)
    assert (lse.view(hk, lq, 16) - s.logsumexp(-1)).abs().max() < 2e-2


def test_function_mode_sees_the_forward_operator():
    from torch.overrides import TorchFunctionMode
    seen = []

    class Recorder(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    hq, hk, d, n = 32, 2, 128, 90
    q, k, v = (det_tensor((n, h, d), 88 + i, 0.25, device=DEV) for i, h in enumerate((hq, hk, hk)))
    args = (cu([n], DEV), cu([n], DEV), n, n)
    plain = infllm_v2.infllmv2_attn_varlen_func(q, k, v, *args, causal=True)
    with Recorder():
        out = infllm_v2.infllmv2_attn_varlen_func(q, k, v, *args, causal=True)
    assert torch.equal(out, plain)
    assert any("_infllmv2_attn_varlen_forward" in s for s in seen)


@pytest.mark.parametrize("lk", [256, 250])
def test_fwd_blocks_that_one_pair_of_tokens_selects(lk):
    # a softmax warp owns two of a tile's eight tokens and skips the blocks that only others selected: its
    # first block, its last one, all but one and, with lk = 250, the ragged block that is never skipped
    hq, hk, d = 32, 2, 128
    q, k, v = (det_tensor((n, h, d), 80 + i, 0.5) for i, (n, h) in enumerate(((16, hq), (lk, hk), (lk, hk))))
    idx = torch.full((hk, 16, 2), -1, dtype=torch.int32)
    for t in range(16):
        pair = (t % 8) // 2
        idx[:, t, 0] = 3 - pair if t < 8 else pair
        if t % 2 and t >= 8:
            idx[:, t, 0], idx[:, t, 1] = min(pair, (pair + 1) % 4), max(pair, (pair + 1) % 4)
    _check(q, k, v, cu([16]), cu([lk]), idx, False)
