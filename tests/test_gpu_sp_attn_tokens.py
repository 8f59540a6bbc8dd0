"""GPU parity of the sp_attn operator (key-token lists at the reference granularity)."""
import pytest
import torch

from helpers import GOLDEN_CASES, OUT_MAX_ABS, OUT_MEAN_ABS, load_golden

pytestmark = pytest.mark.gpu


def _capi():
    from fgattn_tk_cuda_b200 import capi
    return capi


def _close(o, ref, mx=OUT_MAX_ABS, mean=OUT_MEAN_ABS):
    d = (o.float().cpu() - torch.as_tensor(ref).float().cpu()).abs()
    assert torch.isfinite(o.float()).all()
    assert d.max().item() <= mx, d.max().item()
    assert d.mean().item() <= mean, d.mean().item()


@pytest.mark.parametrize("S,D", [(1000, 128), (777, 64), (128, 128)])
def test_identity_and_permuted_lists_equal_dense(S, D):
    """All keys listed, in order and in random order, must reproduce dense attention
    (test/test_sparseattn_asyncgatherload_padded.cu:37-62, python/test/test_extension.py:65-88)."""
    capi = _capi()
    B, H = 1, 2
    g = torch.Generator().manual_seed(S)
    q, k, v = (torch.randn(B, H, S, D, generator=g).to(torch.bfloat16).cuda() for _ in range(3))
    dense = torch.empty_like(q)
    capi.full_attn(dense, q, k, v)
    nb, stride = (S + 127) // 128, 128 * ((S + 127) // 128)
    idx = torch.empty(B, H, nb, stride, dtype=torch.int32, device="cuda")
    cnt = torch.empty(B, H, nb, dtype=torch.int32, device="cuda")
    capi.all_index_mask(idx, cnt, B, H, nb, S)
    o = torch.full_like(q, float("nan"))
    capi.sp_attn(o, q, k, v, idx, cnt)
    capi.check()
    _close(o, dense, 8e-3, 5e-4)
    perm = torch.cat([torch.randperm(S, generator=g), torch.full((stride - S,), stride)]).to(torch.int32)
    idx2 = perm.cuda().expand(B, H, nb, stride).contiguous()
    o2 = torch.full_like(q, float("nan"))
    capi.sp_attn(o2, q, k, v, idx2, cnt)
    capi.check()
    _close(o2, dense, 8e-3, 5e-4)


@pytest.mark.parametrize("name", GOLDEN_CASES)
def test_threshold_token_lists_golden(name):
    """The reference's own token lists (blocksz 128) drive the gather kernel; output against the
    oracle's renormalising sparse attention."""
    from oracle import fgattn_oracle as orc
    capi = _capi()
    g = load_golden(name)
    q, k, v = (g[t].cuda() for t in "qkv")
    idx = torch.from_numpy(g["index_128"]).cuda().contiguous()
    cnt = torch.from_numpy(g["count_128"]).cuda().contiguous()
    o = torch.full_like(q, float("nan"))
    capi.sp_attn(o, q, k, v, idx, cnt)
    capi.check()
    _close(o, orc.sp_attn_tokens(g["q"], g["k"], g["v"], idx.cpu(), cnt.cpu(), 128))


def test_ragged_counts_empty_lists_and_bad_entries():
    from oracle import fgattn_oracle as orc
    capi = _capi()
    B, H, S, D = 1, 2, 900, 128
    g = torch.Generator().manual_seed(11)
    q, k, v = (torch.randn(B, H, S, D, generator=g).to(torch.bfloat16) for _ in range(3))
    nb, stride = (S + 127) // 128, 1024
    idx = torch.full((B, H, nb, stride), stride, dtype=torch.int32)
    cnt = torch.zeros(B, H, nb, dtype=torch.int32)
    for h in range(H):
        for b in range(nb):
            n = int(torch.randint(0, 700, (1,), generator=g))
            if (h, b) == (0, 1):
                n = 0                                   # empty list -> zero rows
            sel = torch.randperm(S, generator=g)[:n].to(torch.int32)
            if n > 10:
                sel[5] = stride                         # out-of-range entry inside the count: ignored
            idx[0, h, b, :n] = sel
            cnt[0, h, b] = n
    o = torch.full((B, H, S, D), float("nan"), dtype=torch.bfloat16, device="cuda")
    capi.sp_attn(o, q.cuda(), k.cuda(), v.cuda(), idx.cuda(), cnt.cuda())
    capi.check()
    _close(o, orc.sp_attn_tokens(q, k, v, idx, cnt, 128))
    # the order in which the thread blocks take the query blocks changes nothing in the result
    o_st = torch.full_like(o, float("nan"))
    capi.sp_attn(o_st, q.cuda(), k.cuda(), v.cuda(), idx.cuda(), cnt.cuda(), ordered=False)
    capi.check()
    assert torch.equal(o_st, o)
    # with the block route switched on the well-filled lists go through whole tiles: same result within rounding
    capi.set_tuning("token_block_route", 1)
    try:
        o_b = torch.full_like(o, float("nan"))
        capi.sp_attn(o_b, q.cuda(), k.cuda(), v.cuda(), idx.cuda(), cnt.cuda(), block_route=True)
        capi.check()
    finally:
        capi.set_tuning("token_block_route", -1)
    _close(o_b, orc.sp_attn_tokens(q, k, v, idx, cnt, 128))


def _routes(capi, ws, B, H, S):
    """Route flags (1 = block route) that the call left in its workspace, per (unit, 128-row query block)."""
    small = (capi.sp_attn_workspace_bytes(B, H, S) + 255) // 256 * 256
    n_rows = B * H * ((S + 127) // 128)
    off = 2 * small + (n_rows * 4 + 255) // 256 * 256
    return ws[off:off + n_rows * 4].view(torch.int32).view(B * H, -1).cpu()


def _lists_from_mask(tm, stride):
    from oracle import fgattn_oracle as orc
    idx, cnt = orc.bitmask_to_indexmask(tm)
    out = torch.full((*idx.shape[:3], stride), stride, dtype=torch.int32)
    n = idx.shape[-1]
    out[..., :n] = torch.where(idx >= n, torch.full_like(idx, stride), idx)
    return out, cnt


@pytest.mark.parametrize("S,D,kv", [(1000, 128, None), (1500, 64, None), (640, 128, 900)])
def test_block_route_mixed_with_row_gather(S, D, kv):
    """Lists that fill the 64-key blocks they touch (what a threshold mask produces) go through whole
    K/V tiles with column masks, scattered lists and lists that name a token twice stay on the row
    gather -- in one call; every query block against the oracle."""
    from oracle import fgattn_oracle as orc
    capi = _capi()
    B, H = 1, 2
    n_kv = kv or S
    g = torch.Generator().manual_seed(S + D)
    q = torch.randn(B, H, S, D, generator=g).to(torch.bfloat16)
    k, v = (torch.randn(B, H, n_kv, D, generator=g).to(torch.bfloat16) for _ in range(2))
    nb, nkb = (S + 127) // 128, (n_kv + 63) // 64
    stride = 128 * ((n_kv + 127) // 128)
    # block-structured mask: a third of the key blocks, 90 % of their columns (ragged last block included)
    blocks = torch.rand(B, H, nb, nkb, generator=g) < 0.35
    tm = blocks.repeat_interleave(64, dim=-1)[..., :n_kv] & (torch.rand(B, H, nb, n_kv, generator=g) < 0.9)
    tm[0, 0, 1] = torch.rand(n_kv, generator=g) < 0.08          # scattered list: row gather
    tm[0, 1, 0] = False                                         # empty list: zero rows
    idx, cnt = _lists_from_mask(tm, stride)
    dup_row = (0, 1, 2)
    n = int(cnt[dup_row])
    if n >= 2:
        idx[dup_row][n - 1] = idx[dup_row][0]                   # a token listed twice: row gather (counts twice)
    ref = orc.sp_attn_tokens(q, k, v, idx, cnt, 128)
    qc, kc, vc, idxc, cntc = q.cuda(), k.cuda(), v.cuda(), idx.cuda(), cnt.cuda()
    ws = torch.empty(capi.sp_attn_token_workspace_bytes(B, H, S, n_kv), dtype=torch.uint8, device="cuda")
    o = torch.full_like(qc, float("nan"))
    capi.set_tuning("token_block_route", 1)
    try:
        capi.sp_attn(o, qc, kc, vc, idxc, cntc, workspace=ws)
        capi.check()
    finally:
        capi.set_tuning("token_block_route", -1)
    _close(o, ref)
    routes = _routes(capi, ws, B, H, S)
    assert routes[0, 1] == 0 and routes[1, 0] == 0              # scattered / empty
    if n >= 2:
        assert routes[1, 2] == 0                                # duplicate
    assert routes.sum() >= 3                                    # well-filled lists took the block route
    # the row gather alone gives the same within rounding
    o_g = torch.full_like(qc, float("nan"))
    capi.sp_attn(o_g, qc, kc, vc, idxc, cntc, block_route=False)
    capi.check()
    _close(o_g, ref)
    assert (o.float() - o_g.float()).abs().max().item() <= 1.6e-2


def test_block_route_large_scores_rerun():
    """Query norms large enough that the sampled exponent hint misses some rows by more than the safe
    range: those query blocks are recomputed by the running-maximum kernel, result unchanged."""
    from oracle import fgattn_oracle as orc
    capi = _capi()
    B, H, S, D = 1, 1, 512, 128
    g = torch.Generator().manual_seed(4)
    q = (torch.randn(B, H, S, D, generator=g) * 12.0).to(torch.bfloat16)
    k = (torch.randn(B, H, S, D, generator=g) * 12.0).to(torch.bfloat16)
    v = torch.randn(B, H, S, D, generator=g).to(torch.bfloat16)
    tm = torch.rand(B, H, 4, S, generator=g) < 0.95
    idx, cnt = _lists_from_mask(tm, S)
    ref = orc.sp_attn_tokens(q, k, v, idx, cnt, 128)
    ws = torch.empty(capi.sp_attn_token_workspace_bytes(B, H, S, S), dtype=torch.uint8, device="cuda")
    o = torch.full((B, H, S, D), float("nan"), dtype=torch.bfloat16, device="cuda")
    capi.set_tuning("token_block_route", 1)
    try:
        capi.sp_attn(o, q.cuda(), k.cuda(), v.cuda(), idx.cuda(), cnt.cuda(), workspace=ws)
        capi.check()
    finally:
        capi.set_tuning("token_block_route", -1)
    _close(o, ref)
    assert _routes(capi, ws, B, H, S).sum() == 4


def test_block_route_with_more_items_than_sms():
    """The queue of the block route with fewer thread blocks than items, of which some are left to the row gather."""
    from oracle import fgattn_oracle as orc
    capi = _capi()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    B, S, D = 1, 1500, 64
    nb, stride = (S + 127) // 128, 128 * ((S + 127) // 128)
    H = sms // nb + 2
    assert H * nb > sms
    g = torch.Generator().manual_seed(8)
    q, k, v = (torch.randn(B, H, S, D, generator=g).to(torch.bfloat16) for _ in range(3))
    keep = torch.rand(B, H, nb, 1, generator=g)                 # list lengths from a few blocks to all
    blocks = torch.rand(B, H, nb, (S + 63) // 64, generator=g) < keep
    tm = blocks.repeat_interleave(64, dim=-1)[..., :S] & (torch.rand(B, H, nb, S, generator=g) < 0.9)
    tm[:, :, ::5] = torch.rand(B, H, (nb + 4) // 5, S, generator=g) < 0.05
    idx, cnt = _lists_from_mask(tm, stride)
    qc, kc, vc, idxc, cntc = q.cuda(), k.cuda(), v.cuda(), idx.cuda(), cnt.cuda()
    ws = torch.empty(capi.sp_attn_token_workspace_bytes(B, H, S, S), dtype=torch.uint8, device="cuda")
    o, o_g = torch.full_like(qc, float("nan")), torch.full_like(qc, float("nan"))
    capi.set_tuning("token_block_route", 1)
    try:
        capi.sp_attn(o, qc, kc, vc, idxc, cntc, workspace=ws)
        capi.check()
    finally:
        capi.set_tuning("token_block_route", -1)
    taken = _routes(capi, ws, B, H, S)
    assert not taken[:, ::5].any() and taken.float().mean().item() > 0.6
    capi.sp_attn(o_g, qc, kc, vc, idxc, cntc, block_route=False)
    capi.check()
    assert (o.float() - o_g.float()).abs().max().item() <= 1.6e-2
    _close(o[:, :3], orc.sp_attn_tokens(q[:, :3], k[:, :3], v[:, :3], idx[:, :3], cnt[:, :3], 128))


@pytest.mark.parametrize("S,D", [(1, 128), (31, 64), (33, 128), (129, 64), (160, 128), (257, 64), (385, 128)])
def test_output_rows_at_the_edges(S, D):
    """The output leaves from the query tile's own buffer in boxes of 32 rows: sequences that end inside a box, at its
    edge, in either query tile, lists of one step and of several, an empty one.  Nothing past the last row of the last
    head may be written, nothing of a head's rows by the one before it."""
    from oracle import fgattn_oracle as orc
    capi = _capi()
    B, H, K = 1, 3, 700
    g = torch.Generator().manual_seed(S)
    q = torch.randn(B, H, S, D, generator=g).to(torch.bfloat16)
    k, v = (torch.randn(B, H, K, D, generator=g).to(torch.bfloat16) for _ in range(2))
    nb, stride = (S + 127) // 128, 768
    tm = torch.rand(B, H, nb, K, generator=g) < torch.tensor([0.1, 0.9, 0.4])[None, :, None, None]
    tm[0, 2, -1] = False
    idx, cnt = _lists_from_mask(tm, stride)
    n = B * H * S * D
    buf = torch.full((n + 40 * D,), 7.0, device="cuda", dtype=torch.bfloat16)
    o = buf[:n].view(B, H, S, D)
    capi.sp_attn(o, q.cuda(), k.cuda(), v.cuda(), idx.cuda(), cnt.cuda())
    capi.check()
    _close(o, orc.sp_attn_tokens(q, k, v, idx, cnt, 128))
    assert torch.all(buf[n:] == 7.0)


@pytest.mark.parametrize("S,D,n_kv,n_valid,row_bytes", [(256, 128, 1500, 1500, 192), (640, 64, 1500, 1400, 188), (1000, 128, 1500, 9999, 189),
                                                       (128, 64, 33, 33, 5), (300, 128, 9000, 9000, 1125)])
def test_packed_mask_and_shared_tiles(S, D, n_kv, n_valid, row_bytes):
    """sp_attn_packed: keys that both blocks of a pair keep are gathered once, in whole tiles of 128 (packed_pairs_kernel).
    Masks with every kind of overlap, rows of whole and of broken words, bits past the last key and past n_valid, against
    the oracle and against sp_attn on the lists of the same bits."""
    import numpy as np
    import fgattn_tk_cuda_b200.spattn  # noqa: F401  (registers torch.ops.cuda_attn)
    from oracle import fgattn_oracle as orc
    capi = _capi()
    # keys of the first block, of the second, of both
    kinds = [(700, 700, 700), (127, 127, 127), (128, 128, 128), (255, 129, 129), (700, 300, 0), (900, 900, 128), (0, 500, 0),
             (513, 640, 400), (n_kv, n_kv, n_kv), (256, 900, 256), (500, 0, 0), (0, 0, 0), (129, 1, 1)]
    nb = (S + 127) // 128
    pairs = (nb + 1) // 2
    B, H = 1, -(-len(kinds) // pairs)
    g = torch.Generator().manual_seed(S + n_kv)
    q = torch.randn(B, H, S, D, generator=g).to(torch.bfloat16)
    k, v = (torch.randn(B, H, n_kv, D, generator=g).to(torch.bfloat16) for _ in range(2))
    bits = torch.zeros(H * 2 * pairs, 8 * row_bytes, dtype=torch.bool)
    for i in range(H * pairs):
        n0, n1, both = (min(n, n_kv) for n in kinds[i % len(kinds)])
        perm = torch.randperm(n_kv, generator=g)
        bits[2 * i, perm[:n0]] = True
        bits[2 * i + 1, torch.cat([perm[:both], perm[n0:n0 + n1 - both]])] = True
    bits[:, n_kv:] = True
    bits = bits.view(H, 2 * pairs, -1)[:, :nb].contiguous()
    packed = torch.from_numpy(np.packbits(bits.numpy(), axis=-1, bitorder="little")).view(B, H, nb, row_bytes)
    limit = min(n_valid, n_kv)
    stride = 128 * ((n_kv + 127) // 128)
    idx, cnt = _lists_from_mask(bits[None, ..., :limit], stride)
    o, again, lists = (torch.full((B, H, S, D), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(3))
    args = (q.cuda(), k.cuda(), v.cuda())
    torch.ops.cuda_attn.sp_attn_packed(o, *args, packed.cuda(), n_valid)
    torch.ops.cuda_attn.sp_attn_packed(again, *args, packed.cuda(), n_valid)
    torch.ops.cuda_attn.sp_attn(lists, *args, idx.cuda(), cnt.cuda())
    capi.check()
    _close(o, orc.sp_attn_tokens(q, k, v, idx, cnt, 128))
    # the keys' order differs, so does the rounding of the probabilities and of the output: 2^-8 of values up to about 1
    _close(o, lists, 8e-3, 5e-4)
    assert torch.equal(o, again)


def test_packed_mask_of_more_than_a_sweep():
    """Rows of more than 32768 bits (packed_pairs_kernel takes 1024 words a sweep): against sp_attn on the lists."""
    import fgattn_tk_cuda_b200.spattn  # noqa: F401  (registers torch.ops.cuda_attn)
    from fgattn_tk_cuda_b200.spattn import mask_utils as mu
    B, H, S, D, n_kv = 1, 3, 300, 64, 70001
    g = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn(B, H, S, D, generator=g, device="cuda").to(torch.bfloat16)
    k, v = (torch.randn(B, H, n_kv, D, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    common = torch.rand(B, H, 1, 70016, generator=g, device="cuda") < 0.02
    bits = common | (torch.rand(B, H, 3, 70016, generator=g, device="cuda") < 0.005)
    bits[..., 30000:31000] = True
    packed = mu.pack(bits)
    o, lists = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    torch.ops.cuda_attn.sp_attn_packed(o, q, k, v, packed, n_kv)
    idx, cnt = mu.packedmask_to_indexmask_cuda(packed, n_kv)
    torch.ops.cuda_attn.sp_attn(lists, q, k, v, idx, cnt)
    _capi().check()
    _close(o, lists.cpu(), 8e-3, 5e-4)


@pytest.mark.parametrize("D,S", [(128, 256), (64, 200)])
def test_items_of_the_last_wave_in_halves(D, S):
    """A few items more than SMs: the last ones are cut into their query blocks, one thread block each.  The same heads in
    calls of at most an item per SM are not cut: the same bits from lists, the same within rounding from a packed mask
    (a query block alone shares no tiles), rows of a block that keeps nothing and of one past the sequence included."""
    import fgattn_tk_cuda_b200.spattn  # noqa: F401  (registers torch.ops.cuda_attn)
    from fgattn_tk_cuda_b200.spattn import mask_utils as mu
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    H, n_kv, nb = sms + 7, 700, (S + 127) // 128
    g = torch.Generator(device="cuda").manual_seed(S)
    q = torch.randn(1, H, S, D, generator=g, device="cuda").to(torch.bfloat16)
    k, v = (torch.randn(1, H, n_kv, D, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    bits = torch.rand(1, H, 1, 704, generator=g, device="cuda") < torch.rand(1, H, 1, 1, generator=g, device="cuda")
    bits = (bits ^ (torch.rand(1, H, nb, 704, generator=g, device="cuda") < 0.1)).contiguous()
    bits[0, sms + 2, 0] = False
    packed = mu.pack(bits)
    idx, cnt = mu.packedmask_to_indexmask_cuda(packed, n_kv)

    def parts(op, *per_head):
        out = torch.full_like(q, float("nan"))
        for a, b in ((0, sms), (sms, H)):
            o = torch.full_like(q[:, a:b], float("nan")).contiguous()
            op(o, *(t[:, a:b].contiguous() for t in (q, k, v) + per_head))
            out[:, a:b] = o
        return out

    o = torch.full_like(q, float("nan"))
    torch.ops.cuda_attn.sp_attn(o, q, k, v, idx, cnt)
    lists = parts(lambda *a: torch.ops.cuda_attn.sp_attn(*a), idx, cnt)
    assert torch.equal(o, lists)
    o2 = torch.full_like(q, float("nan"))
    torch.ops.cuda_attn.sp_attn_packed(o2, q, k, v, packed, n_kv)
    _close(o2, parts(lambda *a: torch.ops.cuda_attn.sp_attn_packed(*a, n_kv), packed).cpu(), 8e-3, 5e-4)
    _close(o2, lists.cpu(), 8e-3, 5e-4)
    _capi().check()


@pytest.mark.parametrize("H,S,D,n_kv", [(3, 256, 128, 1500), (2, 1000, 64, 4205), (5, 129, 128, 33), (2, 300, 64, 70001)])
def test_packed_mask_gives_the_bits_of_its_lists(H, S, D, n_kv):
    """sp_attn_packed takes a block's keys in ascending order, as the lists of the same bits have them: the same output bit
    for bit (another order rounds other probabilities)."""
    import fgattn_tk_cuda_b200.spattn  # noqa: F401  (registers torch.ops.cuda_attn)
    from fgattn_tk_cuda_b200.spattn import mask_utils as mu
    g = torch.Generator(device="cuda").manual_seed(S + n_kv)
    q = torch.randn(1, H, S, D, generator=g, device="cuda").to(torch.bfloat16)
    k, v = (torch.randn(1, H, n_kv, D, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    width = 32 * ((n_kv + 31) // 32)
    common = torch.rand(1, H, 1, width, generator=g, device="cuda") < 0.2
    bits = common ^ (torch.rand(1, H, (S + 127) // 128, width, generator=g, device="cuda") < 0.1)
    packed = mu.pack(bits)
    o, lists = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    torch.ops.cuda_attn.sp_attn_packed(o, q, k, v, packed, n_kv)
    torch.ops.cuda_attn.sp_attn(lists, q, k, v, *mu.packedmask_to_indexmask_cuda(packed, n_kv))
    _capi().check()
    assert torch.equal(o, lists)


@pytest.mark.parametrize("S,D", [(777, 64), (1408, 128)])
def test_token_steps_give_the_bits_of_the_lists(S, D):
    """The threshold step and the replay of kept bits: bit for bit sp_attn on the ascending lists of their masks."""
    from fgattn_tk_cuda_b200 import synth
    from fgattn_tk_cuda_b200.spattn import mask_utils as mu, sparseattn_functionals as sf
    w = synth.Workload("t", 1, 3, S, D, "clustered", centroids=12, run=64, tau=0.5 / S, seed=S)
    q, k, v = synth.make_qkv(w, device="cuda")
    want = sf._sparse(sf._out(q), q, k, v, mu.qk_indexmask_cuda(q, k, w.tau))
    assert torch.equal(sf.attn_computed_with_sparse_mask_cuda(q, k, v, thresh=w.tau, blocksz=128), want)
    cache = mu.CompressedBitMaskCache([0])
    sf.bitmaskcached_attn_cuda(q, k, v, 0, 0, mask_cache=cache, thresh=w.tau)
    q2 = (q + 0.1 * torch.randn_like(q)).contiguous()
    got = sf.bitmaskcached_attn_cuda(q2, k, v, 0, 1, mask_cache=cache, thresh=w.tau)
    _capi().check()
    assert torch.equal(got, sf._sparse(sf._out(q2), q2, k, v, cache.get_mask_from_cache(0)))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("pos", [40, 200, 290])
def test_nan_and_infinity_of_negligible_keys_reach_the_output(D, pos):
    """A listed key whose probability is tiny but not zero (2^-65 to 2^-92 of the row's largest) beside nothing but such keys:
    NaN in its K row makes the output NaN, an infinity in its V row that column infinite, in the first step of a list
    (entry 40), in a full one (200) and in a ragged last one (290 of 300)."""
    import fgattn_tk_cuda_b200.spattn  # noqa: F401  (registers torch.ops.cuda_attn)
    from fgattn_tk_cuda_b200.spattn import mask_utils as mu
    H, S, n_kv, n = 2, 200, 640, 300
    g = torch.Generator().manual_seed(pos)
    q = torch.zeros(1, H, S, D)
    k = torch.zeros(1, H, n_kv, D)
    q[..., 0], k[..., 0] = 16.0, -16.0
    v = torch.randn(1, H, n_kv, D, generator=g)
    idx = torch.stack([torch.sort(torch.randperm(n_kv, generator=g)[:n]).values for _ in range(H * 2)])
    idx = idx.to(torch.int32).view(1, H, 2, n)
    for h in range(H):
        k[0, h, idx[0, h, :, 5].long(), 0] = 16.0          # entry 5 of either block's list outweighs all others
        k[0, h, idx[0, h, :, pos].long(), 0] = -16.0
    cnt = torch.full((1, H, 2), n, dtype=torch.int32)
    k_nan, v_inf = k.clone(), v.clone()
    for h in range(H):
        k_nan[0, h, idx[0, h, :, pos].long(), 1] = float("nan")
        v_inf[0, h, idx[0, h, :, pos].long(), 3] = float("inf")
    q, k, v, k_nan, v_inf = (x.to(torch.bfloat16).cuda() for x in (q, k, v, k_nan, v_inf))
    idx, cnt = idx.cuda(), cnt.cuda()
    bits = mu.indexmask_to_packedmask_cuda(idx, cnt, n_kv)
    for attend in (lambda o, *a: torch.ops.cuda_attn.sp_attn(o, *a, idx, cnt),
                   lambda o, *a: torch.ops.cuda_attn.sp_attn_packed(o, *a, bits, n_kv)):
        o = torch.zeros_like(q)
        attend(o, q, k_nan, v)
        _capi().check()
        assert torch.isnan(o).all()
        attend(o, q, k, v_inf)
        _capi().check()
        assert torch.isinf(o[..., 3]).all()
        assert torch.isfinite(torch.cat([o[..., :3], o[..., 4:]], -1)).all()
