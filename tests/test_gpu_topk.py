"""GPU parity of the top-k key selector (python/spattn/mask_utils.py:389-417 of the reference)."""
import numpy as np
import pytest
import torch

from helpers import GOLDEN, OUT_MAX_ABS, OUT_MEAN_ABS

pytestmark = pytest.mark.gpu

# Scores are fp32 sums of 64..128 products on both sides but in different orders, so two keys whose
# scores differ by less than this (relative to the score scale) may swap places.
SCORE_TOL = 2e-5


def _capi():
    from fgattn_tk_cuda_b200 import capi
    return capi


def _check_lists(idx, cnt, scores, select_k, n_valid):
    """idx [R, stride], cnt [R] from the GPU against fp32 oracle scores [R, n]: exactly select_k
    distinct valid keys; every listed key scores at least the oracle's k-th largest minus the
    tolerance and every unlisted one at most that plus the tolerance; listed in descending order."""
    R = scores.shape[0]
    assert (cnt == select_k).all()
    tol = SCORE_TOL * max(1.0, float(scores.abs().max()))
    kth = torch.sort(scores, dim=-1, descending=True).values[:, select_k - 1]
    for r in range(R):
        sel = idx[r, :select_k].long()
        assert sel.min() >= 0 and sel.max() < n_valid
        assert sel.unique().numel() == select_k
        s_sel = scores[r, sel]
        assert (s_sel >= kth[r] - tol).all()
        rest = torch.ones(scores.shape[1], dtype=torch.bool)
        rest[sel] = False
        assert (scores[r, rest] <= kth[r] + tol).all()
        assert (s_sel[1:] <= s_sel[:-1] + tol).all()
        assert (idx[r, select_k:] == idx.shape[1]).all()


def test_topk_golden_fixture():
    """The fixture made by the reference (ragged last query block); random normal inputs have no
    near-ties at this size, so the lists must match index for index."""
    capi = _capi()
    z = np.load(GOLDEN / "topk_s300_d64_k40.npz")
    q = torch.from_numpy(z["q_bf16"]).view(torch.bfloat16).cuda()
    k = torch.from_numpy(z["k_bf16"]).view(torch.bfloat16).cuda()
    K = int(z["select_k"])
    idx = torch.full((1, 2, 3, 128), -1, dtype=torch.int32, device="cuda")
    cnt = torch.full((1, 2, 3), -1, dtype=torch.int32, device="cuda")
    capi.topk_indices(idx, cnt, q, k, K, blocksz=128)
    capi.check()
    assert np.array_equal(cnt.cpu().numpy(), z["count"])
    assert np.array_equal(idx[..., :K].cpu().numpy(), z["index"])
    assert (idx[..., K:] == 128).all()


@pytest.mark.parametrize("B,H,S,D,blocksz,select_k,kv", [(1, 2, 1024, 128, 128, 100, None), (2, 1, 777, 64, 128, 64, None),
                                                        (1, 1, 2048, 128, 64, 1, None), (1, 2, 1500, 128, 128, 1500, None),
                                                        (1, 1, 4096, 64, 128, 3000, 4000), (1, 3, 640, 128, 256, 333, 600)])
def test_topk_vs_oracle(B, H, S, D, blocksz, select_k, kv):
    from oracle import fgattn_oracle as orc
    capi = _capi()
    g = torch.Generator().manual_seed(S + select_k)
    q = torch.randn(B, H, S, D, generator=g).to(torch.bfloat16)
    k = torch.randn(B, H, S, D, generator=g).to(torch.bfloat16)
    nblk = (S + blocksz - 1) // blocksz
    stride = 128 * ((select_k + 127) // 128)
    idx = torch.full((B, H, nblk, stride), -1, dtype=torch.int32, device="cuda")
    cnt = torch.full((B, H, nblk), -1, dtype=torch.int32, device="cuda")
    capi.topk_indices(idx, cnt, q.cuda(), k.cuda(), select_k, blocksz=blocksz, kv_seq_len=kv)
    capi.check()
    sc = orc.topk_scores(q, k, blocksz, kv_seq_len=kv)
    _check_lists(idx.cpu().view(-1, stride), cnt.cpu().view(-1), sc.reshape(-1, sc.shape[-1]), select_k, kv or S)


def test_topk_ties_take_the_smallest_indices():
    """All keys equal: every score ties, so the list is 0 .. select_k-1 in order."""
    capi = _capi()
    B, H, S, D, K = 1, 1, 512, 64, 37
    q = torch.randn(B, H, S, D).to(torch.bfloat16).cuda()
    k = torch.ones(B, H, S, D, dtype=torch.bfloat16, device="cuda")
    idx = torch.empty(B, H, 4, 128, dtype=torch.int32, device="cuda")
    cnt = torch.empty(B, H, 4, dtype=torch.int32, device="cuda")
    capi.topk_indices(idx, cnt, q, k, K, blocksz=128)
    capi.check()
    assert torch.equal(idx[..., :K].cpu(), torch.arange(K, dtype=torch.int32).expand(B, H, 4, K))


def test_topk_attention_flow():
    """attn_topkmask_cuda (python/spattn/sparseattn_functionals.py:39-48): top-k lists into the
    token-list sparse kernel; select_k = S keeps every key, i.e. dense attention."""
    from fgattn_tk_cuda_b200.spattn import sparseattn_functionals as sf, mask_utils as mu
    from oracle import fgattn_oracle as orc
    g = torch.Generator().manual_seed(3)
    B, H, S, D = 1, 2, 640, 128
    q, k, v = (torch.randn(B, H, S, D, generator=g).to(torch.bfloat16).cuda() for _ in range(3))
    o = sf.attn_topkmask_cuda(q, k, v, 0, 0, select_k=200, blocksz=128)
    idx, cnt = mu.qk_topkmask_indices(q, k, 200, blocksz=128)
    ref = orc.sp_attn_tokens(q.cpu(), k.cpu(), v.cpu(), idx.cpu(), cnt.cpu(), 128)
    d = (o.float().cpu() - ref).abs()
    assert d.max() < OUT_MAX_ABS and d.mean() < OUT_MEAN_ABS
    o_all = sf.attn_topkmask_cuda(q, k, v, 0, 0, select_k=None, blocksz=128)
    d = (o_all.float().cpu() - orc.full_attn(q.cpu(), k.cpu(), v.cpu())).abs()
    assert d.max() < OUT_MAX_ABS and d.mean() < OUT_MEAN_ABS


def test_topk_argument_checks():
    capi = _capi()
    q = torch.zeros(1, 1, 256, 64, dtype=torch.bfloat16, device="cuda")
    idx = torch.empty(1, 1, 2, 128, dtype=torch.int32, device="cuda")
    cnt = torch.empty(1, 1, 2, dtype=torch.int32, device="cuda")
    for bad_k in (0, 257, 129):                      # none, more than the keys, more than the list stride
        with pytest.raises(capi.FgattnError):
            capi.topk_indices(idx, cnt, q, q, bad_k)


@pytest.mark.parametrize("kind", ["spread", "outlier", "steps", "both_signs", "small"])
@pytest.mark.parametrize("select_k", [3, 700, 4096, 8192])
def test_topk_order_of_any_distribution(kind, select_k):
    """The selected scores are put in order by counting where they spread over the bins and by the sort where they
    pile up: one key far above the rest, a few distinct values with many equal scores, scores on both sides of zero,
    and scores in so small a range that the bin width has no inverse (by the sort).  Equal scores: smaller key first."""
    capi = _capi()
    S, D = 8320, 64
    g = torch.Generator().manual_seed(select_k)
    f = torch.randn(S, generator=g)
    if kind == "outlier":
        f[4321] = 3e4
    elif kind == "steps":
        f = torch.floor(2 * f)
    elif kind == "both_signs":
        f = f.sign() * torch.exp2(12 * torch.rand(S, generator=g) - 12)
    elif kind == "small":
        f = 1e-30 * f
    q = torch.zeros(1, 1, 128, D, dtype=torch.bfloat16)
    q[..., 0] = 1.0
    k = torch.zeros(1, 1, S, D, dtype=torch.bfloat16)
    k[0, 0, :, 0] = f.to(torch.bfloat16)
    stride = 128 * ((select_k + 127) // 128)
    idx = torch.full((1, 1, 1, stride), -1, dtype=torch.int32, device="cuda")
    cnt = torch.full((1, 1, 1), -1, dtype=torch.int32, device="cuda")
    capi.topk_indices(idx, cnt, q.cuda(), k.cuda(), select_k, blocksz=128, scale=1.0)
    capi.check()
    # the scores are the first components themselves, exactly, so the list is the stable descending order
    want = torch.sort(k[0, 0, :, 0].float(), descending=True, stable=True).indices[:select_k]
    assert torch.equal(idx[0, 0, 0, :select_k].cpu().long(), want)
    assert (idx[0, 0, 0, select_k:] == stride).all() and int(cnt) == select_k


def _list_of_scores(f, scale_1, select_k, q0=1.0):
    """The top-k list of one query block whose score of key i is q0 * f[i, 0] + scale_1 * f[i, 1], exactly."""
    capi = _capi()
    S, D = f.shape[0], 64
    q = torch.zeros(1, 1, 128, D)
    q[..., 0], q[..., 1] = q0, scale_1
    k = torch.zeros(1, 1, S, D)
    k[0, 0, :, :2] = f
    q, k = q.to(torch.bfloat16), k.to(torch.bfloat16)
    assert torch.equal(k[0, 0, :, :2].float(), f)
    stride = 128 * ((select_k + 127) // 128)
    idx = torch.full((1, 1, 1, stride), -1, dtype=torch.int32, device="cuda")
    cnt = torch.full((1, 1, 1), -1, dtype=torch.int32, device="cuda")
    capi.topk_indices(idx, cnt, q.cuda(), k.cuda(), select_k, blocksz=128, scale=1.0)
    capi.check()
    assert (idx[0, 0, 0, select_k:] == stride).all() and int(cnt) == select_k
    return idx[0, 0, 0, :select_k].cpu().long()


@pytest.mark.parametrize("select_k", [5, 33, 600, 5000])
def test_topk_order_of_scores_a_few_ulps_apart(select_k):
    """256 + n ulps, n in -256 .. 255: the range of the bins is 2^-14 of the scores, and 12 scores or so are equal each."""
    S = 6200
    n = torch.randint(-256, 256, (S,), generator=torch.Generator().manual_seed(select_k)).float()
    got = _list_of_scores(torch.stack([torch.full((S,), 256.0), n], 1), 2.0 ** -15, select_k)
    want = torch.sort(256.0 + n * 2.0 ** -15, descending=True, stable=True).indices[:select_k]
    assert torch.equal(got, want)


@pytest.mark.parametrize("pile", [63, 64, 65, 300])
@pytest.mark.parametrize("S", [700, 2000])
def test_topk_order_with_a_bin_at_its_limit(S, pile):
    """Whole numbers from 0 to 2047 have a bin each (2047 over the range is one), and one of them occurs `pile` times:
    counting takes 64 in a bin, the sort the rest.  Every key is selected, so that no other rule cuts the range."""
    g = torch.Generator().manual_seed(S + pile)
    x = torch.randperm(2046, generator=g)[: S - 2 - pile] + 1
    x = torch.cat([torch.tensor([0, 2047]), x, torch.full((pile,), int(x[7]))])[torch.randperm(S, generator=g)]
    got = _list_of_scores(torch.stack([x - x % 8, x % 8], 1).float(), 1.0, S)
    assert torch.equal(got, torch.sort(x, descending=True, stable=True).indices)


@pytest.mark.parametrize("k_to", [2, 16, 32, 64, 128, 256, 1024, 8192])
@pytest.mark.parametrize("less", [0, 1])
def test_topk_sort_of_every_size(k_to, less):
    """Two values only, so that every selection ends in the sort: list lengths that fill its power of two or fall one
    short of it, from less than a warp's group to the longest."""
    select_k = max(1, k_to - less)
    g = torch.Generator().manual_seed(k_to)
    x = (torch.rand(9000, generator=g) < 0.4).float()
    got = _list_of_scores(torch.stack([x, torch.zeros_like(x)], 1), 0.0, select_k)
    assert torch.equal(got, torch.sort(x, descending=True, stable=True).indices[:select_k])


@pytest.mark.parametrize("select_k", [4, 500, 1990, 2000])
def test_topk_order_with_infinite_scores(select_k):
    """Scores that overflow to infinity on either side, a few or half of them, and finite ones between (select_k up to
    all of them: the range of the bins is then infinite on both sides)."""
    S = 2000
    g = torch.Generator().manual_seed(select_k)
    x = torch.randn(S, generator=g).to(torch.bfloat16).float()
    x[torch.randperm(S, generator=g)[:7]] = 2.0 ** 127
    x[torch.randperm(S, generator=g)[:9]] = -2.0 ** 127
    got = _list_of_scores(torch.stack([x, torch.zeros_like(x)], 1), 0.0, select_k, q0=4.0)
    want = torch.sort(4.0 * x, descending=True, stable=True).indices[:select_k]
    assert torch.equal(got, want)


@pytest.mark.parametrize("select_k", [4, 500, 2000])
def test_topk_with_nan_scores(select_k):
    """NaN scores have no order, but the list stays one of distinct keys, with the others in descending order."""
    S = 2000
    x = torch.randn(S, generator=torch.Generator().manual_seed(select_k)).to(torch.bfloat16).float()
    bad = torch.zeros(S, dtype=torch.bool)
    bad[::97] = True
    k = torch.zeros(1, 1, S, 64)
    k[0, 0, :, 0] = torch.where(bad, torch.tensor(float("nan")), x)
    q = torch.zeros(1, 1, 128, 64)
    q[..., 0] = 1.0
    idx = torch.full((1, 1, 1, 2048), -1, dtype=torch.int32, device="cuda")
    cnt = torch.full((1, 1, 1), -1, dtype=torch.int32, device="cuda")
    capi = _capi()
    capi.topk_indices(idx, cnt, q.to(torch.bfloat16).cuda(), k.to(torch.bfloat16).cuda(), select_k, blocksz=128, scale=1.0)
    capi.check()
    got = idx[0, 0, 0, :select_k].cpu().long()
    assert got.min() >= 0 and got.max() < S and got.unique().numel() == select_k and int(cnt) == select_k
    numbers = got[~bad[got]]
    want = torch.sort(torch.where(bad, torch.tensor(float("-inf")), x), descending=True, stable=True).indices
    assert torch.equal(numbers, want[: numbers.numel()])


@pytest.mark.parametrize("kind", ["normal", "runs", "unlike_its_sample", "steps", "outlier", "nan"])
@pytest.mark.parametrize("S,select_k", [(2000, 1), (3001, 300), (20000, 2000), (20001, 3900), (33000, 8192)])
def test_topk_as_bits(kind, S, select_k):
    """topk_packed sets the bits of the keys that topk_indices lists, whether the threshold comes from a sample of the row
    (16 of every 128 bytes), from the general way because the sample was unlike the row, or from the sort."""
    import fgattn_tk_cuda_b200.spattn  # noqa: F401  (registers torch.ops.cuda_attn)
    capi = _capi()
    g = torch.Generator().manual_seed(S + select_k)
    B, H, rows, D = 1, 2, 300, 64
    f = torch.randn(H, S, generator=g)
    if kind == "runs":
        f = 0.3 * f + 3 * torch.randn(H, S // 250 + 1, generator=g).repeat_interleave(250, 1)[:, :S]
    elif kind == "unlike_its_sample":
        f[:, torch.arange(S) % 32 < 4] += 20
    elif kind == "steps":
        f = torch.floor(2 * f)
    elif kind == "outlier":
        f[:, S // 3] = 3e4
    elif kind == "nan":
        f[:, S // 2] = float("nan")
    q = torch.randn(B, H, rows, D, generator=g)
    q[..., 0] = 2.0
    k = 0.05 * torch.randn(B, H, S, D, generator=g)
    k[0, :, :, 0] = f
    q, k = q.to(torch.bfloat16).cuda(), k.to(torch.bfloat16).cuda()
    stride = 128 * ((select_k + 127) // 128)
    idx = torch.full((B, H, 3, stride), -1, dtype=torch.int32, device="cuda")
    cnt = torch.full((B, H, 3), -1, dtype=torch.int32, device="cuda")
    capi.topk_indices(idx, cnt, q, k, select_k, blocksz=128)
    words = (S + 31) // 32 + 1
    packed = torch.full((B, H, 3, 4 * words), 0xA5, dtype=torch.uint8, device="cuda")
    torch.ops.cuda_attn.topk_packed(packed, q, k, select_k, 128)
    capi.check()
    want = torch.zeros(B * H * 3, 32 * words, dtype=torch.bool)
    want.scatter_(1, idx.view(B * H * 3, stride)[:, :select_k].cpu().long(), True)
    assert (want.sum(1) == select_k).all()
    got = torch.zeros_like(want, dtype=torch.uint8).cuda()
    capi.unpack_mask(got, packed.view(B * H * 3, 4 * words))
    assert torch.equal(got.cpu().bool(), want)


@pytest.mark.parametrize("S,D,select_k", [(2000, 128, 200), (5001, 64, 600), (3000, 128, 1500)])
def test_topk_attention_takes_keys_by_score(S, D, select_k):
    """attn_topkmask_cuda attends to the keys in descending order of their scores, as topk_indices lists them: bit for bit
    what sp_attn gives on those lists.  (Another order rounds the probability that weighs most: a larger error.)"""
    from fgattn_tk_cuda_b200 import synth
    from fgattn_tk_cuda_b200.spattn import mask_utils as mu, sparseattn_functionals as sf
    q, k, v = synth.make_qkv(synth.Workload("t", 1, 3, S, D, "clustered", centroids=16, run=64, seed=S), device="cuda")
    o = sf.attn_topkmask_cuda(q, k, v, select_k=select_k, blocksz=128)
    idx, cnt = mu.qk_topkmask_indices(q, k, select_k)
    want = torch.empty_like(o)
    torch.ops.cuda_attn.sp_attn(want, q, k, v, idx, cnt)
    # the same keys in ascending order are not the same bits, or this test would show nothing
    by_key = torch.empty_like(o)
    ascending = torch.cat([idx[..., :select_k].sort(-1).values, idx[..., select_k:]], -1).contiguous()
    torch.ops.cuda_attn.sp_attn(by_key, q, k, v, ascending, cnt)
    _capi().check()
    assert torch.equal(o, want)
    assert not torch.equal(by_key, want)


@pytest.mark.parametrize("kind", ["above", "below", "outliers", "outlier_in_sample", "infinite", "piled"])
@pytest.mark.parametrize("S,select_k", [(31, 7), (32, 5), (100, 20), (4097, 100), (20001, 2000), (20000, 3300), (33000, 8192)])
def test_topk_of_rows_unlike_their_sample(kind, S, select_k):
    """Scores whose sample (four of every 32, at a place that changes) lies above or below the rest, or holds all or none
    of a few scores far above the others, and scores that pile up just under the largest: every way from the sample to the list."""
    g = torch.Generator().manual_seed(S + select_k)
    x = torch.randn(S, generator=g).to(torch.bfloat16).float()
    i = torch.arange(S)
    sampled = (i // 4 % 8 == (i // 32 * 0x9E3779B1 % (1 << 32)) >> 29) & (i < S // 32 * 32)
    if kind == "above":
        x[sampled] += 16
    elif kind == "below":
        x[sampled] -= 16
    elif kind in ("outliers", "infinite"):
        x[torch.nonzero(~sampled).flatten()[:: max(1, S // 20)][:20]] = 2.0 ** (60 if kind == "outliers" else 127)
    elif kind == "outlier_in_sample":
        x[torch.nonzero(sampled).flatten()[:1]] = 2.0 ** 60
    else:
        x[torch.rand(S, generator=g) < 0.9 * select_k / S] = 2.5
        x[torch.nonzero(sampled).flatten()[:3]] = 64.0
    x = x.to(torch.bfloat16).float()
    got = _list_of_scores(torch.stack([x, torch.zeros_like(x)], 1), 0.0, select_k, q0=4.0)
    assert torch.equal(got, torch.sort(4.0 * x, descending=True, stable=True).indices[:select_k])


def test_topk_as_bits_refuses_rows_beside_which_the_selection_has_no_room():
    """A row's bits are put together in shared memory beside the selected entries: 8 * (1.25 k + 64) + row bytes <= 200 KiB."""
    import fgattn_tk_cuda_b200.spattn  # noqa: F401  (registers torch.ops.cuda_attn)
    g = torch.Generator(device="cuda").manual_seed(1)
    q = torch.randn(1, 1, 128, 64, generator=g, device="cuda").to(torch.bfloat16)
    k = torch.randn(1, 1, 9000, 64, generator=g, device="cuda").to(torch.bfloat16)
    room = 200 * 1024 - 8 * (10240 + 64)
    with pytest.raises(RuntimeError, match="topk_packed failed"):
        torch.ops.cuda_attn.topk_packed(torch.zeros(1, 1, 1, room + 4, dtype=torch.uint8, device="cuda"), q, k, 8192, 128)
    packed = torch.full((1, 1, 1, room), 0xA5, dtype=torch.uint8, device="cuda")
    torch.ops.cuda_attn.topk_packed(packed, q, k, 8192, 128)
    _capi().check()
    bits = torch.zeros(1, 8 * room, dtype=torch.uint8, device="cuda")
    _capi().unpack_mask(bits, packed.view(1, room))
    assert int(bits.sum()) == 8192 and int(bits[:, 9000:].sum()) == 0
