"""GPU parity (bit-exact) of the one-bit-per-entry mask kernels and of the caches built on them."""
import numpy as np
import pytest
import torch

from helpers import GOLDEN

pytestmark = pytest.mark.gpu


def _capi():
    from fgattn_tk_cuda_b200 import capi
    return capi


def test_pack_unpack_golden_fixture():
    """pack / unpack / compressed-cache lists against vectors made by the reference
    (python/spattn/mask_utils.py:421-440, :89-93)."""
    capi = _capi()
    z = np.load(GOLDEN / "packed_2x3x5x136.npz")
    for src in (torch.from_numpy(z["mask"]), torch.from_numpy(z["mask"].astype(np.uint8)),
                torch.from_numpy(z["mask"].astype(np.int32) * 5)):
        packed = torch.full(z["packed"].shape, 0xAA, dtype=torch.uint8, device="cuda")
        capi.pack_mask(packed, src.cuda())
        assert np.array_equal(packed.cpu().numpy(), z["packed"])
    for dt in (torch.bool, torch.uint8, torch.int32):
        mask = torch.empty(z["mask"].shape, dtype=dt, device="cuda")
        capi.unpack_mask(mask, torch.from_numpy(z["packed"]).cuda())
        assert np.array_equal(mask.cpu().numpy().astype(bool), z["mask"])
        assert int(mask.to(torch.int32).max()) == 1
    idx = torch.full(z["index"].shape, -1, dtype=torch.int32, device="cuda")
    cnt = torch.full(z["count"].shape, -1, dtype=torch.int32, device="cuda")
    capi.packedmask_to_indexmask(idx, cnt, torch.from_numpy(z["packed"]).cuda(), 136)
    assert np.array_equal(idx.cpu().numpy(), z["index"]) and np.array_equal(cnt.cpu().numpy(), z["count"])
    back = torch.full(z["packed"].shape, 0x55, dtype=torch.uint8, device="cuda")
    capi.indexmask_to_packedmask(back, idx, cnt)
    assert np.array_equal(back.cpu().numpy(), z["packed"])


@pytest.mark.parametrize("rows,width,dens", [(7, 8, 0.5), (3, 40, 0.3), (5, 4096, 0.08), (2, 75648, 0.02),
                                              (4, 1024, 0.0), (4, 1024, 1.0), (300, 256, 0.15)])
def test_pack_unpack_roundtrip(rows, width, dens):
    from oracle import fgattn_oracle as orc
    capi = _capi()
    g = torch.Generator().manual_seed(rows * 131 + width)
    mask = torch.rand(rows, width, generator=g) < dens
    packed = torch.empty(rows, width // 8, dtype=torch.uint8, device="cuda")
    capi.pack_mask(packed, (mask.to(torch.int32) * 7).cuda())
    assert np.array_equal(packed.cpu().numpy(), orc.pack_mask(mask))
    out = torch.empty(rows, width, dtype=torch.int32, device="cuda")
    capi.unpack_mask(out, packed)
    assert torch.equal(out.cpu(), mask.to(torch.int32))


@pytest.mark.parametrize("rows,width,stride,n_valid,dens", [(6, 384, 384, 384, 0.3), (5, 1280, 1280, 1201, 0.05),
                                                             (3, 40, 40, 33, 0.5), (2, 32768, 32768, 32760, 0.1),
                                                             (4, 256, 256, 256, 0.0), (4, 256, 256, 256, 1.0),
                                                             (9, 264, 260, 257, 0.4), (2, 75648, 75648, 75600, 0.03)])
def test_packed_to_index_and_back(rows, width, stride, n_valid, dens):
    from oracle import fgattn_oracle as orc
    capi = _capi()
    g = torch.Generator().manual_seed(width + rows)
    mask = torch.rand(rows, width, generator=g) < dens
    packed_np = orc.pack_mask(mask)
    packed = torch.from_numpy(packed_np).cuda()
    idx = torch.full((rows, stride), -1, dtype=torch.int32, device="cuda")
    cnt = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    capi.packedmask_to_indexmask(idx, cnt, packed, n_valid)
    ridx, rcnt = orc.packedmask_to_indexmask(packed_np, n_valid=n_valid, stride=stride)
    assert np.array_equal(cnt.cpu().numpy(), rcnt) and np.array_equal(idx.cpu().numpy(), ridx)
    # lists -> bits reproduces the live part of the mask
    back = torch.full((rows, 4 * ((width + 31) // 32)), 0xFF, dtype=torch.uint8, device="cuda")
    capi.indexmask_to_packedmask(back, idx, cnt)
    assert np.array_equal(back.cpu().numpy(), orc.indexmask_to_packedmask(ridx, rcnt, width))
    live = mask.clone()
    live[:, n_valid:] = False
    assert np.array_equal(orc.unpack_mask(back.cpu().numpy())[:, :width], live.numpy())


def test_argument_checks():
    capi = _capi()
    packed = torch.empty(4, 5, dtype=torch.uint8, device="cuda")
    with pytest.raises(capi.FgattnError):
        capi.pack_mask(packed, torch.zeros(4, 40, dtype=torch.float32, device="cuda"))   # dtype
    with pytest.raises(capi.FgattnError):
        capi.pack_mask(packed, torch.zeros(4, 44, dtype=torch.int32, device="cuda"))     # width % 8


def test_compressed_caches_match_plain_caches():
    """CompressedBitMaskCache / CompressedListCache hand back exactly the lists the uncompressed
    caches do (python/spattn/mask_utils.py:70-98)."""
    from fgattn_tk_cuda_b200.spattn import mask_utils as mu
    g = torch.Generator().manual_seed(5)
    B, H, SB, W, S = 1, 3, 4, 512, 500
    mask = ((torch.rand(B, H, SB, W, generator=g) < 0.1).to(torch.int32) * 3).cuda()
    plain, comp = mu.BitMaskCache([0]), mu.CompressedBitMaskCache([0])
    plain.update_cache(0, mask, S)
    comp.update_cache(0, mask, S)
    assert comp.cache[0][0].numel() * 8 == mask.numel()             # one bit per entry instead of 32
    (i0, c0), (i1, c1) = plain.get_mask_from_cache(0), comp.get_mask_from_cache(0)
    assert torch.equal(i0, i1) and torch.equal(c0, c1)
    # block lists: 37 key blocks, list stride 37
    nqb = nkb = 37
    bm = torch.rand(2, 2, nqb, nkb, generator=g) < 0.2
    from oracle import fgattn_oracle as orc
    ridx, rcnt = orc.bitmask_to_indexmask(bm)
    lc = mu.CompressedListCache([0])
    lc.update_cache(3, ridx.cuda(), rcnt.cuda(), nkb)
    i2, c2 = lc.get_mask_from_cache(3)
    assert torch.equal(i2.cpu(), ridx) and torch.equal(c2.cpu(), rcnt)


def test_cached_attention_flow_block_mode():
    """cached_attn_cuda (python/spattn/sparseattn_functionals.py:95-113) in the 64x64 mode: the run that
    builds the mask returns dense attention; a later run with DIFFERENT q / k reuses the cached
    lists and must renormalise over the kept blocks (oracle: softmax restricted to kept keys)."""
    from fgattn_tk_cuda_b200 import synth
    from fgattn_tk_cuda_b200.spattn import mask_utils as mu, sparseattn_functionals as sf
    from oracle import fgattn_oracle as orc
    from helpers import OUT_MAX_ABS, OUT_MEAN_ABS
    w = synth.Workload("t", 1, 2, 1024, 128, "clustered", centroids=16, run=128, tau=1e-4, seed=77)
    q, k, v = synth.make_qkv(w, device="cuda")
    for cache in (mu.NaiveMaskCache([0]), mu.CompressedListCache([0])):
        o0 = sf.cached_attn_cuda(q, k, v, 0, 0, thresh=w.tau, blocksz=64, mask_cache=cache)
        ref0 = orc.full_attn(q.cpu(), k.cpu(), v.cpu())
        assert (o0.float().cpu() - ref0).abs().max() < OUT_MAX_ABS
        q2 = (q.float() * 1.05 + 0.02).to(torch.bfloat16)
        o1 = sf.cached_attn_cuda(q2, k, v, 0, 1, thresh=w.tau, blocksz=64, mask_cache=cache)
        idx, cnt = cache.get_mask_from_cache(0)[:2]
        ref1 = orc.sp_attn_blocks(q2.cpu(), k.cpu(), v.cpu(), idx.cpu(), cnt.cpu())
        d = (o1.float().cpu() - ref1).abs()
        assert d.max() < OUT_MAX_ABS and d.mean() < OUT_MEAN_ABS


@pytest.mark.parametrize("S,K,D", [(1024, 1024, 128), (900, 900, 64), (700, 1500, 128), (130, 97, 64), (1, 33, 128)])
def test_token_lists_by_way_of_bits(S, K, D):
    """The threshold test that writes one bit per entry gives the int mask's bits (same comparison, so the same bits),
    the lists built from them are those of the int mask, and the lists for the attention operators have the same
    entries and counts and leave the slots behind a count alone."""
    import torch
    from fgattn_tk_cuda_b200 import capi, synth
    from fgattn_tk_cuda_b200.spattn import mask_utils as mu
    w = synth.Workload("t", 1, 3, max(S, K), D, "clustered", centroids=12, run=96, tau=2e-3, seed=S + K)
    q, k, _ = synth.make_qkv(w, device="cuda")
    q, k = q[:, :, :S].contiguous(), k[:, :, :K].contiguous()
    mask = mu.qk_token_mask_cuda(q, k, w.tau)[0]
    packed = mu._qk_packed_token_mask(q, k, w.tau)
    assert torch.equal(packed, mu.pack(mask))
    idx, cnt = mu.bitmask_to_indexmask_cuda(mask, K)
    got_idx, got_cnt = mu.qk_indexmask_cuda(q, k, w.tau, blocksz=128)
    assert torch.equal(got_idx, idx) and torch.equal(got_cnt, cnt)
    lists, num = torch.full_like(idx, -7), torch.empty_like(cnt)
    torch.ops.cuda_attn.packedmask_to_lists(lists, num, packed, K)
    capi.check()
    used = torch.arange(idx.shape[-1], device="cuda") < cnt[..., None]
    assert torch.equal(num, cnt) and torch.equal(lists[used], idx[used]) and (lists[~used] == -7).all()


@pytest.mark.parametrize("width,stride,n_valid", [(32768, 32768, 32760), (33000, 9000, 33000), (1096, 1096, 1090), (40, 40, 39)])
@pytest.mark.parametrize("kind", ["runs", "scattered", "mixed", "one per word", "one word"])
def test_packed_to_lists_of_runs_and_scattered_bits(kind, width, stride, n_valid):
    """A warp writes its entries by words or by bits, whichever takes fewer trips: masks that go one way, the other way
    and both ways in one row, lists that the entries overflow, and rows that are no whole number of words."""
    from oracle import fgattn_oracle as orc
    capi = _capi()
    rows = 7
    g = torch.Generator().manual_seed(width + len(kind))
    runs = (torch.rand(rows, width // 8, generator=g) < 0.4).repeat_interleave(8, 1)
    runs[:, width // 3: width // 2] = True
    scattered = torch.rand(rows, width, generator=g) < torch.linspace(0, 0.3, rows)[:, None]
    mask = {"runs": runs, "scattered": scattered, "mixed": torch.where(torch.arange(width) // 700 % 2 == 0, runs, scattered),
            "one per word": (torch.arange(width) % 32 == torch.arange(rows)[:, None] * 5).contiguous(),
            "one word": (torch.arange(width) // 32 == torch.arange(rows)[:, None]).contiguous()}[kind]
    packed_np = orc.pack_mask(mask)
    packed = torch.from_numpy(packed_np).cuda()
    ridx, rcnt = orc.packedmask_to_indexmask(packed_np, n_valid=n_valid, stride=stride)
    idx = torch.full((rows, stride), -1, dtype=torch.int32, device="cuda")
    cnt = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    capi.packedmask_to_indexmask(idx, cnt, packed, n_valid)
    assert np.array_equal(cnt.cpu().numpy(), rcnt) and np.array_equal(idx.cpu().numpy(), ridx)
    import fgattn_tk_cuda_b200.spattn  # noqa: F401  (registers torch.ops.cuda_attn)
    lists, num = torch.full_like(idx, -7), torch.full_like(cnt, -7)
    torch.ops.cuda_attn.packedmask_to_lists(lists, num, packed, n_valid)
    capi.check()
    used = np.arange(stride)[None, :] < rcnt[:, None]
    got = lists.cpu().numpy()
    assert np.array_equal(num.cpu().numpy(), rcnt) and np.array_equal(got[used], ridx[used]) and (got[~used] == -7).all()
