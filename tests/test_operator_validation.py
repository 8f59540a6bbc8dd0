"""Shape and dtype validation of the torch operators, on meta tensors (no GPU needed): the Meta
kernel of every operator is the same check that its CUDA kernel runs first, so a wrong-shaped tensor
is an error before anything reaches the device."""
import pytest
import torch

import fgattn_tk_cuda_b200.spattn  # noqa: F401  (registers torch.ops.cuda_attn)

ops = torch.ops.cuda_attn
B, H, S, D, SKV = 2, 3, 300, 64, 200
NQB, NKB, NQB128, SPAD = 5, 4, 3, 384


def t(*shape, dtype=torch.bfloat16):
    return torch.empty(*shape, dtype=dtype, device="meta")


def good():
    return dict(q=t(B, H, S, D), k=t(B, H, SKV, D), v=t(B, H, SKV, D), o=t(B, H, S, D),
                m=t(B, H, 1, SPAD, dtype=torch.float32), l=t(B, H, 1, SPAD, dtype=torch.float32),
                kb=t(B, H, NQB, NKB, dtype=torch.int32), kc=t(B, H, NQB, dtype=torch.int32),
                ti=t(B, H, NQB128, 256, dtype=torch.int32), tc=t(B, H, NQB128, dtype=torch.int32),
                mask=t(B, H, NQB128, 256, dtype=torch.int32), scratch=t(1024, dtype=torch.float32))


CALLS = {
    "full_attn": lambda a: ops.full_attn(a["o"], a["q"], a["k"], a["v"]),
    "fullattn_maxq_denom": lambda a: ops.fullattn_maxq_denom(a["o"], a["m"], a["l"], a["q"], a["k"], a["v"]),
    "maxq_denom": lambda a: ops.maxq_denom(a["m"], a["l"], a["q"], a["k"]),
    "sp_attn": lambda a: ops.sp_attn(a["o"], a["q"], a["k"], a["v"], a["ti"], a["tc"]),
    "booleanmask_128": lambda a: ops.booleanmask_128(a["mask"], a["m"], a["l"], a["q"], a["k"], 1e-3),
    "booleanmask_128_listed": lambda a: ops.booleanmask_128_listed(a["mask"], a["m"], a["l"], a["q"], a["k"], 1e-3,
                                                                   a["kb"], a["kc"]),
    "booleanmask_to_indexmask": lambda a: ops.booleanmask_to_indexmask(a["ti"], a["tc"], a["mask"], SKV),
    "block_index_lists": lambda a: ops.block_index_lists(a["kb"], a["kc"], a["m"], a["l"], a["o"], a["q"], a["k"],
                                                         a["v"], 1e-3, a["scratch"]),
    "sp_attn_blocks_ml": lambda a: ops.sp_attn_blocks_ml(a["o"], a["q"], a["k"], a["v"], a["kb"], a["kc"], a["m"], a["l"]),
    "sp_attn_blocks": lambda a: ops.sp_attn_blocks(a["o"], a["q"], a["k"], a["v"], a["kb"], a["kc"]),
    "sp_attn_blocks_hint": lambda a: ops.sp_attn_blocks_hint(a["o"], a["q"], a["k"], a["v"], a["kb"], a["kc"], a["m"]),
}

# (operators that take the tensor, replacement that must be refused)
BAD = [
    ("k", t(B, H + 1, SKV, D), None),                             # heads differ from q
    ("k", t(B, H, SKV, 128), None),                               # head dimension differs from q
    ("k", t(B, H, SKV, D, dtype=torch.float16), None),            # dtype
    ("v", t(B, H, SKV - 8, D), None),                             # fewer rows than k
    ("o", t(B, H, S - 1, D), None),                               # not the shape of q
    ("m", t(B, H, 1, S, dtype=torch.float32), None),              # [B,H,1,S] instead of the padded length
    ("l", t(B, H, 1, SPAD, dtype=torch.float16), None),           # dtype
    ("kb", t(B, H, NQB - 1, NKB, dtype=torch.int32), None),       # rows != ceil(S/64)
    ("kb", t(B, H, NQB, NKB - 1, dtype=torch.int32), None),       # stride < number of key blocks
    ("kc", t(B, H, NQB - 1, dtype=torch.int32), None),
    ("ti", t(B, H, NQB128 + 1, 256, dtype=torch.int32), None),    # rows != ceil(S/128)
    ("tc", t(B, H, NQB128 + 2, dtype=torch.int32), None),
    ("mask", t(B, H, NQB128, SKV - 8, dtype=torch.int32), None),  # narrower than the key sequence
    ("mask", t(B, H - 1, NQB128, 256, dtype=torch.int32), None),
]
USES = {
    "full_attn": "qkvo", "fullattn_maxq_denom": ("q", "k", "v", "o", "m", "l"), "maxq_denom": ("q", "k", "m", "l"),
    "sp_attn": ("q", "k", "v", "o", "ti", "tc"), "booleanmask_128": ("q", "k", "m", "l", "mask"),
    "booleanmask_128_listed": ("q", "k", "m", "l", "mask", "kb", "kc"),
    "booleanmask_to_indexmask": ("ti", "tc", "mask"),
    "block_index_lists": ("q", "k", "v", "o", "m", "l", "kb", "kc"),
    "sp_attn_blocks_ml": ("q", "k", "v", "o", "m", "l", "kb", "kc"),
    "sp_attn_blocks": ("q", "k", "v", "o", "kb", "kc"), "sp_attn_blocks_hint": ("q", "k", "v", "o", "m", "kb", "kc"),
}


@pytest.mark.parametrize("name", sorted(CALLS))
def test_well_formed_arguments_pass(name):
    assert CALLS[name](good()) is None


@pytest.mark.parametrize("name", sorted(CALLS))
def test_every_wrong_shape_is_refused(name):
    n = 0
    for key, bad, _ in BAD:
        if key not in USES[name]:
            continue
        if name == "booleanmask_to_indexmask" and key == "mask":
            continue                                  # there the mask defines the shapes; covered below
        args = good()
        args[key] = bad
        with pytest.raises(RuntimeError):
            CALLS[name](args)
        n += 1
    assert n >= 2


def test_compaction_and_packed_mask_shapes():
    a = good()
    with pytest.raises(RuntimeError):
        ops.booleanmask_to_indexmask(t(B, H, NQB128, 128, dtype=torch.int32), a["tc"], a["mask"], SKV)
    with pytest.raises(RuntimeError):
        ops.pack_mask(t(B, 5, dtype=torch.uint8), t(B, 48, dtype=torch.int32))
    assert ops.pack_mask(t(B, 6, dtype=torch.uint8), t(B, 48, dtype=torch.int32)) is None
    with pytest.raises(RuntimeError):
        ops.all_index_mask(a["ti"], a["tc"], B, H, NQB128 + 1, S)
    with pytest.raises(RuntimeError):
        ops.topk_indices(t(B, H, NQB128, 64, dtype=torch.int32), a["tc"], a["q"], a["k"], 100, 128)   # stride < select_k
    assert ops.topk_indices(t(B, H, NQB128, 128, dtype=torch.int32), a["tc"], a["q"], a["k"], 100, 128) is None


def test_noalloc_wrapper_refuses_k_of_another_length():
    """fgattn_block_index_lists_noalloc has no kv_rows argument: the Python layer must not let a k / v of
    another length through (it would be read past its end, or at the wrong per-head stride)."""
    from fgattn_tk_cuda_b200 import capi
    q = torch.zeros(1, 1, 128, 64, dtype=torch.bfloat16)
    k_short = torch.zeros(1, 1, 64, 64, dtype=torch.bfloat16)
    i32 = torch.zeros(1, 1, 2, 2, dtype=torch.int32)
    f32 = torch.zeros(1, 1, 1, 128)
    with pytest.raises(capi.FgattnError, match="shape of q"):
        capi.block_index_lists_noalloc(i32, i32, f32, f32, q, k_short, 1e-3)
    with pytest.raises(capi.FgattnError, match="shape of q"):
        capi.block_index_lists_noalloc(i32, i32, f32, f32, q, q, 1e-3, o=q, v=k_short)


def _bit_cache(seq_len):
    from fgattn_tk_cuda_b200.spattn import mask_utils
    cache = mask_utils.CompressedBitMaskCache([0])
    cache.cache[0] = (t(B, H, NQB128, 256 // 8, dtype=torch.uint8), seq_len)
    return cache


def _replay(cache):
    from fgattn_tk_cuda_b200.spattn import sparseattn_functionals as functionals
    a = good()
    return functionals.bitmaskcached_attn_cuda(a["q"], a["k"], a["v"], 0, 1, mask_cache=cache, thresh=1e-3)


@pytest.mark.parametrize("seq_len", [None, 0, SKV, 256])
def test_kept_bits_of_any_valid_length(seq_len):
    """A kept bit mask whose length is None counts in full width, as packedmask_to_indexmask_cuda takes it."""
    assert _replay(_bit_cache(seq_len)).shape == (B, H, S, D)
    assert _bit_cache(seq_len).get_lists(0)[0].shape == (B, H, NQB128, 256)


def test_replaced_reading_of_a_kept_mask_is_called(monkeypatch):
    """A program's own get_mask_from_cache is the one that an attention step reads, whether it sits on the object, in a
    subclass or in place of the class's."""
    from fgattn_tk_cuda_b200.spattn import mask_utils
    calls = []

    def own(*layer):
        calls.append(layer[-1])
        return good()["ti"], good()["tc"]

    cache = _bit_cache(SKV)
    cache.get_mask_from_cache = own
    _replay(cache)

    class Sub(mask_utils.CompressedBitMaskCache):
        get_mask_from_cache = own

    sub = Sub([0])
    sub.cache = _bit_cache(SKV).cache
    _replay(sub)
    monkeypatch.setattr(mask_utils.CompressedBitMaskCache, "get_mask_from_cache", own)
    _replay(_bit_cache(SKV))
    assert calls == [0, 0, 0]


def _added(name, **change):
    a = dict(good(), packed=t(B, H, NQB128, 28, dtype=torch.uint8), n_valid=SKV, select=100, blocksz=128, tau=1e-3)
    a.update(change)
    if name == "sp_attn_packed":
        return ops.sp_attn_packed(a["o"], a["q"], a["k"], a["v"], a["packed"], a["n_valid"])
    if name == "topk_packed":
        return ops.topk_packed(a["packed"], a["q"], a["k"], a["select"], a["blocksz"])
    return ops.attn_block_mask(a["o"], a["q"], a["k"], a["v"], a["tau"])


_QKV_BAD = [dict(k=t(B, H + 1, SKV, D)), dict(k=t(B, H, SKV, 128)), dict(q=t(B, H, S, 96)), dict(k=t(B, H, 0, D)),
            dict(q=t(B, H, S, D, dtype=torch.float16))]
_VO_BAD = [dict(v=t(B, H, SKV - 8, D)), dict(o=t(B, H, S - 1, D)), dict(o=t(B, H, S, D, dtype=torch.float32))]
_PACKED_BAD = [dict(packed=t(B, H, NQB128 + 1, 28, dtype=torch.uint8)), dict(packed=t(B, H, NQB128, 28, dtype=torch.int32)),
               dict(packed=t(B * H, NQB128, 28, dtype=torch.uint8)), dict(packed=t(B, H, NQB128, 56, dtype=torch.uint8)[..., ::2])]


@pytest.mark.parametrize("name,bad", [("attn_block_mask", _QKV_BAD + _VO_BAD + [dict(tau=0.0), dict(tau=-1.0)]),
                                      ("sp_attn_packed", _QKV_BAD + _VO_BAD + _PACKED_BAD + [dict(n_valid=-1)]),
                                      ("topk_packed", _QKV_BAD + _PACKED_BAD + [
                                          dict(packed=t(B, H, NQB128, 24, dtype=torch.uint8)),        # fewer bits than keys
                                          dict(packed=t(B, H, NQB128, 26, dtype=torch.uint8)),        # not whole words
                                          dict(select=0), dict(select=SKV + 1), dict(blocksz=0), dict(blocksz=64)])])
def test_operators_on_bits_and_in_one_call_refuse_wrong_arguments(name, bad):
    assert _added(name) is None
    for change in bad:
        with pytest.raises(RuntimeError):
            _added(name, **change)


def test_replaced_lists_of_a_kept_mask_are_read(monkeypatch):
    """A step goes by the kept bits only as long as nothing that hands out their lists has been replaced."""
    from fgattn_tk_cuda_b200.spattn import mask_utils
    calls = []

    def own(*layer):
        calls.append(layer[-1])
        return good()["ti"], good()["tc"]

    plain = _bit_cache(SKV)
    assert plain.reads_bits()
    on_object, reader = _bit_cache(SKV), _bit_cache(SKV)
    on_object.get_lists = own
    reader.list_reader = lambda: own

    class Sub(mask_utils.CompressedBitMaskCache):
        get_lists = own

    sub = Sub([0])
    sub.cache = plain.cache
    for cache in (on_object, reader, sub):
        assert not cache.reads_bits()
        _replay(cache)
    monkeypatch.setattr(mask_utils.CompressedBitMaskCache, "get_lists", own)
    assert not plain.reads_bits()
    _replay(plain)
    assert calls == [0, 0, 0, 0]
