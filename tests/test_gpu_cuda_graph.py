"""The sparse step can be captured in a CUDA graph and replayed: no entry point synchronises,
allocates with the CUDA allocator or touches the legacy default stream once it has been called once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_block_sparse_step_replays_from_a_cuda_graph():
    import fgattn_tk_cuda_b200.spattn as spattn  # noqa: F401  registers torch.ops.cuda_attn
    from fgattn_tk_cuda_b200 import capi
    mu = spattn.mask_utils
    import dataclasses
    from fgattn_tk_cuda_b200 import synth
    w = dataclasses.replace(synth.WORKLOADS["c3"], H=4, S=4096)      # clustered: a mix of kept / dropped blocks
    q, k, v = synth.make_qkv(w, device="cuda")
    idx, cnt, max_q, denom = mu.qk_block_indexmask_cuda(q, k, w.tau)
    assert 0 < int(cnt.sum()) < idx.numel()
    eager = torch.empty_like(q)
    torch.ops.cuda_attn.sp_attn_blocks_ml(eager, q, k, v, idx, cnt, max_q, denom)      # also the warm-up call
    eager_rn = torch.empty_like(q)
    torch.ops.cuda_attn.sp_attn_blocks(eager_rn, q, k, v, idx, cnt)
    capi.check()

    out = torch.zeros_like(q)
    out_rn = torch.zeros_like(q)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            torch.ops.cuda_attn.sp_attn_blocks_ml(out, q, k, v, idx, cnt, max_q, denom)
            torch.ops.cuda_attn.sp_attn_blocks(out_rn, q, k, v, idx, cnt)
    torch.cuda.current_stream().wait_stream(side)
    for _ in range(3):
        out.zero_()
        out_rn.zero_()
        graph.replay()
    torch.cuda.synchronize()
    capi.check()
    assert torch.equal(out, eager)
    assert torch.equal(out_rn, eager_rn)


def _step(name):
    from fgattn_tk_cuda_b200.spattn import mask_utils as mu, sparseattn_functionals as sf
    if name == "topk":                   # means, scores, selection, order, attention
        return lambda q, k, v: sf.attn_topkmask_cuda(q, k, v, select_k=300, blocksz=128)
    if name == "tokens":                 # pass, threshold, token mask, lists, order, attention
        return lambda q, k, v: sf.attn_computed_with_sparse_mask_cuda(q, k, v, thresh=2e-4, blocksz=128)
    if name == "blocks":                 # pass, threshold, order, attention
        return lambda q, k, v: sf.attn_computed_with_sparse_mask_cuda(q, k, v, thresh=1e-3, blocksz=64)
    if name == "dense":
        return lambda q, k, v: sf.baseline_attn(q, k, v)
    assert name == "kept_bits"           # lists, order, attention
    cache = mu.CompressedBitMaskCache([0])

    def step(q, k, v):
        if not cache.cache:
            sf.bitmaskcached_attn_cuda(q, k, v, 0, 0, mask_cache=cache, thresh=2e-4)
        return sf.bitmaskcached_attn_cuda(q, k, v, 0, 1, mask_cache=cache, thresh=2e-4)
    return step


@pytest.mark.parametrize("H,S,D", [(12, 3400, 128), (9, 4300, 64), (2, 500, 64)])
@pytest.mark.parametrize("name", ["topk", "tokens", "blocks", "kept_bits", "dense"])
def test_chains_of_kernels_back_to_back_and_from_a_graph(name, H, S, D):
    """The kernels of a step start while the ones before them still run.  Steps on changing inputs without a pause between
    them, and replays of a captured step that also joins another stream, give what steps give that are waited for (with
    more pairs of query blocks than SMs, so that the order of the thread blocks is a link of the chain, and with fewer)."""
    from fgattn_tk_cuda_b200 import capi, synth
    step = _step(name)
    sets = [synth.make_qkv(synth.Workload("t", 1, H, S, D, "clustered", centroids=16, run=64, seed=s), device="cuda") for s in (1, 2)]
    want = []
    for x in sets:
        want.append(step(*x))
        torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    got = [step(*sets[i % 2]) for i in range(6)]
    torch.cuda.synchronize()
    capi.check()
    for i, o in enumerate(got):
        assert torch.equal(o, want[i % 2])

    x = [t.clone() for t in sets[0]]
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    dense = _step("dense")
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        step(*x)                                           # workspaces of this stream
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            other.wait_stream(side)
            with torch.cuda.stream(other):
                beside = dense(*x)
            first = step(*x)
            side.wait_stream(other)
            second = step(*x)                              # behind the step and the other stream
        for i in (1, 0, 1, 1):
            for t, new in zip(x, sets[i]):
                t.copy_(new)
            graph.replay()
            side.synchronize()
            assert torch.equal(first, want[i]) and torch.equal(second, want[i])
            assert torch.equal(beside, dense(*sets[i]))
    torch.cuda.synchronize()
    capi.check()
    del first, second, beside
    graph.reset()
