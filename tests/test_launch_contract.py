"""Kernels that may start while the one in front of them still runs (launch_behind: programmatic dependent launch) wait
for it before they touch memory, and promise the compiler nothing about that memory.  Read off the sources, no GPU needed."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "fgattn_tk_cuda_b200" / "csrc"


def _kernels():
    """name -> (parameters, body) of every kernel."""
    found = {}
    for path in sorted(CSRC.glob("*.cuh")):
        text = path.read_text()
        for m in re.finditer(r"__global__ void(?: __launch_bounds__\((?:[^()]|\([^()]*\))*\))?\s+(\w+)\(([^{]*)\)\s*\{", text):
            end = text.find("\n}", m.end())
            found[m.group(1)] = (m.group(2), text[m.end():end])
    return found


def _launched_behind():
    """Kernels that launch_behind is called with: by name, or as `kern` of the function around the call."""
    text = (CSRC / "fgattn_capi.cu").read_text()
    names = set(re.findall(r"launch_behind\(fg::(\w+)", text))
    for function in re.split(r"\n\}\n", text):
        if "launch_behind(kern" in function:
            names.update(re.findall(r"(?:go\(|kern = )fg::(\w+_kernel)", function))
            names.update(re.findall(r": (?:go\()?fg::(\w+_kernel)", function))
    return names


def test_kernels_launched_behind_wait_first():
    kernels, behind = _kernels(), _launched_behind()
    assert {"dense_attn_kernel", "maxq_pass_kernel", "sparse_ml_persistent_kernel", "sparse_token_attn_kernel",
            "sparse_block_attn_kernel", "topk_scores_kernel", "topk_select_kernel", "sparse_order_kernel"} <= behind
    for name in sorted(behind):
        assert "grid_wait();" in kernels[name][1], name


def test_kernels_that_wait_promise_nothing_about_memory():
    waiting = {name: k for name, k in _kernels().items() if "grid_wait();" in k[1]}
    assert len(waiting) >= 10
    for name, (params, body) in waiting.items():
        assert "__restrict__" not in params, name
        assert "__ldg" not in body and "ld.global.nc" not in body, name
