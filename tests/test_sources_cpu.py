"""Properties of the CUDA sources that no run on one GPU can show."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "mistral_inference_b200" / "csrc"


@pytest.mark.parametrize("path", sorted(CSRC.rglob("*.cu*")), ids=lambda p: p.name)
def test_no_copy_is_multicast_to_a_cluster(path):
    """Processes of a pipeline or of an expert-parallel group run the same kernels as a single one, with other GPUs' memory mapped: every bulk
    copy goes to the one CTA that asked for it (tcgen05.commit, a signal and no copy, may reach both CTAs of a pair)."""
    text = re.sub(r'"\s*\n\s*"', "", path.read_text())  # adjacent string literals are one instruction
    copies = re.findall(r'"[^"\n]*cp\.async\.bulk[^"\n]*"', text)
    assert not [c for c in copies if "multicast" in c]
    assert path.name != "gemm_tcgen05.cuh" or len(copies) >= 3


WEIGHTS = {"w", "w2", "E", "gate_w", "sink"}  # parameters that only loading a model writes


@pytest.mark.parametrize("files", ["*.cu*", "hybrid/*.cu*"])
def test_what_a_predecessor_writes_is_no_read_only_parameter(files):
    """Kernels launched programmatically are resident while their predecessor still writes what they will read.  `const __restrict__` promises that nobody
    does, and lets the compiler read it through the read-only path, or before the wait: only weights may be declared so."""
    text = "\n".join(re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.glob(files)))
    params = dict(re.findall(r"__global__[^;{]*?\b(\w+)\(((?:[^(){}]|\([^()]*\))*)\)\s*\{", text))
    launched = set(re.findall(r"\blaunch_(?:pdl|pairs)\(\s*(\w+)", text)) & set(params)
    assert len(launched) >= 9, launched
    read_only = {k: set(re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params[k])) - WEIGHTS for k in launched}
    assert not {k: v for k, v in read_only.items() if v}


@pytest.mark.parametrize("name,start,wait", [("hybrid/hybrid_linear_f32.cuh", "linear_f32_pair(const", "ft_bar_wait("), ("stream_linear.cuh", "stream_linear_kernel(const", "bar_wait("),
                                             ("stream_tiles.cuh", "stream_tiles_kernel(const", "mbar_wait("), ("gemm_streamk.cuh", "void sk_gemm_body(const", "mbar_wait(")])
def test_limits_of_waits_count_from_the_predecessors_end(name, start, wait):
    """A kernel launched programmatically may be resident for as long as its predecessors run.  Its waits are bounded, and none of its barriers completes before the predecessor has
    ended, so every role waits for that end before its first barrier: else a long predecessor uses the limit up."""
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    body = text[text.index(start):]
    body = body[:body.index("\n}\n")]
    roles = [r for r in re.split(r'\n {2,4}(?:if \(warp|\} else|\}\n(?= +asm volatile\("griddepcontrol\.wait))', body) if wait in r]
    assert len(roles) >= 2
    for role in roles:
        ends = [i for i in (role.find("pdl_wait()"), role.find("griddepcontrol.wait")) if i >= 0]
        assert ends and min(ends) < role.index(wait), role[:300]
