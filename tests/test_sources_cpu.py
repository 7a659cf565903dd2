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
