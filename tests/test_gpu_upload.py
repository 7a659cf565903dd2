"""Prompt metadata on its way to the GPU."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 500, 16384, 16385, 300_000])
def test_upload_takes_its_copy_and_pins_nothing(n):
    """The host may reuse its memory at once, also behind a busy stream, and a first call of a size allocates no pinned memory."""
    from mistral_inference_b200.cache import upload

    d = torch.device("cuda")
    a = torch.randn(4096, 4096, device=d, dtype=torch.bfloat16)
    upload(torch.zeros(3), d)
    pinned = dict(torch.cuda.host_memory_stats())
    kept, got = [], []
    for i in range(4):
        for _ in range(8):
            torch.mm(a, a)
        host = torch.arange(i, i + n, dtype=torch.int32)
        kept.append(host.clone())
        got.append(upload(host, d))
        host.fill_(-1)
        del host
    assert all(torch.equal(g.cpu(), k) for g, k in zip(got, kept))
    assert dict(torch.cuda.host_memory_stats()) == pinned
