"""Prompt kernels of layered decoders against float64 statements, at the sizes where their tiles, plans and masks change."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel(got, ref):
    return ((got.double() - ref).norm() / ref.norm()).item()


def _unit(kind, z, w, limit, alpha):
    if kind == "relu2":
        return z.clamp(min=0) ** 2 * w
    g, u = z[:, 0::2], z[:, 1::2]
    if kind == "glu":  # the weight is on the expert's input
        g, u = (g * w).clamp(max=limit), (u * w).clamp(-limit, limit)
        return g * torch.sigmoid(alpha * g) * (u + 1)
    return (torch.nn.functional.silu(g) if kind == "silu" else torch.nn.functional.gelu(g, approximate="tanh")) * u * w


@pytest.mark.parametrize("kind", ["silu", "gelu", "glu", "relu2"])
@pytest.mark.parametrize("T,width,ff,E,top,idle", [(1, 128, 64, 1, 1, 0), (17, 128, 64, 5, 2, 2), (129, 384, 192, 3, 3, 0), (300, 256, 128, 48, 6, 5), (1100, 128, 128, 2, 2, 1)])
def test_chosen_expert_rows(kind, T, width, ff, E, top, idle, monkeypatch):
    """The grouped form of a mixture: experts nobody chose, choices that name no expert (>= E), segments around the 128-row tile, pairs of tiles
    (the last shape: from 384 rows per expert on), more tokens than one call takes.  The hidden units' three bf16 roundings (gate, up, result;
    2^-9 each) bound the relative error by 3 * 2^-9."""
    from mistral_inference_b200 import _abi, _abi_hybrid as h

    if kind == "relu2" and ff % 128:
        ff = 128
    g = torch.Generator().manual_seed(T)
    units = ff if kind == "relu2" else 2 * ff
    hn = torch.randn(T, width, generator=g).bfloat16().to(DEV)
    w13 = (torch.randn(E * units, width, generator=g) / width ** 0.5).bfloat16().to(DEV)
    w2 = (torch.randn(width, E * ff, generator=g) / ff ** 0.5).bfloat16().to(DEV)
    idx = torch.stack([torch.randperm(E + idle, generator=g)[:top] for _ in range(T)]).int()
    if E > 2:
        idx[idx == 1] = E + idle  # nobody has expert 1
    wts = torch.rand(T, top, generator=g).to(DEV) + 0.1
    base = torch.randn(T, width, generator=g).to(DEV)
    epi = {"silu": h.EPI_SWIGLU, "gelu": h.EPI_GEGLU, "glu": h.EPI_GLU, "relu2": h.EPI_RELU2}[kind]
    ref = torch.zeros(T, width, dtype=torch.float64, device=DEV)
    for e in range(E):
        t, j = torch.nonzero(idx.to(DEV) == e, as_tuple=True)
        z = hn[t].double() @ w13[e * units:(e + 1) * units].double().T
        act = _unit(kind, z, wts[t, j].double()[:, None], 1.5, 1.7)
        ref.index_add_(0, t, act @ w2[:, e * ff:(e + 1) * ff].double().T)
    assert h.moe_grouped_ok(hn, w13, w2, E, ff)
    got = h.moe_grouped(hn, w13, w2, idx.to(DEV), wts, E, ff, epi, 1.5, 1.7)
    assert rel(got, ref) < 3 * 2 ** -9
    monkeypatch.setattr(_abi, "LAYER_MOE_MAX_TOKENS", 100)
    acc = base.clone()
    h.moe_grouped(hn, w13, w2, idx.to(DEV), wts, E, ff, epi, 1.5, 1.7, add_to=acc)
    assert torch.equal(acc, base + got), "blocks of tokens and the sum into a stream change nothing"
