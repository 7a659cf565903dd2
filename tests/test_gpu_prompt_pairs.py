"""The prompt GEMM on pairs of CTAs (csrc/gemm_pair.cuh) through the entry points that run on it, at sizes that fill enough of the chip to take it: its epilogues, weight tiles
of which the second CTA has nothing, walks of several blocks, and last rounds that are cut along k."""
import pytest
import torch

from mistral_inference_b200 import _abi
from mistral_inference_b200.rope import precompute_freqs_cis

pytestmark = pytest.mark.gpu
DEV = "cuda"


def route(T, N, K):
    """The parts that the last round's tiles are cut into, 0: the call does not run on pairs (pairs_fill and cut_plan, for K below 8192)."""
    units = torch.cuda.get_device_properties(0).multi_processor_count // 2
    tiles = -(-T // 256) * -(-N // 256)
    if 2 * tiles < units:
        return 0
    rest = tiles % units
    cut = min(4, units // rest) if rest else 1
    while cut > 1 and ((cut - 1) * rest > 56 or K // 64 < 8 * cut):
        cut -= 1
    return cut


def data(*shapes, seed=0, scale=None):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return [(torch.randn(*s, device=DEV, generator=g) * (1 if i == 0 else s[-1] ** -0.5)).bfloat16() for i, s in enumerate(shapes)]


def workspace(T, K, N):
    return _abi.Workspace(_abi.workspace_bytes(T, K, 32, 8, 128, max(N, 256), N, 1), torch.device(DEV))


def close(got, ref, what=""):
    """bf16 results: within a rounding (2^-8) of the exact sum, beside the fp32 sum's own error where a rounding's edge is near."""
    err = (got.double() - ref).abs()
    assert (err <= 2 ** -8 * ref.abs() + 2 ** -8 * 2 ** -6 * ref.abs().max()).all(), what
    assert (got.double() - ref).norm() < 2 ** -8 * ref.norm(), what


@pytest.mark.parametrize("T,N,K", [(700, 4224, 256), (129, 9600, 64), (700, 6528, 1024), (4200, 2688, 128), (4200, 2432, 1024), (4097, 1280, 2048)])
def test_residual_and_logits(T, N, K):
    """N = 128 (mod 256), one token past a tile, more than 16 token tiles with more than nine of weights (several blocks of the walk), cut last rounds.  In place too."""
    cut = route(T, N, K)
    assert cut >= 1 and (cut > 1) == (K >= 1024)
    x, w, res = data((T, K), (N, K), (T, N), seed=N)
    ws, out, ref = workspace(T, K, N), torch.empty(T, N, dtype=torch.bfloat16, device=DEV), x.double() @ w.double().T
    _abi.linear_residual(x, w, None, out, ws)
    close(out, ref)
    want = out.float() + res.float()
    _abi.linear_residual(x, w, res, res, ws)
    assert torch.equal(res, want.bfloat16())
    nw, logits = torch.ones(K, dtype=torch.bfloat16, device=DEV), torch.empty(T, N, device=DEV)
    if T < 4000:
        _abi.lm_head(x, nw, w, logits, 1e-5, ws)
        close(logits, _abi.rmsnorm(x, nw, 1e-5).double() @ w.double().T)


@pytest.mark.parametrize("T", [513, 700])
def test_the_bits_of_single_ctas(T, monkeypatch):
    """Sums that are not cut run over k in one go on either kernel: projections with rotation and ring, gated units, residual and logits at N = 128 (mod 256)."""
    H, KV, K, N = 31, 1, 256, 4224
    assert route(T, N, K) == 1
    x, w, res = data((T, K), (N, K), (T, N), seed=T)
    nw, ws = torch.rand(K, device=DEV).bfloat16() + 0.5, workspace(T, K, N)
    positions = (torch.arange(T, dtype=torch.int32, device=DEV) * 3) % 500
    rows = torch.tensor([t if t % 5 else -1 for t in range(T)], dtype=torch.int32, device=DEV)
    table, got = torch.view_as_real(precompute_freqs_cis(128, 512, 1e6)).contiguous().to(DEV), []
    for bn in ("", "128"):
        if bn:
            monkeypatch.setenv("MB200_GEMM_BN", bn)
        bf = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device=DEV)  # noqa: E731
        q, k, v, ck, cv, g, out, logits = bf(T, H * 128), bf(T, 128), bf(T, 128), bf(T, KV, 128), bf(T, KV, 128), bf(T, N // 2), bf(T, N), torch.zeros(T, N, device=DEV)
        _abi.attn_qkv(x, nw, w, table, positions, q, k, v, ck, cv, rows, H, KV, 128, 1e-5, ws)
        _abi.ffn_gateup(x, nw, w, g, 1e-5, ws)
        _abi.linear_residual(x, w, res, out, ws)
        _abi.lm_head(x, nw, w, logits, 1e-5, ws)
        got.append((q, k, v, ck, cv, g, out, logits))
    for a, b, what in zip(*got, ("q", "k", "v", "ring keys", "ring values", "gated units", "residual", "logits")):
        assert torch.equal(a, b) and a.any(), what


@pytest.mark.parametrize("T,V,D", [(700, 4224, 128), (700, 6528, 1024), (300, 9600, 128)])
@pytest.mark.parametrize("cols", [None, (64, 96), (96, 128), (0, 64), (-1, 0), (-128, 0), (5, 6), (0, 0)])
@pytest.mark.parametrize("value", ["nan", "-inf"])
def test_scoring(T, V, D, cols, value):
    """Log-probabilities from the epilogue against those of written logits: rows without a target, kept rows, and whole groups of logits that are NaN or -infinity, at
    the seams between the warps that share a group of 64 and in the last, half-empty weight tile."""
    assert route(T, V, D) == (2 if D == 1024 else 1)
    x, w = data((T, D), (V, D), seed=V)
    x = x.abs() + 0.5
    if cols is not None:
        lo, hi = cols[0] % V, cols[1] or V
        w[lo:hi] = float(value)  # x is positive: the logits are NaN or -infinity
    g = torch.Generator(device=DEV).manual_seed(T)
    nw, targets = torch.ones(D, device=DEV, dtype=torch.bfloat16), torch.randint(0, V, (T,), device=DEV, generator=g)
    targets[0], targets[1] = 0, V - 1
    keep, kept_rows = torch.full((T,), -1, dtype=torch.int32, device=DEV), [0, 255, 256, T - 1]
    keep[kept_rows] = torch.tensor([2, 0, 3, 1], dtype=torch.int32, device=DEV)
    ws = workspace(T, D, V)
    logits, ref, got, kept = torch.empty(T, V, device=DEV), torch.zeros(T, device=DEV), torch.zeros(T, device=DEV), torch.empty(4, V, device=DEV)
    _abi.lm_head(x, nw, w, logits, 1e-5, ws)
    _abi.logprob_gather(logits, targets, out=ref)
    none = torch.tensor([7, 300 % T, T - 1], device=DEV)
    targets[none] = -1
    ref[none] = 0
    _abi.lm_head_logprobs(x, nw, w, targets, keep, kept, got, 1e-5, ws)
    assert torch.equal(kept[[2, 0, 3, 1]].nan_to_num(9e9), logits[kept_rows].nan_to_num(9e9))
    if cols is not None and value == "nan":
        assert torch.isnan(ref[targets >= 0]).all()
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.isinf(got), torch.isinf(ref))
    ok = torch.isfinite(ref)
    # the logits are the same bf16 numbers; their exponentials are summed in another order: V 2^-24 of the sum at most, as a difference of logarithms, beside its own rounding
    assert (got - ref)[ok].abs().max() <= V * 2 ** -24 + 2 ** -22 * ref[ok].abs().max() if ok.any() else True
