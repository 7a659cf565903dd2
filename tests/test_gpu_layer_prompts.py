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
@pytest.mark.parametrize("T,width,ff,E,top,idle", [(1, 128, 64, 1, 1, 0), (17, 128, 64, 5, 2, 2), (129, 384, 192, 3, 3, 0), (300, 256, 128, 48, 6, 5), (1100, 128, 128, 2, 2, 1), (450, 256, 128, 1, 1, 0), (2100, 256, 128, 2, 1, 0)])
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


@pytest.mark.parametrize("E,identity,T", [(16, 4, 1030), (40, 8, 700), (3, 1, 129)])
def test_identity_choices_of_grouped_experts(E, identity, T):
    """Choices from E on are the token itself times the choice's weight, summed with the experts; without the flag they count nothing.  More than 32
    experts: the plan's second round of lanes."""
    from mistral_inference_b200 import _abi_hybrid as h

    width, ff, top = 256, 128, min(4, E)
    g = torch.Generator().manual_seed(E)
    hn = torch.randn(T, width, generator=g).bfloat16().to(DEV)
    w13 = (torch.randn(2 * E * ff, width, generator=g) / width ** 0.5).bfloat16().to(DEV)
    w2 = (torch.randn(width, E * ff, generator=g) / ff ** 0.5).bfloat16().to(DEV)
    idx = torch.stack([torch.randperm(E + identity, generator=g)[:top] for _ in range(T)]).int().to(DEV)
    wts = torch.rand(T, top, generator=g).to(DEV) + 0.1
    base = torch.randn(T, width, generator=g).to(DEV)
    plain = h.moe_grouped(hn, w13, w2, idx, wts, E, ff, h.EPI_SWIGLU)
    got = h.moe_grouped(hn, w13, w2, idx, wts, E, ff, h.EPI_SWIGLU, add_to=base.clone(), identity=True)
    own = torch.where(idx >= E, wts, 0.0).double().sum(1, keepdim=True)
    ref = base.double() + plain.double() + own * hn.double()
    assert rel(got, ref) < 2e-7  # a handful of fp32 additions
    ref = torch.zeros(T, width, dtype=torch.float64, device=DEV)
    for e in range(E):
        t, j = torch.nonzero(idx == e, as_tuple=True)
        ref.index_add_(0, t, _unit("silu", hn[t].double() @ w13[2 * e * ff:2 * (e + 1) * ff].double().T, wts[t, j].double()[:, None], 0, 0) @ w2[:, e * ff:(e + 1) * ff].double().T)
    assert rel(plain, ref) < 3 * 2 ** -9


def _route64(x, w, corr, groups, keep, top, score, scale=1.0, renorm=False, group_two=False, w_bias=None):
    """(weights [T, n], 0 where not chosen) in float64, and by how much the closest decision was made."""
    z = x.double() @ w.double().T
    if score == 2:
        z = z + w_bias.double()
        v, i = z.topk(top, 1)
        return torch.zeros_like(z).scatter(1, i, torch.softmax(v, 1) * scale), i
    s = torch.softmax(z, 1) if score == 0 else torch.sigmoid(z)
    c = s + (corr.double() if corr is not None else 0)
    if groups > 1 and keep < groups:
        g = c.view(c.shape[0], groups, -1)
        g = g.topk(2, 2).values.sum(2) if group_two else g.max(2).values
        ok = torch.zeros_like(g, dtype=torch.bool).scatter(1, g.topk(keep, 1).indices, True)
        c = c.masked_fill(~ok.repeat_interleave(c.shape[1] // groups, 1), -float("inf"))
    i = c.topk(top, 1).indices
    v = s.gather(1, i)
    if renorm:
        v = v / (v.sum(1, keepdim=True) + 1e-20)
    return torch.zeros_like(z).scatter(1, i, v * scale), i


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("width", [328, 42, 2052])  # no whole number of steps; no whole 16-byte pieces; fp32 rows of more than 8 KB
@pytest.mark.parametrize("n,groups,keep,top,kw", [(20, 4, 2, 4, dict(score=0)), (8, 1, 1, 2, dict(score=1, scale=2.5, renorm=True)), (33, 3, 2, 5, dict(score=1, group_two=True)),
                                                  (32, 16, 3, 4, dict(score=1, group_two=True)), (16, 1, 1, 3, dict(score=2, always=1)), (7, 1, 1, 7, dict(score=0, gate=True))])
def test_routers_of_prompts_and_of_few_tokens(n, groups, keep, top, kw, dt, width):
    """For many tokens a CTA routes four, below one, in fp32 with more loads in flight or with more CTAs (593 to 740 tokens): every sum in the same order, so the same
    bits; up to 32 outputs are chosen from in registers, more in shared memory.  Against float64: fp32 sums of `width` products, the choices where they are not
    closer than that."""
    from mistral_inference_b200 import _abi_hybrid as h

    T = 1201  # the last CTA has one token
    kw = dict(kw)
    g = torch.Generator().manual_seed(n)
    r = lambda *s: torch.randn(*s, generator=g).to(dt).to(DEV)  # noqa: E731
    x, w, corr = r(T, width), r(n, width) * (5 / width) ** 0.5, r(n) / 10 if kw["score"] != 2 else None
    if kw.pop("gate", False):
        kw["w_gate"] = r(1, width) / 8
    if kw["score"] == 2:
        kw["w_bias"] = r(n)
    whole = h.moe_route(x, w, corr, groups, keep, top, **kw)
    for step in (205, 640):
        parts = [h.moe_route(x[i:i + step], w, corr, groups, keep, top, **kw) for i in range(0, T, step)]
        for a, b in zip(whole, zip(*parts)):
            assert torch.equal(a, torch.cat(b))
    always, gate = kw.pop("always", 0), kw.pop("w_gate", None)
    ref, choice = _route64(x, w, corr, groups, keep, top, **kw)
    dense, idx, wsel = whole[:3]
    same = (idx[:, :top].long().sort(1).values == choice.sort(1).values).all(1)
    assert same.float().mean() > 0.995, "choices differ only where two outputs are as good as equal"
    assert rel(dense[same, :n], ref[same]) < 1e-5
    assert torch.equal(dense[:, n:], torch.ones_like(dense[:, n:])) and (idx[:, top:] == n).all() and dense.shape[1] == n + always
    assert torch.equal(dense.gather(1, idx.long()), wsel)
    if gate is not None:
        assert rel(whole[3], torch.sigmoid(x.double() @ gate.double().T)) < 1e-5


@pytest.mark.parametrize("n", [32, 36])
@pytest.mark.parametrize("T", [3, 701])
def test_groups_one_rounding_apart(n, T):
    """The better of two groups is kept when their scores are neighbouring numbers, whichever comes first: up to 32 outputs (in registers) and more (in shared
    memory)."""
    from mistral_inference_b200 import _abi_hybrid as h

    x, w = torch.randn(T, 64, device=DEV), torch.zeros(n, 64, device=DEV)  # every score is 1/2
    for low in (0, 1, 6):
        for lo, hi in ((1, 5), (5, 1), (0, 7)):
            corr = torch.full((n,), -0.25, device=DEV)
            corr[4 * lo + 1], corr[4 * hi + 2] = low * 2.0 ** -24, (low + 1) * 2.0 ** -24
            _, idx, _ = h.moe_route(x, w, corr, n // 4, 1, 2, score=1)
            assert (idx == torch.tensor([4 * hi + 2, 4 * hi], dtype=torch.int32, device=DEV)).all(), (low, lo, hi)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("form", ["plain", "bias", "window", "chunked", "cap_sink", "gate", "own"])
@pytest.mark.parametrize("lens,past", [([33], [0]), ([1, 64, 31, 90], [5, 0, 40, 3]), ([32, 65], [130, 0])])
def test_fp32_attention_of_prompts(d, form, lens, past):
    """Tiles of 32 queries and 32 keys in fp32 against float64, and against the kernel of one CTA per token and head, than which they may not be less exact than by
    fp32's own rounding.  A token's infinities in keys and values reach no query that does not see it."""
    from mistral_inference_b200 import _abi_hybrid as h

    H, G, W, B = 4, 2, 256, len(lens)
    g = torch.Generator().manual_seed(sum(lens) + d)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)  # noqa: E731
    T = sum(lens)
    q, ring_k, ring_v = r(T, H * d), r(B + 1, W, G, d), r(B + 1, W, G, d)
    slots = torch.tensor([B - b for b in range(B)], dtype=torch.int32, device=DEV)
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    positions = torch.tensor([p + i for n, p in zip(lens, past) for i in range(n)], dtype=torch.int32, device=DEV)
    q_start, seqpos = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in (starts, past))
    scale, window, kw, bias = d ** -0.5, 0, {}, None
    if form == "bias":
        bias = r(20, H)
    elif form == "window":
        window = 37
    elif form == "chunked":
        window, kw = 48, dict(chunked=True)
    elif form == "cap_sink":
        kw = dict(softcap=2.0, sink=r(H))
    elif form == "gate":
        kw = dict(gate=r(T, H * d), gate_entry=True)
    elif form == "own":
        kw = dict(own_k=r(T, G * d), own_v=r(T, G * d), seqpos=seqpos)
    ring_k[slots[0].long(), past[0] + lens[0] - 1] = float("inf")  # the first sequence's last token
    ring_v[slots[0].long(), past[0] + lens[0] - 1] = float("nan")

    def run(tiles):
        out = torch.empty(T, H * d, device=DEV)
        if form == "bias":
            h.attn_bias(q, ring_k, ring_v, bias, positions, q_start, slots, out, B, W, H, G, d, d, scale, n_tiles=tiles)
        else:
            h.attn_window(q, ring_k, ring_v, positions, q_start, slots, out, B, W, H, G, d, d, scale, window, n_tiles=tiles, **kw)
        return out

    got, old = run(sum((n + 63) // 64 for n in lens)), run(0)
    ref = torch.empty(T, H * d, dtype=torch.float64, device=DEV)
    for b in range(B):
        for i in range(lens[b]):
            t, p = starts[b] + i, past[b] + i
            lo = 0 if not window else (p - p % window if kw.get("chunked") else max(0, p - window + 1))
            k, v = (c[slots[b].long(), lo:p + 1].double() for c in (ring_k, ring_v))
            if form == "own":
                m = past[b] - lo
                k = torch.cat([k[:m], kw["own_k"][starts[b]:t + 1].view(-1, G, d).double()])
                v = torch.cat([v[:m], kw["own_v"][starts[b]:t + 1].view(-1, G, d).double()])
            s = torch.einsum("hd,khd->hk", q[t].view(H, d).double(), k.repeat_interleave(H // G, 1)) * scale
            if form == "cap_sink":
                s = torch.cat([2 * torch.tanh(s / 2), kw["sink"].double()[:, None]], 1)
            if bias is not None:
                s = s + bias.double()[(p - torch.arange(lo, p + 1, device=DEV)).clamp(max=19)].T
            w = torch.softmax(s, 1)[:, :k.shape[0]]
            o = torch.einsum("hk,khd->hd", w, v.repeat_interleave(H // G, 1)).flatten()
            ref[t] = o * torch.sigmoid(kw["gate"][t].double()) if form == "gate" else o
    fine = torch.ones(T, dtype=torch.bool, device=DEV)
    fine[starts[1] - 1] = form == "own"  # (own rows: the ring's are not read)
    assert torch.isfinite(got[fine]).all()
    assert rel(got[fine], ref[fine]) < max(1.5 * rel(old[fine], ref[fine]), 3e-7)
    assert not torch.isfinite(got[~fine]).any() or form == "cap_sink"


@pytest.mark.parametrize("lens,past,H", [([16], [900], 4), ([24, 1], [500, 30], 8), ([17, 33], [600, 0], 8)])
def test_fp32_attention_of_few_rows_over_many_keys(lens, past, H):
    """Below 400 rows (tokens and heads) over more than 400 keys every row has a CTA of its own, from there on tiles of 32 queries: both against float64."""
    from mistral_inference_b200 import _abi_hybrid as h

    G, d, W, B = 2, 128, 1024, len(lens)
    g = torch.Generator().manual_seed(H)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)  # noqa: E731
    T, bias = sum(lens), r(30, H)
    q, ring_k, ring_v = r(T, H * d), r(B, W, G, d), r(B, W, G, d)
    dev = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    starts = [sum(lens[:b]) for b in range(B + 1)]
    positions = [p + i for n, p in zip(lens, past) for i in range(n)]
    assert h.f32_rows_alone(T * H, W) == (T * H < 400)
    for splits in (1, 2):
        out = torch.empty(T, H * d, device=DEV)
        h.attn_bias(q, ring_k, ring_v, bias, dev(positions), dev(starts), dev(range(B)), out, B, W, H, G, d, d, d ** -0.5, n_tiles=B, splits=splits)
        for t, p in enumerate(positions):
            b = sum(t >= s for s in starts) - 1
            k, v = (c[b, :p + 1].double().repeat_interleave(H // G, 1) for c in (ring_k, ring_v))
            s = torch.einsum("hd,khd->hk", q[t].view(H, d).double(), k) * d ** -0.5 + bias.double()[(p - torch.arange(p + 1, device=DEV)).clamp(max=29)].T
            assert rel(out[t], torch.einsum("hk,khd->hd", torch.softmax(s, 1), v).flatten()) < 2e-6


@pytest.mark.parametrize("tiled", [True, False])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("form", ["window", "chunked", "bias", "one_distance"])
def test_fp32_attention_of_keys_at_minus_infinity(form, d, tiled):
    """Keys that score -infinity weigh nothing, also where they are all that a query sees of a tile: behind a window's or a chunk's start, and under a bias of
    -infinity for everything far.  A query that sees nothing else has no numbers."""
    from mistral_inference_b200 import _abi_hybrid as h

    H, G, W, lens, past = 4, 2, 512, [90, 40, 33], [0, 47, 300]
    g = torch.Generator().manual_seed(d)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)  # noqa: E731
    T, B = sum(lens), len(lens)
    q, ring_k, ring_v = r(T, H, d), r(B, W, G, d), r(B, W, G, d)
    q[:, :, 0] = q[:, :, 0].abs() + 0.1
    window, kw, bias = 0, {}, None
    if form == "window":
        window = 37
        ring_k[0, 59, :, 0] = ring_k[0, 31, :, 0] = -float("inf")  # the first key that position 95, 67 see: the 32nd of the tiles that start at 28, 0
        ring_k[2, 264:296, :, 0] = -float("inf")                 # a whole tile
    elif form == "chunked":
        window, kw = 48, dict(chunked=True)
        ring_k[:, 48:64, :, 0] = -float("inf")
    else:
        bias = r(20, H)
        bias[-1] = -float("inf")
        if form == "one_distance":
            bias[:] = -float("inf")
            bias[3] = 0.5
    starts = [0, 90, 130, 163]
    dev = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    positions, slots = dev([p + i for n, p in zip(lens, past) for i in range(n)]), dev(range(B))
    out, tiles, scale = torch.empty(T, H * d, device=DEV), sum((n + 63) // 64 for n in lens) if tiled else 0, d ** -0.5
    if bias is not None:
        h.attn_bias(q.flatten(1), ring_k, ring_v, bias, positions, dev(starts), slots, out, B, W, H, G, d, d, scale, n_tiles=tiles)
    else:
        h.attn_window(q.flatten(1), ring_k, ring_v, positions, dev(starts), slots, out, B, W, H, G, d, d, scale, window, n_tiles=tiles, **kw)
    ref = torch.empty(T, H * d, dtype=torch.float64, device=DEV)
    for t, p in enumerate(positions.tolist()):
        b = sum(t >= s for s in starts) - 1
        lo = 0 if not window else (p - p % window if kw else max(0, p - window + 1))
        k, v = (c[b, lo:p + 1].double().repeat_interleave(H // G, 1) for c in (ring_k, ring_v))
        s = torch.einsum("hd,khd->hk", q[t].double(), k) * scale
        if bias is not None:
            s = s + bias.double()[(p - torch.arange(lo, p + 1, device=DEV)).clamp(max=19)].T
        ref[t] = torch.einsum("hk,khd->hd", torch.softmax(s, 1), v).flatten()
    assert torch.equal(out.isnan(), ref.isnan())
    fine = ~ref.isnan()
    assert fine.float().mean() > 0.75 and rel(out[fine], ref[fine]) < 1e-6


def _scan64(q, k, v, decay, state, lens):
    """o [T, H, e] and the final states of sum_j decay^(i-j) (q_i . k_j) v_j in float64, token by token."""
    o, t = torch.empty(*v.shape, dtype=torch.float64, device=v.device), 0
    for b, n in enumerate(lens):
        for _ in range(n):
            state[b] = decay[:, None, None] * state[b] + k[t][:, :, None] * v[t][:, None, :]
            o[t] = (state[b] * q[t][:, :, None]).sum(1)
            t += 1
    return o, state


@pytest.mark.parametrize("H,d,e", [(2, 128, 96), (3, 64, 40), (1, 100, 33), (2, 32, 7)])
@pytest.mark.parametrize("lens", [[8], [17, 1, 16], [33, 40]])
def test_lightning_scan_of_prompts(H, d, e, lens):
    """fp32 prompts: the state's rows in four warps, tiles of 16 tokens, value columns in blocks of 32, against float64 and the scan of a column per thread: the
    same state bit for bit, outputs to the rounding of a sum of d products."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator().manual_seed(d + e)
    T, B = sum(lens), len(lens)
    x = torch.randn(T, 2 * H * d + 2 * H * e, generator=g).to(DEV)
    q, k, v = x[:, :H * d].view(T, H, d).double(), x[:, H * d:2 * H * d].view(T, H, d).double(), x[:, 2 * H * d:2 * H * d + H * e].reshape(T, H, e).double()
    decay = torch.linspace(0.5, 0.99, H).to(DEV)
    start = [0]
    for n in lens:
        start.append(start[-1] + n)
    q_start, seqpos, slots = (torch.tensor(t, dtype=torch.int32, device=DEV) for t in (start, [i % 2 * 5 for i in range(B)], list(range(B))))
    first = torch.randn(B, H, d, e, generator=g).to(DEV)
    states, outs = [first.clone(), first.clone()], [torch.empty(T, H * e, device=DEV) for _ in range(2)]
    h.lightning_scan(x, states[0], decay, q_start, seqpos, slots, outs[0], B, H, d, e, longest=max(8, max(lens)))
    h.lightning_scan(x, states[1], decay, q_start, seqpos, slots, outs[1], B, H, d, e, longest=1)
    want = first.double() * (seqpos > 0)[:, None, None, None]
    o, want = _scan64(q, k, v, decay.double(), want, lens)
    assert torch.equal(states[0], states[1]) and rel(states[0], want) < 1e-6
    assert rel(outs[0], o.flatten(1)) < max(1.2 * rel(outs[1], o.flatten(1)), 2e-7)


@pytest.mark.parametrize("H,d,e", [(3, 128, 128), (2, 64, 96), (5, 32, 32)])
@pytest.mark.parametrize("lens", [[64], [65, 1, 12], [200, 63], [16, 128, 129]])
def test_lightning_chunks(H, d, e, lens):
    """Chunk edges, ragged batches, rows in another order than the batch, states carried on: the chunked kernel against float64 and against the
    token-by-token scan, which it must not be less exact than (products of fp32 numbers in three bf16 parts: 2^-21 on either side)."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator().manual_seed(sum(lens) + d)
    T, B = sum(lens), len(lens)
    x = torch.randn(T, 2 * H * d + 2 * H * e, generator=g).bfloat16().to(DEV)
    decay = torch.linspace(0.3, 1.0, H).to(DEV)
    slots = torch.arange(B).flip(0).int().to(DEV)
    start = torch.randn(B, H, d, e, generator=g).to(DEV)
    seqpos = torch.tensor([0 if b == 0 else 7 for b in range(B)], dtype=torch.int32, device=DEV)
    q_start = torch.tensor([0] + lens).cumsum(0).int().to(DEV)
    q, k = (x[:, i * H * d:(i + 1) * H * d].double().view(T, H, d) for i in (0, 1))
    v = x[:, 2 * H * d: 2 * H * d + H * e].double().view(T, H, e)
    first = start.double()[slots.long()].clone()
    first[0] = 0  # nothing before: whatever the row held does not count
    ref, last = _scan64(q, k, v, decay.double(), first, lens)
    got = []
    for longest in (max(lens), 1):
        state, o = start.clone(), torch.empty(T, H * e, dtype=torch.float32, device=DEV)
        h.lightning_scan(x, state, decay, q_start, seqpos, slots, o, B, H, d, e, longest=max(longest, 12) if longest > 1 else 1)
        got.append((rel(o, ref.flatten(1)), rel(state[slots.long()], last)))
    assert got[0][0] < max(2 ** -21, 1.2 * got[1][0]) and got[0][1] < max(2 ** -21, 1.2 * got[1][1]), got


def test_lightning_infinity_reaches_no_earlier_token():
    from mistral_inference_b200 import _abi_hybrid as h

    T, H, d, e = 150, 2, 64, 64
    g = torch.Generator().manual_seed(3)
    x = torch.randn(T, 2 * H * d + 2 * H * e, generator=g).bfloat16().to(DEV)
    x[100, 2 * H * d + 5] = float("inf")  # head 0, column 5 of the values
    decay, one = torch.full((H,), 0.9, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    q_start = torch.tensor([0, T], dtype=torch.int32, device=DEV)
    outs = []
    for longest in (T, 1):
        state, o = torch.zeros(1, H, d, e, device=DEV), torch.empty(T, H * e, dtype=torch.float32, device=DEV)
        h.lightning_scan(x, state, decay, q_start, one, one, o, 1, H, d, e, longest=longest)
        outs.append((o, state))
    for a, b in zip(*outs):
        assert torch.equal(torch.isfinite(a), torch.isfinite(b)) and torch.equal(torch.isnan(a), torch.isnan(b))
        assert rel(a[torch.isfinite(b)], b[torch.isfinite(b)].double()) < 1e-6


def _attend64(q, k, v, qpos, kpos, scale, window, bias):
    H, G = q.shape[1], k.shape[1]
    dist = qpos[:, None] - kpos[None]
    out = []
    for head in range(H):
        s = q[:, head] @ k[:, head // (H // G)].T * scale
        if bias is not None:
            s = s + bias[dist.clamp(0, len(bias) - 1), head]
        s = s.masked_fill((dist < 0) | (dist >= window), float("-inf"))
        out.append(torch.softmax(s, -1) @ v[:, head // (H // G)])
    return torch.stack(out, 1).flatten(1)


@pytest.mark.parametrize("H,KV", [(4, 2), (3, 1), (2, 2), (8, 1)])
@pytest.mark.parametrize("lens,past,W", [([128], [0], 128), ([129, 60], [5, 0], 300), ([300], [1], 301), ([70, 257, 1], [400, 128, 3], 512), ([200, 48], [777, 90], 256),
                                         ([64], [1000], 70)])
def test_prompt_attention_over_ring_and_own_rows(H, KV, lens, past, W):
    """Portions of prompts on the tcgen05 kernel: rings that wrap, runs around the 128-key tile, windows, rows nothing has written (NaN here),
    one and two heads per CTA; P is rounded to bf16 (2^-9 relative)."""
    from mistral_inference_b200 import _abi

    g = torch.Generator().manual_seed(sum(lens) + W)
    B, T, hd = len(lens), sum(lens), 128
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16().to(DEV)  # noqa: E731
    q, k, v = rnd(T, H, hd), rnd(T, KV, hd), rnd(T, KV, hd)
    ring_k, ring_v = (torch.full((B, W, KV, hd), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2))
    q_start = torch.tensor([0] + lens).cumsum(0).int().to(DEV)
    out, ref = torch.empty(T, H * hd, dtype=torch.bfloat16, device=DEV), []
    for b, (n, m) in enumerate(zip(lens, past)):
        have = min(m, W)
        old = torch.arange(m - have, m, device=DEV)
        ok, ov = rnd(have, KV, hd), rnd(have, KV, hd)
        ring_k[b, old % W], ring_v[b, old % W] = ok, ov
        a, z = int(q_start[b]), int(q_start[b + 1])
        pos = torch.arange(m, m + n, device=DEV)
        ref.append(_attend64(q[a:z].double(), torch.cat((ok, k[a:z])).double(), torch.cat((ov, v[a:z])).double(), pos, torch.cat((old, pos)), hd ** -0.5, W, None))
    _abi.attn_prefill(q, k, v, ring_k, ring_v, q_start, torch.tensor(past, dtype=torch.int32, device=DEV), out, B, max(lens), W, H, KV, hd, causal=True,
                      first_prefill=max(past) == 0)
    assert rel(out, torch.cat(ref)) < 2 ** -8


@pytest.mark.parametrize("H,KV", [(4, 2), (3, 1)])
@pytest.mark.parametrize("lens,past,W,bad", [([100, 60, 20], [9, 7, 30], 200, 0), ([100, 60, 130], [0, 0, 0], 300, 1), ([129, 255], [0, 0], 64, 0), ([40], [500], 64, None),
                                             ([140, 33], [77, 300], 128, None)])
def test_prompt_attention_keeps_bad_values_where_they_are(H, KV, lens, past, W, bad):
    """NaN and infinity in one sequence's own keys and values (`bad`), or in ring rows that have left every query's window (None), reach no other
    token: the others' outputs are the bits that finite values there give."""
    from mistral_inference_b200 import _abi

    g = torch.Generator().manual_seed(sum(lens) + W)
    B, T, hd = len(lens), sum(lens), 128
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16().to(DEV)  # noqa: E731
    q, k, v, ring_k, ring_v = rnd(T, H, hd), rnd(T, KV, hd), rnd(T, KV, hd), rnd(B, W, KV, hd), rnd(B, W, KV, hd)
    q_start = torch.tensor([0] + lens).cumsum(0).int().to(DEV)
    outs = []
    for spoil in (False, True):
        k1, v1, rk, rv = k.clone(), v.clone(), ring_k.clone(), ring_v.clone()
        if spoil and bad is not None:
            a, z = int(q_start[bad]), int(q_start[bad + 1])
            v1[a:z], k1[a:z:2] = float("nan"), float("inf")
        elif spoil:
            for b, m in enumerate(past):
                if m >= W:  # position m - W: the oldest row; the first query, m, sees m - W + 1 and later ones
                    rk[b, (m - W) % W], rv[b, (m - W) % W] = float("inf"), float("nan")
        out = torch.empty(T, H * hd, dtype=torch.bfloat16, device=DEV)
        _abi.attn_prefill(q, k1, v1, rk, rv, q_start, torch.tensor(past, dtype=torch.int32, device=DEV), out, B, max(lens), W, H, KV, hd, causal=True,
                          first_prefill=max(past) == 0)
        outs.append(out)
    for b in range(B):
        if b != bad:
            a, z = int(q_start[b]), int(q_start[b + 1])
            assert torch.isfinite(outs[1][a:z]).all() and torch.equal(outs[0][a:z], outs[1][a:z]), b


@pytest.mark.parametrize("n_tab", [0, 1, 40, 500])
@pytest.mark.parametrize("lens,past", [([64], [0]), ([130, 33], [0, 0]), ([250, 1], [300, 5]), ([128, 128], [128, 1])])
def test_prompt_attention_with_a_bias_over_the_ring(n_tab, lens, past):
    """Every key in the ring (row blocks in another order than the batch, unwritten rows NaN), a bias table shorter and longer than the distances."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator().manual_seed(sum(lens) + n_tab)
    B, T, H, KV, hd = len(lens), sum(lens), 4, 2, 128
    W = max(m + n for m, n in zip(past, lens)) + 3
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16().to(DEV)  # noqa: E731
    q = rnd(T, H * hd)
    ring_k, ring_v = (torch.full((B + 1, W, KV, hd), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2))
    bias = torch.randn(n_tab, H, generator=g).to(DEV) * 2 if n_tab else None
    slots = torch.arange(B).flip(0).add(1).int().to(DEV)
    q_start = torch.tensor([0] + lens).cumsum(0).int().to(DEV)
    seqpos, positions, ref = torch.tensor(past, dtype=torch.int32, device=DEV), [], []
    for b, (n, m) in enumerate(zip(lens, past)):
        kk, vv = rnd(m + n, KV, hd), rnd(m + n, KV, hd)
        ring_k[slots[b].item(), : m + n], ring_v[slots[b].item(), : m + n] = kk, vv
        pos = torch.arange(m, m + n, device=DEV)
        positions.append(pos.int())
        a, z = int(q_start[b]), int(q_start[b + 1])
        ref.append(_attend64(q[a:z].view(n, H, hd).double(), kk.double(), vv.double(), pos, torch.arange(m + n, device=DEV), 0.1, W, bias.double() if n_tab else None))
    out = torch.empty(T, H * hd, dtype=torch.bfloat16, device=DEV)
    tiles = sum((n + 63) // 64 for n in lens)
    h.attn_bias(q, ring_k, ring_v, bias, torch.cat(positions), q_start, slots, out, B, W, H, KV, hd, hd, 0.1, n_tiles=tiles, seqpos=seqpos, longest=max(lens))
    assert rel(out, torch.cat(ref)) < 2 ** -8


@pytest.mark.parametrize("M,N,K", [(9, 130, 64), (127, 96, 100), (128, 128, 7), (129, 257, 300), (33, 2048, 2048), (300, 640, 8192), (17, 6, 1029)])
def test_fp32_linear_in_parts(M, N, K):
    """fp32 Linears of prompts on the tensor cores: tile edges, k parts over clusters, rows that are no multiple of 16 bytes.  The part products
    that are left out are below 2^-21 of a product each; the sum is no further from float64 than a chain of FMAs is."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator().manual_seed(M + N + K)
    x, w, b = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV), torch.randn(N, generator=g).to(DEV)
    ref = x.double() @ w.double().T + b.double()
    got = h.linear(x, w, b, epi=h.EPI_F32)
    chain = torch.zeros(M, N, device=DEV)
    for k in range(K):  # one rounded multiply-add per column, as an FMA chain takes them
        chain = torch.addcmul(chain, x[:, k:k + 1], w[:, k][None])
    assert rel(got, ref) < max(2 ** -22, 1.1 * rel(chain + b, ref))
    base = torch.randn(M, N, generator=g).to(DEV)
    assert rel(h.linear(x, w, None, epi=h.EPI_RESIDUAL, residual=base.clone()), base.double() + x.double() @ w.double().T) < 2 ** -21
    big, tiny = h.linear(x * 1e30, w * 1e-30, epi=h.EPI_F32), h.linear(x * 2.0 ** -60, w * 2.0 ** 60, epi=h.EPI_F32)
    assert rel(big, (x * 1e30).double() @ (w * 1e-30).double().T) < 2 ** -21 and rel(tiny, x.double() @ w.double().T) < 2 ** -21


def _operands(kind, *shape, g):
    if kind == "normal":
        return torch.randn(*shape, generator=g)
    if kind == "positive":
        return 1 + torch.rand(*shape, generator=g)
    if kind == "low bits":  # what truncated parts leave out has one sign
        return torch.full(shape, 1 + 2.0 ** -7 - 2.0 ** -23)
    return torch.randn(*shape, generator=g) * 2.0 ** {"tiny": -118, "huge": 115, "least": -122}[kind]


@pytest.mark.parametrize("K", [1, 3, 8, 15, 16, 17, 64, 100, 2048])
@pytest.mark.parametrize("kx,kw", [("normal", "normal"), ("positive", "positive"), ("low bits", "low bits"), ("tiny", "normal"), ("tiny", "huge"), ("normal", "tiny"), ("huge", "tiny"),
                                   ("least", "huge")])
def test_fp32_linear_is_no_less_exact_than_fmas(kx, kw, K):
    """Either side of the step from FMAs to parts, operands of one sign, with all low bits set, and from both ends of fp32's range: no further from
    float64 than a chain of FMAs is, beside the one step in which the tensor core cuts its sum off, at most 2^-23 of it, and below 16 columns not even that."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator().manual_seed(K)
    x, w = _operands(kx, 40, K, g=g).to(DEV), _operands(kw, 200, K, g=g).to(DEV)
    ref, chain = x.double() @ w.double().T, torch.zeros(40, 200, device=DEV)
    for k in range(K):
        chain = torch.addcmul(chain, x[:, k:k + 1], w[:, k][None])
    assert rel(h.linear(x, w, epi=h.EPI_F32), ref) <= max(2.0 ** -23 if K >= 16 else 0.0, 1.02 * rel(chain, ref))


@pytest.mark.parametrize("M,N,K", [(40, 300, 256), (130, 200, 2048), (128, 128, 1029), (260, 1000, 640)])
def test_fp32_linear_with_infinities_is_a_chain_of_fmas(M, N, K):
    """A tile that holds an infinity or a NaN: exactly the FMA chain's results in all its rows, whatever part of the chip it was spread over."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator().manual_seed(M)
    x, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    x[3, 7], x[M - 1, K - 1], w[N - 1, 8] = float("inf"), float("nan"), float("-inf")
    chain = torch.zeros(M, N, device=DEV)
    for k in range(K):
        chain = torch.addcmul(chain, x[:, k:k + 1], w[:, k][None])
    got = h.linear(x, w, epi=h.EPI_F32)
    assert torch.equal(torch.isnan(got), torch.isnan(chain)) and torch.equal(torch.isinf(got), torch.isinf(chain))
    m0, n0 = (M - 1) // 128 * 128, (N - 1) // 128 * 128
    assert torch.equal(torch.nan_to_num(got[:128]), torch.nan_to_num(chain[:128])) and torch.equal(torch.nan_to_num(got[m0:, n0:]), torch.nan_to_num(chain[m0:, n0:]))


def test_fp32_linear_infinities():
    from mistral_inference_b200 import _abi_hybrid as h

    x, w = torch.ones(40, 256, device=DEV), torch.ones(300, 256, device=DEV)
    x[3, 7], x[4, 9], w[130, 8], w[131, 7] = float("inf"), float("nan"), float("-inf"), 0.0
    got, ref = h.linear(x, w, epi=h.EPI_F32), x.double() @ w.double().T
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.nan_to_num(got).double(), torch.nan_to_num(ref.float()).double())


@pytest.mark.parametrize("H,G,d,e", [(16, 4, 128, 128), (3, 1, 64, 128), (16, 1, 32, 32), (2, 2, 128, 64)])
@pytest.mark.parametrize("pos", [[0], [15, 16, 63], [64, 500, 1, 2047]])
@pytest.mark.parametrize("n_tab", [1, 30, 1200])
def test_decode_attention_with_a_bias(H, G, d, e, pos, n_tab):
    """One token per sequence: against float64, and no further from it than the exact fp32 kernel (the output's bf16 rounding apart, 2^-9); rows
    nothing has written are NaN."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator().manual_seed(H + d + len(pos))
    B, W = len(pos), max(pos) + 2
    q = torch.randn(B, H * d, generator=g).bfloat16().to(DEV)
    ring_k, ring_v = (torch.full((B, W, G, n), float("nan"), dtype=torch.bfloat16, device=DEV) for n in (d, e))
    bias = torch.randn(n_tab, H, generator=g).to(DEV) * 2
    slots, ref = torch.arange(B).flip(0).int().to(DEV), []
    for b, p in enumerate(pos):
        kk, vv = (torch.randn(p + 1, G, n, generator=g).bfloat16().to(DEV) for n in (d, e))
        ring_k[B - 1 - b, : p + 1], ring_v[B - 1 - b, : p + 1] = kk, vv
        ref.append(_attend64(q[b].view(1, H, d).double(), kk.double(), vv.double(), torch.tensor([p], device=DEV), torch.arange(p + 1, device=DEV), 0.2, W, bias.double()))
    ref, positions = torch.cat(ref), torch.tensor(pos, dtype=torch.int32, device=DEV)
    got, exact = (torch.empty(B, H * e, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    assert h.attn_bias_decode_ok(q, ring_k, ring_v, H, G, d, e)
    h.attn_bias_decode(q, ring_k, ring_v, bias, positions, slots, got, B, W, H, G, d, e, 0.2)
    h.attn_bias(q, ring_k, ring_v, bias, positions, torch.arange(B + 1, dtype=torch.int32, device=DEV), slots, exact, B, W, H, G, d, e, 0.2, splits=h.attn_splits(B, H, W))
    assert rel(got, ref) < 2 ** -9 and rel(got, ref) < 1.1 * rel(exact, ref) + 2 ** -16


@pytest.mark.parametrize("lens", [[128], [70, 59, 1], [300, 1, 212], [513, 700]])
def test_scoring_without_written_logits(lens, monkeypatch):
    """Log-probabilities reduced in the lm head's epilogue against the pass over written logits: tile edges, rows without a target, blocks of rows,
    targets at both ends of the vocabulary.  The logits are the same bf16 numbers and only sums of exponentials are taken in another order; at 128
    rows the written logits come from the split-k kernel, whose other order of sums may flip a rounding: one bf16 step of the largest."""
    import mistral_inference_b200 as mi
    from mistral_inference_b200 import _abi, transformer

    args = mi.TransformerArgs(dim=256, n_layers=1, head_dim=128, hidden_dim=512, n_heads=4, n_kv_heads=2, norm_eps=1e-5, vocab_size=640, max_batch_size=4)
    m = transformer.Transformer.empty(args, DEV, torch.bfloat16)
    g = torch.Generator(device=DEV).manual_seed(5)
    for p in m.parameters():
        p.normal_(0, 0.2, generator=g) if p.dim() > 1 else p.fill_(1.0)
    T = sum(lens)
    ids, targets = torch.randint(0, 640, (T,), device=DEV, generator=g), torch.randint(0, 640, (T,), device=DEV, generator=g)
    targets[0], targets[1], targets[T - 1], targets[T // 2] = 0, 639, -1, -1
    got, last = m.forward_logprobs(ids, lens, None, targets)
    monkeypatch.setattr(transformer, "SCORE_BLOCK_TOKENS", 300)
    got2, last2 = m.forward_logprobs(ids, lens, None, targets)
    monkeypatch.setattr(_abi, "lm_head_logprobs_ok", lambda *a: False)
    ref, ref_last = m.forward_logprobs(ids, lens, None, targets)
    step = ref_last.abs().max().item() * 2 ** -7 if T == 128 else 0.0
    assert (last - ref_last).abs().max() <= step and (last2 - ref_last).abs().max() <= step and (got[targets < 0] == 0).all()
    for a in (got, got2):
        assert (a - ref).abs().max() <= 1e-5 * ref.abs().max() + 2 * step


@pytest.mark.parametrize("T", [128, 200, 700])
@pytest.mark.parametrize("cols", [(64, 96), (96, 128), (0, 64), (639, 640), (5, 6), (0, 640)])
@pytest.mark.parametrize("value", ["nan", "-inf"])
def test_scoring_counts_logits_that_are_no_numbers(T, cols, value):
    """Whole groups of NaN logits make the row's log-probability NaN, groups of -infinity add nothing, as in the pass over written logits."""
    from mistral_inference_b200 import _abi

    g = torch.Generator(device=DEV).manual_seed(T)
    D, V = 128, 640
    x, w = torch.rand(T, D, device=DEV, generator=g).bfloat16() + 0.5, (torch.randn(V, D, device=DEV, generator=g) / 8).bfloat16()
    w[cols[0]:cols[1]] = float(value)  # x is positive: the logits are NaN or -infinity
    nw, targets = torch.ones(D, device=DEV, dtype=torch.bfloat16), torch.randint(0, V, (T,), device=DEV, generator=g)
    ws = _abi.Workspace(_abi.workspace_bytes(T, D, 1, 1, 128, 256, V, 1), DEV)
    logits, ref, got = torch.empty(T, V, device=DEV), torch.zeros(T, device=DEV), torch.zeros(T, device=DEV)
    _abi.lm_head(x, nw, w, logits, 1e-5, ws)
    _abi.logprob_gather(logits, targets, out=ref)
    _abi.lm_head_logprobs(x, nw, w, targets, torch.full((T,), -1, dtype=torch.int32, device=DEV), torch.empty(1, V, device=DEV), got, 1e-5, ws)
    assert (torch.isnan(ref).all() if value == "nan" or cols == (0, V) else torch.isfinite(ref[(targets < cols[0]) | (targets >= cols[1])]).all())
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.isinf(got), torch.isinf(ref))
    ok, step = torch.isfinite(ref), logits[torch.isfinite(logits)].abs().max().item() * 2 ** -7 if torch.isfinite(logits).any() else 0.0
    assert (got - ref)[ok].abs().max() <= 1e-5 * 10 + (2 * step if T == 128 else 0.0) if ok.any() else True


@pytest.mark.parametrize("T", [16, 17, 24, 25, 32, 33, 64, 65, 127, 128, 171, 600])
@pytest.mark.parametrize("N,K", [(256, 128), (4096, 8192), (4224, 128), (16384, 1024), (24576, 1024)])  # the third: at 600 rows pairs, half a tile of weights at the end
def test_prompt_linear_steps_by_rows(T, N, K):
    """The steps behind a prompt's Linear at every change of kernel over the rows (whole rows streamed, tiles streamed, single tiles, pairs cut along k): bf16 results
    within a rounding (2^-8) of float64, fp32 ones within 2^-8 of the sum's scale for the rounded sum that is added."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator(device=DEV).manual_seed(T + N)
    x, w = torch.randn(T, K, device=DEV, generator=g).bfloat16(), (torch.randn(N, K, device=DEV, generator=g) / K ** 0.5).bfloat16()
    b, base, rs = torch.randn(N, device=DEV, generator=g).bfloat16(), torch.randn(T, N, device=DEV, generator=g), torch.rand(T, 2, device=DEV, generator=g)
    z = x.double() @ w.double().T
    zb = z + b.double()
    assert h._prompt_gemm_ok(x, T, N, K) and h._prompt_gemm(x, T, N, K) == (T > 32 or (T > 24 and N >= 16384) or (T > 16 and N >= 24576))
    assert rel(h.linear(x, w, b, n_act=N // 2), torch.cat((torch.nn.functional.silu(zb[:, : N // 2]), zb[:, N // 2:]), 1)) < 2 ** -8
    assert rel(h.linear(x, w, b, epi=h.EPI_F32, alpha=0.5), 0.5 * zb) < 1e-5
    assert rel(h.linear(x, w, epi=h.EPI_RESIDUAL, residual=base.clone()) - base, z) < 2 ** -8
    gate, up, s = z[:, 0::2], z[:, 1::2], rs.double().repeat_interleave(N // 4, 1)
    assert rel(h.linear_swiglu(x, w, rs, N // 4), torch.nn.functional.silu(gate) * up * s) < 2 ** -7
    assert rel(h.linear(x, w, epi=h.EPI_GLU, limit=1.5, alpha=1.7), gate.clamp(max=1.5) * torch.sigmoid(1.7 * gate.clamp(max=1.5)) * (up.clamp(-1.5, 1.5) + 1)) < 2 ** -7


@pytest.mark.parametrize("T", [2, 3, 4])
@pytest.mark.parametrize("N,K", [(8, 256), (18, 8), (130, 2056), (512, 4096), (48, 4104), (1024, 5120), (64, 14336)])
def test_linear_of_a_few_tokens(T, N, K):
    """Either side of the step from FMAs to tensor cores (k above 4096, or four tokens with a norm): rows past the last full 16, k past the last full 256 and the
    norm in front.  A Linear's output is bf16 (logits too, held as fp32): within its rounding, 2^-8, of float64, beside 2 K * 2^-24 of the sum
    of the products' sizes (the sum in fp32, and once more where that moves it over a rounding's edge)."""
    from mistral_inference_b200 import _abi

    g = torch.Generator(device=DEV).manual_seed(T * N + K)
    x, w = torch.randn(T, K, device=DEV, generator=g).bfloat16(), (torch.randn(N, K, device=DEV, generator=g) / K ** 0.5).bfloat16()
    nw = torch.rand(K, device=DEV, generator=g).bfloat16()
    ws = _abi.Workspace(_abi.workspace_bytes(8, K, 1, 1, 128, 256, N, 8), DEV)
    logits = torch.full((T, N), float("nan"), device=DEV)
    _abi.lm_head(x, nw, w, logits, 1e-5, ws)
    n = _abi.rmsnorm(x, nw, 1e-5).double()
    ref = n @ w.double().T
    assert ((logits - ref).abs() <= 2 ** -8 * ref.abs() + 2 * K * 2 ** -24 * (n.abs() @ w.double().abs().T)).all()
    res, out = torch.randn(T, N, device=DEV, generator=g).bfloat16(), torch.empty(T, N, dtype=torch.bfloat16, device=DEV)
    _abi.linear_residual(x, w, None, out, ws)
    assert rel(out, x.double() @ w.double().T) < 2 ** -8
    ref = x.double() @ w.double().T + res.double()
    _abi.linear_residual(x, w, res, res, ws)  # in place
    assert rel(res, ref) < 2 ** -7  # the product's rounding and the sum's, 2^-8 of each size


@pytest.mark.parametrize("T,N,K", [(500, 4096, 8192), (100, 4096, 4096)])
def test_two_streams_of_linears_that_share_their_tiles(T, N, K):
    """Pairs cut along k and split stream-K tiles on two streams at once (each call has its own scratch): the bits of one stream alone.  Owners wait
    for blocks that started before them only, so neither launch needs the whole chip."""
    from mistral_inference_b200 import _abi, _abi_hybrid as h

    g = torch.Generator(device=DEV).manual_seed(T)
    assert _abi.lib().mb200_layer_linear_scratch(T, N, K) > 0
    x, w = torch.randn(T, K, device=DEV, generator=g).bfloat16(), (torch.randn(N, K, device=DEV, generator=g) / K ** 0.5).bfloat16()
    ref = h.linear(x, w, epi=h.EPI_F32)
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in range(2)], []
    for _ in range(10):
        for s in streams:
            with torch.cuda.stream(s):
                got.append(h.linear(x, w, epi=h.EPI_F32))
    torch.cuda.synchronize()
    assert all(torch.equal(o, ref) for o in got)


def _f32_step(h, kind, x, w, b, rs, base):
    """(result, the same in float64) of one step after an fp32 Linear"""
    N = w.shape[0]
    y, F = x.double() @ w.double().T, torch.nn.functional
    if kind == "store":
        return h.linear(x, w, b, n_act=N // 2), torch.cat((F.silu((y + b.double())[:, : N // 2]), (y + b.double())[:, N // 2:]), 1)
    if kind == "plain":
        return h.linear(x, w, b), y + b.double()
    if kind == "scaled add":
        return h.linear(x, w, b, epi=h.EPI_RESIDUAL_SCALED, residual=base.clone(), alpha=0.3), base.double() + 0.3 * (y + b.double())
    if kind == "logits":
        return h.linear(x, w, None, epi=h.EPI_F32, limit=5.0, alpha=2.0), 2 * 5 * torch.tanh(y / 5)
    if kind == "relu2":
        return h.linear_relu2(x, w, rs, 8), y.clamp(min=0) ** 2 * rs.double().repeat_interleave(8, 1)[:, :N]
    if kind == "decay":
        a_log = torch.linspace(-1, 1, N // 2, device=DEV)
        return h.linear_decay(x, w, b, a_log, 2), torch.exp(-torch.exp(a_log.double().repeat_interleave(2)) * F.softplus(y + b.double()))
    g, u, r = y[:, 0::2], y[:, 1::2], rs.double().repeat_interleave(8, 1)[:, : N // 2]
    if kind == "glu":
        g, u = (g * r).clamp(max=2.0), (u * r).clamp(-2.0, 2.0)
        return h.linear_glu(x, w, 2.0, 1.7, rs, 8), g * torch.sigmoid(1.7 * g) * (u + 1)
    return h.linear_swiglu(x, w, rs, 8, gelu=kind == "geglu"), (F.gelu(g, approximate="tanh") if kind == "geglu" else F.silu(g)) * u * r


@pytest.mark.parametrize("kind", ["store", "plain", "scaled add", "logits", "relu2", "decay", "glu", "swiglu", "geglu"])
@pytest.mark.parametrize("M,N,K,pad", [(9, 256, 16, 0), (16, 258, 64, 4), (17, 130, 1030, 1), (224, 512, 72, 0), (225, 300, 132, 2), (449, 20480, 192, 0), (130, 2048, 1024, 0)])
def test_fp32_linear_by_pairs(M, N, K, pad, kind):
    """Token tiles of 16 to 224 and one more, weight tiles that end inside either CTA of a pair, k-blocks that end inside a float4 and rows of no whole float4s, tiles cut into parts, several
    rounds, and every step behind: fp32 numbers, so 2^-24 of a result's scale, twice for a step's own rounding, and what the tensor core cuts off a sum (2^-23)."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator().manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)  # noqa: E731
    x, w, b, base = rnd(M, K + pad)[:, :K], rnd(N, K) / K ** 0.5, rnd(N), rnd(M, N)
    if kind not in ("store", "plain", "scaled add", "logits"):
        x = x.contiguous()
    got, ref = _f32_step(h, kind, x, w, b, torch.rand(M, (N + 7) // 8, generator=g).to(DEV), base)
    again, _ = _f32_step(h, kind, x, w, b, torch.rand(M, (N + 7) // 8, generator=torch.Generator().manual_seed(1)).to(DEV), base) if kind in ("plain", "store") else (got, None)
    assert got.dtype == torch.float32 and rel(got, ref) < 2 ** -21 and torch.equal(got, again)


def test_fp32_linear_of_more_rows_than_a_launch_takes():
    """Rows in portions, each with what belongs to them; and the call that brings no memory of its own computes the same bits."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator().manual_seed(1)
    M, N, K = 2 * 4096 + 5, 40, 32
    x, w, rs = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV), torch.rand(M, 5, generator=g).to(DEV)
    got, out = h.linear_relu2(x, w, rs, 8), torch.empty(M, N, device=DEV)
    assert rel(got, (x.double() @ w.double().T).clamp(min=0) ** 2 * rs.double().repeat_interleave(8, 1)) < 2 ** -21
    assert h.lib().mbh_linear_relu2(x.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, rs.data_ptr(), 5, 8, 1, torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(out, got)


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,K,pad", [(1, 8, 0), (130, 72, 8), (1024, 64, 0), (1186, 192, 64), (3072, 2048, 0), (2049, 1416, 0), (8192, 448, 16), (18961, 128, 0), (38000, 320, 0),
                                     (4096, 2112, 0), (4097, 2048, 0), (1184, 4096, 0), (3071, 4160, 0), (3072, 4160, 0), (8192, 1000, 0), (8200, 1000, 0), (40, 264, 0)])
def test_decode_linear_streams_whole_rows(M, N, K, pad):
    """Rows of 8 to 128 a CTA, one and several units of them, the last ones short, k-blocks that end inside a stage and inside a block, x in a wider matrix; matrices of few rows, 16 a CTA, on
    both sides of that line: a bf16 Linear is within its
    rounding (2^-8) of float64, what stays fp32 within 2 K 2^-24 of the products' sizes."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    x, w, b, base = rnd(M, K + pad).bfloat16()[:, :K], (rnd(N, K) / K ** 0.5).bfloat16(), rnd(N).bfloat16(), rnd(M, N)
    ref = x.double() @ w.double().T
    size = x.double().abs() @ w.double().abs().T * (2 * K * 2.0 ** -24)
    assert ((h.linear(x, w, b).double() - ref - b.double()).abs() <= 2 ** -8 * (ref + b.double()).abs() + size + 1e-30).all()
    assert ((h.linear(x, w, None, epi=h.EPI_F32).double() - ref).abs() <= size + 1e-30).all()
    assert ((h.linear(x, w, b, epi=h.EPI_RESIDUAL, residual=base.clone()).double() - base.double() - ref - b.double()).abs()
            <= 2 ** -8 * (ref + b.double()).abs() + size + 2 ** -23 * (base.double().abs() + (ref + b.double()).abs())).all()
    if N % 2 == 0:
        y, F = ref.bfloat16().double(), torch.nn.functional
        got = h.linear_swiglu(x.contiguous(), w, None)
        assert rel(got, F.silu(y[:, 0::2]) * y[:, 1::2]) < 2 ** -7


@pytest.mark.parametrize("T", [2, 8, 9, 17, 24, 25, 32, 33])
def test_decode_steps_linears_against_float64(T):
    """Every step behind the Linears of a decode batch, at the edges of their token groups and one past the last: rotation and ring of q, k, v, gated unit, residual, logits."""
    from mistral_inference_b200 import _abi

    g = torch.Generator(device=DEV).manual_seed(T)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    D, H, KV, hd, F, rows = 640, 4, 2, 128, 1152, 40
    ws = _abi.Workspace(_abi.workspace_bytes(64, D, H, KV, hd, F, D, 64), DEV)
    x, nw = rnd(T, D).bfloat16(), (1 + rnd(D) / 8).bfloat16()
    wqkv, w13, w2 = ((rnd(n, k) / k ** 0.5).bfloat16() for n, k in (((H + 2 * KV) * hd, D), (2 * F, D), (D, F)))
    n = _abi.rmsnorm(x, nw, 1e-5).double()
    pos = torch.randint(0, 100, (T,), device=DEV, generator=g).int()
    ring = torch.randperm(rows, device=DEV, generator=g)[:T].int()
    ring[0] = -1
    ang = torch.rand(100, hd // 2, device=DEV, generator=g) * 6.28
    rope = torch.stack((ang.cos(), ang.sin()), -1).contiguous()
    q, k, v = (torch.empty(T, h * hd, dtype=torch.bfloat16, device=DEV) for h in (H, KV, KV))
    ck, cv = (torch.zeros(rows, KV * hd, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    _abi.attn_qkv(x, nw, wqkv, rope, pos, q, k, v, ck, cv, ring, H, KV, hd, 1e-5, ws)
    y = n @ wqkv.double().T
    c, s = (t.double()[:, None] for t in (rope[pos.long(), :, 0], rope[pos.long(), :, 1]))
    turn = lambda t: torch.stack((t[..., 0::2] * c - t[..., 1::2] * s, t[..., 0::2] * s + t[..., 1::2] * c), -1).flatten(1)  # noqa: E731
    assert rel(q, turn(y[:, : H * hd].view(T, H, hd))) < 2 ** -7 and rel(k, turn(y[:, H * hd:(H + KV) * hd].view(T, KV, hd))) < 2 ** -7  # two roundings to bf16
    assert rel(v, y[:, (H + KV) * hd:]) < 2 ** -8
    there = ring[1:].long()
    assert torch.equal(ck[there], k[1:]) and torch.equal(cv[there], v[1:]) and int((ck != 0).any(1).sum()) == T - 1
    gate = torch.empty(T, F, dtype=torch.bfloat16, device=DEV)
    _abi.ffn_gateup(x, nw, w13, gate, 1e-5, ws)
    u = n @ w13.double().T
    assert rel(gate, torch.nn.functional.silu(u[:, 0::2]) * u[:, 1::2]) < 2 ** -7
    res, out = rnd(T, D).bfloat16(), torch.empty(T, D, dtype=torch.bfloat16, device=DEV)
    _abi.linear_residual(gate, w2, res, out, ws)
    assert rel(out, res.double() + gate.double() @ w2.double().T) < 2 ** -7


@pytest.mark.parametrize("T,N,K", [(33, 128, 64), (48, 384, 128), (49, 1024, 640), (64, 6144, 192), (65, 2176, 1024), (112, 640, 2048), (113, 4096, 320), (127, 20480, 128), (128, 256, 8192),
                                   (129, 1152, 8256), (192, 128, 8192), (193, 1024, 8192), (256, 4096, 8192), (128, 128, 5120), (33, 128, 768), (100, 1664, 832), (129, 768, 8192), (256, 896, 8256), (64, 1536, 704)])
def test_linears_over_streamed_tiles(T, N, K):
    """Fewer and more units than SMs and than twelve a tile, tiles in one piece and in many, tokens at the edges of the MMA's columns and of the accumulators: against float64, for the dense model's steps (bf16
    results: 2^-8) and a layered decoder's (fp32 residual and logits); twice the same bits."""
    from mistral_inference_b200 import _abi, _abi_hybrid as h

    g = torch.Generator(device=DEV).manual_seed(T + N + K)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    x, w, b, res, base = rnd(T, K).bfloat16(), (rnd(N, K) / K ** 0.5).bfloat16(), rnd(N).bfloat16(), rnd(T, N).bfloat16(), rnd(T, N)
    ref, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T * (2 * K * 2.0 ** -24)
    ws, out = _abi.Workspace(_abi.workspace_bytes(T, K, 1, 1, 128, N, N, 8), DEV), torch.empty(T, N, dtype=torch.bfloat16, device=DEV)
    _abi.linear_residual(x, w, res, out, ws)
    assert ((out.double() - res.double() - ref).abs() <= 2 ** -8 * (ref.abs() + (ref + res.double()).abs()) + size).all()
    f32 = h.linear(x, w, b, epi=h.EPI_F32)
    assert ((f32.double() - ref - b.double()).abs() <= size + 2.0 ** -23 * (ref + b.double()).abs()).all() and torch.equal(f32, h.linear(x, w, b, epi=h.EPI_F32))
    got = h.linear(x, w, None, epi=h.EPI_RESIDUAL, residual=base.clone())
    assert ((got.double() - base.double() - ref).abs() <= 2 ** -8 * ref.abs() + size + 2.0 ** -23 * (base.double() + ref).abs()).all()
    y = ref.bfloat16().double()
    assert rel(h.linear_swiglu(x, w), torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2]) < 2 ** -7


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("T,H,G,d,e", [(1, 1, 1, 4, 4), (9, 5, 2, 128, 96), (1100, 7, 1, 64, 132), (33, 3, 2, 132, 4), (33, 3, 1, 100, 6), (17, 2, 2, 30, 32)])
def test_heads_prepared_four_entries_a_lane(T, H, G, d, e, norm, mode, dt):
    """Heads of up to 128 entries in fours; larger ones, odd ones and values of an odd count entry by entry.  A stored number is one rounding of dt from its
    exact value, a query two (it is rounded before its temperature), on top of a few of fp32; lost tokens leave the ring alone."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator().manual_seed(T + d)
    rnd = lambda *s: torch.randn(*s, generator=g).to(dt).to(DEV)
    qkv, qn, kn, first, lam = rnd(T, H * d + G * (d + e)), rnd(d), rnd(d), rnd(T, G * e), rnd(1)
    pos = torch.randint(0, 5000, (T,), generator=g).int().to(DEV)
    rows = torch.randperm(T + 5, generator=g)[:T].int()
    if T > 1:
        rows[T // 2] = -1
    rows = rows.to(DEV)
    q = torch.empty(T, H * d, dtype=dt, device=DEV)
    ck, cv = torch.full((T + 5, G * d), 7.0, dtype=dt, device=DEV), torch.full((T + 5, G * e), 7.0, dtype=dt, device=DEV)
    before = first.clone()
    h.attn_prep(qkv, qn if norm else None, kn if norm else None, pos, rows, q, ck, cv, first, lam, mode, H, G, d, e, 1e-5, 0.1, 64)
    xq, xk, xv = (t.double() for t in qkv.split([H * d, G * d, G * e], 1))
    unit = lambda x, n, w: (x.view(T, n, d) / (x.view(T, n, d).square().mean(-1, keepdim=True) + 1e-5).sqrt() * w.double()).reshape(T, -1) if norm else x
    xq = unit(xq, H, qn) * (1 + 0.1 * torch.log((pos.double() + 1).div(64).floor() + 1))[:, None]
    xk = unit(xk, G, kn)
    if mode == 2:
        xv = (1 - lam.double()) * xv + lam.double() * before.double()
    assert torch.equal(first, qkv[:, -G * e:] if mode == 1 else before)
    step = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -24
    fp32 = 12 * 2.0 ** -23  # the sum of squares, its root and quotient, the logarithm and three products
    kept = rows >= 0
    at = rows[kept].long()
    big = lam.double().abs() * before.double().abs() + (1 + lam.double().abs()) * qkv[:, -G * e:].double().abs()  # what a mixed value's fp32 steps are measured by
    assert ((q.double() - xq).abs() <= (2 * step + step * step + fp32) * xq.abs()).all()
    assert ((ck[at].double() - xk[kept]).abs() <= (step + fp32) * xk[kept].abs()).all()
    assert ((cv[at].double() - xv[kept]).abs() <= step * xv[kept].abs() + (4 * 2.0 ** -24 * big[kept] * (1 + step) if mode == 2 else 0)).all()
    lost = torch.ones(T + 5, dtype=torch.bool, device=DEV)
    lost[at] = False
    assert (ck[lost] == 7).all() and (cv[lost] == 7).all()


@pytest.mark.parametrize("M,N,K", [(9, 300, 64), (300, 2048, 1024), (130, 258, 132)])
def test_fp32_entries_without_room_allocate_nothing(M, N, K):
    """The entries of mistral_b200_hybrid.h bring no room for the parts of x and take none from the device: their results are fp32 numbers all the same, under capture too."""
    from cuda.bindings import runtime as rt

    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator().manual_seed(M)
    x, w, b = torch.randn(M, K, generator=g).to(DEV), (torch.randn(N, K, generator=g) / K ** 0.5).to(DEV), torch.randn(N, generator=g).to(DEV)
    rs, a_log = torch.rand(M, (N + 7) // 8, generator=g).to(DEV), torch.linspace(-1, 1, N // 2, device=DEV)
    y, F = x.double() @ w.double().T, torch.nn.functional
    out = {k: torch.empty(M, N // 2 if k in ("glu", "swiglu") else N, device=DEV) for k in ("store", "glu", "swiglu", "relu2", "decay")}
    lib, p = h.lib(), {k: v.data_ptr() for k, v in out.items()}

    def calls(st):
        X, Wp, B, R = x.data_ptr(), w.data_ptr(), b.data_ptr(), rs.data_ptr()
        return [lib.mbh_linear(X, K, Wp, B, p["store"], None, M, N, K, 0, 0, 0.0, 0.0, 1, st), lib.mbh_linear_glu(X, Wp, p["glu"], M, N, K, 2.0, 1.7, R, rs.shape[1], 8, 1, st),
                lib.mbh_linear_swiglu(X, Wp, p["swiglu"], M, N, K, R, rs.shape[1], 8, 0, 1, st), lib.mbh_linear_relu2(X, Wp, p["relu2"], M, N, K, R, rs.shape[1], 8, 1, st),
                lib.mbh_linear_decay(X, K, Wp, B, a_log.data_ptr(), 2, p["decay"], M, N, K, 1, st)]

    def check():
        r = rs.double().repeat_interleave(8, 1)
        gate, up = (y[:, i::2] * r[:, : N // 2] for i in (0, 1))
        ref = {"store": y + b.double(), "glu": gate.clamp(max=2) * torch.sigmoid(1.7 * gate.clamp(max=2)) * (up.clamp(-2, 2) + 1), "swiglu": F.silu(y[:, 0::2]) * y[:, 1::2] * r[:, : N // 2],
               "relu2": y.clamp(min=0) ** 2 * r[:, :N], "decay": torch.exp(-torch.exp(a_log.double().repeat_interleave(2)) * F.softplus(y + b.double()))}
        for k, v in ref.items():
            assert rel(out[k], v) < 2 ** -21, k

    attr = rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh
    err, pool = rt.cudaDeviceGetDefaultMemPool(torch.cuda.current_device())
    from cuda.bindings import driver

    torch.cuda.synchronize()
    rt.cudaMemPoolSetAttribute(pool, attr, driver.cuuint64_t(0))
    assert calls(torch.cuda.current_stream().cuda_stream) == [0] * 5
    torch.cuda.synchronize()
    assert int(rt.cudaMemPoolGetAttribute(pool, attr)[1]) == 0
    check()
    for o in out.values():
        o.fill_(7)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert calls(torch.cuda.current_stream().cuda_stream) == [0] * 5
    graph.replay()
    check()


def test_fp32_linear_runs_where_its_room_is_not_to_be_had(monkeypatch):
    from mistral_inference_b200 import _abi_hybrid as h

    x, w, base, empty = torch.randn(300, 512, device=DEV), torch.randn(1024, 512, device=DEV) / 512 ** 0.5, torch.randn(300, 1024, device=DEV), torch.empty

    def full(*a, **k):
        if k.get("dtype") == torch.uint8:
            raise torch.OutOfMemoryError("no room")
        return empty(*a, **k)

    monkeypatch.setattr(torch, "empty", full)
    got = h.linear(x, w, None, epi=h.EPI_RESIDUAL, residual=base.clone())
    assert rel(got, base.double() + x.double() @ w.double().T) < 2 ** -21


@pytest.mark.parametrize("kind,epi,kw", [("plain", 0, {}), ("logits", 3, dict(limit=5.0, alpha=2.0)), ("scaled add", 5, dict(alpha=0.3))])
@pytest.mark.parametrize("M,N,K", [(9, 300, 64), (804, 2048, 1024), (449, 20480, 192)])
def test_fp32_room_is_what_the_step_needs(M, N, K, kind, epi, kw):
    """Room for the parts of x and for the slots of the tiles that have any: a plain store keeps none for whole tiles.  So many bytes are enough, nothing behind them is touched,
    and the result is that of the Python call."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator().manual_seed(M)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)  # noqa: E731
    x, w, b, base = rnd(M, K), rnd(N, K) / K ** 0.5, rnd(N), rnd(M, N)
    want, _ = _f32_step(h, kind, x, w, b, None, base)
    limit, alpha = kw.get("limit", 0.0), kw.get("alpha", 0.0)
    need, every = h.lib().mbh_linear_any_scratch(M, N, K, epi, 0, limit, alpha, 1), h.lib().mbh_linear_scratch(M, N, K, 1)
    assert 6 * M * K <= need <= every and (kind != "plain" or N < 20000 or need < every - M * N * 2)  # (the small ones are all cut)
    room = torch.full((need + 4096,), 0x5a, dtype=torch.uint8, device=DEV)
    out = torch.empty(M, N, device=DEV) if kind != "scaled add" else base.clone()
    bias = None if kind == "logits" else b.data_ptr()
    assert h.lib().mbh_linear_any(x.data_ptr(), K, w.data_ptr(), bias, out.data_ptr(), out.data_ptr(), M, N, K, epi, 0, limit, alpha, None, 0, 0, None, room.data_ptr(), need, 1,
                                  torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(out, want) and (room[need:] == 0x5a).all()


@pytest.mark.parametrize("M,N,K", [(255, 64, 1024), (256, 64, 1024), (1024, 33, 1040), (1025, 65, 1024), (2049, 128, 512), (2049, 129, 512), (1153, 384, 1024), (3200, 384, 512), (4097, 128, 16), (4097, 300, 40), (8197, 8200, 32), (16385, 130, 24)])
def test_fp32_linears_of_few_features_and_of_several_launches(M, N, K):
    """Both sides of the lines at which x is no longer split ahead, and prompts of one row more than a launch takes."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator(device=DEV).manual_seed(M)
    x, w, rs = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV) / K ** 0.5, torch.rand(M, (N + 7) // 8, generator=g, device=DEV)
    got = h.linear_relu2(x, w, rs, 8)
    assert rel(got, (x.double() @ w.double().T).clamp(min=0) ** 2 * rs.double().repeat_interleave(8, 1)[:, :N]) < 2 ** -21
    assert torch.equal(got[-5:], h.linear_relu2(x, w, rs, 8)[-5:])


@pytest.mark.parametrize("M", [9, 16, 17, 24, 32])
@pytest.mark.parametrize("K,first,pitch", [(512, 0, 516), (512, 0, 520), (512, 4, 576), (520, 0, 524), (520, 1, 528), (512, 64, 640)])
def test_decode_rows_of_a_wider_matrix(M, K, first, pitch):
    """Rows that start, or follow one another, off the 16-byte grid or off the k-blocks: from 17 on the same bits as rows of their own, which stream (they ran on mma.sync tiles, 25 times
    as long); fewer are read as they lie."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator(device=DEV).manual_seed(M + K)
    x = torch.randn(M, pitch + 8, generator=g, device=DEV).bfloat16().flatten()[: M * pitch].view(M, pitch)[:, first:first + K]
    w = (torch.randn(1024, K, generator=g, device=DEV) / K ** 0.5).bfloat16()
    got, own = (h.linear(t, w, None, epi=h.EPI_F32) for t in (x, x.contiguous()))
    assert rel(got, x.double() @ w.double().T) < 2 * K * 2.0 ** -24
    assert M < 17 or torch.equal(got, own)


_LAUNCHES = """
import torch
from cuda.bindings import runtime as rt
from mistral_inference_b200 import _abi, _abi_hybrid as h
ws = _abi.Workspace(_abi.workspace_bytes(128, 640, 1, 1, 128, 1024, 1024, 8), torch.device("cuda"))
w, wf = torch.randn(1024, 640, device="cuda").bfloat16(), torch.randn(1024, 640, device="cuda")
rows = {m: torch.randn(m, 640, device="cuda").bfloat16() for m in (4, 20, 100)}
fp32, out = torch.randn(300, 640, device="cuda"), {m: torch.empty(m, 1024, device="cuda").bfloat16() for m in rows}
def run():
    for m, x in rows.items():
        h.linear(x, w)
        _abi.linear_residual(x, w, out[m], out[m], ws)
    h.linear(fp32, wf)
run()
graph = torch.cuda.CUDAGraph(keep_graph=True)
with torch.cuda.graph(graph):
    run()
err, *_, count = rt.cudaGraphGetEdges_v2(graph.raw_cuda_graph())
err, _, _, data, count = rt.cudaGraphGetEdges_v2(graph.raw_cuda_graph(), count)
print(count, sum(int(e.type) == int(rt.cudaGraphDependencyType.cudaGraphDependencyTypeProgrammatic) for e in data[:count]))
"""


@pytest.mark.parametrize("pdl", ["0", "1"])
def test_programmatic_launches_can_be_switched_off(pdl):
    """MB200_PDL=0 launches everything the ordinary way, in both libraries: no edge of a captured graph is a programmatic one."""
    import os
    import subprocess
    import sys
    from pathlib import Path

    r = subprocess.run([sys.executable, "-c", _LAUNCHES], capture_output=True, text=True, cwd=Path(__file__).resolve().parents[1], env={**os.environ, "MB200_PDL": pdl}, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    edges, programmatic = (int(v) for v in r.stdout.split())
    assert edges >= 9 and (programmatic == 0 if pdl == "0" else programmatic >= 5)


@pytest.mark.parametrize("M", [9, 16, 17, 32, 33, 128])
def test_rows_of_other_orders_are_copied_or_refused(M):
    """A transposed matrix, one row for all and rows that overlap: from 17 bf16 rows on the bits of a copy, below (and in fp32) refused, never read where they do not lie."""
    from mistral_inference_b200 import _abi_hybrid as h

    g = torch.Generator(device=DEV).manual_seed(M)
    w = (torch.randn(256, 512, generator=g, device=DEV) / 512 ** 0.5).bfloat16()
    flat = torch.randn(512 * M + 512, generator=g, device=DEV).bfloat16()
    for x in (flat[: 512 * M].view(512, M).T, flat[:512].expand(M, 512), flat.as_strided((M, 512), (64, 1))):
        if M >= 17:
            assert torch.equal(h.linear(x, w, None, epi=h.EPI_F32), h.linear(x.contiguous(), w, None, epi=h.EPI_F32))
        else:
            with pytest.raises(AssertionError):
                h.linear(x, w)
        with pytest.raises(AssertionError):
            h.linear(x.float() if x.stride(0) != 0 and x.stride(1) != 1 else flat.float().as_strided(x.shape, x.stride()), w.float())
