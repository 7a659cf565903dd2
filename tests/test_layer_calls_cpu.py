"""What the Python entry points of the prompt kernels refuse before anything is launched."""
import importlib.util

import pytest
import torch

from mistral_inference_b200 import _abi, _abi_hybrid as h


@pytest.mark.parametrize("table", [torch.zeros(9, 4, dtype=torch.bfloat16), torch.zeros(4, 9), torch.zeros(36)])
@pytest.mark.parametrize("longest", [1, 200])
def test_bias_tables_of_another_layout_are_refused(table, longest, monkeypatch):
    monkeypatch.setattr(_abi, "layer_attention", lambda *a: pytest.fail("launched"))
    q, ring = torch.zeros(200, 4 * 128, dtype=torch.bfloat16), torch.zeros(1, 300, 2, 128, dtype=torch.bfloat16)
    i = torch.zeros(2, dtype=torch.int32)
    with pytest.raises(AssertionError, match="bias table"):
        h.attn_bias(q, ring, ring, table, i, i, i, q, 1, 300, 4, 2, 128, 128, 0.1, n_tiles=4, seqpos=i, longest=longest)
    with pytest.raises(AssertionError, match="bias table"):
        h.attn_bias_decode(q[:1], ring, ring, table, i, i, q, 1, 300, 4, 2, 128, 128, 0.1)


@pytest.mark.parametrize("what", ["idx", "rows", "w13", "w2", "add"])
def test_mixtures_of_other_shapes_are_refused(what, monkeypatch):
    monkeypatch.setattr(_abi, "layer_moe", lambda *a: pytest.fail("launched"))
    T, D, E, ff, bf = 40, 256, 3, 128, torch.bfloat16
    x, w13, w2, add = torch.zeros(T, D, dtype=bf), torch.zeros(E * 2 * ff, D, dtype=bf), torch.zeros(D, E * ff, dtype=bf), torch.zeros(T, D)
    idx, wsel = torch.zeros(T, 2, dtype=torch.int32), torch.zeros(T, 2)
    if what == "idx":
        idx = idx.long()
    elif what == "rows":
        idx, wsel = idx[1:], wsel[1:]
    elif what == "w13":
        w13 = w13[:, : D // 2]
    elif what == "w2":
        w2 = w2[:, ff:]
    else:
        add = add.to(bf)
    with pytest.raises(AssertionError, match="choices|experts' weights|add_to"):
        h.moe_grouped(x, w13, w2, idx, wsel, E, ff, h.EPI_SWIGLU, add_to=add)


@pytest.mark.parametrize("what", ["target", "keep", "out"])
def test_scoring_takes_one_target_a_token(what):
    T, V, bf = 130, 128, torch.bfloat16
    target, keep, out = torch.zeros(T, dtype=torch.long), torch.zeros(T, dtype=torch.int32), torch.zeros(T)
    target, keep, out = (t[1:] if what == n else t for t, n in ((target, "target"), (keep, "keep"), (out, "out")))
    with pytest.raises(AssertionError, match="targets and kept rows|results"):
        _abi.lm_head_logprobs(torch.zeros(T, 64, dtype=bf), torch.ones(64, dtype=bf), torch.zeros(V, 64, dtype=bf), target, keep, torch.zeros(1, V), out, 1e-5, None)


@pytest.mark.parametrize("T,H,W,window,own,keys,dtype,tiled", [
    (24, 16, 4096, 0, False, 0, torch.float32, False),      # 384 rows behind a long ring: a CTA each
    (25, 16, 4096, 0, False, 0, torch.float32, True),
    (24, 16, 4096, 0, False, 24, torch.float32, True),      # a first prompt: its own keys only
    (24, 16, 400, 0, False, 0, torch.float32, True),        # a short ring
    (24, 16, 380, 0, True, 0, torch.float32, False),        # ... and the call's own keys beside it
    (24, 16, 4096, 368, True, 0, torch.float32, True),      # a window
    (24, 16, 4096, 369, True, 0, torch.float32, False),
    (24, 16, 4096, 0, False, 0, torch.bfloat16, True),
])
def test_fp32_prompts_of_few_rows_over_many_keys(T, H, W, window, own, keys, dtype, tiled, monkeypatch):
    """Which kernel a prompt's attention takes, by the query tiles that reach the library (none: a CTA per token and head)."""
    seen = []
    record = lambda *a: seen.append(a[17]) or 0  # noqa: E731
    monkeypatch.setattr(h, "lib", lambda: type("Lib", (), {"mbh_attn_bias": staticmethod(record), "mbh_attn_window": staticmethod(record)}))
    monkeypatch.setattr(h, "_ptr", lambda t: None)
    monkeypatch.setattr(h, "_stream", lambda: 0)
    q, ring, i = torch.zeros(T, H * 64, dtype=dtype), torch.zeros(1, W, 1, 64, dtype=dtype), torch.zeros(2, dtype=torch.int32)
    k = q[:, :64].contiguous() if own else None
    h.attn_window(q, ring, ring, i, i, i, q, 1, W, H, 1, 64, 64, 0.1, window, own_k=k, own_v=k, seqpos=i, n_tiles=1, keys=keys)
    if not own and not window:
        h.attn_bias(q, ring, ring, None, i, i, i, q, 1, W, H, 1, 64, 64, 0.1, n_tiles=1, keys=keys)
    assert all((n > 0) == tiled for n in seen) and seen


@pytest.mark.parametrize("B,H,e,longest,dtype,dealt", [
    (1, 16, 128, 8, torch.float32, True), (1, 16, 128, 7, torch.float32, False), (8, 16, 128, 300, torch.float32, True), (8, 16, 129, 300, torch.float32, False),
    (4, 16, 128, 8, torch.bfloat16, True), (8, 16, 96, 100, torch.bfloat16, False), (3, 32, 128, 9, torch.bfloat16, False)])
def test_scans_that_fill_the_chip_keep_a_column_a_thread(B, H, e, longest, dtype, dealt, monkeypatch):
    seen = []
    monkeypatch.setattr(h, "lib", lambda: type("Lib", (), {n: staticmethod(lambda *a, n=n: seen.append(n) or 0) for n in ("mbh_lightning_scan", "mbh_lightning_split")}))
    monkeypatch.setattr(h, "_ptr", lambda t: None)
    monkeypatch.setattr(h, "_stream", lambda: 0)
    x, f = torch.zeros(2, 8, dtype=dtype), torch.zeros(2)
    h.lightning_scan(x, f, f, f, f, f, f, B, H, 100, e, longest=longest)
    assert seen == ["mbh_lightning_split" if dealt else "mbh_lightning_scan"]


def test_the_stream_where_torch_has_no_raw_getter(monkeypatch):
    """The handle by torch's public way."""
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream")
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: type("Stream", (), {"cuda_stream": 77}))
    spec = importlib.util.spec_from_file_location("mistral_inference_b200._abi_without_getter", _abi.__file__)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    assert module._stream() == 77


@pytest.mark.parametrize("epi,missing", [(0, "x"), (1, "w"), (0, "out"), (2, "out"), (1, "out32"), (3, "out32"), (8, "out32")])
def test_linears_without_an_operand_are_refused(epi, missing):
    from mistral_inference_b200 import _abi_hybrid as h

    p = {k: 4096 for k in ("x", "w", "out", "out32", "a_log")}  # never read: the call is refused before any launch
    p[missing] = None
    for dt in (0, 1):
        assert h.lib().mbh_linear_any(p["x"], 64, p["w"], None, p["out"], p["out32"], 32, 64, 64, epi, 0, 0.0, 0.0, None, 0, 8, p["a_log"], None, 0, dt, None) != 0
        assert "null pointer" in h.lib().mbh_last_error().decode()


@pytest.mark.parametrize("B,H,G,d,W,splits", [(1, 8, 8, 128, 4096, 37), (148, 8, 1, 128, 4096, 2), (149, 8, 1, 128, 4096, 2), (221, 8, 1, 128, 4096, 2), (222, 8, 1, 128, 4096, 1), (600, 8, 1, 128, 4096, 1),
                                              (64, 16, 1, 128, 4096, 4), (64, 16, 1, 64, 4096, 9), (64, 8, 1, 64, 4096, 4), (31, 16, 1, 64, 4096, 9), (32, 16, 1, 64, 4096, 18), (443, 16, 1, 64, 4096, 2),
                                              (444, 16, 1, 64, 4096, 1), (1, 8, 1, 128, 64, 1), (1, 8, 1, 128, 65, 2), (1, 1, 1, 64, 100000, 64)])
def test_decode_attention_fills_the_places_there_are(B, H, G, d, W, splits):
    from mistral_inference_b200 import _abi_hybrid as h

    got = h.attn_decode_splits(B, G, W, per_sm=h._decode_ctas(B, H, G, d, d, 1))
    assert got == splits and 1 <= got <= 64
    assert got <= 2 or got * B * G <= 148 * h._decode_ctas(B, H, G, d, d, 1)
