"""The few-row products (16 or 32 rows a tile, the weight stream dealt to the SMs in k-steps) where they can go wrong: row counts around a
tile, inner and outer sizes that end inside a k-step or a tile, the common part of a batch's prompts.  Against the decode engine, whose products
run row by row (and which reads a single request's prompt of fewer than 33 tokens itself)."""
import numpy as np
import pytest

from helpers import make_model, prompt_tokens

pytestmark = pytest.mark.gpu

# sizes that end inside a 64-wide k-step and a 128-wide column tile; one head of 40 values
SMALL = dict(vocab=163, hidden=160, layers=2, heads=4, inter=264)
WIDE = dict(vocab=161, hidden=384, layers=1, heads=3, inter=1096)
# the integer products are exact; norms, attention and softmax are fp32 sums in another order: a few 2^-24 of the largest value per sum and layer
TOL = 64 * 2.0 ** -24


def model(meta, qt, **kw):
    import turboinfer_b200 as tb
    tb.init(0)
    return tb.Model(meta, qt, attn_mode=1, rope_mode=1, max_seq=160, **kw).load(make_model(meta, norm_jitter=0.1))


@pytest.mark.parametrize("qt", ["Q_INT8", "Q_INT4"])
@pytest.mark.parametrize("meta", [SMALL, WIDE], ids=["small", "wide"])
def test_short_prompts_equal_the_decode_engine(monkeypatch, meta, qt):
    import turboinfer_b200 as tb
    out = []
    for path in ("", "decode"):
        monkeypatch.setenv("TURBOINFER_B200_PREFILL", path)
        m = model(meta, getattr(tb, qt))
        out.append([m.prefill(prompt_tokens(n, meta["vocab"], offset=n)) for n in (5, 6, 7, 15, 16, 17, 31, 32, 33)])
        m.free()
    for got, want in zip(*out):
        assert np.abs(got - want).max() <= TOL * np.abs(want).max()


@pytest.mark.parametrize("qt", ["Q_INT8", "Q_INT4"])
@pytest.mark.parametrize("meta", [SMALL, WIDE], ids=["small", "wide"])
def test_common_part_of_one_prompt(monkeypatch, meta, qt):
    import turboinfer_b200 as tb
    monkeypatch.setenv("TURBOINFER_B200_PREFILL", "")
    m = model(meta, getattr(tb, qt))
    prompts = [prompt_tokens(n, meta["vocab"], offset=n) for n in (3, 6, 7, 16, 17, 18, 32, 33, 34)]   # 2 .. 33 rows at once
    got = [m.generate_batch_greedy(np.array([p], dtype=np.int32), 1, want_logits=True)[1][0] for p in prompts]
    monkeypatch.setenv("TURBOINFER_B200_PREFILL", "decode")
    want = [m.prefill(p) for p in prompts]
    m.free()
    for g, w in zip(got, want):
        assert np.abs(g - w).max() <= TOL * np.abs(w).max()


@pytest.mark.parametrize("qt", ["Q_INT8", "Q_INT4"])
@pytest.mark.parametrize("lens", [[1], [2, 2], [9] * 15, [3] * 16, [4, 70] * 8 + [5], [12] * 31, [6] * 32, [2] * 33, [40, 41, 39]], ids=lambda v: f"{len(v)}x{min(v)}")
def test_batches_equal_the_decode_engine(monkeypatch, lens, qt):
    import turboinfer_b200 as tb
    meta = SMALL if len(lens) != 16 else WIDE
    prompts = [prompt_tokens(n, meta["vocab"], offset=3 * b) for b, n in enumerate(lens)]
    m = model(meta, getattr(tb, qt))
    equal = len(set(lens)) == 1
    if equal:
        toks, logits, _ = m.generate_batch_greedy(np.array(prompts, dtype=np.int32), 5, want_logits=True)
    else:
        toks = m.generate_batch_ragged(prompts, 5)[0]
    monkeypatch.setenv("TURBOINFER_B200_PREFILL", "decode")
    for b, p in enumerate(prompts):
        st, sl, _ = m.generate_greedy(p, 5, want_logits=True)
        assert np.array_equal(toks[b], st)
        if equal:
            assert np.abs(logits[b] - sl[-1]).max() <= TOL * np.abs(sl[-1]).max()
    m.free()
