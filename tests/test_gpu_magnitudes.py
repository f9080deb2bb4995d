"""Prompt rows whose attention is fp32 whatever the size of their queries, keys and values: the common part of a batch's prompts, and the last row
of a prompt.  A factor of a power of two on one projection and its inverse on another leaves the model as it is."""
import numpy as np
import pytest

from helpers import make_model, prompt_tokens

pytestmark = pytest.mark.gpu

# fp32 sums in another order: a few 2^-24 of the largest value per sum and layer
TOL = 64 * 2.0 ** -24


def scaled(meta, q, k, v):
    w = make_model(meta, norm_jitter=0.1)
    for l in range(meta["layers"]):
        for name, e in (("q", q), ("k", k), ("v", v), ("o", -v)):
            w["layers.%d.attention.%s_proj.weight" % (l, name)] *= np.float32(2.0 ** e)
    return w


SIZES = [(0, 0, 0), (20, -20, 0), (-20, 20, 0), (0, 0, 20), (0, 0, -14), (-12, 12, -20)]


def load(meta, sizes, qt="Q_INT8"):
    import turboinfer_b200 as tb
    tb.init(0)
    return tb.Model(meta, getattr(tb, qt), attn_mode=1, rope_mode=1, max_seq=320).load(scaled(meta, *sizes))


@pytest.mark.parametrize("sizes", SIZES, ids=str)
@pytest.mark.parametrize("heads,hidden", [(2, 128), (1, 128), (3, 120)])   # heads of 64, 128 and 40
@pytest.mark.parametrize("n", [6, 17, 18, 34, 70, 150])   # 5, 16, 17, 33, 69 and 149 common tokens
def test_common_part_of_a_batch(monkeypatch, sizes, heads, hidden, n):
    common_part(monkeypatch, sizes, heads, hidden, n, 3)


@pytest.mark.parametrize("batch", [1, 2])
@pytest.mark.parametrize("n", [3, 4])
def test_two_common_tokens(monkeypatch, batch, n):
    common_part(monkeypatch, (0, 0, 0), 2, 128, n, batch)


def common_part(monkeypatch, sizes, heads, hidden, n, batch):
    meta = dict(vocab=160, hidden=hidden, layers=2, heads=heads, inter=256)
    prompts = [prompt_tokens(n, meta["vocab"], offset=3 * b) for b in range(batch)]
    m = load(meta, sizes)
    toks, logits, _ = m.generate_batch_greedy(np.array(prompts, dtype=np.int32), 3, want_logits=True)
    monkeypatch.setenv("TURBOINFER_B200_PREFILL", "decode")
    for b, p in enumerate(prompts):
        st, sl, _ = m.generate_greedy(p, 3, want_logits=True)
        assert np.array_equal(toks[b], st)
        assert np.abs(logits[b] - sl[-1]).max() <= TOL * np.abs(sl[-1]).max()
    m.free()


@pytest.mark.parametrize("sizes", SIZES, ids=str)
@pytest.mark.parametrize("heads,hidden", [(2, 128), (1, 128), (3, 120)])
@pytest.mark.parametrize("n", [33, 64, 129, 300])
def test_last_row_of_a_prompt(monkeypatch, sizes, heads, hidden, n):
    # one layer: the logits hang on the last row's attention alone
    meta = dict(vocab=160, hidden=hidden, layers=1, heads=heads, inter=256)
    out = []
    for path in ("", "decode"):
        monkeypatch.setenv("TURBOINFER_B200_PREFILL", path)
        m = load(meta, sizes)
        out.append(m.prefill(prompt_tokens(n, meta["vocab"])))
        m.free()
    assert np.abs(out[0] - out[1]).max() <= TOL * np.abs(out[1]).max()


@pytest.mark.parametrize("qt", ["Q_INT8", "Q_INT4"])
@pytest.mark.parametrize("sizes", SIZES, ids=str)
def test_short_prompts_run_token_by_token(monkeypatch, sizes, qt):
    meta = dict(vocab=160, hidden=128, layers=2, heads=2, inter=256)
    lens = (1, 5, 6, 7, 16, 31, 32)
    out = []
    for path in ("", "decode"):
        monkeypatch.setenv("TURBOINFER_B200_PREFILL", path)
        m = load(meta, sizes, qt)
        out.append([m.prefill(prompt_tokens(n, meta["vocab"], offset=n)) for n in lens])
        m.free()
    for got, want in zip(*out):
        assert np.array_equal(got, want)
