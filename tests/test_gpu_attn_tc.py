"""The tcgen05 attention of prompt rows (attn_tc.cuh) at the edges of its tiles, in both engines."""
import numpy as np
import pytest

import binusun_cases
import binusun_plain
from helpers import make_model, prompt_tokens

pytestmark = pytest.mark.gpu

# products round their rows to bf16 (2^-9 of a value), a dozen in a row; the attention itself is accurate to 2^-22 of a value
TOL = 12 * 2.0 ** -9


@pytest.mark.parametrize("dim,vdim", [(64, 64), (128, 128), (40, 100), (100, 40)])
@pytest.mark.parametrize("rows,window", [(9, 1000), (64, 64), (65, 63), (127, 1), (129, 128), (193, 65), (300, 1000)])
def test_query_and_key_tiles(dim, vdim, rows, window):
    cfg = binusun_cases.make_config([binusun_cases.attn_layer(heads=4, kv_heads=2, dim=dim, vdim=vdim, rot_dims=8, window=window)], width=64)
    W = binusun_cases.random_weights(cfg, seed=rows + dim)
    toks = [int(t) for t in np.random.default_rng(rows).integers(0, cfg["vocab"], rows + 70)]
    m = binusun_cases.build_engine(cfg, W, "bfloat16")
    s = m.open()   # a portion, then one that starts inside a page behind it
    got = np.concatenate([m.step([(s, toks[:70])], [range(70)]), m.step([(s, toks[70:])], [range(rows)])])
    m.free()
    want = binusun_plain.forward(cfg, W, toks)
    assert np.abs(got - want).max() <= TOL * np.abs(want).max()


def test_more_keys_than_the_image_buffer_holds():
    # 9000 tokens x 64 key/value heads of 64: 295 MB of split keys and values, done in groups of heads.  The last row as part of the prompt
    # must agree with the same token decoded behind it.
    cfg = binusun_cases.make_config([binusun_cases.attn_layer(heads=64, kv_heads=64, dim=64, vdim=64, rot_dims=8, window=20000)], width=64)
    W = binusun_cases.random_weights(cfg, seed=4)
    toks = [int(t) for t in np.random.default_rng(5).integers(0, cfg["vocab"], 9000)]
    m = binusun_cases.build_engine(cfg, W, "bfloat16", max_tokens=2 * 9088, max_seqs=2)
    a, b = m.open(), m.open()
    whole = m.step([(a, toks)], [[8999]])
    m.step([(b, toks[:-1])])
    last = m.step([(b, toks[-1:])], [[0]])
    m.free()
    assert np.abs(whole - last).max() <= TOL * np.abs(last).max()


@pytest.mark.parametrize("heads", [1, 2])
@pytest.mark.parametrize("page", [0, 48])   # pages that are no multiple of a key tile
@pytest.mark.parametrize("n", [34, 65, 129, 193, 258])
def test_prefill_logits_equal_the_decode_engines(monkeypatch, heads, page, n):
    import turboinfer_b200 as tb
    tb.init(0)
    meta = dict(vocab=160, hidden=128, layers=2, heads=heads, inter=256)
    weights = make_model(meta, norm_jitter=0.1)
    prompt = prompt_tokens(n, meta["vocab"])
    out = []
    for path in ("", "decode"):
        monkeypatch.setenv("TURBOINFER_B200_PREFILL", path)
        m = tb.Model(meta, tb.Q_INT8, attn_mode=1, rope_mode=1, max_seq=320, kv_page_tokens=page).load(weights)
        out.append(m.prefill(prompt))
        m.free()
    # fp32 sums in another order: a few 2^-24 of the largest value per sum, two layers
    assert np.abs(out[0] - out[1]).max() <= 64 * 2.0 ** -24 * np.abs(out[1]).max()
