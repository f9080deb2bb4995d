"""Many-row products of the layered sequence engine (bf16 mode, CTA pairs on tcgen05) at the edges of their tiles: row counts around 128 and
256, column counts that are no multiple of a tile, of 32 or of 4, inner sizes that end inside a k-step, activated columns that start off a
16-byte boundary.  Against the plain float64 implementation."""
import numpy as np
import pytest

import binusun_cases
import binusun_plain
import nubipel_cases
import nubipel_plain

pytestmark = pytest.mark.gpu

# every product rounds its rows to bf16 (2^-9 of a value); a dozen such roundings in a row, largest error over the largest logit
TOL = 12 * 2.0 ** -9


def one_step(m, toks):
    s = m.open()
    out = m.step([(s, toks)], [range(len(toks))])
    m.close(s)
    return out


@pytest.mark.parametrize("rows", [33, 64, 127, 128, 129, 255, 256, 257, 520])
@pytest.mark.parametrize("width,ff,vocab", [(72, 328, 133), (264, 1000, 300), (64, 64, 64)])
def test_rows_and_columns_around_tiles(rows, width, ff, vocab):
    cfg = binusun_cases.make_config([binusun_cases.attn_layer(heads=3, kv_heads=1, dim=40, vdim=24, rot_dims=8, window=50, ff=ff)], vocab=vocab, width=width)
    W = binusun_cases.random_weights(cfg, seed=rows)
    toks = [int(t) for t in np.random.default_rng(rows).integers(0, vocab, rows)]
    m = binusun_cases.build_engine(cfg, W, "bfloat16")
    got = one_step(m, toks)
    m.free()
    want = binusun_plain.forward(cfg, W, toks)
    assert np.abs(got - want).max() <= TOL * np.abs(want).max()


@pytest.mark.parametrize("rows", [40, 200, 257])
@pytest.mark.parametrize("heads,ff", [(4, 64), (3, 72), (5, 200)])   # q, k, v columns in front of the activated ones: 176, 132, 220
def test_activated_columns(rows, heads, ff):
    cfg = nubipel_cases.make_config([nubipel_cases.attn(heads=heads, kv_heads=1, dim=12, vdim=20, chunk=24, mlp=nubipel_cases.dense(ff)),
                                     nubipel_cases.latent(mlp=nubipel_cases.dense(ff))], width=136, vocab=140)
    W = nubipel_cases.random_weights(cfg, seed=rows + ff)
    toks = [int(t) for t in np.random.default_rng(rows).integers(0, cfg["vocab"], rows)]
    m = nubipel_cases.build_engine(cfg, W, "bfloat16")
    got = one_step(m, toks)
    m.free()
    want, _ = nubipel_plain.run(cfg, W, toks)
    assert np.abs(got - want).max() <= TOL * np.abs(want).max()


@pytest.mark.parametrize("dim", [32, 64, 128])
@pytest.mark.parametrize("first,rows", [(0, 64), (0, 79), (5, 65), (33, 96), (70, 200)])
def test_recurrence_in_chunks_equals_tokens(dim, first, rows):
    """Portions of 64 rows and more run the wkv recurrence in chunks of 16 tokens, shorter ones token by token: the same rows both ways, from a
    fresh state and behind earlier tokens, with a second request of its own length in the step."""
    cfg = binusun_cases.make_config([binusun_cases.wkv_layer(heads=2, dim=dim, rank=8), binusun_cases.wkv_layer(heads=2, dim=dim, rank=8, ff=64)], width=64)
    W = binusun_cases.random_weights(cfg, seed=first + rows, decay_bias=-2.0)
    rng = np.random.default_rng(rows)
    toks, other = [[int(t) for t in rng.integers(0, cfg["vocab"], n)] for n in (first + rows, 17)]
    m = binusun_cases.build_engine(cfg, W, "float32")
    s, o = m.open(), m.open()
    got = []
    if first:
        got.append(m.step([(s, toks[:first])], [range(first)]))
    both = m.step([(o, other), (s, toks[first:])], [range(17), range(rows)])
    got.append(both[17:])
    m.free()
    # fp32 throughout; sums of up to 16 tokens and 128 channels in another order
    for want, g in ((binusun_plain.forward(cfg, W, toks), np.concatenate(got)), (binusun_plain.forward(cfg, W, other), both[:17])):
        assert np.abs(g - want).max() <= 2e-4 * np.abs(want).max()


@pytest.mark.parametrize("rows", [33, 130])
@pytest.mark.parametrize("width,rank,ff", [(72, 64, 72), (136, 72, 200), (264, 64, 1032), (136, 32, 200), (68, 64, 68)])   # the last two: mixes in fp32
def test_mixes_and_gated_rows_in_bf16(rows, width, rank, ff):
    """Token-shift mixes and gated feed-forward rows that go to their products as bf16, for rows behind an earlier portion and of two requests."""
    cfg = binusun_cases.make_config([binusun_cases.wkv_layer(heads=2, dim=40, rank=rank, ff=ff)], width=width)
    W = binusun_cases.random_weights(cfg, seed=rows + ff, decay_bias=-2.0)
    rng = np.random.default_rng(rows)
    toks, other = [[int(t) for t in rng.integers(0, cfg["vocab"], n)] for n in (20 + rows, 35)]
    m = binusun_cases.build_engine(cfg, W, "bfloat16")
    s, o = m.open(), m.open()
    head = m.step([(s, toks[:20])], [range(20)])
    both = m.step([(o, other), (s, toks[20:])], [range(35), range(rows)])
    m.free()
    for want, got in ((binusun_plain.forward(cfg, W, toks), np.concatenate([head, both[35:]])), (binusun_plain.forward(cfg, W, other), both[:35])):
        assert np.abs(got - want).max() <= TOL * np.abs(want).max()


@pytest.mark.parametrize("rows", [1, 3, 8])
@pytest.mark.parametrize("width,ff,vocab", [(256, 4736, 4753), (256, 9488, 14209), (288, 2400, 9473)])   # 16 columns x 296 blocks = 4736: one, two, three turns a block
def test_few_rows_with_several_column_tiles_a_block(rows, width, ff, vocab):
    cfg = binusun_cases.make_config([binusun_cases.attn_layer(heads=3, kv_heads=1, dim=40, vdim=24, rot_dims=8, window=50, ff=ff)], vocab=vocab, width=width)
    W = binusun_cases.random_weights(cfg, seed=rows)
    toks = [int(t) for t in np.random.default_rng(rows).integers(0, vocab, rows)]
    m = binusun_cases.build_engine(cfg, W, "bfloat16")
    got = one_step(m, toks)
    m.free()
    want = binusun_plain.forward(cfg, W, toks)
    assert np.abs(got - want).max() <= TOL * np.abs(want).max()
