"""A token whose values are not finite touches the rows that see it, not the ones in front of it."""
import numpy as np
import pytest

import binusun_cases
import binusun_plain

pytestmark = pytest.mark.gpu

# rows of bf16 products (2^-9 of a value), a dozen roundings; fp32 sums in another order otherwise
TOL = {"bfloat16": 12 * 2.0 ** -9, "float32": 2e-4}


def rows_in_front(cfg, dtype, n, at, value):
    """The first `at` rows of a portion of n tokens whose token number `at` has an embedding of `value`, and what they ought to be."""
    W = binusun_cases.random_weights(cfg, seed=n + at, decay_bias=-2.0)
    bad = cfg["vocab"] - 1
    toks = [int(t) for t in np.random.default_rng(at).integers(0, bad, n)]
    toks[at] = bad
    want = binusun_plain.forward(cfg, W, toks[:at])
    W["embed"][bad] = value
    m = binusun_cases.build_engine(cfg, W, dtype)
    s = m.open()
    got = m.step([(s, toks)], [range(n)])
    m.free()
    return got[:at], want


@pytest.mark.parametrize("dim", [32, 64, 128])
@pytest.mark.parametrize("at,value", [(37, np.inf), (63, np.nan), (65, -np.inf)])   # inside, at the end and at the beginning of a chunk of 16
def test_recurrence_in_chunks_is_causal(dim, at, value):
    cfg = binusun_cases.make_config([binusun_cases.wkv_layer(heads=2, dim=dim, rank=8)], width=64)
    got, want = rows_in_front(cfg, "float32", 90, at, value)
    assert np.abs(got - want).max() <= TOL["float32"] * np.abs(want).max()


@pytest.mark.parametrize("window", [1000, 40])
@pytest.mark.parametrize("at,rows,free", [(100, 130, 64), (70, 128, 64), (127, 200, 64), (128, 200, 128), (200, 300, 192)])
def test_attention_of_earlier_key_tiles(window, at, rows, free):
    # rows in front of the 64-key tile that holds the token do not multiply its values, not even by zero
    cfg = binusun_cases.make_config([binusun_cases.attn_layer(heads=4, kv_heads=2, dim=64, vdim=64, rot_dims=8, window=window)], width=64)
    got, want = rows_in_front(cfg, "bfloat16", rows, at, np.inf)
    assert np.abs(got[:free] - want[:free]).max() <= TOL["bfloat16"] * np.abs(want[:free]).max()


def test_attention_of_rows_behind_the_window():
    # ... and rows whose window begins behind that tile neither, although the first rows of their block of 128 see it
    cfg = binusun_cases.make_config([binusun_cases.attn_layer(heads=4, kv_heads=2, dim=64, vdim=64, rot_dims=8, window=30)], width=64)
    W = binusun_cases.random_weights(cfg, seed=3)
    toks = [int(t) for t in np.random.default_rng(3).integers(0, cfg["vocab"] - 1, 128)]
    want = binusun_plain.forward(cfg, W, toks)
    toks[20] = cfg["vocab"] - 1
    W["embed"][cfg["vocab"] - 1] = np.nan
    m = binusun_cases.build_engine(cfg, W, "bfloat16")
    got = m.step([(m.open(), toks)], [range(128)])
    m.free()
    assert np.abs(got[94:] - want[94:]).max() <= TOL["bfloat16"] * np.abs(want[94:]).max()   # (row 93 sees key 64)
