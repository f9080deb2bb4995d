"""Calls on a GPU that has no room for their larger buffers, and what calls allocate at all.  A shim in front of the CUDA runtime's allocation
functions (preloaded into a child process) refuses requests above a size, the device ones with the runtime's own out-of-memory error, and keeps
count."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static size_t device_limit = ~(size_t)0, pinned_limit = ~(size_t)0;
static long n_refused, n_pinned, total;
static size_t largest;
void shim_limits(size_t device, size_t pinned) { device_limit = device; pinned_limit = pinned; n_refused = n_pinned = 0; total = 0; largest = 0; }
long shim_refused(void) { return n_refused; }
long shim_pinned(void) { return n_pinned; }
long shim_total(void) { return total; }
long shim_largest(void) { return (long)largest; }
static void* real(const char* name) { return dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), name); }
int cudaMalloc(void** p, size_t n) {
    int (*f)(void**, size_t) = (int (*)(void**, size_t))real("cudaMalloc");
    if (n > device_limit) { ++n_refused; return f(p, (size_t)1 << 50); }
    total += (long)n;
    if (n > largest) largest = n;
    return f(p, n);
}
int cudaHostAlloc(void** p, size_t n, unsigned int flags) {
    int (*f)(void**, size_t, unsigned int) = (int (*)(void**, size_t, unsigned int))real("cudaHostAlloc");
    ++n_pinned;
    if (n > pinned_limit) { ++n_refused; return 2; }
    return f(p, n, flags);
}
"""

COMMON = r"""
import ctypes, os, sys
sys.path[:0] = [ROOT, os.path.join(ROOT, "tests")]
import numpy as np
shim = ctypes.CDLL(None)
NONE = 2 ** 63
def limits(device=NONE, pinned=NONE): shim.shim_limits(ctypes.c_size_t(device), ctypes.c_size_t(pinned))
for f in ("refused", "pinned", "total", "largest"): getattr(shim, "shim_" + f).restype = ctypes.c_long
import binusun_cases, binusun_plain
import turboinfer_b200 as tb
from turboinfer_b200.seq import SeqError as seq_error
from helpers import make_model, prompt_tokens
TOL16 = 12 * 2.0 ** -9   # a dozen roundings to bf16

META = dict(vocab=160, hidden=256, layers=2, heads=4, inter=1024)
def llama(**kw): return tb.Model(META, tb.Q_INT8, attn_mode=1, rope_mode=1, max_seq=160).load(make_model(META, norm_jitter=0.1))
def prompts(n, batch=4): return np.array([prompt_tokens(n, META["vocab"], offset=3 * b) for b in range(batch)], dtype=np.int32)
def alone(n, new):   # the same answers, a request at a time through the decode engine
    os.environ["TURBOINFER_B200_PREFILL"] = "decode"
    m = llama()
    out = np.array([m.generate_greedy(list(p), new)[0] for p in prompts(n)])
    m.free()
    del os.environ["TURBOINFER_B200_PREFILL"]
    return out
def seq(layers, dtype, **kw):
    cfg = binusun_cases.make_config(layers, width=64)
    W = binusun_cases.random_weights(cfg, seed=7, decay_bias=-2.0)
    return cfg, W, binusun_cases.build_engine(cfg, W, dtype, **kw)
def tokens(n, seed=1): return [int(t) for t in np.random.default_rng(seed).integers(0, 97, n)]
def close(got, want, tol): assert np.abs(got - want).max() <= tol * np.abs(want).max(), np.abs(got - want).max() / np.abs(want).max()
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("shim")
    src, lib = d / "shim.c", d / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(lib), str(src), "-ldl"], check=True)
    return str(lib)


def child(shim, code):
    p = subprocess.run([sys.executable, "-c", "ROOT = %r\n" % ROOT + COMMON + code], env=dict(os.environ, LD_PRELOAD=shim), capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout[-2000:] + p.stderr[-3000:]


def test_recurrence_without_room_for_chunks(shim):
    # 96 rows both times, in 6 chunks of 16 tokens and then in 12: there is no room for the products inside the second step's chunks
    child(shim, """
cfg, W, m = seq([binusun_cases.wkv_layer(heads=2, dim=32, rank=8)], "float32", max_seqs=10)
a = tokens(96)
s = m.open()
close(m.step([(s, a)], [range(96)]), binusun_plain.forward(cfg, W, a), 2e-4)
m.close(s)
parts = [tokens(64, 2)] + [tokens(4, 3 + i) for i in range(8)]
ids = [m.open() for _ in parts]
limits(device=20000)
got = m.step(list(zip(ids, parts)), [range(len(p)) for p in parts])
assert shim.shim_refused() > 0
close(got, np.concatenate([binusun_plain.forward(cfg, W, p) for p in parts]), 2e-4)
""")


def test_batch_after_one_without_room(shim):
    # scratch that could not be made: the call fails, and nothing of it may be left for the next one -- neither for one of the same shape,
    # whose captured steps hold the old addresses, nor for one with fewer rows
    child(shim, """
tb.init(0)
want = alone(2, 5)
m = llama()
assert np.array_equal(m.generate_batch_greedy(prompts(2), 5)[0], want)
limits(device=2000)
try:
    m.generate_batch_greedy(prompts(50), 5)
    raise SystemExit("no error")
except tb.B200Error:
    pass
limits()
assert np.array_equal(m.generate_batch_greedy(prompts(2), 5)[0], want)
assert np.array_equal(m.generate_batch_greedy(prompts(50), 5)[0], alone(50, 5))
""")


def test_first_batch_without_room(shim):
    child(shim, """
tb.init(0)
want = alone(50, 5)
m = llama()
for room in (300000, 100000, 10000, 1000):   # the failure moves forward through what a batch allocates
    limits(device=room)
    try:
        m.generate_batch_greedy(prompts(50), 5)
        raise SystemExit("no error")
    except tb.B200Error:
        pass
limits()
assert np.array_equal(m.generate_batch_greedy(prompts(50), 5)[0], want)
""")


def test_step_after_one_without_room(shim):
    child(shim, """
cfg, W, m = seq([binusun_cases.attn_layer(dim=32), binusun_cases.wkv_layer(heads=2, dim=32, rank=8)], "float32")
toks = tokens(400)
s = m.open()
got = [m.step([(s, toks[:60])], [range(60)])]
for room in (300000, 100000, 20000):   # the failure moves forward through the step's buffers
    limits(device=room)
    try:
        m.step([(s, toks[60:])], [range(340)])
        raise SystemExit("no error")
    except seq_error:
        pass
limits()
got.append(m.step([(s, toks[60:70])], [range(10)]))
got.append(m.step([(s, toks[70:])], [range(330)]))
close(np.concatenate(got), binusun_plain.forward(cfg, W, toks), 2e-4)
""")


def test_a_short_prompt_needs_no_second_copy_of_the_weights(shim):
    child(shim, """
tb.init(0)
m = llama()
limits()
for n in (5, 6, 8, 16, 31, 32):
    m.prefill(prompt_tokens(n, META["vocab"]))
    m.generate_greedy(prompt_tokens(n, META["vocab"]), 3)
assert shim.shim_total() < 100000, shim.shim_total()   # (the weights: 2 million)
""")


@pytest.mark.parametrize("room,what", [(1000000, "two sequences' rows"), (500000, "one sequence's rows"), (480000, "a step's rows only")])
def test_batch_prompts_without_room_for_their_rows(shim, room, what):
    # four prompts of 59 common tokens at once want 1.9 MB for the inner rows, one of them 483 KB; a step of the batch wants 393 KB
    child(shim, """
tb.init(0)
want2, want = alone(2, 5), alone(60, 5)
m = llama()
assert np.array_equal(m.generate_batch_greedy(prompts(2), 5)[0], want2)
limits(device=%d)
for _ in range(2): assert np.array_equal(m.generate_batch_greedy(prompts(60), 5)[0], want)
assert shim.shim_refused() > 0
assert np.array_equal(m.generate_batch_greedy(prompts(2), 5)[0], want2)
""" % room)


def test_split_keys_of_visible_pages_only(shim):
    # portions of 128 rows with windows of 100 and 300 behind up to 9000 tokens: the pages in front of the windows are neither split nor stored
    child(shim, """
layers = [binusun_cases.attn_layer(heads=4, kv_heads=4, dim=64, vdim=64, rot_dims=8, window=w) for w in (100, 300)]
cfg, W, m = seq(layers, "bfloat16", max_tokens=2 * 9088, max_seqs=2)
toks = tokens(9000)
s = m.open()
m.step([(s, toks[:512])])
limits()
for i in range(512, 8704, 512): m.step([(s, toks[i:i + 512])])
got = m.step([(s, toks[8704:8832])], [range(128)])
assert shim.shim_largest() < 3000000, shim.shim_largest()   # 512 + 300 rows in 14 pages of four heads of 32 KB; all pages: 18 MB
close(got, binusun_plain.forward(cfg, W, toks[8000:8832])[-128:], TOL16)   # (the windows reach 398 tokens back)
""")


@pytest.mark.parametrize("room", [140000, 100000])   # two key/value heads of four pages: 262 KB; one: 131 KB, then none
def test_attention_without_room_for_split_keys(shim, room):
    child(shim, """
cfg, W, m = seq([binusun_cases.attn_layer(heads=4, kv_heads=2, dim=64, vdim=64, rot_dims=8, window=1000) for _ in range(3)], "bfloat16")
toks = tokens(256)
s = m.open()
got = [m.step([(s, toks[:128])], [range(128)])]
limits(device=%d)
got.append(m.step([(s, toks[128:])], [range(128)]))
assert 0 < shim.shim_refused() <= 2, shim.shim_refused()   # (asked once a step, not once a layer)
close(np.concatenate(got), binusun_plain.forward(cfg, W, toks), TOL16)
""" % room)


def test_prompt_without_room_for_split_keys(shim):
    # a batch leaves scratch of 236 rows behind (and no images): the prompt then only lacks room for its keys and values, 262 KB for all four heads
    child(shim, """
tb.init(0)
os.environ["TURBOINFER_B200_PREFILL"] = "decode"
m = llama()
want = m.prefill(prompt_tokens(128, META["vocab"]))
m.free()
del os.environ["TURBOINFER_B200_PREFILL"]
for room in (140000, 70000, 60000):   # two heads, one, none
    m = llama()
    m.generate_batch_greedy(prompts(60), 2)
    limits(device=room)
    got = m.prefill(prompt_tokens(128, META["vocab"]))
    assert shim.shim_refused() in (1, 2, 3), shim.shim_refused()   # (asked once a prompt, not once a layer)
    limits()
    close(got, want, 64 * 2.0 ** -24)
    m.free()
""")


def test_results_without_a_pinned_buffer(shim):
    child(shim, """
limits(pinned=300000)
tb.init(0)
m = llama()
got = m.prefill(prompt_tokens(20, META["vocab"]))
cfg, W, e = seq([binusun_cases.attn_layer(dim=32)], "float32")
toks = tokens(40)
out = e.step([(e.open(), toks)], [range(40)])
assert shim.shim_refused() >= 2, shim.shim_refused()   # (one buffer a library)
close(out, binusun_plain.forward(cfg, W, toks), 2e-4)
tb.shutdown()
limits()
tb.init(0)
assert np.array_equal(got, llama().prefill(prompt_tokens(20, META["vocab"])))
""")


def test_models_pin_no_memory_of_their_own(shim):
    child(shim, """
tb.init(0)
first = llama()
_, _, e = seq([binusun_cases.attn_layer(dim=32)], "float32")
limits()
keep = [llama() for _ in range(3)] + [seq([binusun_cases.attn_layer(dim=32)], "float32")[2] for _ in range(3)]
assert shim.shim_pinned() == 0, shim.shim_pinned()
""")
