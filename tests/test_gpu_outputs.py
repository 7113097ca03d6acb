"""Caller-owned buffers of a pass: which calls touch them, what a refusal leaves behind, the cache of pinned blocks."""
import ctypes

import numpy as np
import pytest

import modelgen
from modelgen import config

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def model(pkg):
    return pkg.Model.open(modelgen.cached_gguf(config.variant(config.TINY, name="tiny-draft", vocab=4096, has_draft=1)))


def ids_of(model, n, seed):
    return np.random.default_rng(seed).integers(0, model.cfg["vocab"], n).astype(np.int32)


def test_a_refused_draft_call_does_not_read_the_rows(pkg, model):
    """The rows' copy is asynchronous when they are pinned, so a call that is refused may not have begun it: the caller is free to give the
    memory back. Here it lies in a page that cannot be read at all."""
    libc = ctypes.CDLL(None)
    libc.mmap.restype, libc.mmap.argtypes = ctypes.c_void_p, [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_long]
    page = libc.mmap(None, 1 << 16, 0, 0x22, -1, 0)   # PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS
    assert page and page != ctypes.c_void_p(-1).value
    g, L = pkg.Graph(model, n_kv=64, max_tokens=16), pkg.lib.load()
    lg, rs = ctypes.c_void_p(), ctypes.c_void_p()
    bad = np.array([model.cfg["vocab"]], dtype=np.int32)
    assert L.b200_draft_rows(g._h, page, bad.ctypes.data, 1, 0, ctypes.byref(rs), ctypes.byref(lg)) == pkg.lib.EINVAL
    small = np.empty(16, dtype=np.float32)
    good = ids_of(model, 1, 0)
    pkg.lib.check(L.b200_graph_set_outputs(g._h, small.ctypes.data, small.size, None, 0))
    assert L.b200_draft_rows(g._h, page, good.ctypes.data, 1, 0, ctypes.byref(rs), ctypes.byref(lg)) == pkg.lib.ECAPACITY
    assert g.draft_past() == 0
    h = np.random.default_rng(1).standard_normal((1, model.cfg["n_embd"])).astype(np.float32)
    got, want = g.draft_rows(h, good), pkg.Graph(model, n_kv=64, max_tokens=16).draft_rows(h, good)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_outputs_hold_for_one_call_even_one_with_null_arguments(pkg, model):
    L = pkg.lib.load()
    g = pkg.Graph(model, n_kv=64, max_tokens=16)
    V = model.cfg["vocab"]
    lg, rs = ctypes.c_void_p(), ctypes.c_void_p()
    out, one = (ctypes.byref(lg), ctypes.byref(rs)), ids_of(model, 1, 2)
    calls = (lambda: L.b200_graph_forward(g._h, None, 1, *out), lambda: L.b200_graph_extend(g._h, None, 1, *out), lambda: L.b200_graph_extend_input(g._h, None, *out),
             lambda: L.b200_graph_extend_rows(g._h, None, 1, *out), lambda: L.b200_graph_extend_residual(g._h, None, 1, *out),
             lambda: L.b200_graph_decode_rows(g._h, None, one.ctypes.data, 1, out[0]), lambda: L.b200_draft_rows(g._h, None, one.ctypes.data, 1, 0, *out))
    for call in calls:
        mine = np.full(V, 7.0, dtype=np.float32)
        pkg.lib.check(L.b200_graph_set_outputs(g._h, mine.ctypes.data, V, None, 0))
        assert call() == pkg.lib.EINVAL
        pkg.lib.check(L.b200_graph_extend(g._h, one.ctypes.data, 1, *out))
        assert lg.value != mine.ctypes.data and (mine == 7.0).all()


def test_outputs_of_a_call_that_was_not_made_are_dropped(pkg, model):
    g = pkg.Graph(model, n_kv=64, max_tokens=16)
    blocks = []

    def interrupted(lg, rs):
        blocks.append(True)
        raise KeyboardInterrupt

    big = (16, model.cfg["vocab"])   # large enough for a pinned block
    with pytest.raises(KeyboardInterrupt):
        g._results(interrupted, big)
    one = ids_of(model, 1, 3)
    lg, rs = ctypes.c_void_p(), ctypes.c_void_p()
    pkg.lib.check(pkg.lib.load().b200_graph_extend(g._h, one.ctypes.data, 1, ctypes.byref(lg), ctypes.byref(rs)))
    first = lg.value
    pkg.lib.check(pkg.lib.load().b200_graph_extend(g._h, one.ctypes.data, 1, ctypes.byref(lg), ctypes.byref(rs)))
    assert blocks and first == lg.value   # the graph's own buffer both times


@pytest.mark.parametrize("call", ["forward", "extend", "extend_residual"])
def test_a_prompt_whose_outputs_do_not_fit_leaves_the_slot_alone(pkg, model, call):
    """Twenty tokens are three passes of at most eight: the refusal comes before the first, not with the logits of the last."""
    L = pkg.lib.load()
    V, H = model.cfg["vocab"], model.cfg["n_embd"]
    head, ids = ids_of(model, 5, 4), ids_of(model, 20, 5)
    g, plain = (pkg.Graph(model, n_kv=64, max_tokens=8, use_cuda_graph=False) for _ in range(2))
    for x in (g, plain):
        x.forward(head)
    lg, rs = ctypes.c_void_p(), ctypes.c_void_p()
    n = 8 if call == "extend_residual" else 20   # a pass returns every row's residual, so all of them in one
    small = np.empty(V, dtype=np.float32)
    if call == "extend_residual":
        rows = np.empty(n * H - 1, dtype=np.float32)
        pkg.lib.check(L.b200_graph_set_outputs(g._h, small.ctypes.data, V, rows.ctypes.data, rows.size))
    else:
        pkg.lib.check(L.b200_graph_set_outputs(g._h, small.ctypes.data, V - 1, None, 0))
    assert getattr(L, "b200_graph_" + call)(g._h, ids.ctypes.data, n, ctypes.byref(lg), ctypes.byref(rs)) == pkg.lib.ECAPACITY
    assert g.past() == 5
    assert np.array_equal(g.extend(ids)[0], plain.extend(ids)[0])


def test_a_block_given_back_twice_is_handed_out_once(pkg, model):
    g, L = pkg.Graph(model, n_kv=16, max_tokens=8), pkg.lib.load()
    a = L.b200_host_acquire(g._h, 3 << 20)
    L.b200_host_release(a)
    L.b200_host_release(a)
    two = [L.b200_host_acquire(g._h, 3 << 20) for _ in range(2)]
    assert all(two) and two[0] != two[1]
    for p in two:
        L.b200_host_release(p)
    L.b200_host_release(None)
    L.b200_host_release(ctypes.c_void_p(12345))   # nobody's block


def test_the_cache_of_blocks_is_bounded(pkg, model):
    g, L = pkg.Graph(model, n_kv=16, max_tokens=8), pkg.lib.load()
    blocks = []
    while len(blocks) < 9 and (p := L.b200_host_acquire(g._h, 256 << 20)):
        blocks.append(p)
    assert 1 <= len(blocks) <= 4 and len(set(blocks)) == len(blocks)   # 1 GiB in all, whatever other tests hold of it
    ids = ids_of(model, 16, 6)
    got = g.extend_rows(ids[:8])                                       # no block to be had: the graph's own buffers, copied
    assert all(np.array_equal(a, b) for a, b in zip(got, pkg.Graph(model, n_kv=16, max_tokens=8).extend_rows(ids[:8])))
    for p in blocks:
        L.b200_host_release(p)
    p = L.b200_host_acquire(g._h, 256 << 20)
    assert p
    L.b200_host_release(p)


def test_pageable_and_pinned_buffers_get_the_same_results(pkg, model):
    L = pkg.lib.load()
    V, H, n = model.cfg["vocab"], model.cfg["n_embd"], 3
    ids = ids_of(model, n, 7)
    want = pkg.Graph(model, n_kv=16, max_tokens=8).extend_rows(ids)
    g = pkg.Graph(model, n_kv=16, max_tokens=8)
    block = L.b200_host_acquire(g._h, 4 * n * (V + H))
    pinned = np.ctypeslib.as_array(ctypes.cast(block, ctypes.POINTER(ctypes.c_float)), (n * (V + H),))
    for buf in (np.zeros(n * (V + H), dtype=np.float32), pinned):
        g.reset()
        at = buf.ctypes.data
        pkg.lib.check(L.b200_graph_set_outputs(g._h, at, n * V, at + 4 * n * V, n * H))
        lg, rs = ctypes.c_void_p(), ctypes.c_void_p()
        pkg.lib.check(L.b200_graph_extend_rows(g._h, ids.ctypes.data, n, ctypes.byref(lg), ctypes.byref(rs)))
        assert (lg.value, rs.value) == (at, at + 4 * n * V)
        assert np.array_equal(buf[:n * V].reshape(n, V), want[0]) and np.array_equal(buf[n * V:].reshape(n, H), want[1])
    L.b200_host_release(block)
