"""Kernels and dispatch rules at the sizes where they change hands: rows per pass, ends of tiles and chunks, cut keys."""
import numpy as np
import pytest

import modelgen
from parity import compare

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tiny(pkg, tiny_path):
    return pkg.Model.open(tiny_path)


def ids_of(model, n, seed):
    return np.random.default_rng(seed).integers(0, model.cfg["vocab"], n).astype(np.int32)


@pytest.mark.parametrize("typ", [12, 13, 14])
@pytest.mark.parametrize("rows,k,m", [(1, 256, 1), (15, 512, 2), (17, 768, 3), (130, 1024, 5), (4752, 2048, 8), (2048, 4096, 1)])
def test_projection_of_at_most_eight_rows(pkg, orc, typ, rows, k, m):
    rng = np.random.default_rng(rows + k + m)
    q = orc.quantize(typ, (0.02 * rng.standard_normal((rows, k))).astype(np.float32))
    x = rng.standard_normal((m, k)).astype(np.float32)
    got = pkg.qgemv(typ, q, rows, k, x)
    want = x.astype(np.float16).astype(np.float64) @ orc.dequantize(typ, q, rows * k).reshape(rows, k).astype(np.float64).T
    # Q6_K integers above 2048 are rounded to fp16; the others are exact
    assert np.abs(got - want).max() <= (1e-3 if typ == 14 else 1e-5) * max(np.abs(want).max(), 1e-3)


@pytest.mark.parametrize("n", [9, 15, 16, 17, 63, 64, 65, 127, 128, 129, 193, 257, 513])
def test_one_pass_is_the_passes_of_eight_rows(pkg, tiny, n):
    ids = ids_of(tiny, n, 20 + n)
    want, _ = pkg.Graph(tiny, n_kv=640, max_tokens=8, use_cuda_graph=False).forward(ids)
    big = pkg.Graph(tiny, n_kv=640, max_tokens=640, use_cuda_graph=False)
    got, _ = big.forward(ids)
    r = compare(got, want)
    # the bounds of fp16-rounded weights with a router near-tie (as for the 300-row pass)
    assert r["rms"] <= 1e-2 * float(np.sqrt(np.mean(np.square(want)))) and r["max_abs"] <= 5e-2 * r["ref_max"], r


@pytest.mark.parametrize("context,n", [(0, 16), (100, 16), (511, 33), (1000, 24), (1003, 130)])
def test_few_query_rows_over_a_long_context_cut_the_keys(pkg, tiny, context, n):
    ids = ids_of(tiny, n, context + n)
    outs = []
    for rows in (512, 8):
        g = pkg.Graph(tiny, n_kv=1280, max_tokens=rows, use_cuda_graph=False)
        if context:
            g.synth_context(context, seed=5)
        outs.append(g.extend(ids)[0])
    r = compare(*outs)
    assert r["rms"] <= 1e-2 * float(np.sqrt(np.mean(np.square(outs[1])))) and r["max_abs"] <= 5e-2 * r["ref_max"], r


@pytest.mark.parametrize("n", [1, 2, 3, 5, 8])
def test_batched_rows_are_the_solo_rows_and_results_stay(pkg, tiny, n):
    g = pkg.Graph(tiny, n_kv=64, max_tokens=16, slots=8)
    ids = ids_of(tiny, 8, 3)
    solo, kept = [], []
    for s in range(n):
        g.use_slot(s); g.reset(); g.extend(ids[: 2 + s])
        ck = g.checkpoint()
        lg, hd = g.extend([int(ids[s])])
        solo.append(lg); kept.append((lg.copy(), hd, hd.copy()))
        g.restore(ck); g.checkpoint_free(ck)
    batched = g.decode_rows(list(range(n)), ids[:n])
    for s in range(n):
        assert np.array_equal(batched[s].view(np.uint32), solo[s].view(np.uint32)), s
        # what earlier calls returned is the caller's: later passes leave it alone
        assert np.array_equal(solo[s], kept[s][0]) and np.array_equal(kept[s][1], kept[s][2]), s
