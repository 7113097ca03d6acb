"""Expert kernels by weight type: Q4_K, Q5_K (rows, work lists, GEMMs) and Q6_K (work lists of the column-tiled kernel, GEMMs)."""
import numpy as np
import pytest

import modelgen
from modelgen import config, gguf
from parity import follow_pass

pytestmark = pytest.mark.gpu

TYPES = {"q4": (gguf.Q4_K, gguf.Q4_K), "q5": (gguf.Q5_K, gguf.Q5_K), "q6": (gguf.Q6_K, gguf.Q6_K)}


@pytest.fixture(scope="module", params=list(TYPES))
def typed(request, pkg):
    expert, shared = TYPES[request.param]
    cfg = config.variant(config.TINY, name=f"tiny-{request.param}-experts", vocab=4096, n_expert=8, types=dict(expert=expert, shared=shared))
    path = modelgen.cached_gguf(cfg)
    return request.param, pkg.Model.open(path), modelgen.oracle_model(path)[0]


def ids_of(n, seed):
    return np.random.default_rng(seed).integers(0, 4096, n).astype(np.int32)


@pytest.mark.parametrize("n", [1, 3, 8])
def test_streams_are_counted_once(pkg, typed, n):
    kind, model, _ = typed
    c = model.cfg
    g = pkg.Graph(model, n_kv=16, max_tokens=16, slots=n, trace=True)
    g.stats_reset()
    g.decode_rows(np.arange(n), ids_of(n, n))
    topk = g.trace(n)["topk"]
    # the row kernels stream an expert per row and slot, a work list every expert once
    want = c["n_layer"] * n * c["n_expert_used"] if kind != "q6" else sum(len(set(layer.ravel().tolist())) for layer in topk)
    assert g.stats()["expert_streams"] == want
    g.stats_reset()
    g.generate_greedy(np.arange(n), ids_of(n, n), 1)
    if kind != "q6":
        assert g.stats()["expert_streams"] == want
    else:
        assert c["n_layer"] * c["n_expert_used"] <= g.stats()["expert_streams"] <= c["n_layer"] * n * c["n_expert_used"]


# rows per pass on both sides of every change of kernel: rows on their own up to 8, work lists with exact projections to 15, with fp16-rounded ones
# from 16, GEMMs over expert-sorted rows from 32 rows per expert (64 here)
@pytest.mark.parametrize("n", [1, 9, 16, 63, 65])
def test_every_row_matches_the_oracle(pkg, orc, typed, n):
    kind, model, oracle = typed
    if kind == "q4" and n != 65:
        pytest.skip("the other tests' models have Q4_K experts")
    g, seq = pkg.Graph(model, n_kv=640, max_tokens=512, trace=True), oracle.seq()
    first = ids_of(5, 90)
    follow_pass(g, orc, seq, first, f"{kind}: five rows")
    follow_pass(g, orc, seq, ids_of(n, n), f"{kind}: {n} rows after them")


@pytest.fixture(scope="module")
def many(pkg, orc):
    """640 experts (more than one CTA's threads take two of), values drawn and quantised on the device."""
    cfg = config.variant(config.TINY, name="tiny-640-experts", n_embd=512, vocab=4096, n_expert=640, n_expert_used=6)
    model = pkg.Model.synthetic(cfg, seed=3)
    tensors = {name: (typ, tuple(dims), model.read_tensor(name)) for name, typ, dims, _ in config.manifest(cfg)}
    return model, orc.Model(config.graph_fields(cfg), tensors)


@pytest.mark.parametrize("n", [1, 7, 12, 40, 520])
def test_more_than_512_experts(pkg, orc, many, n):
    model, oracle = many
    g = pkg.Graph(model, n_kv=640, max_tokens=640, trace=True)
    follow_pass(g, orc, oracle.seq(), ids_of(n, n), f"640 experts: {n} rows")
