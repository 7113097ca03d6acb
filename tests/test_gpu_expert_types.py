"""Expert kernels by weight type: Q4_K, Q5_K (rows, work lists, GEMMs) and Q6_K (work lists of the column-tiled kernel, GEMMs)."""
import numpy as np
import pytest

import modelgen
from modelgen import config, gguf

pytestmark = pytest.mark.gpu

TYPES = {"q4": (gguf.Q4_K, gguf.Q4_K), "q5": (gguf.Q5_K, gguf.Q5_K), "q6": (gguf.Q6_K, gguf.Q6_K)}


@pytest.fixture(scope="module", params=list(TYPES))
def typed(request, pkg):
    expert, shared = TYPES[request.param]
    cfg = config.variant(config.TINY, name=f"tiny-{request.param}-experts", vocab=4096, types=dict(expert=expert, shared=shared))
    return request.param, pkg.Model.open(modelgen.cached_gguf(cfg))


def ids_of(n, seed):
    return np.random.default_rng(seed).integers(0, 4096, n).astype(np.int32)


@pytest.mark.parametrize("n", [1, 3, 8])
def test_streams_are_counted_once(pkg, typed, n):
    kind, model = typed
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
