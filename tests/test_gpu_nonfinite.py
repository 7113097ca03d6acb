"""Rows that are not finite (a damaged embedding, a damaged router) spoil their own results and nothing else: whatever the logits, the
selected experts stay in range, since they index counters, work lists and weights."""
import numpy as np
import pytest

import modelgen
from modelgen import gguf

pytestmark = pytest.mark.gpu

BAD = 77   # the token whose embedding is NaN


@pytest.fixture(scope="module")
def models(pkg, tiny_path):
    r = gguf.Reader(tiny_path)
    cfg = gguf.model_config(r.kv, r.tensors)
    tensors = {t: (typ, tuple(dims), np.array(data, dtype=np.uint8).ravel()) for t, (typ, dims, data) in r.tensors.items()}

    def with_nan(name, row, offset, every):
        """A copy of `tensors` in which the fp16 block scales of one row are NaN."""
        typ, dims, data = tensors[name]
        rb = gguf.row_bytes(typ, dims[0])
        data = data.copy()
        for b in range(row * rb, (row + 1) * rb, every):
            data[b + offset:b + offset + 2] = (0x00, 0x7E)
        return {**tensors, name: (typ, dims, data)}

    return dict(good=pkg.Model.from_tensors(cfg, tensors), embedding=pkg.Model.from_tensors(cfg, with_nan("token_embd.weight", BAD, 208, 210)),
                router=pkg.Model.from_tensors(cfg, with_nan("blk.1.ffn_gate_inp.weight", 5, 0, 34)))


def in_range(g, rows, model):
    topk = g.trace(rows)["topk"]
    assert topk.min() >= 0 and topk.max() < model.cfg["n_expert"], (topk.min(), topk.max())
    assert all(len(set(r)) == len(r) for r in topk.reshape(-1, topk.shape[-1]).tolist())


# rows per pass where the routing and the experts change kernels: per row, work lists, GEMMs over expert-sorted rows, a warp per row
@pytest.mark.parametrize("n", [1, 5, 12, 40, 300, 512])
def test_a_damaged_row_leaves_the_others_alone(pkg, models, n):
    ids = np.random.default_rng(n).integers(100, 2000, n).astype(np.int32)
    spoilt = ids.copy()
    spoilt[n // 2] = BAD
    others = np.arange(n) != n // 2
    want = pkg.Graph(models["good"], n_kv=16, max_tokens=max(n, 16), slots=n).decode_rows(np.arange(n), ids)
    for trace in (True, False):
        g = pkg.Graph(models["embedding"], n_kv=16, max_tokens=max(n, 16), slots=n, trace=trace)
        got = g.decode_rows(np.arange(n), spoilt)
        assert not np.isfinite(got[n // 2]).any()
        assert np.array_equal(got[others].view(np.uint32), want[others].view(np.uint32))
        if trace:
            in_range(g, n, models["embedding"])


@pytest.mark.parametrize("n", [1, 3, 12, 40, 200, 600])
def test_a_damaged_router_selects_experts_that_exist(pkg, models, n):
    ids = np.random.default_rng(n).integers(100, 2000, n).astype(np.int32)
    g = pkg.Graph(models["router"], n_kv=640, max_tokens=640, trace=True)
    logits, _ = g.forward(ids)
    assert not np.isfinite(logits).any()
    in_range(g, n, models["router"])
    want, _ = pkg.Graph(models["good"], n_kv=640, max_tokens=640).forward(ids)
    assert np.isfinite(want).all()
