"""Attention of many-row passes alone, against f64: query tiles, key tiles and cut keys that end whole or ragged, on both head shapes.
Scores and sums are f32; what rounds are the probabilities, the result (fp16 both, 2.1e-4 of a value each on average) and nothing else, so
a relative 2-norm of 2^-11.5 (3.4e-4) over all rows and twice that over any one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = {256: (16, 2), 128: (8, 2)}   # head dims: query heads, KV heads


def inputs(dims, rows, cells, sharp):
    heads, kv = SHAPES[dims]
    rng = np.random.default_rng(rows + cells + dims)

    def f(std, *shape):
        return (std * rng.standard_normal(shape)).astype(np.float16).astype(np.float32)

    return f(sharp, rows, heads, dims), f(1.0, cells, kv, dims), f(0.5, cells, kv, dims), rng.standard_normal((rows, heads, dims)).astype(np.float32)


def attention(q, k, v, gate):
    rows, heads, dims = q.shape
    cells, kv = k.shape[:2]
    out = np.empty(q.shape)
    for h in range(heads):
        s = q[:, h].astype(np.float64) @ k[:, h * kv // heads].astype(np.float64).T / np.sqrt(dims)
        s[np.arange(cells)[None] > np.arange(cells - rows, cells)[:, None]] = -np.inf
        p = np.exp(s - s.max(-1, keepdims=True))
        out[:, h] = p @ v[:, h * kv // heads].astype(np.float64) / p.sum(-1, keepdims=True)
    return out / (1 + np.exp(-gate.astype(np.float64)))


def errors(got, want):
    d, n = np.linalg.norm(got - want, axis=-1), np.linalg.norm(want, axis=-1)
    return float(np.linalg.norm(d) / np.linalg.norm(n)), float((d / n).max())


@pytest.mark.parametrize("dims", [256, 128])
@pytest.mark.parametrize("rows,cells,parts", [(16, 16, 1), (16, 128, 1), (17, 129, 1), (33, 256, 1), (100, 255, 1), (128, 128, 1), (64, 512, 1), (40, 513, 1), (256, 1024, 1),
                                              (200, 1003, 1), (16, 1024, 8), (24, 1152, 8), (31, 2048, 8), (130, 3000, 4), (16, 4096, 32), (300, 4095, 8)])
def test_every_row_in_full(pkg, dims, rows, cells, parts):
    x = inputs(dims, rows, cells, 1.0)
    total, worst = errors(pkg.attention(*x, parts=parts), attention(*x))
    print(dims, rows, cells, parts, total, worst)
    assert total <= 2.0 ** -11.5 and worst <= 2.0 ** -10.5, (total, worst)


@pytest.mark.parametrize("dims", [256, 128])
@pytest.mark.parametrize("cells", [512, 2048])
def test_large_probabilities_lose_nothing(pkg, dims, cells):
    """Peaked scores: a few cells have nearly all the weight, the largest probability is exactly 1 and the sum is of rounded ones, so little
    more is left than the rounding of the result. (A largest probability that is anything up to 256 leaves 1.3 times that.)"""
    x = inputs(dims, 64, cells, 4.0)
    want = attention(*x)
    total, _ = errors(pkg.attention(*x), want)
    rounding, _ = errors(want.astype(np.float16).astype(np.float64), want)
    print(dims, cells, total, rounding)
    assert total <= 1.08 * rounding, (total, rounding)


def test_attention_refusals(pkg):
    q, k, v, gate = inputs(128, 16, 32, 1.0)
    for bad in ((q[:8], k, v, gate[:8], 1), (q, k[:8], v[:8], gate, 1), (q, k, v, gate, 0), (q[:, :6], k, v, gate[:, :6], 1)):
        with pytest.raises(pkg.lib.B200Error):
            pkg.attention(*bad)
