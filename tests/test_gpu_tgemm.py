"""The exact tensor-core projection (more than eight rows): K-quant integers in fp16, block scales applied in f32 per
super-block. Against the product over the oracle's dequantised weights only the summation differs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("typ", [12, 13])
@pytest.mark.parametrize("rows,k,m", [(128, 256, 9), (16, 256, 16), (200, 512, 17), (384, 2048, 32), (144, 4096, 33), (2048, 512, 64), (272, 1024, 65), (19200, 768, 12)])
def test_exact_projection(pkg, orc, typ, rows, k, m):
    rng = np.random.default_rng(rows + 3 * k + m)
    q = orc.quantize(typ, (0.02 * rng.standard_normal((rows, k))).astype(np.float32))
    x = rng.standard_normal((m, k)).astype(np.float32)
    got = pkg.qgemv(typ, q, rows, k, x)
    w = orc.dequantize(typ, q, rows * k).reshape(rows, k).astype(np.float64)
    want = x.astype(np.float16).astype(np.float64) @ w.T
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max(), (np.abs(got - want).max(), np.abs(want).max())


def test_more_rows_than_a_grid_is_high(pkg, orc):
    rng = np.random.default_rng(9)
    q = orc.quantize(12, (0.02 * rng.standard_normal((16, 256))).astype(np.float32))
    x = rng.standard_normal((65600, 256)).astype(np.float32)
    want = x.astype(np.float16).astype(np.float64) @ orc.dequantize(12, q, 16 * 256).reshape(16, 256).astype(np.float64).T
    assert np.abs(pkg.qgemv(12, q, 16, 256, x) - want).max() <= 1e-5 * np.abs(want).max()
