"""How far the exact K-quant projections are from f64. A row's sum of scale x quant x activation and its min term are each two to three times
their difference, and each is carried through a few f32 roundings: seven roundings of the result, 2^-24 each, as a relative 2-norm.
(Measured: up to 2.6e-7 for eight rows and fewer, 3.6e-7 above. Quants 24 binary places down, where the tensor core drops low bits of
subnormals: 4e-7 to 1.1e-6; tcgen05 over quants that are not centred: 5e-7 to 8e-7.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 8, 12, 64])
@pytest.mark.parametrize("rows,k", [(512, 512), (2048, 2048), (1024, 4096)])
@pytest.mark.parametrize("typ", [12, 13])
def test_exact_projections_in_f32_precision(pkg, orc, typ, rows, k, m):
    rng = np.random.default_rng(typ * rows + k + m)
    q = orc.quantize(typ, (0.02 * rng.standard_normal((rows, k))).astype(np.float32))
    x = rng.standard_normal((m, k)).astype(np.float16).astype(np.float32)
    want = x.astype(np.float64) @ orc.dequantize(typ, q, rows * k).reshape(rows, k).astype(np.float64).T
    error = np.linalg.norm(pkg.qgemv(typ, q, rows, k, x) - want) / np.linalg.norm(want)
    print(typ, rows, k, m, error)
    assert error <= 7 * 2.0 ** -24, error
