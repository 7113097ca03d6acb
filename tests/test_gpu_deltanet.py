"""The recurrence of many-row passes (conv, gates, L2 norms, delta rule) against the token-by-token recurrence in f64
(llm/deltanet.go:305-418), at the ends of chunks and of the token-by-token form. Everything is f32 in the reference's device path, so the
bound is that of f32: a read-out is formed from k, v, the state's product with k, the update, q and the state's product with q, each with
an error of about one rounding, 2^-24, as a relative 2-norm: six of them, 3.6e-7. (Measured: up to 3.1e-7. With the chunks' large products
summed by the tensor core 4.1e-7 to 4.7e-7, with their decays' logarithms in f32 too 9e-7, and 1.4e-5 for a state.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D, TOL = 128, 6 * 2.0 ** -24


def inputs(rows, hk, hv, n_embd, slow, seed):
    rng = np.random.default_rng(seed)

    def f(std, *shape):
        return (std * rng.standard_normal(shape)).astype(np.float32)

    cw = (2 * hk + hv) * D
    return dict(proj=f(0.9, rows, cw + hv * D), x=f(1.0, rows, n_embd).astype(np.float16).astype(np.float32), alpha_w=f(0.02, hv, n_embd),
                beta_w=f(0.02, hv, n_embd), conv_w=f(0.5, cw, 4), ssm_a=(-np.exp(rng.uniform(0, np.log(16), hv)) * slow).astype(np.float32),
                dt_bias=f(0.02, hv), state=f(0.05, hv, D, D))


def recurrence(hk, proj, x, alpha_w, beta_w, conv_w, ssm_a, dt_bias, state):
    t = {k: np.asarray(v, dtype=np.float64) for k, v in locals().items() if k != "hk"}
    rows, hv = proj.shape[0], alpha_w.shape[0]
    cw = (2 * hk + hv) * D
    past = np.vstack([np.zeros((3, cw)), t["proj"][:, :cw]])
    c = sum(past[i:i + rows] * t["conv_w"][:, i] for i in range(4))
    c = c / (1 + np.exp(-c))
    q, k, v = (a.reshape(rows, -1, D) for a in np.split(c, [hk * D, 2 * hk * D], axis=1))
    q, k = (a / np.sqrt((a * a).sum(-1, keepdims=True) + 1e-6) for a in (q, k))
    alpha, beta = t["x"] @ t["alpha_w"].T, 1 / (1 + np.exp(-(t["x"] @ t["beta_w"].T)))
    g = np.exp(np.log1p(np.exp(alpha + t["dt_bias"])) * t["ssm_a"])
    head = np.arange(hv) % hk
    s, out = t["state"].copy(), np.zeros((rows, hv, D))
    for i in range(rows):
        s *= g[i][:, None, None]
        d = (v[i] - np.einsum("hji,hi->hj", s, k[i][head])) * beta[i][:, None]
        s += d[:, :, None] * k[i][head][:, None, :]
        out[i] = np.einsum("hji,hi->hj", s, q[i][head]) / np.sqrt(D)
    return out.reshape(rows, -1), s


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("slow", [1.0, 0.01])
@pytest.mark.parametrize("rows,hk,hv,n_embd", [(2, 2, 4, 256), (17, 2, 4, 512), (63, 2, 4, 256), (64, 2, 4, 256), (65, 4, 4, 256), (129, 2, 6, 768), (701, 2, 4, 256), (320, 16, 32, 2048)])
def test_recurrence_in_f32_precision(pkg, rows, hk, hv, n_embd, slow):
    d = inputs(rows, hk, hv, n_embd, slow, rows)
    want, want_state = recurrence(hk, **d)
    out, state = pkg.deltanet(hk, **d)
    errors = rel(out, want), rel(state, want_state)
    print(rows, slow, errors)
    assert max(errors) <= TOL, errors
