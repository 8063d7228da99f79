"""The network's activation at the ends of its range, through the public calls: a hidden layer whose
sixteen units all see the same pre-activation z = 2 x, summed by weights of one, for z from -inf
to +inf. silu(z) is z / (1 + exp(-z)): zero, not z times a smallest reciprocal, far below zero,
and infinite, not NaN, at +inf."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# BF16 values: the inputs are rounded to BF16 on the way in
X = np.array([0.5, 20.0, 1e30, 2.9e38, np.inf, -8.0, -32.0, -43.0, -43.75, -44.0, -44.25, -44.5, -50.0, -1e4, -1e30, -5e36,
              -np.inf, np.nan], np.float32)


def bf16(a):
    u = np.asarray(a, np.float32).view(np.uint32).astype(np.uint64)
    r = ((u + 0x7FFF + ((u >> 16) & 1)) >> 16 << 16).astype(np.uint32).view(np.float32)
    return np.where(np.isfinite(a), r, np.asarray(a, np.float32))


@pytest.mark.parametrize("rows", [len(X), 1040, 2100, 4200])
def test_activation_over_its_whole_range(rows):
    """rows: 8, 16, 32 and 64 rows a CTA. Bound of the finite values: the hidden value and the exact
    one may round to neighbouring BF16 values, 2^-7 of it at most."""
    from nofluidx3d_gb300.mlp import MLP

    x = np.resize(bf16(X), rows).reshape(-1, 1)
    with np.errstate(over="ignore", invalid="ignore"):
        z = np.float32(2.0) * x[:, 0]
        e = np.exp(-z.astype(np.float32))  # in FP32: overflows below -88.7, where silu is zero
        want = 16.0 * (z.astype(np.float64) / (1.0 + e.astype(np.float64)))
    with MLP(1, 16, 1, 8, max_batch=rows) as m:
        p = np.zeros(m.num_params, np.float32)
        p[:16] = 2.0  # W_0; b_0 stays zero
        p[32:32 + 128] = 1.0  # W_1
        m.set_params(p)
        y = m.forward(x)[:, 0].astype(np.float64)
        finite = np.isfinite(want)
        np.testing.assert_allclose(y[finite], want[finite], rtol=2.0 ** -7, atol=0)
        assert np.array_equal(y[~finite], want[~finite], equal_nan=True)
        # the derivative: zero where exp(-z) overflows, so neither gradient nor descent moves such a row
        low = (z < -89.0) & np.isfinite(z)
        t = np.ones((rows, 8), np.float32)
        w = low.astype(np.float32)  # the other rows out of the loss
        xs = np.where(low[:, None], x, np.float32(0.0))
        loss, dx = m.backward(xs, t, w, scale=1.0, want_dx=True)
        assert np.all(loss[low] == 8.0) and np.all(dx[low] == 0.0)
        got, fit_loss = m.fit_inputs(xs, t, [True], [-3e38], [3e38], steps=2, lr=1e-2, weight=w)
        assert np.all(fit_loss[low] == 8.0) and np.array_equal(got[low], xs[low])
