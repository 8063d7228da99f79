"""The row-wise network kernels at the sizes where they can go wrong: the smallest and widest
layers, output widths that are not multiples of 16, every number of rows a CTA takes, and batches
that leave a CTA partly filled — against the CPU oracle (same bf16 rounding points)."""

import numpy as np
import pytest

from oracle import mlp as M

pytestmark = pytest.mark.gpu

# n_in, width, depth, n_out, rows
SHAPES = [(1, 16, 1, 8, 1), (16, 48, 2, 24, 9), (6, 256, 3, 64, 65), (5, 272, 7, 40, 33), (3, 1024, 1, 1024, 17),
          (6, 64, 2, 72, 1025), (6, 32, 2, 8, 2100), (2, 80, 1, 16, 4100)]


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("n_in,width,depth,n_out,rows", SHAPES)
def test_rows_match_oracle(n_in, width, depth, n_out, rows):
    """The kernels and the oracle round activations and gradients to bf16 at the same points; the
    FP32 sums differ in order only, which can move a rounded value by one bf16 step, 2^-8 of it. At
    most every value of every layer moves: (depth + 1) 2^-8 forward, and as much again backward."""
    from nofluidx3d_gb300.mlp import MLP

    shape = M.MLPShape(n_in=n_in, width=width, depth=depth, n_out=n_out)
    rng = np.random.default_rng(width + rows)
    p = shape.init(width)
    x = rng.uniform(-1, 1, (rows, n_in)).astype(np.float32)
    t = rng.normal(0, 1, (rows, n_out)).astype(np.float32)
    w = rng.uniform(0.5, 2, rows).astype(np.float32)
    tol = (depth + 1) * 2.0 ** -8
    with MLP(n_in, width, depth, n_out, max_batch=rows) as m:
        m.set_params(p)
        assert np.array_equal(m.params(), p)
        y_ref, _ = M.forward(shape, p, x)
        assert rel(m.forward(x), y_ref) < tol
        loss, dx = m.backward(x, t, w, scale=1.0 / rows, want_dx=True)
        rows_ref, g_ref, dx_ref = M.loss_and_grads(shape, p, x, t, w, scale=1.0 / rows)
        assert rel(loss, rows_ref) < 2 * tol
        assert rel(dx, dx_ref) < 2 * tol
        assert rel(m.grads(), g_ref) < 2 * tol
        assert np.array_equal(m.backward(x, t, w, scale=1.0 / rows), loss)  # without the input gradient
        # one Adam step on the inputs: both moments are the gradient's own, so every free input moves
        # by lr g / (|g| + eps) up to a few float roundings of the step and of the input
        free = np.arange(n_in) % 3 != 2
        lo, hi = np.full(n_in, -0.9, np.float32), np.full(n_in, 0.9, np.float32)
        dxu = m.backward(x, t, w, scale=1.0, want_dx=True)[1].astype(np.float64)
        got, _ = m.fit_inputs(x, t, free, lo, hi, steps=1, lr=1e-2, eps=1e-4, weight=w)
        want = np.where(free, np.clip(x - 1e-2 * dxu / (np.abs(dxu) + 1e-4), -0.9, 0.9), x)
        np.testing.assert_allclose(got, want, rtol=0, atol=4 * 2.0 ** -24)
