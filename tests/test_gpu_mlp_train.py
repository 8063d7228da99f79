"""The training loop (two launches a step, AdamW in the weight gradients' epilogue) against the same
steps made by single calls — backward of the rows drawn, then AdamW — with the index stream and the
learning rates formed here."""

import numpy as np
import pytest

from oracle import mlp as M

pytestmark = pytest.mark.gpu


def drawn(n, count, seed):
    """Rows of the epochs of a PCG32-driven Fisher-Yates shuffle."""
    state = (seed * 6364136223846793005 + 1442695040888963407) % 2 ** 64

    def draw():
        nonlocal state
        old = state
        state = (old * 6364136223846793005 + 1442695040888963407) % 2 ** 64
        xs, rot = (((old >> 18) ^ old) >> 27) & 0xFFFFFFFF, old >> 59
        return (xs >> rot | xs << ((32 - rot) & 31)) & 0xFFFFFFFF

    perm, out, pos = list(range(n)), [], n
    while len(out) < count:
        if pos >= n:
            for k in range(n - 1, 0, -1):
                j = draw() % (k + 1)
                perm[k], perm[j] = perm[j], perm[k]
            pos = 0
        out.append(perm[pos])
        pos += 1
    return out


@pytest.mark.parametrize("width,depth,n_out,n,batch", [(64, 2, 24, 40, 24), (256, 3, 64, 1300, 1250), (1024, 2, 1024, 1240, 1233)])
def test_training_loop_is_its_steps(width, depth, n_out, n, batch):
    """Both ways run the same products; bias corrections and updates may differ by some float roundings, which can
    move a weight's BF16 value by one step. Gradients then differ by (depth + 1) 2^-8 forward and as much
    again backward, as in the row kernels' test, and the parameters' change with them."""
    from nofluidx3d_gb300.mlp import MLP

    steps, lr, lr_min, wd = 5, 1e-3, 1e-4, 0.01
    shape = M.MLPShape(n_in=6, width=width, depth=depth, n_out=n_out)
    rng = np.random.default_rng(n)
    p0 = shape.init(3)
    x = rng.uniform(-1, 1, (n, 6)).astype(np.float32)
    t = rng.normal(0, 1, (n, n_out)).astype(np.float32)
    w = rng.uniform(0.5, 2, n).astype(np.float32)
    idx = drawn(n, steps * batch, 11)
    with MLP(6, width, depth, n_out, max_batch=batch) as a, MLP(6, width, depth, n_out, max_batch=batch) as b:
        a.set_params(p0)
        losses = a.train(x, t, steps=steps, batch=batch, lr=lr, lr_min=lr_min, weight_decay=wd, weight=w, seed=11)
        b.set_params(p0)
        want = []
        for s in range(steps):
            rows = idx[s * batch:(s + 1) * batch]
            want.append(b.backward(x[rows], t[rows], w[rows], scale=1.0 / batch).astype(np.float64).mean())
            b.adamw(lr_min + 0.5 * (lr - lr_min) * (1 + np.cos(np.pi * s / (steps - 1))), weight_decay=wd)
        pa, pb = a.params().astype(np.float64), b.params().astype(np.float64)
    tol = 2 * (depth + 1) * 2.0 ** -8
    np.testing.assert_allclose(losses, want, rtol=tol)
    assert np.linalg.norm(pa - pb) < 2 * tol * np.linalg.norm(pb - p0)
