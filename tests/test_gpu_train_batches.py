"""One Adam step of the epoch launch (csrc/learned.cu) over a batch of every
shape of its groups: a single row, a partial group, full groups, more groups than
blocks.  The first step moves a parameter by lr g / (|g| + eps) against the
gradient g, whose value comes from gqm_mlp_grad (checked against the CPU oracle
elsewhere).  Where |g| >= 1e-4 the order of the rows (shuffled in training)
cannot change its sign (fp32 sums of at most 8,192 terms), and eps = 1e-8 takes
less than 1e-4 of the step: within 1e-3 of lr, plus the rounding of the
parameter."""
import numpy as np
import pytest

from gpu_cdt_refine_b200 import refine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(1, 64), (33, 64), (64, 64), (1000, 1024), (4736, 4736), (5000, 8192)])
def test_first_step(gpu, n, batch):
    rng = np.random.default_rng(n)
    x = rng.normal(0, 1, (n, refine.MLP_FEATURES)).astype(np.float32)
    t = rng.uniform(0, 4, n).astype(np.float32)
    p = refine.mlp_init(n, 0.3)
    lr = 1e-3
    loss0, g = refine.mlp_grad(p, x, t)
    q, loss = refine.mlp_train(p, x, t, epochs=1, batch=batch, lr=lr, seed=3)
    assert abs(loss - loss0) <= 1e-5 * max(1.0, abs(loss0))
    big = np.abs(g) >= 1e-4
    assert big.any()
    want = p[big] - lr * np.sign(g[big])
    assert np.all(np.abs(q[big] - want) <= 1e-3 * lr + 4 * np.spacing(np.abs(want).astype(np.float32)))
    # a second call repeats it bit for bit (sums in a fixed order)
    q2, _ = refine.mlp_train(p, x, t, epochs=1, batch=batch, lr=lr, seed=3)
    assert np.array_equal(q, q2)
