"""The layer-by-layer surrogate's training step at sizes where its tiles and row maps end: rows of one
tile more or less, more rows than the row map a tile keeps in shared memory (1,024), hidden widths that
are no power of two; and AdamW in the gradient product's epilogue against the plain update."""
from __future__ import annotations

import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))
import surrogate_wide_oracle as sw  # noqa: E402

pytestmark = pytest.mark.gpu

GRAD_RTOL = 2e-3        # FP32 accumulation in another order than float64, per tensor's largest entry


@pytest.mark.parametrize("in_dim,hidden,rows", [(1, 128, 5), (130, 384, 127), (130, 384, 129), (257, 128, 1025),
                                                (1441, 256, 1300)])
def test_gradients_match_the_checker(in_dim, hidden, rows):
    from tetris_ai3_b200.surrogate import Surrogate
    d = sw.Dims(in_dim, hidden)
    rng = np.random.default_rng(rows)
    s = Surrogate(in_dim=in_dim, hidden=hidden)
    p = sw.init_params(d, 3)
    s.params = p
    x = rng.normal(size=(rows, in_dim)).astype(np.float32)
    y = rng.normal(size=rows).astype(np.float32)
    g, loss = s.gradients(x, y)
    want, want_loss = sw.gradients(d, p, x, y)
    assert abs(loss - want_loss) <= 1e-3 * abs(want_loss) + 1e-3
    for lo, hi in ((d.w1, d.w2), (d.w2, d.w3), (d.w3, d.b1), (d.b1, d.b2), (d.b2, d.b3), (d.b3, d.n)):
        assert np.abs(g[lo:hi] - want[lo:hi]).max() <= GRAD_RTOL * np.abs(want[lo:hi]).max() + 1e-9, (lo, hi)


@pytest.mark.parametrize("in_dim,hidden", [(130, 384), (4929, 256)])
def test_a_step_is_adamw_on_the_gradients(in_dim, hidden):
    """One row, so that shuffling changes nothing: the updated parameters are AdamW's first step on
    gradients()'s result, in float32 with the kernel's order of operations (one unit in the last place
    of the parameter allowed for the host's pow)."""
    from tetris_ai3_b200.surrogate import Surrogate
    d = sw.Dims(in_dim, hidden)
    rng = np.random.default_rng(1)
    lr, wd, f = np.float32(1e-3), np.float32(1e-2), np.float32
    s = Surrogate(in_dim=in_dim, hidden=hidden, lr=float(lr), weight_decay=float(wd))
    p = np.asarray(sw.init_params(d, 4), np.float32)
    s.params = p
    x = rng.normal(size=(1, in_dim)).astype(np.float32)
    y = np.array([0.7], np.float32)
    g, _ = s.gradients(x, y)
    s.train(x, y, epochs=1, batch=1, standardized=True)
    b1, b2 = f(0.9), f(0.999)
    m, v = (f(1) - b1) * g, (f(1) - b2) * g * g
    want = p - lr * (m / (f(1) - b1)) / (np.sqrt(v / (f(1) - b2)) + f(1e-8)) - lr * wd * p
    got = s.params
    assert (np.abs(got - want) <= np.spacing(np.abs(want)) + 1e-12).all()
    assert not np.array_equal(got, p)
