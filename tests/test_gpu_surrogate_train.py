"""The v11 surrogate's training launches: a whole run of steps in one launch of a cluster (minibatches of
up to eight 128-row tiles) or two launches a step beyond that."""
from __future__ import annotations

import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))
import surrogate_oracle as so  # noqa: E402

pytestmark = pytest.mark.gpu

LR, WD = 1e-3, 1e-2


def _data(rows, seed=0):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(rows, 97)).astype(np.float32)
    return x, (x[:, 0] - 0.5 * x[:, 1] ** 2).astype(np.float32)


def _model(seed=3):
    from tetris_ai3_b200.surrogate import Surrogate
    return Surrogate(device=0, seed=seed, lr=LR, weight_decay=WD)


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 300, 1024, 1025, 1300])
def test_first_step_follows_the_gradients(rows):
    """AdamW's first step is lr * sign(g) (plus the decay) wherever |g| is far above eps; the shuffled
    minibatch sums the same gradients in another order, so entries near zero are left out."""
    s = _model()
    x, y = _data(rows)
    p = s.params
    g, _ = s.gradients(x, y)
    s.train(x, y, epochs=1, batch=rows, standardized=True)
    step = s.params - p
    clear = np.abs(g) > max(1e-2 * np.abs(g).max(), 1e-4)
    assert clear.sum() > 10
    want = -LR * np.sign(g) - LR * WD * p
    assert np.abs(step - want)[clear].max() <= 2e-6 + np.spacing(np.abs(p)).max()
    assert not step[g == 0].any() or np.abs(step[g == 0] + LR * WD * p[g == 0]).max() <= 1e-6


def test_one_run_equals_its_steps_one_by_one():
    """One row, so that shuffling changes nothing: five epochs in one call equal five calls bit for bit
    (weights, moments and the step count carry over)."""
    x, y = _data(1)
    a, b = _model(), _model()
    a.train(x, y, epochs=5, batch=64, standardized=True)
    for _ in range(5):
        b.train(x, y, epochs=1, batch=64, standardized=True)
    assert a.params.tobytes() == b.params.tobytes()
    assert a.predict(x).tobytes() == b.predict(x).tobytes()


@pytest.mark.parametrize("rows,batch", [(1000, 256), (700, 100), (2500, 1024), (2500, 1100)])
def test_training_with_a_ragged_last_minibatch_learns(rows, batch):
    x, y = _data(rows)
    s = _model()
    held, true = _data(400, seed=9)
    s.train(x, y, epochs=60, batch=batch)
    assert np.isfinite(s.params).all() and np.isfinite(s.last_loss)
    assert so.spearman(s.predict(held), true) > 0.5


@pytest.mark.parametrize("rows,batch", [(100, 1200), (300, 5000)])
def test_minibatch_larger_than_the_rows(rows, batch):
    """A minibatch is never larger than the rows there are, however large the argument (here beyond the eight
    tiles that a cluster holds): one step an epoch over the same shuffle, so the results are bit-identical."""
    x, y = _data(rows)
    a, b = _model(), _model()
    a.train(x, y, epochs=3, batch=batch, standardized=True)
    b.train(x, y, epochs=3, batch=rows, standardized=True)
    assert a.params.tobytes() == b.params.tobytes() and a.last_loss == b.last_loss
