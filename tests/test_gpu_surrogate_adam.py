"""Several AdamW steps in a row, where moments, weights and the minibatches' rows carry over from step to step:
the v11 surrogate's cluster launch over ragged epochs and over more steps than one launch takes, and the
widened surrogate's update in the epilogue. A step's gradients (which other tests hold against float64) are
those of gradients() over the same rows in the same order, and AdamW is float32 operations rounded one by one, so
the parameters are equal bit for bit."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, ptr

pytestmark = pytest.mark.gpu

F = np.float32
LR, WD = F(1e-3), F(1e-2)


@pytest.fixture(scope="module")
def order(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("shuffle") / "libshuffle.so")
    subprocess.run(["g++", "-std=c++20", "-O2", "-fPIC", "-shared", "-o", lib,
                    os.path.join(ROOT, "tests", "cpp", "shuffle.cpp")], check=True)
    fn = C.CDLL(lib).epochs_order

    def rows_of(n, epochs, seed):
        out = np.zeros((epochs, n), np.int32)
        fn(n, epochs, seed, ptr(out))
        return out
    return rows_of


def _adam(p, gradient, minibatches):
    """AdamW in the kernels' order of operations; powf as the library calls it."""
    powf = C.CDLL("libm.so.6").powf
    powf.restype, powf.argtypes = C.c_float, [C.c_float, C.c_float]
    m, v = np.zeros_like(p), np.zeros_like(p)
    b1, b2 = F(0.9), F(0.999)
    for t, rows in enumerate(minibatches, 1):
        g = gradient(p, rows)
        m = b1 * m + (F(1) - b1) * g
        v = b2 * v + (F(1) - b2) * g * g
        c1, c2 = F(1) - F(powf(b1, t)), F(1) - F(powf(b2, t))
        p = p - LR * (m / c1) / (np.sqrt(v / c2) + F(1e-8)) - LR * WD * p
        assert p.dtype == np.float32
    return p


# v11: minibatches of 3, 3 and 1 tiles; of 8 and 1; two launches a step. Widened: several tiles of rows, of inputs
# and of hidden units; more rows than a tile's row map holds.
@pytest.mark.parametrize("in_dim,hidden,rows,batch,epochs", [
    (97, 128, 300, 300, 3), (97, 128, 700, 300, 2), (97, 128, 1100, 1024, 2), (97, 128, 1500, 1100, 2),
    (130, 384, 300, 300, 3), (257, 128, 700, 300, 2), (1441, 256, 1300, 1300, 3)])
def test_steps_follow_the_shuffled_minibatches(order, in_dim, hidden, rows, batch, epochs):
    from tetris_ai3_b200.surrogate import Surrogate
    rng = np.random.default_rng(rows)
    x, y = rng.normal(size=(rows, in_dim)).astype(np.float32), rng.normal(size=rows).astype(np.float32)
    s, t = (Surrogate(in_dim=in_dim, hidden=hidden, seed=5, lr=float(LR), weight_decay=float(WD)) for _ in range(2))
    p0 = s.params
    s.train(x, y, epochs=epochs, batch=batch, standardized=True)

    def gradient(p, r):
        t.params = p
        return t.gradients(x[r], y[r])[0]

    mini = [o[k:k + batch] for o in order(rows, epochs, 5) for k in range(0, rows, batch)]
    want = _adam(p0, gradient, mini)
    assert s.params.tobytes() == want.tobytes()
    # the BF16 copies are those of the updated weights: set from the parameters, they predict the same
    t.params = want
    t._set_data(x, y, True)
    assert s.predict(x).tobytes() == t.predict(x).tobytes()


def test_more_steps_than_one_launch_takes():
    """One row, so that shuffling changes nothing: 4,100 steps are two launches (4,096 and 4) in one call, and
    4,000 and 100 are one each; weights, moments and bias corrections carry over alike."""
    from tetris_ai3_b200.surrogate import Surrogate
    rng = np.random.default_rng(0)
    x, y = rng.normal(size=(1, 97)).astype(np.float32), np.array([0.3], np.float32)
    a, b = (Surrogate(seed=3, lr=1e-4, weight_decay=WD) for _ in range(2))
    a.train(x, y, epochs=4100, batch=64, standardized=True)
    b.train(x, y, epochs=4000, batch=64, standardized=True)
    b.train(x, y, epochs=100, batch=64, standardized=True)
    assert np.isfinite(a.params).all() and a.params.tobytes() == b.params.tobytes()


@pytest.mark.parametrize("batch", [2**31, 2**32 - 1])
def test_a_minibatch_beyond_an_int_is_all_rows(batch):
    from tetris_ai3_b200.surrogate import Surrogate
    rng = np.random.default_rng(1)
    x, y = rng.normal(size=(100, 97)).astype(np.float32), rng.normal(size=100).astype(np.float32)
    a, b = (Surrogate(seed=3) for _ in range(2))
    a.train(x, y, epochs=2, batch=batch, standardized=True)
    b.train(x, y, epochs=2, batch=100, standardized=True)
    assert a.params.tobytes() == b.params.tobytes() and a.last_loss == b.last_loss
