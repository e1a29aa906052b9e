"""Input standardisation: narrow or small training sets take the host's column statistics, the others the
device's. Both are FP64 sums in row order, so predictions do not depend on which of them it was."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _standardised(x):
    """The plain loop's statistics: sequential float64 sums down each column, rounded to float32 at the end."""
    v = x.astype(np.float64)
    mu = np.add.accumulate(v, axis=0)[-1] / len(x)
    sd = np.sqrt(np.add.accumulate((v - mu) ** 2, axis=0)[-1] / len(x))
    inv = np.divide(1.0, sd, out=np.ones_like(sd), where=sd > 1e-12)
    return (x - mu.astype(np.float32)) * inv.astype(np.float32)


# (inputs, rows) on both sides of the rule's two edges: 48 inputs, 16,384 values
@pytest.mark.parametrize("in_dim,rows", [(1, 1), (3, 1000), (7, 40_000), (48, 700), (49, 334), (49, 335), (97, 168),
                                         (97, 169), (97, 1), (130, 900)])
def test_statistics_equal_the_plain_loop(in_dim, rows):
    from tetris_ai3_b200.surrogate import Surrogate
    hidden = 128
    rng = np.random.default_rng(rows)
    x = (rng.standard_normal((rows, in_dim)) * 3 + 5).astype(np.float32)
    x[:, 0] = 2.5                                            # a constant column: deviation 0, left as it is
    y = np.zeros(rows, np.float32)
    a, b = (Surrogate(in_dim=in_dim, hidden=hidden, seed=1) for _ in range(2))
    a._set_data(x, y, False)                                 # (a constant target has mean 0 and deviation 1)
    b._set_data(x, y, True)
    assert a.predict(x[:300]).tobytes() == b.predict(_standardised(x)[:300]).tobytes()

