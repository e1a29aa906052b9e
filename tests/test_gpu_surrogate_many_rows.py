"""Predictions of more rows than go into page-locked memory (262,144) are those of their parts, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [262_144, 262_145, 300_001])
def test_large_predictions_equal_their_parts(rows):
    from tetris_ai3_b200.surrogate import Surrogate
    x = np.random.default_rng(rows).standard_normal((rows, 97), dtype=np.float32)
    s = Surrogate(seed=2)
    s._set_data(x[:500], x[:500, 0], False)
    mean, lv = s.predict(x, with_logvar=True)
    for k in range(0, rows, 60_000):
        m, v = s.predict(x[k:k + 60_000], with_logvar=True)
        assert m.tobytes() == mean[k:k + 60_000].tobytes() and v.tobytes() == lv[k:k + 60_000].tobytes()
