"""W1's padding columns are zero whatever a training run meets: a target that overflows the loss makes the
gradients of whole rows infinite or NaN, and a padding column's gradient (their product with zero) NaN too."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("in_dim,hidden", [(97, 128), (1, 128), (126, 128), (130, 256), (4929, 256)])
@pytest.mark.parametrize("target", [0.5, 1e30, np.inf, np.nan])
def test_padding_columns_stay_zero(in_dim, hidden, target):
    from tetris_ai3_b200.surrogate import Surrogate
    s = Surrogate(in_dim=in_dim, hidden=hidden, weight_decay=0.01)
    x = np.random.default_rng(0).standard_normal((5, in_dim), dtype=np.float32)
    y = x[:, 0].copy()
    y[2] = target
    before = s.params
    s.train(x, y, epochs=2, batch=5, standardized=True)
    after = s.params
    inp = 112 if in_dim == 97 else -(-in_dim // 128) * 128
    assert not after[:hidden * inp].reshape(hidden, inp)[:, in_dim:].any()      # (NaN counts as non-zero)
    assert after.tobytes() != before.tobytes()
