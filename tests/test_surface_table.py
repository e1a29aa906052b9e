"""The surface input sqrt(s) / 100 the kernels read from a table: both operations rounded to nearest
float32 for every surface sum a 10 x 23 board can have (at most 9 * 23^2)."""
from __future__ import annotations

import ctypes as C

import numpy as np

from conftest import ptr
from test_core_host import core  # noqa: F401  (fixture)


def test_every_surface_input_is_correctly_rounded(core):  # noqa: F811
    got = np.zeros(9 * 23 * 23 + 1, np.float32)
    core.ta3bt_surface_table(ptr(got))
    want = np.sqrt(np.arange(got.size, dtype=np.float32)) / np.float32(100)     # IEEE float32 operations
    assert want.dtype == np.float32 and got.tobytes() == want.tobytes()
