"""The surrogates' host side without a GPU, on a stand-in for the CUDA runtime."""
from __future__ import annotations

import pytest

import fake_cuda


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("fake_cuda"))


@pytest.fixture(autouse=True)
def _reset(lib):
    lib.fake_reset()
    yield
    lib.fake_reset()


@pytest.mark.parametrize("in_dim,rows,device", [(1, 100_000, 0), (48, 5000, 0), (49, 334, 0), (49, 335, 1), (97, 168, 0),
                                                (97, 169, 1), (256, 1000, 1)])
def test_narrow_or_small_training_sets_take_the_host_statistics(lib, in_dim, rows, device):
    """The device's chain of additions takes as long for one column as for a hundred."""
    m = fake_cuda.Model(lib, "ta3s" if in_dim == 97 else "ta3w", in_dim)
    lib.fake_reset()
    assert m.set_data(rows) == 0
    assert m.launches("column_stats_kernel") == device
    m.close()
