"""The evaluator's host side without a GPU, on a stand-in for the CUDA runtime."""
from __future__ import annotations

import numpy as np
import pytest

import fake_cuda
from tetris_ai3_b200 import evaluator


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("fake_cuda"), ("ta3b_eval.cu",))


@pytest.mark.parametrize("trace,nth", [(False, n) for n in range(2, 6)] + [(True, n) for n in range(6, 9)])
def test_no_memory_for_a_larger_batch_leaves_the_smaller_ones_working(lib, monkeypatch, trace, nth):
    """The result buffers grow one by one, each freed before its larger one is allocated: when one of them fails,
    a smaller batch needs fresh buffers too, and no kernel gets a null pointer."""
    monkeypatch.setattr(evaluator, "_lib", lib)
    lib.fake_reset()
    w = np.zeros((40, 97), np.float32)
    seeds = np.arange(3, dtype=np.uint64)
    with evaluator.ModelEvaluator() as ev:
        play = ev.eval_trace if trace else ev.eval_full
        play(w[:2], 2, seeds, 5)
        lib.fake_reset()
        lib.fake_fail(b"cudaMalloc", nth)             # the first two: weights and seeds
        with pytest.raises(evaluator.EvaluatorError):
            play(w, 40, np.arange(9, dtype=np.uint64), 5)
        lib.fake_reset()
        play(w[:2], 2, seeds, 5)
    lib.fake_reset()
