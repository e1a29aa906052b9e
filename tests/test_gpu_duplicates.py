"""Boards that several kept nodes share: the kernels evaluate each distinct child list once and let it
stand for its copies. Models with few distinct values (zero, sign and small-integer weights) make ties
between copies and other candidates the rule, so every position and order decides; traces, scores and
evaluation counts have to equal the oracle's."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import ptr

pytestmark = pytest.mark.gpu

CAP = 40
# (launch variant or None for the default choice, games per model): teams of four, pairs and single warps
KERNELS = [(None, 2), (10, 2), (11, 2), (7, 2), (2, 2), (None, 97)]


def _oracle(lib, w, hidden, seeds):
    out = []
    for m in w:
        for s in seeds:
            sc, p, l, e, nm = C.c_float(), C.c_uint32(), C.c_uint32(), C.c_uint64(), C.c_uint32()
            tr, bd = np.zeros(3 * CAP, np.uint8), np.zeros(10, np.uint32)
            lib.ta3o_play_net(ptr(m), *hidden, C.c_uint64(int(s)), CAP, C.byref(sc), C.byref(p), C.byref(l),
                              C.byref(e), ptr(tr), C.byref(nm), ptr(bd))
            out.append((np.float32(sc.value).tobytes(), p.value, l.value, e.value, nm.value,
                        tr[:3 * nm.value].tobytes(), bd.tolist()))
    return out


def _device(ev, w, seeds):
    o = ev.eval_trace(w, len(w), seeds, CAP)
    return [(o["score"][i].tobytes(), int(o["pieces"][i]), int(o["lines"][i]), int(o["evals"][i]), int(o["moves"][i]),
             o["trace"][i][:3 * int(o["moves"][i])].tobytes(), o["board"][i].tolist()) for i in range(len(o["score"]))]


def _tied_models(params, seed):
    rng = np.random.default_rng(seed)
    w = np.stack([np.zeros(params), rng.integers(-1, 2, params), rng.integers(-2, 3, params) * 0.5,
                  -np.ones(params), rng.integers(0, 2, params) * -1.0, rng.normal(size=params) * 0.3])
    return np.ascontiguousarray(w + 0.0, np.float32)          # + 0.0: no negative zeros


@pytest.mark.parametrize("variant,games", KERNELS)
def test_tied_models_match_the_oracle(oracle, variant, games):
    from tetris_ai3_b200 import ModelEvaluator
    w = _tied_models(97, 5)
    seeds = np.arange(100, 100 + games, dtype=np.uint64)
    with ModelEvaluator(device=0) as ev:
        if variant is not None:
            ev.select_variant(variant)
        got = _device(ev, w, seeds)
    few = min(games, 3)                                       # the oracle plays the first games of each model
    want = _oracle(oracle, w, (8, 0), seeds[:few])
    for m in range(len(w)):
        assert got[m * games:m * games + few] == want[m * few:(m + 1) * few], m


@pytest.mark.parametrize("hidden", [32, 64])
def test_tied_widened_models_match_the_oracle(oracle, hidden):
    from tetris_ai3_b200 import ModelEvaluator
    from tetris_ai3_b200.workload import wide_params
    w = _tied_models(wide_params(hidden), 6)
    seeds = np.arange(7, 9, dtype=np.uint64)
    with ModelEvaluator(device=0) as ev:
        assert _device(ev, w, seeds) == _oracle(oracle, w, (hidden, hidden), seeds)


def test_large_widened_batch_plays_the_small_ones_games():
    """Width 32 has a launch shape of its own for large batches (at least four games per slot of 12 warps
    an SM): the same games as batches below that, bit for bit."""
    from tetris_ai3_b200 import ModelEvaluator, workload
    b = workload.wide_batch(islands=1, pop=80, games=90, max_moves=6, hidden=32)
    with ModelEvaluator(device=0) as ev:
        assert b.sims >= 4 * 12 * ev.launch_info()["sms"]
        many = ev.eval_full(b.weights, b.models, b.seeds, b.max_moves)
        assert ev.launch_info()["warps_per_block"] == 12
        for m in (0, 41, 79):
            few = ev.eval_full(b.weights[m:m + 1], 1, b.seeds, b.max_moves)
            assert ev.launch_info()["warps_per_block"] == 4
            for x, y in zip(many, few):
                assert x[m * 90:(m + 1) * 90].tobytes() == y.tobytes()
