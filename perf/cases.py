"""What this framework's users have it do, as measurable cases.

Three paths, each through its public entry point:

* games: a population of value-model weight vectors plays seeded games with the depth-4 beam
  search (`ModelEvaluator`), from the 8-game check of one model to the 10,000-game CMA-ES
  generation, for the v11 network and the two widened ones;
* surrogate: the MLP that predicts a weight vector's mean score (`Surrogate`): prediction,
  gradients and training, for the v11 size (97 inputs) and the widened one (4,929);
* training: a short island CMA-ES run (`Trainer`), which calls the first path from C++.

Sizes are those of the benchmark's batches, the default trainer configuration and the tests, or
shortened versions of them (fewer models or a lower move cap) where a whole one takes minutes.
"""
import math

import numpy as np
import torch

from tetris_ai3_b200 import workload
from tetris_ai3_b200.evaluator import ModelEvaluator
from tetris_ai3_b200.surrogate import Surrogate
from tetris_ai3_b200.trainer import Trainer, default_config

PLACEMENTS_PER_MOVE = 3_500      # evaluated boards of one searched move (measured: 3,300 to 3,530)


def listed():
    return [
        # one small model's games, the smallest call (the framework's smoke and parity size)
        {"name": "games_single", "kind": "games", "net": 8, "models": "random", "islands": 1, "pop": 1, "games": 8,
         "cap": 500, "entry": "host"},
        # a finished model's quality check: 30 games of the shipped champion, cap 300 (few long games: latency)
        {"name": "games_champion", "kind": "games", "net": 8, "models": "champion", "islands": 1, "pop": 1, "games": 30,
         "cap": 300, "entry": "host"},
        # one generation of the default trainer configuration: 4 islands x 50 x 30 games, cap 300
        {"name": "games_default_generation", "kind": "games", "net": 8, "models": "generation", "islands": 4, "pop": 50,
         "games": 30, "cap": 300, "entry": "host"},
        # the benchmark's generation: 4 islands x 50 x 50 games, cap 2,000
        {"name": "games_generation", "kind": "games", "net": 8, "models": "generation", "islands": 4, "pop": 50,
         "games": 50, "cap": 2000, "entry": "host"},
        # very uneven lengths, device-resident: 10 % champions to the cap, 90 % dying early
        {"name": "games_uneven", "kind": "games", "net": 8, "models": "uneven", "islands": 1, "pop": 110, "games": 91,
         "cap": 1000, "entry": "device"},
        # the widened evaluators' generations with fewer models and a lower cap
        {"name": "games_wide64", "kind": "games", "net": 64, "models": "wide", "islands": 8, "pop": 25, "games": 10,
         "cap": 200, "entry": "host"},
        {"name": "games_wide32", "kind": "games", "net": 32, "models": "wide", "islands": 8, "pop": 25, "games": 10,
         "cap": 300, "entry": "host"},
        # a pre-screening: 4 islands x 200 sampled candidates ranked by the v11 surrogate
        {"name": "surrogate_predict", "kind": "predict", "in_dim": 97, "hidden": 128, "rows": 800},
        # the v11 surrogate retrained on the archive of 40 generations (4 x 50 candidates each)
        {"name": "surrogate_train", "kind": "train", "in_dim": 97, "hidden": 128, "rows": 8000, "batch": 256,
         "epochs": 10},
        # the widened surrogate: gradients over a ragged number of rows, and a retrain
        {"name": "wide_surrogate_gradients", "kind": "gradients", "in_dim": 4929, "hidden": 256, "rows": 1000},
        {"name": "wide_surrogate_train", "kind": "train", "in_dim": 4929, "hidden": 256, "rows": 4000, "batch": 256,
         "epochs": 4},
        # the first generations of a training run with the default islands, games and cap
        {"name": "training_run", "kind": "training", "islands": 4, "pop": 50, "games": 30, "cap": 300,
         "generations": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["games", "games", "games", "wide", "predict", "gradients", "train", "training"])
    if kind == "games":
        models = rng.choice(["random", "champion", "generation", "generation", "uneven"])
        cap = _log_int(rng, 20, 2000)
        islands = 1 if models != "generation" else rng.randint(1, 8)
        pop = 1 if models == "champion" else _log_int(rng, 10 if models == "uneven" else 1, 110)
        most = 10_000 // (islands * pop)
        if models == "champion":                 # every game plays to the cap
            most = min(most, 3_000_000 // cap)
        games = _log_int(rng, 1, max(1, min(100, most)))
        return {"kind": "games", "net": 8, "models": models, "islands": islands, "pop": pop, "games": games,
                "cap": cap, "entry": rng.choice(["host", "device"])}
    if kind == "wide":
        return {"kind": "games", "net": rng.choice([32, 64]), "models": "wide", "islands": rng.randint(1, 8),
                "pop": _log_int(rng, 1, 25), "games": _log_int(rng, 1, 10), "cap": _log_int(rng, 20, 200),
                "entry": rng.choice(["host", "device"])}
    if kind == "training":
        return {"kind": "training", "islands": rng.randint(1, 4), "pop": rng.randint(6, 50),
                "games": rng.randint(2, 30), "cap": _log_int(rng, 40, 300), "generations": 2}
    in_dim, hidden = rng.choice([(97, 128), (4929, 256), (1441, 128)])
    case = {"kind": kind, "in_dim": in_dim, "hidden": hidden, "rows": _log_int(rng, 1, 8000 if in_dim == 97 else 4000)}
    if kind == "train":
        case |= {"batch": rng.choice([64, 100, 128, 256, 300]), "epochs": rng.randint(1, 4)}
    return case


def _weights(case, seed):
    """The models' weights [islands * pop][params] and the games' seeds [islands][games]."""
    islands, pop, games = case["islands"], case["pop"], case["games"]
    seeds = np.stack([workload.xoshiro_seeds(seed * 1000 + i, games) for i in range(islands)])
    n = islands * pop
    if case["models"] == "wide":
        sc = workload.wide_scale(case["net"])
        z = workload.normal(seed, n * sc.size).reshape(n, sc.size)
        w = np.where(sc[None, :] > 0, z * sc[None, :], 0.0)            # N(0, 1 / fan_in), biases +0
    elif case["models"] == "champion":
        w = np.repeat(workload.champion()[None, :], n, axis=0)
    elif case["models"] == "random":
        w = 0.5 * workload.normal(seed, n * workload.NUM_PARAMS).reshape(n, -1)
    elif case["models"] == "uneven":
        w = workload.uneven_batch(n, games, case["cap"], seed).weights
    else:
        # candidates N(m, 0.5^2) around the benchmark's own island mean (its seed 1)
        m = 0.5 * workload.normal(1, workload.NUM_PARAMS)
        w = m[None, :] + 0.5 * workload.normal(seed, n * workload.NUM_PARAMS).reshape(n, -1)
    return np.ascontiguousarray(w, np.float32), seeds


def _rows(case, seed):
    """Surrogate inputs (standard normal weight vectors) and targets (a quadratic of 8 directions)."""
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((case["rows"], case["in_dim"]), dtype=np.float32)
    a = rng.standard_normal((case["in_dim"], 8), dtype=np.float32) / np.float32(math.sqrt(case["in_dim"]))
    return x, (-(x @ a) ** 2).sum(1).astype(np.float32)


def _params(case, seed):
    """A surrogate's parameters as its initialisation draws them (He-uniform, biases zero)."""
    d, h = case["in_dim"], case["hidden"]
    pad = 112 if (d, h) == (97, 128) else -(-d // 128) * 128
    rng = np.random.default_rng(seed + 77)
    w1 = np.zeros((h, pad), np.float32)
    w1[:, :d] = rng.uniform(-1, 1, (h, d)) * math.sqrt(6 / d)
    w2 = (rng.uniform(-1, 1, (h, h)) * math.sqrt(6 / h)).astype(np.float32)
    w3 = (rng.uniform(-1, 1, (2, h)) * math.sqrt(1 / h)).astype(np.float32)
    return w1, w2, w3, np.zeros(h, np.float32), np.zeros(h, np.float32), np.zeros(2, np.float32)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "games":
        w, s = _weights(case, seed)
        state["evaluator"] = ModelEvaluator()
        if case["entry"] == "device":
            n = w.shape[0] * s.shape[1]
            state["stream"] = torch.cuda.Stream()
            state["weights"] = torch.from_numpy(w).cuda()
            state["seeds"] = torch.from_numpy(s.view(np.int64)).cuda()
            state["out"] = [torch.zeros(n, dtype=t, device="cuda") for t in
                            (torch.float32, torch.int32, torch.int32, torch.int32)]
        else:
            state["weights"], state["seeds"] = w, s
    elif kind == "training":
        state["config"] = default_config(islands=case["islands"], population=case["pop"], games=case["games"],
                                         max_moves=case["cap"], training_seed=seed)
    else:
        state["x"], state["y"] = _rows(case, seed)
        state["params"] = np.concatenate([p.reshape(-1) for p in _params(case, seed)])
        state["model"] = Surrogate(seed=0, in_dim=case["in_dim"], hidden=case["hidden"])
        state["model"].params = state["params"]
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "games":
        if case["entry"] == "device":
            state["evaluator"].eval_device(state["weights"], state["seeds"], case["cap"], *state["out"],
                                           num_islands=case["islands"], stream=state["stream"])
            return state["out"]
        if case["islands"] == 1:
            return state["evaluator"].eval_full(state["weights"], case["pop"], state["seeds"], case["cap"])
        return state["evaluator"].eval_islands(state["weights"], state["seeds"], case["cap"])
    if kind == "training":
        t = Trainer(state["config"])
        for _ in range(case["generations"]):
            t.run_generation()
        champions = [t.champion(i) for i in range(case["islands"])]
        return {"champions": [c[0] for c in champions], "fitness": [c[1] for c in champions],
                "means": [t.island_mean(i) for i in range(case["islands"])], "pieces": t.stats()["pieces"]}
    model = state["model"]
    if kind == "predict":
        return model.predict(state["x"], with_logvar=True)
    if kind == "gradients":
        return model.gradients(state["x"], state["y"])
    model.params = state["params"]               # a retrain from the same start, with the same shuffles
    model.trainings = 0
    loss = model.train(state["x"], state["y"], epochs=case["epochs"], batch=case["batch"])
    return {"loss": loss, "params": model.params}


def work(case):
    kind = case["kind"]
    if kind in ("games", "training"):
        islands, pop, games, cap = case["islands"], case["pop"], case["games"], case["cap"]
        sims = islands * pop * games
        if kind == "training":
            sims *= case["generations"] + 1
        # mean moves of a game: champions play to the cap, random models die after about 30 pieces, a tenth
        # or a fifth of a batch lives long
        moves = {"champion": cap, "random": min(cap, 30), "uneven": min(cap, 40) + cap // 10,
                 "wide": cap // 2}.get(case.get("models"), min(cap, 40) + cap // 5)
        net = case.get("net", 8)
        macs = 10 * net + net if net == 8 else 10 * net + net * net + net
        params = macs + (net + 1 if net == 8 else 2 * net + 1)
        return {"bytes": 4 * islands * pop * params + 8 * islands * games + 12 * sims,
                "flops": float(sims) * moves * PLACEMENTS_PER_MOVE * (2 * macs + 40)}
    d, h, rows = case["in_dim"], case["hidden"], case["rows"]
    macs = d * h + h * h + 2 * h
    params = macs + 2 * h + 2
    passes = {"predict": 2, "gradients": 6, "train": 6 * case.get("epochs", 1)}[kind]
    out = 8 * rows if kind == "predict" else 4 * params
    return {"bytes": 4 * rows * (d + (kind != "predict")) + 4 * params + out, "flops": float(passes) * macs * rows}


def exact(case, seed):
    """The surrogate's outputs and gradients in float64. Games and training runs have no such value (a game's
    score follows from its discrete moves, which both sides have to find bit for bit); a retrain's minibatches
    come from the library's own shuffle."""
    if case["kind"] not in ("predict", "gradients"):
        return None
    d = case["in_dim"]
    x, y = (v.astype(np.float64) for v in _rows(case, seed))
    w1, w2, w3, b1, b2, b3 = (p.astype(np.float64) for p in _params(case, seed))
    z1 = x @ w1[:, :d].T + b1
    h1 = np.maximum(z1, 0)
    z2 = h1 @ w2.T + b2
    h2 = np.maximum(z2, 0)
    o = h2 @ w3.T + b3
    if case["kind"] == "predict":
        return o[:, 0], o[:, 1]
    s = np.clip(o[:, 1], -12, 12)
    e = np.exp(-s)
    r = y - o[:, 0]
    loss = float((0.5 * (s + r * r * e)).sum())
    g = np.stack([-r * e, np.where(np.abs(o[:, 1]) < 12, 0.5 * (1 - r * r * e), 0)], 1) / len(y)
    d2 = (g @ w3) * (z2 > 0)
    d1 = (d2 @ w2) * (z1 > 0)
    gw1 = np.zeros_like(w1)
    gw1[:, :d] = d1.T @ x
    parts = [gw1, d2.T @ h1, g.T @ h2, d1.sum(0), d2.sum(0), g.sum(0)]
    return np.concatenate([p.reshape(-1) for p in parts]), loss
