"""The work that a user of the library has it do, as cases to be timed.

A case is a plain dict; ``api`` names the public entry point:

* ``class``    ``IncrementalNNFeatureSelection(...).train()``: host arrays in, the finished selection out (buffers,
               uploads and the whole greedy loop are part of the pass, as they are for its users);
* ``batch``    ``Batch(problems).run()``: many independent selections in one call;
* ``resume``   a loaded ``Selector`` that takes up a known prefix (``commit_sequence``) and scores the next step;
* ``step``     ``snn_score_step_noalloc`` on the caller's own device buffers.

Data come from the seeded generators of ``speedynn_b200.datagen`` (correlated magnitudes, their differences, noise).
"""
import ctypes
import math
import random

import numpy as np
import torch

from speedynn_b200 import _lib, datagen
from speedynn_b200._lib import _i32p, check, ptr
from speedynn_b200.base import IncrementalNNFeatureSelection
from speedynn_b200.batch import Batch
from speedynn_b200.selector import Selector

STEP_SCRATCH = 4_194_304  # predictions that the allocation-free step holds
EXACT_LIMIT = 3.0e10      # (row, column, candidate) triples that exact() goes through in 64 bits


def _case(name, api, **kw):
    c = dict(n_train=0, n_val=0, p=0, n_mag=5, n_heavy=0, k="10", steps=0, method="forward", folds=10, auto=False,
             losses="rmse", model="regression", mixture=False, dup=0.0, standardize=False)
    c.update(kw)
    return {"name": name, "api": api, **c} if name else {"api": api, **c}


def listed():
    return [
        # the smallest call: speedynn's own example (100 x 10, k from 2 to 50, three features, ten folds)
        _case("example-100", "class", n_train=100, p=10, k="2-50", steps=3),
        # the class's defaults (backward, k from 1 to 9, ten folds), stopped by the error's rise
        _case("cv-backward-1501", "class", n_train=1501, p=14, k="1-9", steps=4, method="backward", auto=True),
        # cross-validated forward selection at the reference's CPU size (the pooled 3000 x 20 workload)
        _case("cv-forward-3000", "class", n_train=3000, p=20, steps=8, folds=3),
        # the same problem as a train / validation split (the fwd-2k workload)
        _case("holdout-2k", "class", n_train=2000, n_val=1000, p=20, steps=8),
        # classification: the mode of the neighbours' labels, three losses of which the first decides
        _case("classes-5k", "class", n_train=5003, n_val=2501, p=24, k="1,5,15", steps=6, losses="zero_one,rmse_norm,mad",
              model="classification"),
        # long neighbour lists (k up to 150), as when the best k is searched for over a wide range
        _case("wide-k-8k", "class", n_train=8192, n_val=4096, p=20, k="16,64,150", steps=4),
        # one step scored on another runtime's device buffers
        _case("device-step-33k", "step", n_train=32771, n_val=16001, p=40, n_mag=6, k="10", steps=7),
        # a stopped forward selection of the fwd-64k workload taken up again after seven features
        _case("resume-64k", "resume", n_train=65536, n_val=32768, p=60, n_mag=8, n_heavy=10, k="10", steps=7),
        # backward elimination down to 20 of 120 features (the bwd-50k workload at a quarter of its pairs)
        _case("backward-25k", "class", n_train=25003, n_val=12502, p=120, n_mag=7, k="5", steps=20, method="backward",
              standardize=True),
        # long lists on mixture data with duplicated rows (the fwd-200k workload at a sixteenth of its pairs)
        _case("mixture-50k", "class", n_train=50021, n_val=24989, p=100, n_mag=8, k="50", steps=20, mixture=True, dup=0.02),
        # many uneven problems in one call (batch-64x5 with an eighth of its pools)
        _case("batch-8x5", "batch", n_train=1024, n_val=40000, p=40, n_mag=6, k="1,5,10,20", steps=15, folds=5),
        # the headline workload: 15 of 60 features from 65,536 training and 32,768 validation rows
        _case("forward-64k", "class", n_train=65536, n_val=32768, p=60, n_mag=8, n_heavy=10, k="10", steps=15),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_once(rng):
    kind = rng.choice(["cv", "cv", "holdout", "holdout", "large", "large", "classes", "wide", "step", "resume", "batch"])
    if kind == "cv":
        n, p = _log_int(rng, 100, 6000), rng.randint(10, 40)
        back = rng.random() < 0.5
        return _case(None, "class", n_train=n, p=p, k=rng.choice(["1-9", "2-50", "10", "5", "20"]),
                     steps=rng.randint(2, 8) if not back else rng.randint(2, p // 2), folds=rng.choice([3, 5, 10]),
                     method="backward" if back else "forward", auto=rng.random() < 0.25)
    if kind == "holdout":
        n, p = _log_int(rng, 1024, 30000), rng.randint(16, 60)
        return _case(None, "class", n_train=n, n_val=max(2, int(n * rng.uniform(0.3, 0.7))), p=p,
                     k=rng.choice(["1", "5", "10", "20", "1-9", "40"]), steps=rng.randint(4, 15),
                     n_heavy=rng.choice([0, 3]))
    if kind == "large":
        back = rng.random() < 0.5
        n = _log_int(rng, 12000, 65536)
        p = rng.randint(40, 120)
        return _case(None, "class", n_train=n, n_val=int(n * rng.uniform(0.4, 0.6)), p=p, n_mag=rng.choice([6, 7, 8]),
                     n_heavy=rng.choice([0, 0, 10]), k=rng.choice(["5", "10", "10", "20", "50"]),
                     steps=rng.randint(8, 20) if not back else rng.randint(p // 3, p - 8),
                     method="backward" if back else "forward", standardize=back, mixture=rng.random() < 0.3,
                     dup=rng.choice([0.0, 0.02]))
    if kind == "classes":
        n = _log_int(rng, 500, 12000)
        return _case(None, "class", n_train=n, n_val=max(2, n // 2), p=rng.randint(12, 40), k=rng.choice(["1,5,15", "3", "1-9"]),
                     steps=rng.randint(3, 8), model="classification",
                     losses=rng.choice(["zero_one", "zero_one,rmse_norm,mad", "mad_norm,std"]))
    if kind == "wide":
        n = _log_int(rng, 1024, 10000)
        return _case(None, "class", n_train=n, n_val=max(2, n // 2), p=rng.randint(12, 24), k=rng.choice(["16,64,150", "100", "80,200"]),
                     steps=rng.randint(2, 4))
    if kind == "step":
        n, p = _log_int(rng, 2000, 50000), rng.randint(20, 60)
        s = rng.randint(2, 9)
        return _case(None, "step", n_train=n, n_val=min(n // 2, STEP_SCRATCH // (p - s)), p=p, n_mag=6,
                     k=rng.choice(["1", "5", "10", "16", "50"]), steps=s)
    if kind == "resume":
        n = _log_int(rng, 8000, 65536)
        return _case(None, "resume", n_train=n, n_val=n // 2, p=rng.randint(30, 60), n_mag=6, k=rng.choice(["5", "10", "20"]),
                     steps=rng.randint(2, 12))
    return _case(None, "batch", n_train=1024, n_val=_log_int(rng, 4000, 40000), p=rng.randint(20, 40), n_mag=6,
                 k=rng.choice(["1,5,10,20", "10", "5,20"]), steps=rng.randint(8, 15), folds=rng.choice([2, 3, 5]))


def draw(rng):
    top = max(_weight(c) for c in listed())
    while True:
        c = _draw_once(rng)
        if _weight(c) <= top:
            return c


# -- sizes -----------------------------------------------------------------

def _kv(c):
    if "-" in c["k"]:
        lo, hi = c["k"].split("-")
        return list(range(int(lo), int(hi) + 1))
    return [int(x) for x in c["k"].split(",")]


def _pools(c):
    """A batch's pools: (generator seed, n_train) of each, sizes log-uniform in [n_train, n_val] of the case."""
    out = []
    for i in range(8):
        r = random.Random(1000 + i)
        out.append(_log_int(r, c["n_train"], c["n_val"]))
    return out


def _candidates(c):
    """Candidates over all steps: those of the whole selection, without an early stop."""
    p, s = c["p"], c["steps"]
    if c["api"] in ("step", "resume"):
        return p - s
    if c["method"] == "backward":
        return sum(range(s + 1, p + 1))
    return sum(p - t for t in range(p if c["auto"] else s))


def _evals(c):
    if c["api"] == "batch":
        return sum(n * (n // 2) for n in _pools(c)) * c["folds"] * _candidates(c)
    return c["n_train"] * (c["n_val"] or c["n_train"]) * _candidates(c)


def _weight(c):
    """What a case costs beside another: its evaluations, more for longer neighbour lists, and its committed distances."""
    k = max(_kv(c))
    pairs = c["n_train"] * (c["n_val"] or c["n_train"]) if c["api"] != "batch" else 0
    return _evals(c) * (1.0 if k <= 16 else 1.6 if k <= 64 else 8.0) * (1.5 if c["api"] == "batch" else 1.0) + 60.0 * pairs


def work(case):
    """Inputs read once, results written once; sub, mul and add of each candidate distance."""
    c = case
    n = c["n_train"] + c["n_val"]
    if c["api"] == "batch":
        rows = c["folds"] * sum(m + m // 2 for m in _pools(c))
        return {"bytes": 4.0 * rows * (c["p"] + 1), "flops": 3.0 * _evals(c)}
    b = 4.0 * n * (c["p"] + 1) + 4.0 * c["p"] * 5
    if c["api"] == "step":
        b += 4.0 * c["n_train"] * c["n_val"] + 12.0 * (c["p"] - c["steps"]) * len(_kv(c))
    return {"bytes": b, "flops": 3.0 * _evals(c)}


# -- inputs ----------------------------------------------------------------

def _split(c, seed, n_train=None, n_val=None):
    n_train = c["n_train"] if n_train is None else n_train
    n_val = c["n_val"] if n_val is None else n_val
    s = datagen.generate(n_train, max(1, n_val), c["p"], n_mag=c["n_mag"], n_heavy=c["n_heavy"], seed=seed,
                         mixture=c["mixture"], dup_frac=c["dup"], standardize=c["standardize"],
                         n_col=min(c["n_mag"] - 1, 5) if c["method"] == "backward" else None)
    if c["model"] == "classification":
        s.ytrain = np.floor(2.0 * s.ytrain).astype(np.float32)
        s.yval = np.floor(2.0 * s.yval).astype(np.float32)
    return s


def _prefix(c, split):
    """The features already chosen: informative ones first, then others."""
    inf = [int(f) for f in split.informative]
    rest = [f for f in range(c["p"]) if f not in set(inf)]
    return (inf[::2] + rest + inf[1::2])[: c["steps"]]


def _problems(c, seed):
    probs = []
    kv = _kv(c)
    for i, n in enumerate(_pools(c)):
        pool = _split(c, seed * 64 + i, n, n // 2)
        X, y = np.concatenate([pool.Xtrain, pool.Xval]), np.concatenate([pool.ytrain, pool.yval])
        for s in range(c["folds"]):
            perm = np.random.default_rng((seed * 64 + i) * 31 + s).permutation(X.shape[0])
            tr, va = perm[:n], perm[n:]
            probs.append(dict(Xtrain=np.ascontiguousarray(X[tr]), ytrain=np.ascontiguousarray(y[tr]),
                              Xval=np.ascontiguousarray(X[va]), yval=np.ascontiguousarray(y[va]),
                              k_vals=[kv[i % len(kv)]], num_features=c["steps"], method=c["method"]))
    return probs


def prepare(case, seed):
    c = dict(case)
    if c["api"] == "batch":
        return {"case": c, "problems": _problems(c, seed)}
    s = _split(c, seed)
    if c["api"] == "class":
        return {"case": c, "split": s}
    prefix = _prefix(c, s)
    if c["api"] == "resume":
        sel = Selector(s.Xtrain, s.ytrain, s.Xval, s.yval, k_vals=_kv(c), num_features=len(prefix) + 1)
        return {"case": c, "split": s, "prefix": prefix, "selector": sel}
    # the caller's device buffers: feature-major points and the distances committed so far
    dev = torch.device("cuda", 0)
    n, m, p = c["n_train"], c["n_val"], c["p"]
    ld = (n + 63) // 64 * 64
    XT = torch.zeros((p, ld), dtype=torch.float32, device=dev)
    XT[:, :n] = torch.from_numpy(np.ascontiguousarray(s.Xtrain.T)).to(dev)
    XV = torch.from_numpy(np.ascontiguousarray(s.Xval.T)).to(dev)
    D = torch.zeros((m, ld), dtype=torch.float32, device=dev)
    for f in prefix:
        t = XV[f][:, None] - XT[f][None, :]
        D += t.mul_(t)
    D[:, n:] = float("inf")
    kv = np.asarray(_kv(c), np.int32)
    cands = np.asarray([f for f in range(p) if f not in set(prefix)], np.int32)
    out = torch.zeros((cands.size, kv.size), dtype=torch.float32, device=dev)
    out64 = torch.zeros((cands.size, kv.size), dtype=torch.float64, device=dev)
    return {"case": c, "XT": XT, "XV": XV, "D": D, "ld": ld, "kv": kv, "cands": cands, "out": out, "out64": out64,
            "yt": torch.from_numpy(s.ytrain).to(dev), "yv": torch.from_numpy(s.yval).to(dev)}


# -- one pass --------------------------------------------------------------

def _losses(c):
    return c["losses"].split(",")


def run(state):
    c = state["case"]
    if c["api"] == "class":
        s = state["split"]
        m = IncrementalNNFeatureSelection(s.Xtrain, s.ytrain, k_vals=_kv(c), auto_feature=c["auto"], num_features=c["steps"],
                                          k_fold=c["folds"], method=c["method"], loss_functions=_losses(c),
                                          model_type=c["model"], Xval=s.Xval if c["n_val"] else None,
                                          Yval=s.yval if c["n_val"] else None)
        m.train()
        return {"ordering": m.get_selected_ordering(), "mask": m.get_selected_dimensions(), "errors": m.get_selected_errors(),
                "errors64": m.selected_errors64, "best_k": m.get_optimal_model_k(), "num_final": m.num_final_features}
    if c["api"] == "batch":
        with Batch(state["problems"]) as b:
            r = b.run()
        return {key: np.stack([np.asarray(x[key]) for x in r])
                for key in ("ordering", "mask", "errors", "errors64", "step_best_k", "best_k", "num_final")}
    if c["api"] == "resume":
        sel = state["selector"]
        sel.commit_sequence(state["prefix"])
        sel.step()
        r = sel.results()
        return {key: r[key] for key in ("ordering", "mask", "errors", "errors64", "step_best_k", "best_k", "num_final")}
    st = state
    check(_lib.lib().snn_score_step_noalloc(
        st["D"].data_ptr(), st["ld"], st["XT"].data_ptr(), st["XV"].data_ptr(), c["n_val"], st["yt"].data_ptr(),
        st["yv"].data_ptr(), c["n_val"], c["n_train"], c["p"], ptr(st["cands"], _i32p), st["cands"].size,
        ptr(st["kv"], _i32p), st["kv"].size, 0, st["out"].data_ptr(), st["out64"].data_ptr(),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return {"errors": st["out"], "errors64": st["out64"]}


# -- the same in 64 bits ----------------------------------------------------

def _mode(lab):
    """Per row the label with the largest count, the earliest in rank order where several have it."""
    n = lab.shape[1]
    cnt = (lab[:, :, None] == lab[:, None, :]).sum(2)
    return lab.gather(1, (cnt * n - torch.arange(n, device=lab.device)).argmax(1, keepdim=True))[:, 0]


def _loss64(name, y, pred):
    e = y - pred
    if name == "rmse":
        return e.square().mean().sqrt()
    if name == "rmse_norm":
        return (e / (1.0 + y)).square().mean().sqrt()
    if name in ("mad", "mad_norm"):
        e = e / (1.0 + y) if name == "mad_norm" else e
        med = e.sort().values[e.numel() // 2]
        return (e - med).abs().sort().values[e.numel() // 2]
    if name == "zero_one":
        return (e.abs() >= 1.0).double().mean()
    if name == "std":  # the reference's: only the last row's term remains
        return ((e[-1] - e.mean()).square() / (e.numel() - 1)).sqrt()
    raise ValueError(name)


def _neighbour_labels(d, yc, k):
    """The labels of each row's k nearest columns in rank order (rows in parts: the sort needs room)."""
    part = max(1, int(2.0e8 // d.shape[1]))
    return torch.cat([yc[d[r:r + part].topk(k, dim=1, largest=False, sorted=True).indices] for r in range(0, d.shape[0], part)])


def _values64(c, lab, y):
    """[k][loss] values of one candidate from its neighbours' labels."""
    out = []
    for k in _kv(c):
        pred = _mode(lab[:, :k]) if c["model"] == "classification" else lab[:, :k].mean(1)
        out.append([float(_loss64(n, y, pred)) for n in _losses(c)])
    return out


def exact(case, seed):
    c = dict(case)
    if c["api"] == "batch" or _evals(c) > EXACT_LIMIT or max(_kv(c)) >= c["n_train"] * 0.8:
        return None
    s = _split(c, seed)
    dev = torch.device("cuda", 0)
    X = torch.from_numpy(s.Xtrain).to(dev)
    yc = torch.from_numpy(s.ytrain).to(dev).double()
    Xr, yr = (torch.from_numpy(s.Xval).to(dev), torch.from_numpy(s.yval).to(dev).double()) if c["n_val"] else (X, yc)
    n, p, kmax = X.shape[0], c["p"], max(_kv(c))
    back = c["method"] == "backward"

    def sq(f):
        return (Xr[:, f].double()[:, None] - X[:, f].double()[None, :]).square()

    D = torch.zeros((Xr.shape[0], n), dtype=torch.float64, device=dev)
    if c["api"] == "step":  # D is an input there: the sums in 32 bits
        D32 = torch.zeros((Xr.shape[0], n), dtype=torch.float32, device=dev)
        prefix = _prefix(c, s)
        for f in prefix:
            t = Xr[:, f][:, None] - X[:, f][None, :]
            D32 += t.mul_(t)
        D = D32.double()
        del D32
        vals = [[v[0] for v in _values64(c, _neighbour_labels(D + sq(f), yc, kmax), yr)] for f in range(p) if f not in set(prefix)]
        vals = np.asarray(vals)
        return {"errors": vals, "errors64": vals}
    if not c["n_val"]:
        fold = torch.arange(n, device=dev) // (n // c["folds"])
        D.masked_fill_(fold[:, None] == fold[None, :], float("inf"))
    left = list(range(p))
    if back:
        for f in left:
            D += sq(f)
    errors, errors64 = np.zeros((p, len(_losses(c)))), np.zeros(p)
    total = p if c["auto"] else (p - c["steps"] if back else c["steps"])
    forced = _prefix(c, s) if c["api"] == "resume" else []
    if c["api"] == "resume":
        total = len(forced) + 1
    for t in range(total):
        it = p - 1 - t if back else t
        if t < len(forced):
            win = forced[t]
        else:
            best, win, row = math.inf, -1, None
            for f in left:
                d = D - sq(f) if back else D + sq(f)
                for v in _values64(c, _neighbour_labels(d, yc, kmax), yr):
                    if v[0] < best:
                        best, win, row = v[0], f, v
            errors[it], errors64[it] = row, row[0]
        left.remove(win)
        D = D - sq(win) if back else D + sq(win)
        if c["auto"] and t > 0 and errors[it + 1 if back else it - 1][0] < errors[it][0]:
            break
    if c["api"] == "resume":
        return {"ordering": None, "mask": None, "errors": errors[:, 0], "errors64": errors64, "step_best_k": None, "best_k": None,
                "num_final": None}
    return {"ordering": None, "mask": None, "errors": errors, "errors64": errors64, "best_k": None, "num_final": None}
