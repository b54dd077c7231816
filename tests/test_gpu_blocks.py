"""Handles that reuse an earlier handle's memory block, stream and events give
the results of handles made first: problems of different sizes, models and
directions in turn, then from several threads at once; and a run right after a
load or a reset, which starts from the distances that are already there."""
import threading

import numpy as np
import pytest

from speedynn_b200 import datagen
from speedynn_b200.selector import Selector

pytestmark = pytest.mark.gpu

KEYS = ("ordering", "mask", "errors", "errors64", "step_best_k", "best_k", "num_final", "errors_all")
PROBLEMS = [
    dict(n=700, m=300, p=14, k=[5, 9], nf=5, method="forward"),
    dict(n=300, m=0, p=11, k=[4], nf=4, method="backward"),
    dict(n=3000, m=1000, p=16, k=[20], nf=4, method="forward"),
    dict(n=500, m=200, p=12, k=[3], nf=3, method="forward", loss_functions=(2, 0), classes=True),
]


def _run(q, seed=91):
    s = datagen.generate(q["n"], max(q["m"], 1), q["p"], n_mag=5, seed=seed)
    y, yv = (np.floor(2 * s.ytrain), np.floor(2 * s.yval)) if q.get("classes") else (s.ytrain, s.yval)
    with Selector(s.Xtrain, y, s.Xval if q["m"] else None, yv if q["m"] else None, k_vals=q["k"], num_features=q["nf"],
                  method=q["method"], k_fold=5, loss_functions=q.get("loss_functions", (0,)),
                  model_type=int(q.get("classes", False))) as sel:
        a = sel.run()
        b = sel.run()
        sel.reset()
        c = sel.run()
    for r in (b, c):
        _same(r, a)
    return a


def _same(a, b):
    for k in KEYS:
        np.testing.assert_array_equal(np.asarray(a[k]), np.asarray(b[k]), err_msg=k)


def test_reused_blocks_and_threads_give_the_same_results():
    want = [_run(q) for q in PROBLEMS]
    for i in (2, 0, 3, 1, 1, 0):
        _same(_run(PROBLEMS[i]), want[i])
    errors = []

    def work(first):
        try:
            for j in range(4):
                i = (first + j) % len(PROBLEMS)
                _same(_run(PROBLEMS[i]), want[i])
        except Exception as e:  # noqa: BLE001 -- reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
