"""Engines of different sizes run from host threads of their own: the kernels whose dynamic shared memory follows the
number of tiles (the cascade's and the learned engine's warps in step) launch whatever other threads' engines asked for."""
import threading

import pytest

from ballasim_b200 import fields as F
from ballasim_b200 import workloads as W
from ballasim_b200.params import resolve

pytestmark = pytest.mark.gpu

# kind: a frame with few warps to a block (three engines) and one with many (one engine)
KINDS = {"cascade": ((100, 100), (346, 260)), "learned": ((320, 120), (400, 350))}
RUNS = 600  # one-window runs of the larger engine


def make(kind, size, net):
    from ballasim_b200.engine import Engine
    from ballasim_b200.sensor import SensorModel

    r, (w, h) = W.Rules(), size
    rows = {**W.MISMATCH, "noise": False} if kind == "cascade" else W.MISMATCH
    m = SensorModel(resolve("prophesee_gen3" if kind == "cascade" else "ideal", rows), w, h, 7, [{"type": "constant"}], 0)
    eng = Engine([(m, F.blobs(w, h, 7, 1))], tol=r.tol, dark=r.dark, min_dt_ns=r.min_dt_ns,
                 max_refine_levels=r.max_refine_levels, l_min=0, l_max=r.l_max)
    if net is not None:
        eng.set_proposal(net, margin=-3.0)
    eng.set_graph(False)
    return eng


@pytest.mark.parametrize("kind", sorted(KINDS))
def test_two_sizes_at_once(cuda_lib, kind):
    from ballasim_b200.learned import StepMLP

    few, many = KINDS[kind]
    net = StepMLP(seed=3) if kind == "learned" else None
    engines = [make(kind, size, net) for size in (many, few, few, few)]
    errors, done = [], threading.Event()

    def work(i):
        try:
            engines[i].start(0)
            n = 0
            while not done.is_set() and (i > 0 or n < RUNS):
                engines[i].run(1)
                n += 1
        except Exception as e:  # reported by the main thread
            errors.append(f"{(few, many)[i == 0]}: {e}")
        if i == 0:
            done.set()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(engines))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
