"""The fused engine with the cascade, its noise lattice and a learned proposal where the windows' lengths differ a lot (blobs
of many pixels per window, fine lattices, fine tolerances): the cascade and the lattice against the two-kernel route on
the same windows, the learned engine's forms against one another, bit for bit."""
from dataclasses import replace

import numpy as np
import pytest

from ballasim_b200 import fields as F
from ballasim_b200 import workloads as W
from ballasim_b200.params import resolve

pytestmark = pytest.mark.gpu

RULES = W.Rules()
# name: (frames, field of a frame, rules, windows)
CASES = {
    "fast blobs": ([(75, 43), (33, 9)], lambda w, h, i: F.blobs(w, h, 50 + i, 6, v_sigma=1500.0), RULES, 4),
    "fast blobs, large": ([(346, 260)], lambda w, h, i: F.blobs(w, h, 50 + i, 40, v_sigma=600.0), RULES, 2),
    "fine lattice": ([(40, 22)], lambda w, h, i: F.blobs(w, h, 50 + i, 3), replace(RULES, l_min=6), 3),
    "fine tolerance": ([(60, 40)], lambda w, h, i: F.blobs(w, h, 50 + i, 4), replace(RULES, tol=1e-5), 3),
    # a slow edge under a fine tolerance: taken for even windows, with some past every stage
    "edge past the stages": ([(60, 40)], lambda w, h, i: F.tanh_edge(w, h, 4), replace(RULES, tol=1e-6), 4),
    "edge past the stages, large": ([(346, 260)], lambda w, h, i: F.tanh_edge(w, h, 4), replace(RULES, tol=1e-6), 2),
}


def play_engine(sensors, rules, windows, proposal=None):
    from ballasim_b200.engine import Engine

    eng = Engine(sensors, **kw(rules))
    if proposal is not None:
        eng.set_proposal(proposal, margin=0.0)
    eng.start(0)
    got = [[] for _ in sensors]
    for n in (1, windows - 1):
        eng.run(n)
        for i, ev in enumerate(eng.take_events(with_pixel=True)):
            got[i].append(ev)
    return eng, got


def kw(rules):
    return dict(tol=rules.tol, dark=rules.dark, min_dt_ns=rules.min_dt_ns, max_refine_levels=rules.max_refine_levels,
                l_min=rules.l_min, l_max=rules.l_max)


def make(sizes, field, preset, rows):
    from ballasim_b200.sensor import SensorModel

    return [(SensorModel(resolve(preset, rows), w, h, 50 + i, [{"type": "constant"}], i), field(w, h, i))
            for i, (w, h) in enumerate(sizes)]


@pytest.mark.parametrize("lattice", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_photoreceptors_against_the_runs_route(cuda_lib, name, lattice):
    from ballasim_b200.windows import DeviceWindows

    sizes, field, rules, windows = CASES[name]
    rows = {**W.MISMATCH, "noise": lattice, "leak_rate_hz": 1.0}
    a, b = (make(sizes, field, "prophesee_gen3", rows) for _ in range(2))
    _, got = play_engine(a, rules, windows)
    dw = DeviceWindows(b, **kw(rules))
    dw.start(0)
    want = [[] for _ in sizes]
    dw.run(windows, on_events=lambda i, m, ev: want[i].append(m.download_events(ev, with_pixel=True)), concurrent=False)
    for i in range(len(sizes)):
        g, w = ({k: np.concatenate([p[k] for p in parts[i]]) for k in parts[i][0]} for parts in (got, want))
        for k in g:
            assert g[k].tobytes() == w[k].tobytes(), k
        assert a[i][0].save_state() == b[i][0].save_state()


@pytest.mark.parametrize("name", sorted(CASES))
def test_learned_forms_agree(cuda_lib, name):
    """The first sensor on its own (warps apart on few tiles) and beside one of 5,000 tiles, over fields that keep the
    blocks in step or let them run: the same events and state."""
    from ballasim_b200.learned import StepMLP

    sizes, field, rules, windows = CASES[name]
    net, got = StepMLP(seed=3), []
    for beside in (None, lambda w, h, i: F.blobs(w, h, 3, 20), lambda w, h, i: F.blobs(w, h, 3, 20, v_sigma=1500.0)):
        sensors = make(sizes[:1], field, "ideal", {**W.MISMATCH, **W.NOISE})
        if beside is not None:
            sensors += make([(400, 400)], beside, "ideal", W.MISMATCH)
        eng, ev = play_engine(sensors, rules, windows, net)
        got.append(([{k: v.tobytes() for k, v in e.items()} for e in ev[0]], sensors[0][0].save_state()))
    assert got[0] == got[1] == got[2]
