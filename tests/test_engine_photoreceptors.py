"""The fused engine with the cascade photoreceptor (its warps in step) and with its noise lattice against the two-kernel
route on the same windows (sample runs in device memory, the one-thread-per-pixel model), bit for bit: whole rounds of
blocks and a last one that is partly filled, single pixels, windows past the stage, several sensors, two calls."""
from dataclasses import replace

import numpy as np
import pytest

from ballasim_b200 import fields as F
from ballasim_b200 import workloads as W
from ballasim_b200.params import resolve

pytestmark = pytest.mark.gpu

RULES = W.Rules()
CASES = {
    "one round in step": ([(200, 120)], False, RULES, 3),
    "two rounds": ([(400, 250)], False, RULES, 2),
    "one pixel": ([(1, 1)], False, RULES, 12),
    "ragged": ([(75, 43), (33, 9)], False, RULES, 6),
    "past the stage": ([(40, 22)], False, replace(RULES, l_min=5), 3),
    "some past the stage": ([(40, 22)], False, replace(RULES, tol=2e-4), 4),
    "lattice": ([(75, 43), (33, 9)], True, RULES, 3),
    "lattice, capped": ([(332, 244)], True, RULES, 2),
    "lattice past the stage": ([(24, 16)], True, replace(RULES, l_min=6), 2),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_against_the_runs_route(cuda_lib, name):
    from ballasim_b200.engine import Engine
    from ballasim_b200.sensor import SensorModel
    from ballasim_b200.windows import DeviceWindows

    sizes, lattice, rules, windows = CASES[name]
    rows = {**W.MISMATCH, "noise": lattice, "leak_rate_hz": 1.0}

    def sensors():
        return [(SensorModel(resolve("prophesee_gen3", rows), w, h, 50 + i, [{"type": "constant"}], i),
                 F.blobs(w, h, 50 + i, max(3, w * h // 2000), v_sigma=120.0)) for i, (w, h) in enumerate(sizes)]

    kw = dict(tol=rules.tol, dark=rules.dark, min_dt_ns=rules.min_dt_ns, max_refine_levels=rules.max_refine_levels,
              l_min=rules.l_min, l_max=rules.l_max)
    a, b = sensors(), sensors()
    eng = Engine(a, **kw)
    eng.start(0)
    got = [[] for _ in sizes]
    for n in (1, windows - 1):
        eng.run(n)
        for i, ev in enumerate(eng.take_events(with_pixel=True)):
            got[i].append(ev)
    dw = DeviceWindows(b, **kw)
    dw.start(0)
    want = [[] for _ in sizes]
    dw.run(windows, on_events=lambda i, m, ev: want[i].append(m.download_events(ev, with_pixel=True)), concurrent=False)
    total = 0
    for i in range(len(sizes)):
        g, w = ({k: np.concatenate([p[k] for p in parts[i]]) for k in parts[i][0]} for parts in (got, want))
        for k in g:
            x, y = (v.view(np.uint32) if v.dtype.kind == "f" else v for v in (g[k], w[k]))
            assert np.array_equal(x, y), k
        total += len(g["p"])
        assert a[i][0].save_state() == b[i][0].save_state()
    assert total > 0 or name == "one pixel"


@pytest.mark.parametrize("alone, beside", [((75, 43), (400, 250)), ((1, 1), (320, 160)), ((128, 74), (300, 130))])
def test_learned_warps_apart_and_in_step(cuda_lib, alone, beside):
    """A sensor on its own (few tiles: its warps run apart) and beside a larger one (the blocks' warps in step) gives the
    same events and state."""
    from ballasim_b200.engine import Engine
    from ballasim_b200.learned import StepMLP
    from ballasim_b200.sensor import SensorModel

    net, r, got = StepMLP(seed=3), RULES, []
    for sizes in ([alone], [alone, beside]):
        sensors = [(SensorModel(resolve("ideal", W.NOISE), w, h, 60 + i, [{"type": "constant"}], i),
                    F.blobs(w, h, 60 + i, max(3, w * h // 2000), v_sigma=120.0)) for i, (w, h) in enumerate(sizes)]
        eng = Engine(sensors, tol=r.tol, dark=r.dark, min_dt_ns=r.min_dt_ns, max_refine_levels=r.max_refine_levels,
                     l_min=r.l_min, l_max=r.l_max)
        eng.set_proposal(net, margin=0.0)
        eng.start(0)
        eng.run(6)
        got.append((eng.take_events(with_pixel=True)[0], sensors[0][0].save_state()))
    for k in got[0][0]:
        assert got[0][0][k].tobytes() == got[1][0][k].tobytes(), k
    assert got[0][1] == got[1][1]
