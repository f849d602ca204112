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
    "two rounds": ([(400, 250)], False, RULES, 2),
    "one pixel": ([(1, 1)], False, RULES, 12),
    "ragged": ([(75, 43), (33, 9)], False, RULES, 6),
    "past the stage": ([(40, 22)], False, replace(RULES, l_min=5), 3),
    "some past the stage": ([(40, 22)], False, replace(RULES, tol=2e-4), 4),
    "lattice": ([(75, 43), (33, 9)], True, RULES, 3),
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
