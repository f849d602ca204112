"""The split engine's form of two launches per window, which calls of more than 4,736 tiles take, on the small sensors of
test_split_engine: a second sensor of 5,000 tiles and no blobs beside each takes the call over that line."""
from dataclasses import replace

import numpy as np
import pytest

from ballasim_b200 import fields as F
from ballasim_b200 import workloads as W
from ballasim_b200.params import resolve
from test_split_engine import CASES, NOISY, RULES, engine, run, same

pytestmark = pytest.mark.gpu

BESIDE = W.SensorSpec(400, 400, 91, 30, dict(W.MISMATCH), F.blobs(400, 400, 91, 0))


@pytest.mark.parametrize("name", sorted(CASES))
def test_events_and_states(cuda_lib, name):
    from oracle.oracle import simulate_port

    w, h, overrides, field, rules, windows = CASES[name]
    spec = W.SensorSpec(w, h, 31, 2, dict(overrides), field)
    chunks = (windows // 2, windows - windows // 2)
    ora, _ = simulate_port(spec, rules, windows)
    # the sensor under test before the other one and after it
    for specs, i in (([spec, BESIDE], 0), ([BESIDE, spec], 1)):
        events, states, samples = run(*engine(specs, rules, 1), chunks)
        want = run(*engine(specs, rules, 0), chunks)
        assert samples == want[2] and states == want[1] and len(ora["t_cross_ns"]) > 0
        same(events[i], ora)
        same(events[1 - i], want[0][1 - i])


@pytest.mark.parametrize("l_min,windows", [(5, 6), (3, 10)])
def test_windows_past_the_stage(cuda_lib, l_min, windows):
    from oracle.oracle import simulate_port

    wl = W.small("noise", 40, 30, windows)
    rules = replace(wl.rules, l_min=l_min, l_max=max(l_min, wl.rules.l_max))
    rates = {"noise_shot_rate_hz": 40.0, "noise_ba_median_hz": 30.0, "leak_rate_hz": 3.0}
    spec = replace(wl.sensors[0], overrides={**wl.sensors[0].overrides, **rates})
    ora, _ = simulate_port(spec, rules, windows, params=resolve("ideal", spec.overrides))
    events, _, _ = run(*engine([spec, BESIDE], rules, 1), (windows,))
    same(events[0], ora)
    assert len(ora["t_cross_ns"]) > 20


def test_more_sensors_than_kernel_arguments_and_given_frames(cuda_lib):
    specs = [W.SensorSpec(8 + i, 5 + i % 3, 40 + i, i, dict(NOISY), F.blobs(8 + i, 5 + i % 3, 40 + i, 3))
             for i in range(18)]
    specs.insert(9, BESIDE)
    rng = np.random.default_rng(1)
    frames = [rng.uniform(0.0, 200.0, s.width * s.height).astype(np.float32) for s in specs]
    got, want = (run(*engine(specs, RULES, stage), (3, 9), frames) for stage in (1, 0))
    assert got[2] == want[2] and sum(len(e["p"]) for e in got[0]) > 100
    for a, b in zip(got[0], want[0], strict=True):
        same(a, b)
    assert got[1] == want[1]


def test_a_call_run_again_for_its_events(cuda_lib):
    """More events than the buffers have room for at first (65,536): the call starts again from its input state."""
    spec = W.SensorSpec(480, 360, 33, 1, {**NOISY, "noise_ba_median_hz": 200.0}, F.blobs(480, 360, 33, 60))
    got = []
    for stage in (1, 0):
        eng, models = engine([spec], RULES, stage)
        got.append(run(eng, models, (30, 8)))
        assert models[0].stats()["gpu_reruns"] >= 1
    assert len(got[1][0][0]["p"]) > 1 << 16
    same(got[0][0][0], got[1][0][0])
    assert got[0][1:] == got[1][1:]
