"""The split engine (stage 1) where its quick test, blob lists, noise stops and crossing search change their path: the
events against the oracle chain, and the events and saved states against the streaming engine (stage 0), bit for bit."""
from dataclasses import replace

import numpy as np
import pytest

from ballasim_b200 import fields as F
from ballasim_b200 import workloads as W
from ballasim_b200.params import resolve

pytestmark = pytest.mark.gpu

NOISY = {**W.MISMATCH, **W.NOISE, "noise_shot_rate_hz": 40.0, "noise_ba_median_hz": 20.0, "leak_rate_hz": 2.0}
RULES = W.Rules()


def dim(field: F.Field, base: float, scale: float) -> F.Field:
    b = field.blobs.copy()
    b[:, 0] *= np.float32(scale)
    return replace(field, base=float(np.float32(base)), blobs=b)


def signed(field: F.Field) -> F.Field:
    b = field.blobs.copy()
    b[::2, 0] *= np.float32(-0.2)
    return replace(field, blobs=b)


# name: (width, height, overrides, field, rules, windows)
CASES = {
    # one tile's list: a few slot groups, more blobs than centres, more than a list holds
    "slot groups": (41, 30, NOISY, F.blobs(41, 30, 5, 24), RULES, 12),
    "over 64 listed": (24, 20, NOISY, F.blobs(24, 20, 6, 90), replace(RULES, l_max=3), 6),
    "over 256 listed": (16, 9, NOISY, F.blobs(16, 9, 7, 300), RULES, 6),
    # noise stops: none skipped (a dim field accepts nearly every candidate), bounds from negative amplitudes
    "dim": (33, 21, {**NOISY, "noise_shot_rate_hz": 20.0, "noise_ba_median_hz": 0.0},
            dim(F.blobs(33, 21, 8, 6), 0.01, 0.002), RULES, 20),
    "signed": (40, 24, NOISY, signed(F.blobs(40, 24, 9, 12)), RULES, 16),
    # refined windows, some past the stage; segments down to 2 ns
    "refined": (32, 24, W.MISMATCH, F.blobs(32, 24, 10, 8, v_sigma=400.0), replace(RULES, tol=2e-4, l_max=2), 6),
    "fine": (20, 12, W.MISMATCH, F.blobs(20, 12, 11, 4, v_sigma=400.0),
             replace(RULES, tol=1e-4, min_dt_ns=1, max_refine_levels=3, l_max=3), 4),
    "level 0": (20, 12, NOISY, F.blobs(20, 12, 12, 6), replace(RULES, l_min=0, l_max=0), 10),
    # resets and references
    "ideal refractory": (40, 24, {**NOISY, "reset_mode": "ideal", "refractory_s": 2e-3}, F.blobs(40, 24, 13, 8), RULES, 16),
    "long refractory": (40, 24, {**NOISY, "refractory_s": 2e-2}, F.blobs(40, 24, 14, 8), RULES, 16),
    "no refractory": (40, 24, {**NOISY, "refractory_s": 0.0}, F.blobs(40, 24, 15, 8), RULES, 12),
    "strong leak": (40, 24, {**W.MISMATCH, "leak_rate_hz": 40.0, "leak_sigma_log10": 0.3}, F.blobs(40, 24, 16, 8, v_sigma=5.0),
                    RULES, 20),
    # single pixels and partial tiles
    "one pixel": (1, 1, NOISY, F.blobs(1, 1, 17, 3), RULES, 40),
    "one row": (35, 1, NOISY, F.blobs(35, 1, 18, 4), RULES, 20),
    "edge": (30, 21, {**W.MISMATCH, "leak_rate_hz": 1.0}, F.tanh_edge(30, 21, 3), RULES, 16),
}


def engine(specs, rules, stage):
    from ballasim_b200.engine import Engine
    from ballasim_b200.sensor import SensorModel

    models = [SensorModel(resolve(s.preset, s.overrides), s.width, s.height, s.seed, [{"type": "constant"}], s.camera)
              for s in specs]
    eng = Engine([(m, s.field) for m, s in zip(models, specs)], tol=rules.tol, dark=rules.dark,
                 min_dt_ns=rules.min_dt_ns, max_refine_levels=rules.max_refine_levels, l_min=rules.l_min,
                 l_max=rules.l_max)
    eng.set_launch(0, 0, stage, 8)
    return eng, models


def run(eng, models, chunks, frames=None):
    """Each model's events over the chunks and its saved state after them, and the samples."""
    eng.start(0, frames=frames)
    samples, parts = 0, [[] for _ in models]
    for n in chunks:
        samples += eng.run(n)[0]
        for i, m in enumerate(models):
            parts[i].append(m.take_events(with_pixel=True))
    events = [{k: np.concatenate([p[k] for p in ps]) for k in ps[0]} for ps in parts]
    return events, [m.save_state() for m in models], samples


def same(a: dict, b: dict) -> None:
    for k in ("pixel", "p", "label", "flags", "t_cross_ns", "ds", "dn", "dl", "l_first"):
        x, y = np.asarray(a[k]), np.asarray(b[k])
        if x.dtype.kind == "f":
            x, y = x.view(np.uint32), y.view(np.uint32)
        assert np.array_equal(x, y), k


@pytest.mark.parametrize("name", sorted(CASES))
def test_events_and_states(cuda_lib, name):
    from oracle.oracle import simulate_port

    w, h, overrides, field, rules, windows = CASES[name]
    spec = W.SensorSpec(w, h, 31, 2, dict(overrides), field)
    ora, st = simulate_port(spec, rules, windows)
    split, states, samples = run(*engine([spec], rules, 1), (windows // 2, windows - windows // 2))
    assert samples == st["pixel_samples"] and len(ora["t_cross_ns"]) > 0
    same(split[0], ora)
    assert states == run(*engine([spec], rules, 0), (windows // 2, windows - windows // 2))[1]


def test_more_sensors_than_kernel_arguments_and_given_frames(cuda_lib):
    """19 sensors (their first tiles looked up in device memory), started from frames below and above the fields, so
    that the noise bound comes from the carried sample: as the streaming engine from the same frames."""
    specs = [W.SensorSpec(8 + i, 5 + i % 3, 40 + i, i, dict(NOISY), F.blobs(8 + i, 5 + i % 3, 40 + i, 3))
             for i in range(19)]
    rng = np.random.default_rng(1)
    frames = [rng.uniform(0.0, 200.0, s.width * s.height).astype(np.float32) for s in specs]
    got, want = (run(*engine(specs, RULES, stage), (3, 9), frames) for stage in (1, 0))
    assert got[2] == want[2] and sum(len(e["p"]) for e in got[0]) > 100
    for a, b in zip(got[0], want[0]):
        same(a, b)
    assert got[1] == want[1]
