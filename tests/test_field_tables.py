"""Blob tables that the fields' own generator does not make, as the C ABI takes them."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from ballasim_b200 import fields as F
from ballasim_b200 import workloads as W
from ballasim_b200.params import resolve

ROOT = Path(__file__).resolve().parents[1]
RULES = W.Rules()


def sensors(sizes, rows):
    from ballasim_b200.sensor import SensorModel

    return [SensorModel(resolve("ideal", rows), w, h, 70 + i, [{"type": "constant"}], i) for i, (w, h) in enumerate(sizes)]


def play(models, structs, stage, frames=None, windows=(3, 9)):
    """Every model's events and saved state over the runs of a C ABI engine on these field structs."""
    from ballasim_b200 import _lib

    L, n, r = _lib.lib(), len(models), RULES
    rules = _lib.SampleRules(r.tol, r.dark, 1, 1, r.max_refine_levels, r.min_dt_ns, r.l_min, r.l_max)
    handles = (C.c_void_p * n)(*[m.handle.value for m in models])
    h = C.c_void_p()
    _lib.check(L.bs_engine_create(handles, (_lib.Field * n)(*structs), n, C.byref(rules), C.byref(h)))
    try:
        _lib.check(L.bs_engine_set_launch(h, 0, 0, stage, 0))
        if frames is None:
            _lib.check(L.bs_engine_start(h, 0, None))
        else:
            arrs = [np.ascontiguousarray(f, np.float32).reshape(-1) for f in frames]
            _lib.check(L.bs_engine_start_frames(h, 0, (C.c_void_p * n)(*[a.ctypes.data for a in arrs]), None))
        events = []
        for w in windows:
            _lib.check(L.bs_engine_run(h, w, None, None, None))
            events += [m.take_events(with_pixel=True) for m in models]
    finally:
        L.bs_engine_destroy(h)
    return events, [m.save_state() for m in models]


def same(a, b):
    for x, y in zip(a[0], b[0], strict=True):
        for k in x:
            assert np.asarray(x[k]).tobytes() == np.asarray(y[k]).tobytes(), k
    assert a[1] == b[1]


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [[(40, 24)], [(40, 24), (400, 400)]])
def test_a_negative_count_is_an_empty_table(cuda_lib, sizes):
    """In the call of one launch (few tiles) and in the one of two launches per window."""
    from ballasim_b200.sampling import field_struct

    rows = {**W.MISMATCH, **W.NOISE, "noise_shot_rate_hz": 40.0}
    got = []
    for count in (-1, 0, -(2**31)):
        structs = []
        for i, (w, h) in enumerate(sizes):
            s = field_struct(F.blobs(w, h, 70 + i, 3))
            if i == 0:
                s.n_blobs, s.blobs = count, None
            structs.append(s)
        got.append(play(sensors(sizes, rows), structs, 1))
    assert sum(len(e["p"]) for e in got[1][0]) > 0
    same(got[0], got[1])
    same(got[2], got[1])


# name: (word of the blob row, its value) on the first blob of the first sensor
TABLES = {
    "an amplitude of NaN": {0: np.nan},
    "an infinite amplitude": {0: -np.inf},
    "a term that grows": {0: -5.0, 5: -0.01, 6: 1600.0},  # below 0 from 15 px out to its rim at 40
    "a NaN falloff": {5: np.nan},
    "an infinite falloff": {5: np.inf},
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(TABLES))
def test_noise_under_a_table_out_of_the_ordinary(cuda_lib, name):
    """The shot candidates that the bound on the field's values lets the split engine skip are ones that the model
    rejects, whatever the table holds: the streaming engine (which skips none) gives the same events and states."""
    from ballasim_b200.sampling import field_struct

    rows = {**W.MISMATCH, **W.NOISE, "noise_shot_rate_hz": 60.0}
    got = []
    for stage in (1, 0):
        f = F.blobs(48, 32, 90, 4)
        b = f.blobs.copy()
        b[0, 1:5] = (24.0, 16.0, 60.0, -40.0)
        for k, v in TABLES[name].items():
            b[0, k] = np.float32(v)
        f.blobs = b
        got.append(play(sensors([(48, 32)], rows), [field_struct(f)], stage, [np.full(48 * 32, f.base, np.float32)], (4, 12)))
    assert sum(np.count_nonzero(e["label"] == 1) for e in got[1][0]) > 20
    same(got[0], got[1])


def test_bounds_hold_every_sample(tmp_path):
    """field_bounds on the CPU over random fields (tests/native/field_bounds.cc)."""
    exe = tmp_path / "field_bounds"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT / 'ballasim_b200' / 'csrc'}",
                    str(ROOT / "tests" / "native" / "field_bounds.cc"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
