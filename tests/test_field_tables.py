"""Blob tables that the fields' own generator does not make, as the C ABI takes them."""
import ctypes as C

import numpy as np
import pytest

from ballasim_b200 import fields as F
from ballasim_b200 import workloads as W
from ballasim_b200.params import resolve

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
