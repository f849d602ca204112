"""An engine's launch shape: what launch reports is what set_launch takes, and the autotuner leaves the engine whole."""
from dataclasses import replace

import pytest

from ballasim_b200 import fields as F
from ballasim_b200 import workloads as W
from ballasim_b200.params import resolve

pytestmark = pytest.mark.gpu


def engine(preset, rows, w=60, h=40, field=None, r=W.Rules()):
    from ballasim_b200.engine import Engine
    from ballasim_b200.sensor import SensorModel

    m = SensorModel(resolve(preset, rows), w, h, 9, [{"type": "constant"}], 0)
    eng = Engine([(m, field or F.blobs(w, h, 9, 5))], tol=r.tol, dark=r.dark, min_dt_ns=r.min_dt_ns,
                 max_refine_levels=r.max_refine_levels, l_min=r.l_min, l_max=r.l_max)
    return eng, m


@pytest.mark.parametrize("kind", ["instantaneous", "learned", "cascade", "lattice"])
def test_launch_goes_back_in(cuda_lib, kind):
    from ballasim_b200.learned import StepMLP

    preset = "ideal" if kind in ("instantaneous", "learned") else "prophesee_gen3"
    eng, _ = engine(preset, {**W.MISMATCH, "noise": kind == "lattice"})
    before = eng.launch
    if kind == "learned":
        eng.set_proposal(StepMLP(seed=1))
        with pytest.raises(ValueError):
            eng.set_launch(stage=1)  # no split engine with a proposal
    shape = eng.launch
    eng.set_launch(**shape)
    assert eng.launch == shape
    if kind == "learned":
        eng.set_proposal(None)
    assert eng.launch == before
    eng.start(0)
    assert eng.run(2)[0] > 0


@pytest.mark.parametrize("kind, shapes", [("learned", 3), ("cascade", 3), ("lattice", 12)])
def test_the_autotuner_tries_a_shape_once(cuda_lib, kind, shapes):
    from ballasim_b200.learned import StepMLP

    eng, _ = engine("ideal" if kind == "learned" else "prophesee_gen3", {**W.MISMATCH, "noise": kind == "lattice"})
    if kind == "learned":
        eng.set_proposal(StepMLP(seed=1))
    eng.start(0)
    rows = eng.autotune(2)
    assert len(rows) == shapes == len({(r["tile_width"], r["warps_per_block"], r["stage"]) for r in rows})
    assert eng.launch["tile_width"] == min(rows, key=lambda r: r["ms"])["tile_width"]


def test_a_failed_autotune_leaves_the_shape(cuda_lib):
    eng, m = engine("ideal", {**W.MISMATCH, "noise": False})
    eng.set_launch(2, 3, 16, 16)
    shape = eng.launch
    with pytest.raises(RuntimeError):  # before start()
        eng.autotune(2)
    assert eng.launch == shape


@pytest.mark.parametrize("size, field, rules, stage", [
    ((346, 260), dict(), dict(), 1),
    ((346, 260), dict(v_sigma=600.0), dict(), 0),  # levels past 4
    ((346, 260), dict(v_sigma=600.0), dict(l_max=4), 1),  # 0.8 px a step: within the tolerance
    ((346, 260), dict(v_sigma=600.0), dict(l_max=4, tol=1e-4), 0),
    ((346, 260), dict(), dict(tol=1e-5), 0),  # refined past the stage
    ((346, 260), dict(), dict(tol=1e-5, max_refine_levels=0), 1),
    ((346, 260), dict(), dict(l_min=5), 0),
    ((97, 61), dict(v_sigma=600.0), dict(), 1),  # few tiles
    ((97, 61), dict(), dict(l_min=5), 0),
    ((346, 260), dict(n_blobs=256, v_sigma=600.0), dict(), 0),
    ((346, 260), dict(n_blobs=257, v_sigma=600.0), dict(), 1),  # more blobs than the streaming engine lists
])
def test_the_stage_an_engine_starts_with(cuda_lib, size, field, rules, stage):
    """The split engine where the windows are expected to fit its stage or the tiles are few, and the streaming engine's
    events whichever it is."""
    w, h = size
    r = replace(W.Rules(), **rules)
    f = F.blobs(w, h, 9, **{"n_blobs": 12, **field})
    got = []
    for chosen in (None, 0):
        eng, m = engine("ideal", {**W.MISMATCH, **W.NOISE}, w, h, f, r)
        if chosen is None:
            assert eng.launch["stage"] == stage
        else:
            eng.set_launch(stage=chosen)
        eng.start(0)
        got.append((eng.run(3), m.take_events(with_pixel=True), m.save_state()))
    assert got[0][0] == got[1][0] and got[0][2] == got[1][2]
    for k in got[0][1]:
        assert got[0][1][k].tobytes() == got[1][1][k].tobytes(), k


@pytest.mark.parametrize("speed, stage", [(40.0, 1), (-40.0, 1), (600.0, 0), (-600.0, 0)])
def test_the_stage_of_an_edge(cuda_lib, speed, stage):
    eng, _ = engine("ideal", W.MISMATCH, 346, 260, replace(F.tanh_edge(346, 260, 3), speed=speed))
    assert eng.launch["stage"] == stage


@pytest.mark.parametrize("field, rules, stage", [
    (dict(), dict(), 32), (dict(), dict(tol=1e-5), 32), (dict(), dict(l_min=4), 32), (dict(), dict(l_min=5), 0),
    (dict(v_sigma=1500.0), dict(), 0), (dict(v_sigma=1500.0), dict(l_max=4), 32),
])
def test_the_stage_of_the_lattice(cuda_lib, field, rules, stage):
    eng, _ = engine("prophesee_gen3", W.MISMATCH, 60, 40, F.blobs(60, 40, 9, 5, **field), replace(W.Rules(), **rules))
    assert eng.launch["stage"] == stage


@pytest.mark.parametrize("speed, tol, stage", [(40.0, 1e-2, 32), (40.0, 1e-4, 32), (40.0, 1e-6, 0), (2000.0, 1e-2, 0)])
def test_the_stage_of_the_lattice_at_an_edge(cuda_lib, speed, tol, stage):
    eng, _ = engine("prophesee_gen3", W.MISMATCH, 60, 40, replace(F.tanh_edge(60, 40, 3), speed=speed),
                    replace(W.Rules(), tol=tol))
    assert eng.launch["stage"] == stage
