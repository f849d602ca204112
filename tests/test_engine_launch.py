"""An engine's launch shape: what launch reports is what set_launch takes, and the autotuner leaves the engine whole."""
import pytest

from ballasim_b200 import fields as F
from ballasim_b200 import workloads as W
from ballasim_b200.params import resolve

pytestmark = pytest.mark.gpu


def engine(preset, rows, w=60, h=40):
    from ballasim_b200.engine import Engine
    from ballasim_b200.sensor import SensorModel

    r = W.Rules()
    m = SensorModel(resolve(preset, rows), w, h, 9, [{"type": "constant"}], 0)
    eng = Engine([(m, F.blobs(w, h, 9, 5))], tol=r.tol, dark=r.dark, min_dt_ns=r.min_dt_ns,
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
