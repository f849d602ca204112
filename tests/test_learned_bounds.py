"""The learned engine's quiet windows (kept from the pixel model by two bounds on their samples) where the window's first
sample, the one carried over from the window before, is not a number: the model takes such a sample as 0."""
import numpy as np
import pytest

from ballasim_b200 import fields as F
from ballasim_b200.params import resolve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["learned, apart", "learned, in step", "split"])
def test_a_carried_sample_that_is_no_number(cuda_lib, form):
    """One sample a window (no lattice level, no refinement) of a field that is 100 but for one pixel at each window's
    end, where it is no number: ln I falls by 25 from the instant before the end to the end itself, which is the next
    window's to find. Against the streaming engine."""
    from ballasim_b200.engine import Engine
    from ballasim_b200.learned import StepMLP
    from ballasim_b200.sensor import SensorModel

    w, h, windows = (33, 1, 12) if form != "learned, in step" else (330, 120, 12)  # 8 tiles a multiprocessor: 1,184
    step = 2.0 / (2**23 * 1e-9)  # two pixels a window, a reach of half a pixel
    f = F.blobs(w, h, 3, 1)
    f.base = 100.0
    f.blobs = np.array([[np.nan, 0.5, 0.5, step, 0.0, 1.0, 0.25, 0.0, 0.0, 0.0]], np.float32)
    rows = {"theta_on": 20.0, "theta_off": 20.0, "dark_current_fA": 1e-9, "leak_rate_hz": 0.0, "noise": False}
    got = []
    for learned in (form.startswith("learned"), None):
        m = SensorModel(resolve("ideal", rows), w, h, 5, [{"type": "constant"}], 0)
        eng = Engine([(m, f)], tol=0.01, dark=0.01, min_dt_ns=2**23, max_refine_levels=0, l_min=0, l_max=0)
        if learned is None:
            eng.set_launch(0, 0, 0, 8)
        elif learned:
            eng.set_proposal(StepMLP(seed=3), margin=-40.0)
        eng.start(0, frames=[np.full(w * h, 100.0, np.float32)])
        samples = eng.run(windows)[0]
        got.append((samples, m.take_events(with_pixel=True), m.save_state()))
    assert got[0][0] == got[1][0] == 2 * w * h * windows
    assert len(got[1][1]["p"]) > 5
    for k in got[0][1]:
        assert got[0][1][k].tobytes() == got[1][1][k].tobytes(), k
    assert got[0][2] == got[1][2]
