"""The split engine where most windows hold more samples than it stages (motion of many pixels per window, a fine tolerance,
a fine lattice): pixels posted whole, walked again over their tile's blob list by warps that take their records as they
come. Against the streaming engine, bit for bit, in the call of one launch and in that of two launches per window; blob
lists of none, some, more than the slot groups' 64 and more than a list's 256."""
from dataclasses import replace

import pytest

from ballasim_b200 import fields as F
from ballasim_b200 import workloads as W
from test_split_engine import NOISY, RULES, engine, run, same

pytestmark = pytest.mark.gpu

# name: (width, height, field, rules, windows)
CASES = {
    "fast": (64, 48, F.blobs(64, 48, 3, 6, v_sigma=1500.0), RULES, 10),
    "fast, many blobs": (40, 24, F.blobs(40, 24, 4, 120, v_sigma=1500.0), RULES, 4),
    "fast, over a list": (24, 16, F.blobs(24, 16, 5, 300, v_sigma=1500.0), RULES, 3),
    "fine tolerance": (64, 48, F.blobs(64, 48, 6, 6, v_sigma=300.0), replace(RULES, tol=1e-5), 6),
    "fine lattice": (64, 48, F.blobs(64, 48, 7, 6), replace(RULES, l_min=6), 6),
    "fast edge": (64, 48, replace(F.tanh_edge(64, 48, 8), speed=1500.0), replace(RULES, tol=1e-4), 8),
    "no blobs": (33, 17, F.blobs(33, 17, 9, 0), replace(RULES, l_min=5), 4),
}


@pytest.mark.parametrize("beside", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_against_the_streaming_engine(cuda_lib, name, beside):
    w, h, field, rules, windows = CASES[name]
    specs = [W.SensorSpec(w, h, 31, 2, dict(NOISY), field)]
    if beside:  # 5,000 tiles more: two launches per window, and more posted pixels than one pass of their kernel takes
        specs.append(W.SensorSpec(400, 400, 91, 30, dict(W.MISMATCH), F.blobs(400, 400, 91, 30, v_sigma=1500.0)))
    got, want = (run(*engine(specs, rules, stage), (1, windows - 1)) for stage in (1, 0))
    assert got[2] == want[2] and got[1] == want[1]
    assert sum(len(e["p"]) for e in want[0]) > 0
    for a, b in zip(got[0], want[0], strict=True):
        same(a, b)


def test_windows_past_the_stage_and_then_none(cuda_lib):
    """Blobs that leave the frame: the windows past the stage are the first ones only."""
    f = F.blobs(64, 48, 3, 4, v_sigma=2000.0)
    specs = [W.SensorSpec(64, 48, 31, 2, dict(NOISY), f)]
    got, want = (run(*engine(specs, RULES, stage), (3, 30)) for stage in (1, 0))
    same(got[0][0], want[0][0])
    assert got[1:] == want[1:]
