"""A captured engine step and the buffers that it holds by address: sequences in which a call outside the graph makes the
split engine's buffers grow between two calls of one graph key, against the same calls without a graph."""
import numpy as np
import pytest

from ballasim_b200 import fields as F
from ballasim_b200 import workloads as W
from ballasim_b200.params import resolve

pytestmark = pytest.mark.gpu

# (tile width, windows, recording: the step outside the graph) per call, on 61 x 41 px: 82 tiles 32 px wide, 96 tiles 4 px
# wide.
SEQUENCES = {
    "more windows": [(8, 10, False), (8, 60, True), (8, 10, False), (8, 10, False)],
    "more tiles": [(32, 6, False), (4, 6, True), (32, 6, False)],
    "both": [(32, 6, False), (4, 40, True), (32, 6, False), (4, 6, False)],
}


def play(calls, graph):
    from ballasim_b200.engine import Engine
    from ballasim_b200.sensor import SensorModel

    r = W.Rules()
    m = SensorModel(resolve("ideal", {**W.MISMATCH, **W.NOISE}), 61, 41, 5, [{"type": "constant"}], 0)
    eng = Engine([(m, F.blobs(61, 41, 5, 6))], tol=r.tol, dark=r.dark, min_dt_ns=r.min_dt_ns,
                 max_refine_levels=r.max_refine_levels, l_min=r.l_min, l_max=r.l_max)
    eng.set_graph(graph)
    eng.start(0)
    events = []
    for width, windows, record in calls:
        eng.set_launch(0, 0, 1, width)
        eng.set_record(1024 if record else 0)
        eng.run(windows)
        events.append(m.take_events(with_pixel=True))
    return events, m.save_state()


@pytest.mark.parametrize("name", sorted(SEQUENCES))
def test_a_replay_finds_its_buffers(cuda_lib, name):
    (got, state), (want, want_state) = (play(SEQUENCES[name], graph) for graph in (True, False))
    assert sum(len(e["p"]) for e in want) > 100
    for a, b in zip(got, want):
        for k in a:
            assert np.asarray(a[k]).tobytes() == np.asarray(b[k]).tobytes(), k
    assert state == want_state


def test_a_network_in_place_of_another(cuda_lib):
    """Each network dies before the next one is made, which may then stand at its address. Their last biases differ by
    a step's length (log2), so that each proposes other steps than the one before."""
    from ballasim_b200.engine import Engine
    from ballasim_b200.learned import StepMLP
    from ballasim_b200.sensor import SensorModel

    r, got = W.Rules(), []
    for graph in (True, False):
        m = SensorModel(resolve("ideal", {**W.MISMATCH, **W.NOISE}), 48, 32, 5, [{"type": "constant"}], 0)
        eng = Engine([(m, F.blobs(48, 32, 5, 6))], tol=r.tol, dark=r.dark, min_dt_ns=r.min_dt_ns,
                     max_refine_levels=r.max_refine_levels, l_min=r.l_min, l_max=r.l_max)
        eng.set_graph(graph)
        eng.start(0)
        rows = []
        for seed in range(6):
            eng.set_proposal(None)
            net = StepMLP(seed=seed)
            net.params = np.append(net.params[:-1], np.float32(seed + 6))
            eng.set_proposal(net, margin=0.0)
            del net
            eng.start(0)
            rows.append((eng.run(5), m.take_events(with_pixel=True)["t_cross_ns"].tobytes(), m.save_state()))
        got.append(rows)
    assert got[0] == got[1]
    assert len({samples for (samples, _), _, _ in got[1]}) > 1  # the networks do propose other steps
