"""What the event-camera path is timed on: calls that programs using this package make, through its public entry
points, from one window of a small array to a rig of large sensors.

A case is a dict of plain values. ``kind`` picks the entry points:

- ``engine``: the fused engine (engine.Engine): the sensors' first frames from pinned host memory in, ``calls`` runs
  of ``windows`` windows each, every run's events out into the program's recording (bs_engine_take_events).
  ``photo`` picks the photoreceptor (the instantaneous response, the cascade, the cascade with its noise lattice),
  ``law`` the comparator's rows, ``tuned`` whether the program has run the autotuner once.
- ``runs``: the two-kernel route with the sample runs in device memory (windows.DeviceWindows), every window's events
  downloaded into the recording as they come (bs_model_download_events).
- ``host``: the host-array interface: per window sampling.sample_window, then SensorModel.advance on its runs.
- ``learned``: the engine sampling with a trained step proposal (learned.StepMLP).
- ``train``: training that proposal on traced pairs.
- ``sink``: writing an event file (export.RawWriter / DatWriter) from host columns.

A recording is a set of host event columns of a fixed capacity, kept from pass to pass as a recorder keeps its
buffers, with the number of events in it.

Frame sizes, comparator laws, fields, densities and sampler rules are those of workloads.py; a duration is a number of
8.389 ms windows. ``draw`` gives more cases of the same ranges.
"""
from __future__ import annotations

import ctypes as C
import dataclasses
import math
import os
import tempfile

import numpy as np
import torch

from ballasim_b200 import _lib
from ballasim_b200 import fields as F
from ballasim_b200 import workloads as W
from ballasim_b200.engine import Engine
from ballasim_b200.export import DatWriter, RawWriter
from ballasim_b200.learned import StepMLP, trace_pairs
from ballasim_b200.params import resolve
from ballasim_b200.sampling import MidpointTest, field_frame, field_levels, sample_window
from ballasim_b200.sensor import EVENT_COLUMNS, SensorModel, column_struct
from ballasim_b200.windows import DeviceWindows, carried_samples

WINDOW_NS = W.WINDOW_NS
RULES = W.Rules()
LAWS = {"ideal": W.IDEAL, "mismatch": W.MISMATCH, "noise": {**W.MISMATCH, **W.NOISE}}
LIGHT = [{"type": "constant"}]
TRAIN_BATCH, TRAIN_LR, TRAIN_TAU = 8192, 1e-3, 0.25


def listed() -> list[dict]:
    return [
        # A live viewer of a small array: the events of each window fetched before the next one is asked for.
        {"name": "edge_64x48_live", "kind": "engine", "sensors": "64x48", "blobs": 0, "law": "ideal",
         "photo": "instant", "windows": 1, "calls": 5, "tuned": False},
        # A batch run of one DAVIS-sized sensor (2.0 s), after the program's autotune.
        {"name": "blobs_346x260", "kind": "engine", "sensors": "346x260", "blobs": 16, "law": "mismatch",
         "photo": "instant", "windows": 239, "calls": 1, "tuned": True},
        # A short run of an odd-sized crop with every noise source on, at the engine's own launch shape.
        {"name": "odd_333x187_noise", "kind": "engine", "sensors": "333x187", "blobs": 31, "law": "noise",
         "photo": "instant", "windows": 37, "calls": 1, "tuned": False},
        # A batch run of one HD sensor with every noise source on (0.5 s).
        {"name": "blobs_1280x720_noise", "kind": "engine", "sensors": "1280x720", "blobs": 256, "law": "noise",
         "photo": "instant", "windows": 60, "calls": 1, "tuned": True},
        # A rig of five sensors in one launch, from a DAVIS to a full-HD one (0.5 s): the largest call.
        {"name": "rig_5_noise", "kind": "engine", "sensors": "346x260,640x480,1280x720,1280x720,1920x1080",
         "blobs": 128, "law": "noise", "photo": "instant", "windows": 60, "calls": 1, "tuned": True},
        # The cascade photoreceptor, its noise lattice off.
        {"name": "cascade_346x260", "kind": "engine", "sensors": "346x260", "blobs": 16, "law": "mismatch",
         "photo": "cascade", "windows": 60, "calls": 1, "tuned": False},
        # The full photoreceptor model with its noise lattice.
        {"name": "lattice_346x260", "kind": "engine", "sensors": "346x260", "blobs": 16, "law": "mismatch",
         "photo": "lattice", "windows": 8, "calls": 1, "tuned": False},
        # An engine of one's own around the device boundary: three sensors, runs in device memory, each window's
        # events downloaded.
        {"name": "runs_3_noise", "kind": "runs", "sensors": "346x260,640x480,1280x720", "blobs": 128, "law": "noise",
         "windows": 12},
        # A simulation loop that keeps its runs on the host.
        {"name": "host_346x260", "kind": "host", "sensors": "346x260", "blobs": 16, "law": "mismatch", "windows": 3},
        # A run sampled by a trained step proposal.
        {"name": "learned_640x360", "kind": "learned", "sensors": "640x360", "blobs": 64, "law": "noise",
         "windows": 30},
        # Part of training the step proposal.
        {"name": "train_512", "kind": "train", "sensors": "320x180", "blobs": 16, "law": "noise", "windows": 24,
         "steps": 512},
        # Writing the events of a busy HD sensor as an EVT 3.0 file.
        {"name": "sink_evt3_4Mi", "kind": "sink", "format": "evt3", "events": 4 << 20, "sensors": "1280x720"},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _frame_size(rng, px_hi: int) -> tuple[int, int]:
    """A frame of about 4:3 to 16:9 with 3,072 to px_hi pixels, odd sizes among them; one in four a stock size."""
    stock = [s for s in ((64, 48), (320, 180), (346, 260), (640, 480), (1280, 720), (1920, 1080))
             if s[0] * s[1] <= px_hi]
    if rng.random() < 0.25:
        return stock[rng.randrange(len(stock))]
    px = _log_int(rng, 3072, px_hi)
    w = max(48, int(round(math.sqrt(px * rng.uniform(1.3, 1.8)))))
    return w, max(32, px // w)


def _blobs(rng, px: int) -> int:
    """Blobs of the workloads' densities (one per 700 to 16,000 px), at most their 256."""
    return max(3, min(256, int(px * math.exp(rng.uniform(math.log(1 / 16000), math.log(1 / 700))))))


def _windows(rng, px: int, most: int, hi: int) -> int:
    """Windows for px pixels: at most `hi`, at most `most` pixel-windows, at least enough for events to occur."""
    hi = max(1, min(hi, most // px))
    return _log_int(rng, min(hi, max(1, 6000 // px)), hi)


def draw(rng) -> dict:
    kind = rng.choices(["engine", "cascade", "lattice", "runs", "host", "learned", "train", "sink"],
                       [12, 3, 2, 3, 2, 2, 1, 2])[0]
    if kind == "train":
        return {"kind": "train", "sensors": "320x180", "blobs": rng.randint(8, 32), "law": "noise",
                "windows": rng.randint(12, 24), "steps": _log_int(rng, 64, 1024)}
    if kind == "sink":
        w, h = _frame_size(rng, 1280 * 720)
        return {"kind": "sink", "format": rng.choice(["evt2", "evt21", "evt3", "dat"]),
                "events": _log_int(rng, 1 << 16, 4 << 20), "sensors": f"{w}x{h}"}
    if kind == "engine":
        law = rng.choice(["ideal", "mismatch", "noise", "noise"])
        edge = law == "ideal" and rng.random() < 0.5
        sizes = [_frame_size(rng, 1920 * 1080) for _ in range(1 if edge else rng.choice([1, 1, 1, 2, 3]))]
        px = sum(w * h for w, h in sizes)
        windows = _windows(rng, px, 150_000_000, 239)
        live = len(sizes) == 1 and windows <= 8
        return {"kind": "engine", "sensors": ",".join(f"{w}x{h}" for w, h in sizes),
                "blobs": 0 if edge else _blobs(rng, min(w * h for w, h in sizes)), "law": law, "photo": "instant",
                "windows": windows, "calls": rng.randint(1, 5) if live else 1, "tuned": rng.random() < 0.5}
    if kind in ("cascade", "lattice"):
        w, h = _frame_size(rng, 640 * 480)
        most, hi = (10_000_000, 120) if kind == "cascade" else (720_000, 12)
        return {"kind": "engine", "sensors": f"{w}x{h}", "blobs": _blobs(rng, w * h), "law": "mismatch",
                "photo": kind, "windows": _windows(rng, w * h, most, hi), "calls": 1, "tuned": rng.random() < 0.3}
    law = rng.choice(["mismatch", "noise"])
    if kind == "runs":
        sizes = [_frame_size(rng, 1280 * 720) for _ in range(rng.randint(1, 4))]
        px = sum(w * h for w, h in sizes)
        return {"kind": "runs", "sensors": ",".join(f"{w}x{h}" for w, h in sizes), "blobs": _blobs(rng, min(w * h for w, h in sizes)),
                "law": law, "windows": _windows(rng, px, 20_000_000, 40)}
    w, h = _frame_size(rng, 346 * 260 if kind == "host" else 640 * 480)
    if kind == "host":
        return {"kind": "host", "sensors": f"{w}x{h}", "blobs": _blobs(rng, w * h), "law": law,
                "windows": rng.randint(1, 4)}
    return {"kind": "learned", "sensors": f"{w}x{h}", "blobs": _blobs(rng, w * h), "law": "noise",
            "windows": _windows(rng, w * h, 8_000_000, 60)}


# ---- inputs ----

def _sizes(case: dict) -> list[tuple[int, int]]:
    return [tuple(int(v) for v in s.split("x")) for s in case["sensors"].split(",")]


def _edge(w: int, h: int, seed: int) -> F.Field:
    """workloads.edge_64x48's edge, placed so that it starts on a seeded point of the array's middle half (most
    seeds' edges miss a small array)."""
    f = F.tanh_edge(w, h, seed)
    g = F.SplitMix64(seed + 1)
    c = f.nx * w * (0.25 + 0.5 * g.uniform()) + f.ny * h * (0.25 + 0.5 * g.uniform())
    return dataclasses.replace(f, c=float(np.float32(c)))


def _sensors(case: dict, seed: int) -> list[tuple[SensorModel, F.Field]]:
    """The case's sensors with their fields; with several sensors each has its own threshold, as a rig has."""
    g = F.SplitMix64(seed)
    preset = "ideal" if case.get("photo", "instant") == "instant" else "prophesee_gen3"
    out = []
    for cam, (w, h) in enumerate(_sizes(case)):
        rows = dict(LAWS[case["law"]])
        if cam > 0:
            th = 0.15 + 0.15 * g.uniform()
            rows.update(theta_on=th, theta_off=th)
        if preset != "ideal":
            rows["noise"] = case["photo"] == "lattice"
        s = seed * 100 + cam
        f = F.blobs(w, h, s, case["blobs"]) if case["blobs"] else _edge(w, h, s)
        out.append((SensorModel(resolve(preset, rows), w, h, s, LIGHT, cam), f))
    return out


def _pinned_frames(sensors) -> list[np.ndarray]:
    return [torch.from_numpy(field_frame(f, 0)).pin_memory().numpy() for _, f in sensors]


def _engine(sensors) -> Engine:
    return Engine(sensors, tol=RULES.tol, dark=RULES.dark, min_dt_ns=RULES.min_dt_ns,
                  max_refine_levels=RULES.max_refine_levels, l_min=RULES.l_min, l_max=RULES.l_max)


def _pairs(case: dict, seed: int):
    """Training pairs traced on a field of the case's frame size and blob density."""
    w, h = _sizes(case)[0]
    f = F.blobs(w, h, seed * 100 + 50, case["blobs"])
    return trace_pairs(f, RULES, case["windows"], stride=2 if case["kind"] == "train" else 4)[:2]


def _capacity(case: dict, w: int, h: int) -> int:
    """Room for a sensor's events: several times what the workloads' fields of the case's blob density give."""
    per_window = 0.03 + 300.0 * case["blobs"] / (w * h) + (0.6 if case.get("photo") == "lattice" else 0.0)
    return int(w * h * (1.0 + per_window * case["windows"] * case.get("calls", 1)))


class Recording:
    def __init__(self, capacity: int):
        self.columns = {name: np.zeros(capacity, dtype) for name, dtype in EVENT_COLUMNS}
        self.count = 0

    def room(self, n: int):
        """The C columns of the next n events, which then count as recorded."""
        at, self.count = self.count, self.count + n
        if self.count > len(self.columns["x"]):
            raise MemoryError("the recording is full")
        return column_struct({k: v[at:at + n] for k, v in self.columns.items()})

    def output(self) -> dict:
        return {**self.columns, "count": self.count}


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "train":
        x, y = _pairs(case, seed)
        net = StepMLP(seed)
        return {"case": case, "x": x, "y": y, "net": net, "p0": net.params, "seed": seed}
    if kind == "sink":
        w, h = _sizes(case)[0]
        ev = W.event_stream(case["events"], w, h, seed=seed)
        folder = tempfile.TemporaryDirectory(prefix="events_")
        return {"case": case, "ev": ev, "folder": folder, "path": os.path.join(folder.name, "cam0.raw")}
    sensors = _sensors(case, seed)
    st = {"case": case, "sensors": sensors, "frames": _pinned_frames(sensors),
          "recordings": [Recording(_capacity(case, m.width, m.height)) for m, _ in sensors]}
    if kind == "runs":
        st["windows"] = DeviceWindows(sensors, tol=RULES.tol, dark=RULES.dark, min_dt_ns=RULES.min_dt_ns,
                                      max_refine_levels=RULES.max_refine_levels, l_min=RULES.l_min,
                                      l_max=RULES.l_max)
    elif kind == "host":
        n = sensors[0][0].width * sensors[0][0].height
        st["ids"] = np.arange(n, dtype=np.uint32)
        st["test"] = MidpointTest(RULES.tol, RULES.dark, [1.0], [1.0])
    else:
        st["engine"] = _engine(sensors)
        if kind == "learned":
            x, y = _pairs({**case, "sensors": "320x180", "blobs": 16, "windows": 12}, seed)
            st["net"] = StepMLP(seed)
            st["net"].train(x, y, steps=600, batch=TRAIN_BATCH, lr=TRAIN_LR, seed=seed, tau=TRAIN_TAU)
            st["engine"].set_proposal(st["net"], 0.25)
        elif case["tuned"]:
            st["engine"].start(0)
            st["engine"].autotune(windows=4)
    return st


# ---- one pass ----

def _outputs(st: dict) -> list[dict]:
    return [r.output() for r in st["recordings"]]


def _run_engine(st: dict):
    eng, case, recs = st["engine"], st["case"], st["recordings"]
    for r in recs:
        r.count = 0
    eng.start(0, frames=st["frames"])
    for _ in range(case.get("calls", 1)):
        eng.run(case["windows"])
        columns = (_lib.EventColumns * len(recs))()
        for i, (m, _) in enumerate(st["sensors"]):
            n = C.c_size_t()
            _lib.check(_lib.lib().bs_model_event_count(m.handle, C.byref(n)))
            columns[i] = recs[i].room(n.value)
        _lib.check(_lib.lib().bs_engine_take_events(eng._h, columns))
    return _outputs(st)


def _run_windows(st: dict):
    dw, recs = st["windows"], st["recordings"]
    for r in recs:
        r.count = 0

    def record(i, m, ev):
        columns = recs[i].room(int(ev.count))
        _lib.check(_lib.lib().bs_model_download_events(m.handle, C.byref(ev), C.byref(columns)))

    dw.start(0, frames=st["frames"])
    dw.run(st["case"]["windows"], on_events=record)
    return _outputs(st), [carried_samples(dw, i) for i in range(len(recs))]


def _run_host(st: dict):
    (model, f), ids, rec = st["sensors"][0], st["ids"], st["recordings"][0]
    irr = st["frames"][0].reshape(-1, 1)
    sig = np.zeros(len(ids), np.uint64)
    rec.count = 0
    model.init(0, irr)
    for k in range(st["case"]["windows"]):
        t_w = k * WINDOW_NS
        runs = sample_window(t_w, ids, field_levels(f, t_w, RULES.l_min, RULES.l_max), ids, irr, sig, f,
                             refine_signature=True, midpoint=st["test"], max_refine_levels=RULES.max_refine_levels,
                             min_dt_ns=RULES.min_dt_ns)
        events = model.advance(runs.pixel_ids, runs.t_ns, runs.irradiance, t_w + WINDOW_NS, offsets=runs.offsets)
        irr, sig = runs.last_irradiance, runs.last_signature
        at = rec.count
        rec.room(len(events["x"]))
        for name, column in rec.columns.items():
            column[at:rec.count] = events[name]
    return {"events": rec.output(), "carried": irr, "offsets": runs.offsets}


def _run_train(st: dict):
    net = st["net"]
    net.params = st["p0"]
    losses = net.train(st["x"], st["y"], steps=st["case"]["steps"], batch=TRAIN_BATCH, lr=TRAIN_LR, seed=st["seed"],
                       tau=TRAIN_TAU)
    return {"losses": losses, "params": net.params}


def _run_sink(st: dict):
    ev, fmt = st["ev"], st["case"]["format"]
    if fmt == "dat":
        writer = DatWriter(st["path"], ev.width, ev.height, 0, 0)
    else:
        writer = RawWriter(st["path"], fmt, ev.width, ev.height, 0, 0)
    writer.append(ev.x, ev.y, ev.p, ev.t_ns)
    info = writer.close()
    # The file is the output: mapped, after a sparse tail that brings it to the same length for every stream.
    room = 4096 + 9 * len(ev.t_ns)
    os.truncate(st["path"], room)
    return {"file": np.memmap(st["path"], np.uint8, "r", shape=(room,)), "bytes": info["bytes"]}


_RUN = {"engine": _run_engine, "learned": _run_engine, "runs": _run_windows, "host": _run_host, "train": _run_train,
        "sink": _run_sink}


def run(st: dict):
    return _RUN[st["case"]["kind"]](st)


# ---- what a pass cannot do without ----

EVENTS_PER_PX_WINDOW = 0.017  # the six-sensor and 346x260 workloads' event rate
SAMPLES_PER_PX_WINDOW = 4.0   # and their pixel-samples
EVENT_BYTES = 40              # one event's host columns
MODEL_BYTES = 4 + 40 + 2 * 72  # a pixel's first frame, its map, its state in and out
# Operations of one pixel-sample: a field evaluation over the one or two blobs in reach (an exp each), the midpoint
# test, the log and the two comparator bounds.
SAMPLE_FLOPS = 100
CELL_FLOPS = 150              # one noise-lattice cell: the draw, the tables, the step and the hull
MLP_FLOPS = 2 * (16 * 64 + 64 * 64 + 64)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "train":
        rows = case["steps"] * TRAIN_BATCH
        return {"bytes": rows * 36.0, "flops": 3.0 * rows * MLP_FLOPS}
    if kind == "sink":
        return {"bytes": case["events"] * (13 + {"evt2": 4, "evt21": 2.3, "evt3": 2.5, "dat": 8}[case["format"]]),
                "flops": 0.0}
    px = sum(w * h for w, h in _sizes(case))
    pw = px * case["windows"] * case.get("calls", 1)
    samples = SAMPLES_PER_PX_WINDOW * pw
    out = {"bytes": px * MODEL_BYTES + pw * EVENTS_PER_PX_WINDOW * EVENT_BYTES, "flops": samples * SAMPLE_FLOPS}
    if kind == "host":
        out["bytes"] += 2 * 12 * samples  # the runs out to the host and back in
    elif kind == "learned":
        out["flops"] += pw * 2 * MLP_FLOPS
    elif case.get("photo") == "lattice":
        out["flops"] += pw * 128 * CELL_FLOPS
    return out


# ---- 64-bit values ----

def _batch_rows(seed: int, step: int, n: int) -> np.ndarray:
    """The rows of training step `step`: two words of Philox4x32-10 under the batch stream's counter layout."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [np.full(TRAIN_BATCH, 0x0091 << 8, np.uint64), np.arange(TRAIN_BATCH, dtype=np.uint64),
         np.full(TRAIN_BATCH, step, np.uint64), np.zeros(TRAIN_BATCH, np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32,
             (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return ((c[0] << np.uint64(32)) | c[1]) % np.uint64(n)


def exact(case: dict, seed: int):
    """Training in 64 bits: the same batches and Adam steps, no operand rounded. The other kinds return what a
    bit-exact integer-time comparator or a file format defines, or columns whose length it decides: no 64-bit value."""
    if case["kind"] != "train":
        return None
    st = prepare(case, seed)
    dev = st["x"].device
    x = (st["x"].view(torch.int16).to(torch.int32) << 16).view(torch.float32).double()
    target = st["y"].double()
    shapes = ((16, 64), (64,), (64, 64), (64,), (64,), ())
    flat = torch.from_numpy(st["p0"]).to(dev).double()
    m, v, losses = torch.zeros_like(flat), torch.zeros_like(flat), []
    for s in range(case["steps"]):
        rows = torch.from_numpy(_batch_rows(st["seed"], s, len(target)).astype(np.int64)).to(dev)
        flat.requires_grad_(True)
        w1, b1, w2, b2, w3, b3 = (t.reshape(sh) for t, sh in
                                  zip(flat.split([math.prod(sh) for sh in shapes]), shapes))
        e = torch.relu(torch.relu(x[rows] @ w1 + b1) @ w2 + b2) @ w3 + b3 - target[rows]
        weight = torch.where(e < 0, 2 * TRAIN_TAU, 2 * (1 - TRAIN_TAU))
        loss = (weight * e * e).sum() / (2 * TRAIN_BATCH)
        grad, = torch.autograd.grad(loss, flat)
        losses.append(loss.detach())
        m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
        up = (m / (1 - 0.9 ** (s + 1))) / ((v / (1 - 0.999 ** (s + 1))).sqrt() + 1e-8)
        flat = (flat - TRAIN_LR * up).detach()
    return {"losses": torch.stack(losses).cpu(), "params": flat.cpu()}
