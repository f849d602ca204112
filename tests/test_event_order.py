"""The device's event order (t_cross, pixel) at the sizes where its sort changes form, against NumPy's lexsort: short
lists in one block, longer ones of unknown times in two radix passes (foreign device records), a model's own in one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RAW = np.dtype([("pixel", "<u4"), ("p", "u1"), ("label", "u1"), ("flags", "<u2"), ("t", "<i8"), ("ds", "<f4"),
                ("dn", "<f4"), ("dl", "<f4"), ("l_first", "<f4")])


@pytest.mark.parametrize("n", [1, 2, 3, 63, 64, 65, 1000, 2047, 2048, 2049, 5000])
def test_foreign_records(cuda_lib, n):
    import torch

    from ballasim_b200 import _lib
    from ballasim_b200.params import resolve
    from ballasim_b200.sensor import SensorModel

    rng = np.random.default_rng(n)
    w, h = 640, 480
    rec = np.zeros(n, RAW)
    rec["t"] = rng.integers(-50, 50, n) * 10**17 // 10  # many equal times, both signs, a span of 59 bits
    rec["pixel"] = rng.permutation(w * h)[:n]
    rec["p"], rec["label"], rec["flags"] = rng.integers(0, 2, n), rng.integers(0, 3, n), rng.integers(0, 4096, n)
    for k in ("ds", "dn", "dl", "l_first"):
        rec[k] = rng.normal(size=n)
    dev = torch.from_numpy(rec.view(np.uint8).copy()).cuda()
    m = SensorModel(resolve("ideal", {}), w, h, 1, [{"type": "constant"}], 0)
    torch.cuda.synchronize()  # the model reads on its own stream
    got = m.download_events(_lib.DeviceEvents(dev.data_ptr(), n), with_pixel=True)
    want = rec[np.lexsort((rec["pixel"], rec["t"]))]
    assert np.array_equal(got["pixel"], want["pixel"]) and np.array_equal(got["t_cross_ns"], want["t"])
    assert np.array_equal(got["x"], want["pixel"] % w) and np.array_equal(got["y"], want["pixel"] // w)
    for k in ("p", "label", "flags", "ds", "dn", "dl", "l_first"):
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("windows", [1, 12])
def test_a_call_s_own_events(cuda_lib, windows):
    """Taken from the model (one radix sort over the call's span, or the short form) and downloaded through a copy of
    its device records (nothing known of them): the same columns."""
    import torch

    from ballasim_b200 import _lib
    from ballasim_b200 import workloads as W
    from ballasim_b200.params import resolve
    from ballasim_b200.sensor import SensorModel
    from ballasim_b200.windows import DeviceWindows

    spec = W.small("noise", 120, 90, windows).sensors[0]
    m = SensorModel(resolve("ideal", {**spec.overrides, "noise_ba_median_hz": 20.0}), 120, 90, 7,
                    [{"type": "constant"}], 0)
    dw = DeviceWindows([(m, spec.field)])
    dw.start(1 << 40)
    seen = []

    def check(_i, model, ev):
        own = model.download_events(ev, with_pixel=True)
        n = int(ev.count)
        copy = torch.empty(32 * max(1, n), dtype=torch.uint8, device="cuda")
        if n:
            torch.cuda.synchronize()
            src = torch.as_tensor(_Raw(ev.data, 32 * n), device="cuda")
            copy[:32 * n].copy_(src)
            torch.cuda.synchronize()
        other = model.download_events(_lib.DeviceEvents(copy.data_ptr(), n), with_pixel=True)
        for k in own:
            assert np.array_equal(own[k], other[k]), k
        seen.append(n)

    dw.run(windows, on_events=check)
    assert sum(seen) > 100


class _Raw:
    """Device bytes at an address, as torch takes them."""

    def __init__(self, ptr: int, nbytes: int):
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (int(ptr), False), "version": 3}
