"""Translation maps of a small image over a large one, and of images with flat halves, ramps and steps: their
moment sums cancel from tables whose entries sum a whole plane, over covariances that are near singular. The
map's peak is the float64 oracle's cell, within 1e-4 of its value, as for any other pair. The same at turned
poses, whose overlap is a transform's sum: the moments are exact, and dividing them by a sum with a
transform's error leaves a flat part with a covariance of that error times its mean squared (there the cell
alone is held: scores so close to singular keep 1e-4 in no float32 transform)."""
import math

import numpy as np
import pytest

import zcmir_b200 as zc
from oracle import smi_oracle as O
from zcmir_b200 import synth

pytestmark = pytest.mark.gpu


def image(rng, h, w, kind):
    f = synth.blob_field(max(h, 64) + 8, max(w, 64) + 8, rng)[:h, :w]
    x = np.arange(w)[None] / max(w - 1, 1)
    f = {"ramp": 0.4 * f + 0.6 * x, "step": 0.4 * f + 0.6 * (x > 0.5), "half": np.where(x < 0.5, f, 0.25)}[kind]
    return np.ascontiguousarray(f, np.float32)


def peaks(mw, mh, fw, fh, kind, mode, seed, H, calibrated=False):
    rng = np.random.default_rng(seed)
    m, f = image(rng, mh, mw, kind), image(rng, fh, fw, kind)
    with zc.Engine(half=False, smi_features=mode) as reg:
        reg.set_images(m, f, preprocess=False)
        pa, pb = ({"w": x.shape[2], "h": x.shape[1], "mode": mode, "feat": x, "acf": O.acf(x),
                   "stack": np.concatenate([np.ones((1,) + x.shape[1:], np.float32), x])} for x in (reg.features(0), reg.features(1)))
        sm = reg.shift_map(H, exact=True, calibrated=calibrated, cap=2048)
    ref = O.shift_map(pa, pb, H, exact=True, calibrated=calibrated, cap=2048)
    assert sm.map.shape == ref["map"].shape
    return sm, ref


T = lambda x, y: np.array([[1, 0, x], [0, 1, y], [0, 0, 1.0]])


@pytest.mark.parametrize("mw,mh,fw,fh,kind,mode,seed", [
    (8, 9, 118, 73, "ramp", "laplacian", 77031), (66, 10, 40, 108, "step", "laplacian", 77159),
    (39, 12, 17, 35, "half", "cubic", 77164), (21, 54, 172, 309, "ramp", "laplacian", 77175),
    (42, 15, 310, 166, "step", "laplacian", 77255),
])
def test_the_peak_is_the_oracles(mw, mh, fw, fh, kind, mode, seed):
    sm, ref = peaks(mw, mh, fw, fh, kind, mode, seed, T((fw - mw) // 2, (fh - mh) // 2))
    assert sm.peak_index == ref["peak_index"]
    assert abs(sm.peak - ref["peak"]) <= 1e-4 * abs(ref["peak"])


@pytest.mark.parametrize("mw,mh,fw,fh,kind,mode,cal,deg,scale,seed", [
    (23, 11, 21, 11, "half", "cubic", False, 31.920643042480606, 1.063623676183559, 77044),
    (193, 27, 20, 159, "ramp", "three", False, -36.29954584778869, 0.9264467620867614, 77067),
    (335, 290, 147, 63, "half", "cubic", True, -4.542457536365696, 1.0348408156781983, 77206),
    (40, 18, 8, 413, "ramp", "three", False, -0.823287183861801, 0.9760298781751318, 77211),
    (158, 64, 13, 21, "step", "laplacian", False, -2.3422982112263853, 1.0873577712876905, 77231),
])
def test_the_peak_is_the_oracles_when_turned(mw, mh, fw, fh, kind, mode, cal, deg, scale, seed):
    a, c = math.radians(deg), ((fw + 1) / 2, (fh + 1) / 2)
    R = np.array([[scale * math.cos(a), -scale * math.sin(a), 0], [scale * math.sin(a), scale * math.cos(a), 0], [0, 0, 1.0]])
    sm, ref = peaks(mw, mh, fw, fh, kind, mode, seed, T(*c) @ R @ T(-c[0], -c[1]) @ T((fw - mw) / 2, (fh - mh) / 2), cal)
    assert sm.peak_index == ref["peak_index"]
