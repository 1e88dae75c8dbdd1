"""Translation maps of a small image over a large one, and of images with flat halves, ramps and steps: their
moment sums cancel from tables whose entries sum a whole plane, over covariances that are near singular. The
map's peak is the float64 oracle's cell, within 1e-4 of its value, as for any other pair."""
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


@pytest.mark.parametrize("mw,mh,fw,fh,kind,mode,seed", [
    (8, 9, 118, 73, "ramp", "laplacian", 77031), (66, 10, 40, 108, "step", "laplacian", 77159),
    (39, 12, 17, 35, "half", "cubic", 77164), (21, 54, 172, 309, "ramp", "laplacian", 77175),
    (42, 15, 310, 166, "step", "laplacian", 77255),
])
def test_the_peak_is_the_oracles(mw, mh, fw, fh, kind, mode, seed):
    rng = np.random.default_rng(seed)
    m, f = image(rng, mh, mw, kind), image(rng, fh, fw, kind)
    H = np.array([[1, 0, (fw - mw) // 2], [0, 1, (fh - mh) // 2], [0, 0, 1.0]])
    with zc.Engine(half=False, smi_features=mode) as reg:
        reg.set_images(m, f, preprocess=False)
        pa, pb = ({"w": x.shape[2], "h": x.shape[1], "mode": mode, "feat": x, "acf": O.acf(x),
                   "stack": np.concatenate([np.ones((1,) + x.shape[1:], np.float32), x])} for x in (reg.features(0), reg.features(1)))
        sm = reg.shift_map(H, exact=True, calibrated=False, cap=2048)
    ref = O.shift_map(pa, pb, H, exact=True, calibrated=False, cap=2048)
    assert sm.map.shape == ref["map"].shape and sm.peak_index == ref["peak_index"]
    assert abs(sm.peak - ref["peak"]) <= 1e-4 * abs(ref["peak"])
