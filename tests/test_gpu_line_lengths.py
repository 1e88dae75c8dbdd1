"""Shift maps at every FFT line length with a compile-time schedule (and some without), as rows of a
wide pair and as columns of a tall one, against the float64 oracle on the GPU's own features.

The bounds are the shift-map tests': the same argmax, the peak within 1e-4, cells with at least 20 %
of the largest overlap within 1e-4 of the peak and the others within 1e-2 (float32 FFT round-off,
which grows with log2 of the length and where the overlap is small); cells that one side zeroes and
the other does not lie within 1 % of the 8 % overlap floor."""
import numpy as np
import pytest

import zcmir_b200 as zc
from oracle import smi_oracle as O
from zcmir_b200 import synth

pytestmark = pytest.mark.gpu

LADDER = sorted(2 ** a * 3 ** b for a in range(14) for b in range(9) if 48 <= 2 ** a * 3 ** b <= 8192)


def pair(w, h, seed):
    """A field and its inverted remap, the moving image showing it 5 px right and 2 px up."""
    scale = max(w, h) / 256.0
    big = synth.blob_field(h + 16, w + 16, np.random.default_rng(seed), n_blobs=64 / max(scale, 1.0), sigma=(2.0, 8.0))
    rng = np.random.default_rng(seed + 1)
    moving = 1.0 - big[6:6 + h, 13:13 + w] ** 2 + 0.02 * rng.standard_normal((h, w))
    return moving.astype(np.float32), big[8:8 + h, 8:8 + w].astype(np.float32)


@pytest.mark.parametrize("mode", ["laplacian", "three"])
@pytest.mark.parametrize("length", LADDER)
def test_map_of_each_line_length(monkeypatch, length, mode):
    # the oracle's plan stops at 2048 points, the reference's longest line; this build's at 8192
    monkeypatch.setattr(O, "map_plan", lambda w, h, cap=0, sizes="ladder": O.linear_corr_plan_rect(w, h, cap, sizes))
    side, thin = (length + 1) // 2, 22
    tall = length % 4 == 0 if mode == "laplacian" else length % 4 != 0
    w, h = (thin, side) if tall else (side, thin)
    m, f = pair(w, h, length)
    with zc.Engine(half=False, smi_features=mode) as reg:
        reg.set_images(m, f, preprocess=False)
        pa, pb = ({"w": w, "h": h, "mode": mode, "feat": x, "acf": O.acf(x),
                   "stack": np.concatenate([np.ones((1, h, w), np.float32), x])} for x in (reg.features(0), reg.features(1)))
        sm = reg.shift_map(np.eye(3), exact=True, calibrated=False, cap=8192)
    ref = O.shift_map(pa, pb, np.eye(3), exact=True, calibrated=False, cap=8192, return_corr=True)
    assert length in sm.map.shape and sm.map.shape == ref["map"].shape
    assert sm.peak_index == ref["peak_index"] and abs(sm.peak - ref["peak"]) <= 1e-4 * abs(ref["peak"])
    n, err = ref["corr"][0], np.abs(sm.map.astype(np.float64) - ref["map"]) / abs(ref["peak"])
    differ = (sm.map == 0) != (ref["map"] == 0)
    assert np.all(np.abs(n[differ] - 0.08 * n[0, 0]) <= 0.01 * 0.08 * n[0, 0])
    assert err[(n >= 0.2 * n.max()) & ~differ].max() <= 1e-4
    assert err[~differ].max() <= 1e-2
