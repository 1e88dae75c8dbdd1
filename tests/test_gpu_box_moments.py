"""Shift maps whose moment sums come from summed-area tables (grids of whole pixels: the fixed
image's box at any pose, the moving image's too at translations) against the float64 oracle.

The bounds are the shift-map tests': the same argmax, the peak within 1e-4, cells with at least 20 %
of the largest overlap within 1e-4 of the peak and the others within 1e-2; a cell that only one side
zeroes has under 20 % of the largest overlap (on the 8 % floor, or a covariance of so few pixels that
its smallest pivot is float32 round-off). Sizes run over the tables' tile edges
(32 columns, 8 rows): below one tile, a whole one, one more and one less; boxes inside, beside and
across each other; and whole- and half-pixel translations, at which the moving weight is still 1."""
import numpy as np
import pytest

import zcmir_b200 as zc
from oracle import smi_oracle as O
from zcmir_b200 import synth

pytestmark = pytest.mark.gpu

T = lambda x, y: np.array([[1, 0, x], [0, 1, y], [0, 0, 1.0]])


def turn(deg, w, h):
    c, s = np.cos(np.deg2rad(deg)), np.sin(np.deg2rad(deg))
    return T((w + 1) / 2, (h + 1) / 2) @ np.array([[c, -s, 0], [s, c, 0], [0, 0, 1.0]]) @ T(-(w + 1) / 2, -(h + 1) / 2)


CASES = [
    ((32, 24), (32, 24), T(0, 0)), ((31, 23), (33, 25), T(1, 1)), ((64, 40), (65, 41), T(0, 0)),
    ((97, 33), (64, 64), T(-20, 11)), ((60, 70), (131, 129), T(35, 20)), ((131, 129), (60, 70), T(-30, -25)),
    ((70, 64), (64, 70), T(2.5, -3.5)), ((64, 64), (64, 64), T(50, -45)), ((90, 66), (80, 75), turn(7.0, 80, 75)),
    ((45, 91), (88, 52), turn(-31.0, 88, 52)),
]


@pytest.mark.parametrize("mode", ["laplacian", "three", "cubic"])
@pytest.mark.parametrize("k", range(len(CASES)))
def test_tabled_moments_match_the_oracle(k, mode):
    (mw, mh), (fw, fh), H = CASES[k]
    rng = np.random.default_rng(k)
    big = synth.blob_field(160, 160, rng, n_blobs=200, sigma=(2.0, 8.0))
    f = big[8:8 + fh, 8:8 + fw].astype(np.float32)
    m = (1.0 - big[5:5 + mh, 12:12 + mw] ** 2 + 0.02 * rng.standard_normal((mh, mw))).astype(np.float32)
    with zc.Engine(half=False, smi_features=mode) as reg:
        reg.set_images(m, f, preprocess=False)
        pa, pb = ({"w": x.shape[2], "h": x.shape[1], "mode": mode, "feat": x, "acf": O.acf(x),
                   "stack": np.concatenate([np.ones((1,) + x.shape[1:], np.float32), x])} for x in (reg.features(0), reg.features(1)))
        sm = reg.shift_map(H, exact=True, calibrated=False, cap=2048)
        cal = reg.shift_map(H, exact=True, calibrated=True, cap=2048)
    ref = O.shift_map(pa, pb, H, exact=True, calibrated=False, cap=2048, return_corr=True)
    rc = O.shift_map(pa, pb, H, exact=True, calibrated=True, cap=2048)
    n, err = ref["corr"][0], np.abs(sm.map.astype(np.float64) - ref["map"]) / abs(ref["peak"])
    differ = (sm.map == 0) != (ref["map"] == 0)
    assert sm.map.shape == ref["map"].shape and sm.peak_index == ref["peak_index"]
    assert abs(sm.peak - ref["peak"]) <= 1e-4 * abs(ref["peak"])
    assert np.all(n[differ] < 0.2 * n.max())
    assert err[(n >= 0.2 * n.max()) & ~differ].max() <= 1e-4
    assert err[~differ].max() <= 1e-2
    big_n = n >= 0.2 * n.max()
    assert np.max(np.abs(cal.map - rc["map"])[big_n]) <= 1e-4 * max(abs(rc["peak"]), 1e-30)
