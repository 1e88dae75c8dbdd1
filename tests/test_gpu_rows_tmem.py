"""The fused last pass (sums in tensor memory, scored in the same kernel), which maps with 2048-point rows
and no moment tables take: grids coarser than a pixel, and global whitening.

Against ZCMIR_B200_ROW_PASS=split (the rows pass and the score pass): the same float32 line FFT on the
same spectra, so within 1e-5 of the peak and the same argmax; a cell that only one of the two zeroes sits
on the overlap floor (under one in ten thousand). Against the float64 oracle: the shift-map tests' bounds.
The map read back comes in chunks of rows, the peak alone without them: both agree."""
import numpy as np
import pytest

import zcmir_b200 as zc
from oracle import smi_oracle as O
from zcmir_b200 import synth

pytestmark = pytest.mark.gpu

CASES = [  # side, mode, exact, calibrated
    (1300, "laplacian", True, False), (1300, "laplacian", True, True), (1300, "three", True, False),
    (1300, "three", True, True), (1024, "laplacian", False, False), (1024, "three", False, False),
]


@pytest.mark.parametrize("n,mode,exact,calibrated", CASES)
def test_fused_rows_match_the_two_passes(monkeypatch, n, mode, exact, calibrated):
    m, f, _ = synth.pair_segmented(n=n, seed=4, max_shift=n // 6)
    maps, launches = {}, {}
    for route in ("tmem", "split"):
        monkeypatch.setenv("ZCMIR_B200_ROW_PASS", route)
        with zc.Engine(half=False, smi_features=mode) as reg:
            reg.set_images(m, f, preprocess=False)
            at = dict(exact=exact, calibrated=calibrated, cap=2048)
            maps[route] = reg.shift_map(np.eye(3), **at)
            reg.set_images(m, f, preprocess=False)
            reg.gpu_counts()
            peak = reg.shift_map(np.eye(3), want_map=False, **at)
            launches[route] = reg.gpu_counts()["launches"]
            assert (peak.peak, peak.peak_index, peak.zero) == (maps[route].peak, maps[route].peak_index, maps[route].zero)
    a, b = maps["tmem"], maps["split"]
    assert a.map.shape == b.map.shape and a.map.shape[1] == 2048
    assert launches["split"] == launches["tmem"] + 1  # rows and score apart
    assert a.peak_index == b.peak_index
    floor = (a.map == 0) != (b.map == 0)
    assert floor.mean() < 1e-4
    assert np.max(np.abs(a.map - b.map)[~floor]) <= 1e-5 * abs(a.peak)


@pytest.mark.parametrize("n,mode,exact,calibrated", [CASES[1], CASES[2], CASES[4]])
def test_fused_rows_match_the_oracle(n, mode, exact, calibrated):
    m, f, _ = synth.pair_segmented(n=n, seed=4, max_shift=n // 6)
    with zc.Engine(half=False, smi_features=mode) as reg:
        reg.set_images(m, f, preprocess=False)
        pa, pb = ({"w": x.shape[2], "h": x.shape[1], "mode": mode, "feat": x, "acf": O.acf(x),
                   "stack": np.concatenate([np.ones((1,) + x.shape[1:], np.float32), x])} for x in (reg.features(0), reg.features(1)))
        sm = reg.shift_map(np.eye(3), exact=exact, calibrated=calibrated, cap=2048)
    ref = O.shift_map(pa, pb, np.eye(3), exact=exact, calibrated=calibrated, cap=2048, return_corr=True)
    n0, err = ref["corr"][0], np.abs(sm.map.astype(np.float64) - ref["map"]) / abs(ref["peak"])
    differ = (sm.map == 0) != (ref["map"] == 0)
    assert sm.map.shape == ref["map"].shape and sm.peak_index == ref["peak_index"]
    assert abs(sm.peak - ref["peak"]) <= 1e-4 * abs(ref["peak"])
    assert differ.mean() < 1e-3 and np.all(n0[differ] < 0.2 * n0.max())
    assert err[(n0 >= 0.2 * n0.max()) & ~differ].max() <= 1e-4
