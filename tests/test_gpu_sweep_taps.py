"""The sweep's packed windows at every count of taps per cell side (1 to 6) and at image sides that
are no multiple of the stacks' 4 × 2 tiles, against the CPU oracle.

Tolerance: the sweep tests' own. An oracle lane clear of the others by 1e-3 of its candidate's top
score is found at the same map index, its score within 1e-4 of the top (float32 transforms and taps
against float64); the oracle places the taps in float32, so that none leaves the image on one side
only by its rounding."""
import numpy as np
import pytest

import zcmir_b200 as zc
from oracle import sweep_oracle as S
from test_gpu_sweep import check_lanes, prep_from
from zcmir_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,grid,taps", [
    ((101, 83, 93, 110), 32, {4, 6}), ((130, 97, 97, 131), 32, {5, 6}), ((101, 83, 93, 110), 64, {2, 4, 6}),
    ((130, 97, 97, 131), 64, {3, 5, 6}), ((101, 83, 93, 110), 128, {1, 2, 4}),
])
def test_windows_of_each_tap_count(sizes, grid, taps):
    mw, mh, fw, fh = sizes
    f = synth.blob_field(160, 160, np.random.default_rng(grid)).astype(np.float32)
    m, fx = np.ascontiguousarray(f[:mh, :mw]), np.ascontiguousarray(f[20:20 + fh, 10:10 + fw])
    # scales 0.5, 1, 2: the range's ends must lie on either side of 1
    with zc.Engine(half=False, sw_nth=4, sw_ns=3, sw_smin=0.5, sw_smax=2.0, sw_rot_range=True, sw_rot_lo=-170.0,
                   sw_rot_hi=160.0, sw_grid=grid) as eng:
        eng.set_images(m, fx, preprocess=False)
        pa, pb = prep_from(eng.features(0)), prep_from(eng.features(1))
        sw = eng.sweep(np.eye(3), n_peak=4)
    gv = S.sweep_grid(rot_lo=-170.0, rot_hi=160.0, n_theta=4, n_sigma=3, s_min=0.5, s_max=2.0)
    ref = S.sweep(pa, pb, np.eye(3), gv, G=grid, min_overlap=0.05, f32_positions=True)
    cands, cell = ref["setup"]["cands"], ref["setup"]["cell"]
    assert {c["taps"] for c in cands} == taps and len(cands) == sw.info["candidates"]
    assert abs(sw.info["cell"] - cell) < 1e-12
    assert check_lanes(sw.scores.astype(np.float64), sw.index, ref, len(cands), 4, cell) >= len(cands) // 2
