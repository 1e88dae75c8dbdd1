"""Moment tables kept between maps: a table is read again only while it holds what its side's key names.
A graph replay (zcb_sweep_stack) rewrites the map buffers without running the engine's own map code, so
everything known of them is forgotten, the tables as well as the spectra."""
import numpy as np
import pytest

import zcmir_b200 as zc
from zcmir_b200 import synth

pytestmark = pytest.mark.gpu

T = lambda x, y: np.array([[1, 0, x], [0, 1, y], [0, 0, 1.0]])


def test_tables_after_a_graph_replay_are_the_pairs_own():
    """Sweep and stack captured, a map at a translation, the graph replayed (its last slices' tables are
    now in the buffers), a map at a turned pose in the same frame (it refills the fixed side's spectra
    and reads no table of that side), then the translation again: the same map, value for value."""
    rng = np.random.default_rng(3)
    big = synth.blob_field(320, 320, rng)
    f = big[20:276, 20:276].astype(np.float32)
    m = (1.0 - big[50:240, 60:260] ** 2).astype(np.float32)  # 200 × 190, inside the fixed image
    slices = [np.ascontiguousarray(big[a:a + 264, a:a + 260], np.float32) for a in (0, 20, 41)]
    H = T(35, 25)
    c, s = np.cos(0.02), np.sin(0.02)
    turned = T(140, 120) @ np.array([[c, -s, 0], [s, c, 0], [0, 0, 1.0]]) @ T(-140, -120) @ H
    at = dict(exact=True, calibrated=False, cap=1024)
    with zc.Engine(half=False, sw_nth=36, sw_ns=3, sw_grid=64) as reg:
        reg.set_images(m, f, preprocess=False)
        reg.stack_load(slices, exact=True, calibrated=False, cap=1024)
        reg.sweep_stack(n_peak=4)
        first = reg.shift_map(H, **at)
        reg.sweep_stack(n_peak=4)
        turn = reg.shift_map(turned, **at)
        assert turn.canvas == first.canvas == (256, 256) and turn.offset == first.offset
        again = reg.shift_map(H, **at)
    with zc.Engine(half=False) as reg:
        reg.set_images(m, f, preprocess=False)
        fresh = reg.shift_map(H, **at)
    np.testing.assert_array_equal(first.map, fresh.map)
    np.testing.assert_array_equal(again.map, fresh.map)
    assert (again.peak, again.peak_index, again.zero) == (fresh.peak, fresh.peak_index, fresh.zero)
