"""The bench line's whole-map bytes and operations count the transforms and tables that the timed map ran,
so a map that transforms fewer planes and correlations is credited with fewer."""
import numpy as np
import pytest

import bench


def plan(n_real, n_corr):
    return dict(nx=2048, ny=1536, cw=1024, ch=700, canvas_w=1024, canvas_h=700, n_real=n_real, n_corr=n_corr)


# transformed planes of both sides and correlations, tabled sides: exact plans of four and three features
# at any pose on a coarse grid, at a turned pose and at a translation; the global score
@pytest.mark.parametrize("n_real,n_corr,tables", [(30, 45, 0), (20, 32, 1), (10, 18, 2), (20, 28, 0), (14, 20, 1), (8, 11, 2),
                                                  (10, 25, 0), (8, 16, 0)])
def test_a_map_is_credited_with_what_it_transforms(n_real, n_corr, tables):
    p = plan(n_real, n_corr)
    b, f = bench.map_work(p)
    half = p["ny"] * (p["nx"] // 2 + 1) * 8
    assert b == 2 * 5 * 1024 * 700 * 4 + 2 * n_real * half + 2 * tables * 1024 * 700 * (80 if n_corr in (20, 11) else 112) + 2048 * 1536 * 4
    plane = 2.5 * 2048 * (11 * 700 + np.log2(1536) * 1536)
    corr = (2.5 * np.log2(2048 * 1536) + 10) * 2048 * 1536
    assert f == pytest.approx(n_real * plane + n_corr * corr + 300 * 2048 * 1536, rel=1e-12)
