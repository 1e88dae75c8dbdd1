"""A pose's sums do not depend on the launch that makes them: refining a pose alone (few blocks: several
pixels' taps in flight per thread) gives, bit for bit, what refining it among many does (a full grid:
one pixel at a time), for images from a few tiles (8 × 4 pixels) with remainders to several waves."""
import numpy as np
import pytest

import zcmir_b200 as zc
from zcmir_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", ["homography", "affine"])
@pytest.mark.parametrize("mw,mh,fw,fh", [(33, 31, 36, 29), (64, 64, 64, 64), (257, 129, 130, 260), (500, 420, 433, 391)])
def test_alone_equals_among_many(mw, mh, fw, fh, group):
    rng = np.random.default_rng(mw)
    big = synth.blob_field(max(mh, fh), max(mw, fw), rng, n_blobs=64, sigma=(2.0, 9.0))
    m = (1.0 - big[:mh, :mw] ** 2 + 0.02 * rng.standard_normal((mh, mw))).astype(np.float32)
    T = lambda x, y: np.array([[1, 0, x], [0, 1, y], [0, 0, 1.0]])
    poses = [T(0.4 * k - 1.0, 0.7 - 0.3 * k) for k in range(24)]
    with zc.Engine(half=False, group=group) as reg:
        reg.set_images(m, big[:fh, :fw].astype(np.float32), preprocess=False)
        P, S = reg.refine_poses(poses, 3)
        for k in (0, 11, 23):
            p, s = reg.refine_poses([poses[k]], 3)
            np.testing.assert_array_equal(p[0], P[k])
            assert s[0] == S[k]
