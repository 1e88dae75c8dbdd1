"""The features of images at the edges of the tiles that form them, against the CPU oracle.

Tolerance: the feature tests' own, 2e-6 (float32 arithmetic restated operation by operation; the
image-wide sums are float64 in another order on the two sides, so the whitening may round apart), and
all but one value in a thousand equal."""
import numpy as np
import pytest

import zcmir_b200 as zc
from oracle import smi_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["laplacian", "cubic"])
@pytest.mark.parametrize("w,h", [(16, 16), (33, 9), (31, 65), (300, 17), (32, 8 * 593), (701, 513)])
def test_features_of_odd_sizes(w, h, mode):
    rng = np.random.default_rng(w * h)
    m, f = (rng.random((h, w), dtype=np.float32) for _ in range(2))
    with zc.Engine(half=False, smi_features=mode) as eng:
        eng.set_images(m, f, preprocess=False)
        for side, img in ((0, m), (1, f)):
            gpu, ora = eng.features(side), O.prepare(img, mode)["feat"]
            np.testing.assert_allclose(gpu, ora, rtol=0, atol=2e-6)
            assert np.mean(gpu == ora) > 0.999
