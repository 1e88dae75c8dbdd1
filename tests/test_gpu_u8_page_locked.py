"""8-bit pixels in page-locked memory are the caller's again when the upload call returns: a buffer refilled
at once, or used for both sides in turn, gives the images it held at each call. The uploads queue behind a
large build, so a copy that the call did not wait for would read the refilled buffer."""
import numpy as np
import pytest
import torch

import zcmir_b200 as zc
from zcmir_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [1, 3, 4])
@pytest.mark.parametrize("rgba", [False, True])
def test_a_page_locked_buffer_may_be_refilled_on_return(c, rgba):
    rng = np.random.default_rng(c)
    c = 4 if rgba else c
    a, b = (rng.integers(0, 256, (700, 900, c), dtype=np.uint8) for _ in range(2))
    big = rng.integers(0, 256, (4096, 4096), dtype=np.uint8)
    buf = torch.empty(a.shape, dtype=torch.uint8, pin_memory=True).numpy()

    def put(eng, side, img):
        if rgba:
            eng.call("zc_set_image_rgba", side, img.ctypes.data_as(N.u8p), img.shape[1], img.shape[0])
        else:
            eng.set_image(side, img)

    with zc.Engine() as eng:
        for side, img in ((0, a), (1, b)):
            put(eng, side, img)
        want = [eng.work_image(s) for s in (0, 1)]
        eng.set_image(0, big)
        for side, img in ((0, a), (1, b)):
            buf[:] = img
            put(eng, side, buf)
            buf[:] = 255 - img
        for s in (0, 1):
            np.testing.assert_array_equal(eng.work_image(s), want[s])
