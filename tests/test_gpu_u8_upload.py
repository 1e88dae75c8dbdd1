"""8-bit images of one, three and four channels go up as they are (zcb_set_image_u8) and give, bit for
bit, the work image and features that the same image expanded to RGBA8 gives (zc_set_image_rgba); what
was refused stays refused."""
import ctypes

import numpy as np
import pytest

import zcmir_b200 as zc
from zcmir_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half,clahe", [(True, True), (False, True), (False, False)])
@pytest.mark.parametrize("w,h", [(8, 8), (33, 17), (129, 250)])
@pytest.mark.parametrize("c", [0, 1, 3, 4])
def test_u8_equals_rgba(w, h, c, half, clahe):
    rng = np.random.default_rng(w + c)
    img = rng.integers(0, 256, (h, w, c) if c else (h, w), dtype=np.uint8)
    if c == 3:
        img = img[:, ::-1]  # not contiguous
    with zc.Engine(half=half, clahe=clahe) as eng:
        eng.set_images(img, img[::-1])
        got = [eng.work_image(s) for s in (0, 1)] + [eng.features(s) for s in (0, 1)]
        for s, a in ((0, img), (1, img[::-1])):
            px = zc.rgba8(a)
            eng.call("zc_set_image_rgba", s, px.ctypes.data_as(N.u8p), w, h)
        want = [eng.work_image(s) for s in (0, 1)] + [eng.features(s) for s in (0, 1)]
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)


def test_u8_refusals():
    a = np.zeros((16, 16, 2), np.uint8)
    with zc.Engine() as eng:
        with pytest.raises(ValueError):
            eng.set_image(0, a)
        with pytest.raises(ValueError):
            eng.set_image(0, a[..., 0], preprocess=False)
        for side, w, h, c in ((2, 16, 16, 1), (0, 7, 16, 1), (0, 16, 16, 2)):
            with pytest.raises(zc.EngineError):
                eng.call("zcb_set_image_u8", side, a.ctypes.data_as(N.u8p), w, h, c)
        with pytest.raises(zc.EngineError):
            eng.call("zcb_set_image_u8", 0, ctypes.cast(None, N.u8p), 16, 16, 1)
