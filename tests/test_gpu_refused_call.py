"""A call that the engine refuses fails alone: the next call, on the same engine or on another, is not
blamed for it. (A roto-scale map of 7776 angles needs more shared memory than a block has: the launch's
set-up is refused on the host and nothing runs.)"""
import numpy as np
import pytest

import zcmir_b200 as zc
from zcmir_b200 import synth

pytestmark = pytest.mark.gpu


def test_the_call_after_a_refused_one_runs():
    m, f, H = synth.pair_remap(n=1700, shift=(6, -4), seed=2)
    with zc.Engine(half=False, map_res=7776) as reg, zc.Engine(half=False) as other:
        reg.set_images(m, f, preprocess=False)
        want = reg.score(H)
        for eng in (reg, other):
            with pytest.raises(zc.EngineError, match="invalid argument"):
                reg.rs_map(H, symmetric=False)
            eng.set_images(m, f, preprocess=False)
            assert eng.score(H) == want
