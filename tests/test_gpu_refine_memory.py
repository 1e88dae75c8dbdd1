"""A batched refine's device memory: the blocks' partial sums of many candidates are kept for as many
poses as a bounded scratch holds, the launches taking that many poses at a time. A pose's sums, and so
the refined poses, do not depend on which poses share its launch."""
import numpy as np
import pytest
import torch

import zcmir_b200 as zc
from zcmir_b200 import synth

pytestmark = pytest.mark.gpu

N = 1000


def poses(n):
    rng = np.random.default_rng(7)
    out = np.tile(np.eye(3), (n, 1, 1))
    out[:, :2, 2] = rng.uniform(-3, 3, (n, 2))
    return out


def refine(symmetric, pair):
    with zc.Engine(half=False, symmetric=symmetric) as reg:
        reg.set_images(*pair, preprocess=False)
        reg.refine_poses(poses(1), iters=1)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        H, s = reg.refine_poses(poses(N), iters=1)
        grown = before - torch.cuda.mem_get_info()[0]
        few = [reg.refine_poses(poses(N)[k:k + 3], iters=1) for k in (0, N // 2, N - 3)]
    for k, (h, v) in zip((0, N // 2, N - 3), few):
        np.testing.assert_array_equal(h, H[k:k + 3])
        np.testing.assert_array_equal(v, s[k:k + 3])
    return grown


def test_a_symmetric_refine_takes_no_more_scratch_than_a_one_sided_one():
    m, f, _ = synth.pair_remap(n=1024, shift=(3, 2), seed=4)
    one, both = refine(False, (m, f)), refine(True, (m, f))
    # the poses' own sums, coefficients and scores are doubled: 0.8 KB of the 80 KB a candidate's scratch took
    assert both <= one + (64 << 20), (one >> 20, both >> 20)
