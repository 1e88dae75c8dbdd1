"""Roto-scale maps of 5832 to 6912 angles: their grids fill a row (as many cells as the transform has
points), so the forward pass's staged row and its line must fit shared memory together.

The forward map against the sums formed directly in float64 from the oracle's log-polar planes, at the
zero lag, the peak and lags spread over every angle: the bound is the roto-scale tests', 1e-4 of the
peak where the overlap is at least 20 % of the zero lag's."""
import numpy as np
import pytest
import torch

import zcmir_b200 as zc
from oracle import rs_oracle as R
from oracle import smi_oracle as O
from zcmir_b200 import synth

pytestmark = pytest.mark.gpu


def planes(s, rho):
    """The 15 real planes of premultiplied samples s = [w, w f0..w f3] (5, rows, n_θ), times the ρ weight."""
    w = torch.where(s[0] > 1e-6, s[0], 1.0)
    pairs = [torch.where(s[0] > 1e-6, s[1 + i] * s[1 + j] / w, 0.0) for i, j in O.TRI]
    return torch.stack([*s, *pairs]) * rho


def lag_sums(la, lb, rho, lags, rows=256):
    """(45, lags) sums Σ a(λ + k, θ + l)·b(λ, θ), θ cyclic, from the log-polar planes (float64 on the GPU)."""
    la, lb, rho = (torch.as_tensor(v, dtype=torch.float64, device="cuda") for v in (la, lb, rho))
    out = np.zeros((45, len(lags)))
    ids, corrs = O.corr_plan(True, False)
    assert list(ids) == list(range(15))
    for q, (k, l) in enumerate(lags):
        G = torch.zeros((15, 15), dtype=torch.float64, device="cuda")
        y0, y1 = max(0, -k), min(la.shape[1], la.shape[1] - k)
        for r in range(y0, y1, rows):
            e = min(y1, r + rows)
            A = planes(torch.roll(la[:, r + k:e + k], -l, dims=2), rho[r + k:e + k]).flatten(1)
            G += A @ planes(lb[:, r:e], rho[r:e]).flatten(1).T
        G = G.cpu().numpy()
        for a, b, c in corrs:
            out[c, q] = G[a, b]
    return out


@pytest.mark.parametrize("n,side", [(5832, 1240), (6912, 1520)])
def test_rs_map_of_rows_that_fill_their_line(n, side):
    m, f, H = synth.pair_remap(n=side, shift=(6, -4), seed=2)
    with zc.Engine(half=False, calibrated=False, map_res=n) as reg:
        reg.set_images(m, f, preprocess=False)
        r = reg.rs_map(H, symmetric=False)
        pa, pb = ({"feat": x, "acf": None, "stack": np.concatenate([np.ones((1,) + x.shape[1:], np.float32), x])}
                  for x in (reg.features(0), reg.features(1)))
    assert (r.n, r.n_th) == (n, n)
    ox, oy, W, Hh = O.reg_frame(H, side, side, side, side)
    p = R.rs_plan(W, Hh, ox, oy, R.moving_centroid(H, side, side), cap=n)
    assert p["n"] == n
    la, rho = R.logpolar(O.warp_stack(pa["stack"], O.canvas_H(H, ox, oy), W, Hh), p)
    lb, _ = R.logpolar(O.paste_stack(pb["stack"], ox, oy, W, Hh), p)
    y, x = divmod(int(np.argmax(r.fwd)), n)
    signed = lambda v: v if v <= n // 2 else v - n
    lags = [(0, 0), (signed(y), signed(x)), (3, n // 4), (-7, -n // 3), (20, n // 2 - 1), (-40, 1)]
    raw = lag_sums(la, lb, rho, lags)
    scale = np.array([np.exp(k * p["dlam"]) for k, _ in lags]) * p["dlam"] * p["dth"]
    want = O.combine(raw * scale, exact=True, calibrated=False, min_n=O.MIN_N, n00=(raw * scale)[0, 0])
    got = np.array([r.fwd[k % n, l % n] for k, l in lags], np.float64)
    full = raw[0] >= 0.2 * raw[0, 0]
    assert full.sum() >= 4
    assert np.max(np.abs(got - want)[full]) <= 1e-4 * abs(r.fwd.max()), (got, want)
