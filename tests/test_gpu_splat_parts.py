"""Frames of many particles (copied and drawn in parts, spheres behind what a
pixel already holds dropped early) against the oracle, bit for bit.

Only some particles lie in front of the camera, so the oracle draws those
alone: indices at both sides of every part, spheres 1 to 60 pixels wide in
dense layers, touching and grazing ones among them, and equal spheres in
different parts (the lower index wins)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import splat_ref
from tests.test_splat import _params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65535, 131072, 196609, 270001])
def test_parts_equal_the_oracle(n):
    from moldyn_gb300 import render as rnd
    rng = np.random.default_rng(n)
    w, h = 160, 90
    cam = rnd.Camera((0.0, 0.0, 0.0), 70.0, w, h)
    p = np.zeros((n, 12), dtype=np.float32)
    p[:, 0:3] = [-50.0, 0.0, 0.0]           # behind the camera
    p[:, 3] = p[:, 7] = p[:, 8] = 1.0
    p[:, 9] = 0.5
    parts = max(1, min(4, n >> 16))
    per = -(-n // parts)
    seen = {0, n - 1}
    for k in range(1, parts):
        seen |= {k * per - 1, k * per}
    seen |= set(rng.choice(n, 260, replace=False).tolist())
    idx = np.array(sorted(seen))
    m = len(idx)
    p[idx, 0] = rng.uniform(4.0, 60.0, m)
    p[idx, 1:3] = rng.uniform(-0.5, 0.5, (m, 2)) * p[idx, 0:1]
    p[idx, 4:7] = rng.normal(0.0, 0.6, (m, 3))
    p[idx, 9] = np.exp(rng.uniform(np.log(0.01), np.log(2.0), m))
    p[idx, 10] = rng.integers(0, 6, m)
    # the same sphere in the first and the last part, and tangent neighbours
    p[idx[-1], :10] = p[idx[0], :10]
    p[idx[-1], 10] = (p[idx[0], 10] + 1) % 6
    p[idx[5], 0:3] = p[idx[4], 0:3] + np.float32([0.0, 0.0, 1.0]) * (p[idx[4], 9] + p[idx[5], 9])
    prm = rnd.splat_params(cam, 0)
    got = rnd.splat(p, prm, w, h)
    want = splat_ref.render(p[idx], _params(cam), w, h)
    bad = np.argwhere(np.any(got != want, axis=2))
    assert len(bad) == 0, f"{len(bad)} pixels differ, first {bad[:5].tolist()}"
    for k in range(parts):                  # every part draws something seen
        rest = p[idx[(idx < k * per) | (idx >= (k + 1) * per)]]
        assert np.any(splat_ref.render(rest, _params(cam), w, h) != want)
