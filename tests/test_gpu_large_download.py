"""Downloads large enough that the host settles the output pages first: buffers
that start and end inside a page, mapped and not yet mapped, written whole and
not a byte further."""
from __future__ import annotations

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu


def test_large_download_into_ragged_buffers():
    from moldyn_gb300.engine import Engine
    pos, vel, box = gs.fcc((74, 74, 74), jitter=0.03, seed=3)      # 1,620,896 atoms: 143 MB
    n = len(pos)
    e = Engine(precision="mixed", threads_per_atom=1)
    e.set_potential(0, 0, 1.0, 1.0)
    e.upload(np.zeros(n, dtype=np.uint16), pos, vel, [1.0], box)
    e.compute_forces()
    pad = 1025
    for mapped in (False, True):
        out, whole = {}, {}
        for k, m in (("pos", 3), ("vel", 3), ("force", 3), ("potential", 1), ("temp", 1)):
            w = whole[k] = np.full(m * n + 2 * pad, -7.0) if mapped else np.empty(m * n + 2 * pad)
            w[:pad] = w[-pad:] = -7.0
            out[k] = w[pad:-pad].reshape((n, 3) if m == 3 else (n,))
        ids = {k: id(v) for k, v in out.items()}
        got = e.download(out)
        assert all(id(got[k]) == i for k, i in ids.items())
        assert all((w[:pad] == -7.0).all() and (w[-pad:] == -7.0).all() for w in whole.values())
        assert np.array_equal(got["pos"], pos) and np.array_equal(got["vel"], vel)
        for k in ("force", "potential", "temp"):
            assert np.array_equal(got[k], e.download(fields=(k,))[k])
    e.close()
