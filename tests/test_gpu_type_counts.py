"""Uploads of several types on both sides of the size up to which the types are
counted on the host: the ranks shown by the momentum's bits, and the refusals."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_gpu_type_ranks import MASS, _engine, _momentum, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(16384,), (16385,), (5, 12288, 127, 300), (5, 16000, 128, 300)])
def test_beside_the_line(oracle, sizes):
    from moldyn_gb300._lib import MdgbError
    parts = [_system(n, 9) for n in sizes]
    offs = np.cumsum([0] + list(sizes))
    ids, pos, vel = (np.concatenate([p[k] for p in parts]) for k in range(3))
    boxes = np.full((len(sizes), 3), 9.0)
    e = _engine()
    e.upload_ensemble(offs, ids, pos, vel, MASS, boxes)
    for t in range(5):
        got = e.macro(t)
        for p, m in zip(parts, got if len(sizes) > 1 else [got]):
            assert m["count"] == (p[0] == t).sum()
            assert np.array_equal(m["momentum"], _momentum(oracle, p[0], p[2], t)), t
    bad, lone = ids.copy(), ids.copy()
    bad[-1] = 5
    first = lone[:offs[1]]
    first[first == 3] = 2            # the first replica without type 3
    for wrong in (bad, lone):
        with pytest.raises(MdgbError) as x:
            e.upload_ensemble(offs, wrong, pos, vel, MASS, boxes)
        assert x.value.status == 1
        assert np.array_equal(e.download(fields=("vel",))["vel"], vel)    # the state held before stays
    e.close()
