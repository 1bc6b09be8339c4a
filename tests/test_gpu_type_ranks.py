"""Uploads of several types: the device's ranks (type-major within a replica,
the caller's order within a type) at the edges of a tile, for one system and
for replicas.  A type's momentum is a serial sum in rank order in a
reference-order engine, so its bits show the order."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine():
    from moldyn_gb300.engine import Engine
    e = Engine(precision="fp64", reference_order=True)
    for a in range(5):
        for b in range(a, 5):
            e.set_potential(a, b, 0.3, 1.0)
    return e


def _system(n, seed):
    rng = np.random.default_rng([n, seed])
    ids = rng.integers(0, 5, n).astype(np.uint16)
    ids[:5] = rng.permutation(5)
    return ids, rng.random((n, 3)) * 9.0, rng.standard_normal((n, 3))


MASS = np.array([1.0, 0.7, 2.1, 3.3, 1.9])


def _momentum(oracle, ids, vel, t):
    v = vel[ids == t]
    st = oracle.OracleState([len(v)], np.zeros_like(v), v, [MASS[t]], np.full(3, 9.0), oracle.pot_table(1))
    return st.momentum(0)


@pytest.mark.parametrize("n", [5, 127, 128, 129, 3001])
def test_single_system(oracle, n):
    ids, pos, vel = _system(n, 1)
    e = _engine()
    e.upload(ids, pos, vel, MASS, [9.0, 9.0, 9.0])
    for t in range(5):
        m = e.macro(t)
        assert m["count"] == (ids == t).sum()
        assert np.array_equal(m["momentum"], _momentum(oracle, ids, vel, t)), t
    e.close()


def test_replicas_and_refused_uploads(oracle):
    from moldyn_gb300._lib import MdgbError
    parts = [_system(n, 7) for n in (5, 260, 128, 40000, 131)]
    offs = np.cumsum([0] + [len(p[0]) for p in parts])
    ids, pos, vel = (np.concatenate([p[k] for p in parts]) for k in range(3))
    boxes = np.full((5, 3), 9.0)
    e = _engine()
    e.upload_ensemble(offs, ids, pos, vel, MASS, boxes)
    want = [[_momentum(oracle, p[0], p[2], t) for p in parts] for t in range(5)]
    for t in range(5):
        for r, m in enumerate(e.macro(t)):
            assert np.array_equal(m["momentum"], want[t][r]), (t, r)
    bad = ids.copy()
    bad[777] = 5
    lone = ids.copy()
    lone[offs[2]:offs[3]][lone[offs[2]:offs[3]] == 3] = 2     # a replica without type 3
    for wrong in (bad, lone):
        with pytest.raises(MdgbError) as x:
            e.upload_ensemble(offs, wrong, pos, vel, MASS, boxes)
        assert x.value.status == 1
        assert np.array_equal(e.download(fields=("vel",))["vel"], vel)    # the state held before stays
    e.close()
