"""FP64 in tree order with one thread per atom: the three force passes -- over
pair records, without them, and the one-launch kernel of small systems -- give
the same bits, so the memory that happens to be free, or a system's size, only
changes the time."""
from __future__ import annotations

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "force", "potential", "temp")


def _engine(state, **kw):
    from moldyn_gb300.engine import Engine
    pos, vel, box, types = state
    e = Engine(precision="fp64", **kw)
    for (a, b), (s, ep) in {(0, 0): (1.0, 1.0), (0, 1): (0.95, 0.9), (1, 1): (0.9, 0.8)}.items():
        e.set_potential(a, b, s, ep)
    e.upload(types, pos, vel, [1.0, 2.0][:int(types.max()) + 1], box)
    e.compute_forces()
    return e


def _state(cells, rho, two):
    pos, vel, box = gs.fcc(cells, rho=rho, jitter=0.04, seed=21, t_star=1.1)
    types = np.zeros(len(pos), dtype=np.uint16)
    if two:
        types[::3] = 1
    return pos, vel, box, types


def _same(a, b):
    a, b = a.download(), b.download()
    for k in FIELDS:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("cells,rho,two", [((11, 11, 9), 0.8442, False), ((13, 14, 15), 0.6, True)])
def test_records_or_not(cells, rho, two):
    state = _state(cells, rho, two)
    a, b = _engine(state, threads_per_atom=1), _engine(state, threads_per_atom=1, pair_records=False)
    _same(a, b)
    for n in (1, 30):
        a.step(n, 0.003)
        b.step(n, 0.003)
    _same(a, b)
    assert a.stats().kernel_launches != b.stats().kernel_launches
    a.close()
    b.close()


@pytest.mark.parametrize("cells,two", [((4, 4, 4), False), ((6, 7, 8), True)])
def test_one_launch_or_several(cells, two):
    state = _state(cells, 0.8442, two)
    a, b = _engine(state), _engine(state, trace=True, threads_per_atom=1)
    for n in (1, 30):
        a.step(n, 0.003)
        b.step(n, 0.003)
    _same(a, b)
    assert a.stats().kernel_launches < b.stats().kernel_launches
    a.close()
    b.close()
