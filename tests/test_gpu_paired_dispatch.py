"""Which replicas take the paired list build: 32,768 atoms and more, and from
8,192 those that average at most 24 atoms a cell.  A cell of more than 32 atoms
among them sends the rebuild to the direct build, which mdgb_stats counts; the
same cell in a replica that does not take the paired build is not counted.  (An
upload builds the lists and nothing else, so the crowd may overlap.)"""
from __future__ import annotations

import math

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu

SKIN, R_CUT = 0.3, 2.5


def _grid(n, box):
    """The engine's cells: one list radius wide at least, about 8 atoms at least."""
    nc = [int(L / ((R_CUT + SKIN) * (1.0 + 1e-6))) for L in box]
    cap = int(max(27.0, min(math.ceil(np.prod(nc) * 1.3) + 27.0, n / 8.0 + 27.0)))
    while np.prod(nc) > cap:
        a = 0
        if nc[1] > nc[a]:
            a = 1
        if nc[2] > nc[a]:
            a = 2
        nc[a] -= 1
    return nc


def _crowded(cells, n, rho):
    """n atoms of an FCC lattice, 40 of them moved into one cell."""
    pos, vel, box = gs.fcc(cells, rho=rho, jitter=0.03, seed=n)
    pos, vel = pos[:n], vel[:n]
    side = box / np.array(_grid(n, box))
    rng = np.random.default_rng(n)
    pos[rng.choice(n, 40, replace=False)] = (np.array([1, 2, 1]) + 0.5 + rng.uniform(-0.3, 0.3, (40, 3))) * side
    return pos, vel, box


def _direct_builds(systems):
    from moldyn_gb300.engine import Engine
    offs = np.cumsum([0] + [len(s[0]) for s in systems])
    e = Engine(precision="mixed", threads_per_atom=1, skin=SKIN)
    e.set_potential(0, 0, 1.0, 1.0)
    e.upload_ensemble(offs, np.zeros(offs[-1], dtype=np.uint16), np.concatenate([s[0] for s in systems]),
                      np.concatenate([s[1] for s in systems]), [1.0], np.array([s[2] for s in systems]))
    n = e.stats().direct_list_builds
    e.close()
    return n


@pytest.mark.parametrize("cells,n,rho,paired", [
    ((13, 13, 13), 8191, 0.1, False), ((13, 13, 13), 8192, 0.1, True),
    ((13, 13, 13), 8788, 0.8442, False),                        # 25.6 atoms a cell
    ((16, 16, 17), 17408, 0.8442, True),                        # 21.5
    ((20, 20, 21), 32767, 0.8442, True), ((16, 16, 32), 32768, 0.8442, True)])
def test_line_of_the_paired_build(cells, n, rho, paired):
    s = _crowded(cells, n, rho)
    average = n / np.prod(_grid(n, s[2]))
    assert paired == (n >= 32768 or (n >= 8192 and average <= 24))
    assert (_direct_builds([s]) > 0) == paired
    # beside a replica that takes the paired build but is not crowded
    assert (_direct_builds([gs.fcc((17, 17, 29), jitter=0.02, seed=1), s]) > 0) == paired


def test_dense_replica_below_32768_atoms():
    """A dense replica that takes the paired build: the direct build's trajectory."""
    from moldyn_gb300.engine import Engine
    pos, vel, box = gs.fcc((16, 16, 17), jitter=0.04, seed=8, t_star=1.2)
    outs = []
    for direct in (False, True):
        e = Engine(precision="mixed", threads_per_atom=1, direct_list=direct, trace=True)
        e.set_potential(0, 0, 1.0, 1.0)
        e.upload(np.zeros(len(pos), dtype=np.uint16), pos, vel, [1.0], box)
        e.compute_forces()
        e.step(40, 0.005)
        assert e.stats().rebuilds > 2 and (e.stats().direct_list_builds > 0) == direct
        outs.append(e.download())
        e.close()
    for k in ("pos", "vel", "force", "potential", "temp"):
        assert np.array_equal(outs[0][k], outs[1][k]), k
