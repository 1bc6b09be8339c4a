"""Cells whose neighbours' atoms fill the one-launch kernel's window once, exactly,
and more than twice: the trajectory of single launches (a traced engine), bit for
bit."""
from __future__ import annotations

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu


# 27 cells an axis of three: every cell sees all atoms -- 1,372, 1,800, 2,048, 4,000
@pytest.mark.parametrize("cells,n,skin,precision,ref", [
    ((7, 7, 7), 1372, 1.3, "mixed", False), ((8, 8, 8), 1800, 1.9, "mixed", False), ((8, 8, 8), 1801, 1.9, "mixed", False),
    ((10, 10, 10), 4000, 3.0, "mixed", False), ((10, 10, 10), 4000, 3.0, "fp64", True)])
def test_windows(cells, n, skin, precision, ref):
    from moldyn_gb300.engine import Engine
    pos, vel, box = gs.fcc(cells, jitter=0.04, seed=14, t_star=3.0)
    keep = np.random.default_rng(n).permutation(len(pos))[:n]
    pos, vel = pos[keep], vel[keep]
    outs, launches = [], []
    for trace in (False, True):
        e = Engine(precision=precision, reference_order=ref, skin=skin, threads_per_atom=1, trace=trace)
        e.set_potential(0, 0, 1.0, 1.0)
        e.upload(np.zeros(n, dtype=np.uint16), pos, vel, [1.0], box)
        e.compute_forces()
        n0 = e.stats()
        e.step(120, 0.005)
        e.step(100, 0.005)
        assert e.stats().rebuilds > n0.rebuilds
        launches.append(e.stats().kernel_launches - n0.kernel_launches)
        outs.append(e.download())
        e.close()
    assert launches[0] < launches[1]
    for k in ("pos", "vel", "force", "potential", "temp"):
        assert np.array_equal(outs[0][k], outs[1][k]), k
