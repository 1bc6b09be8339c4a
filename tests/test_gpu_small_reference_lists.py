"""Lists of more than 128 entries in the reference's order inside k_steps, where
all lanes of a warp write an atom's list before one of them sorts it: the same
trajectory as single launches (a traced engine takes those), bit for bit, over
several rebuilds."""
from __future__ import annotations

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,skin,r_cut", [((7, 8, 9), 1.1, 2.5), ((8, 8, 8), 0.3, 3.5), ((9, 9, 9), 1.6, 2.5)])
def test_long_reference_lists(cells, skin, r_cut):
    from moldyn_gb300.engine import Engine
    pos, vel, box = gs.fcc(cells, jitter=0.04, seed=12, t_star=3.0)
    perm = np.random.default_rng(2).permutation(len(pos))
    pos, vel = pos[perm], vel[perm]
    outs, launches = [], []
    for trace in (False, True):
        e = Engine(precision="fp64", reference_order=True, skin=skin, trace=trace)
        e.set_potential_raw(0, 0, 1.0, 1.0, r_cut, 0.0)
        e.upload(np.zeros(len(pos), dtype=np.uint16), pos, vel, [1.0], box)
        e.compute_forces()
        n0 = e.stats()
        for n in (1, 64, 120):
            e.step(n, 0.004)
        st = e.stats()
        assert st.max_neighbors > 128 and st.rebuilds > n0.rebuilds + 1
        launches.append(st.kernel_launches - n0.kernel_launches)
        outs.append(e.download())
        e.close()
    assert launches[0] < launches[1]
    for k in ("pos", "vel", "force", "potential", "temp"):
        assert np.array_equal(outs[0][k], outs[1][k]), k
