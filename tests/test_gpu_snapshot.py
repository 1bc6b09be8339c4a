"""The state a chunk of steps starts from, put back when the chunk fails in a later
step: every array, below and above 262,144 atoms, and the run after it."""
from __future__ import annotations

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "force", "potential", "temp", "box")


@pytest.mark.parametrize("cells", [(5, 6, 7), (30, 31, 32), (40, 41, 42)])
def test_failed_chunk_puts_the_state_back(cells):
    from moldyn_gb300 import _lib
    from moldyn_gb300.engine import Engine
    from moldyn_gb300.initializer import Barostat, Thermostat
    pos, vel, box = gs.fcc(cells, jitter=0.04, seed=41, t_star=1.2)
    e = Engine(precision="mixed", threads_per_atom=1)
    e.set_potential(0, 0, 1.0, 1.0)
    e.upload(np.zeros(len(pos), dtype=np.uint16), pos, vel, [1.0], box)
    e.compute_forces()

    def step(n):
        e.step(n, 0.004, thermostat=Thermostat.Berendsen(0.5), target_temperature=gs.t_ref(0.8),
               barostat=Barostat.Berendsen(1.0, 5.0), target_pressure=1.0)

    step(5)
    before = e.download()
    e.test_barrier_timeout(hold_block=1, wait_cycles=4_000_000, step=3)
    with pytest.raises(_lib.MdgbError) as err:
        step(6)
    assert err.value.status == 7          # MDGB_ERR_DEVICE_TIMEOUT
    after = e.download()
    for k in FIELDS:
        assert np.array_equal(before[k], after[k]), k
    step(6)
    assert not np.array_equal(e.download()["pos"], before["pos"])
    e.close()
