"""A step call that fails in the middle of a chunk puts the state back; the
coupling state read afterwards is the one put back too, not the failed chunk's."""
from __future__ import annotations

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single_launches", [False, True])
@pytest.mark.parametrize("kind", ["berendsen", "nose_hoover"])
def test_coupling_after_a_failed_chunk(kind, single_launches):
    from moldyn_gb300 import _lib
    from moldyn_gb300.engine import Engine
    from moldyn_gb300.initializer import Barostat, Thermostat
    pos, vel, box = gs.fcc((7, 8, 9), jitter=0.04, seed=4, t_star=1.3)
    e = Engine(precision="mixed", threads_per_atom=1, trace=single_launches)
    e.set_potential(0, 0, 1.0, 1.0)
    e.upload_ensemble([0, len(pos)], np.zeros(len(pos), dtype=np.uint16), pos, vel, [1.0], box)
    e.compute_forces()
    th = Thermostat.Berendsen(0.5) if kind == "berendsen" else Thermostat.NoseHoover(0.5)
    ba = Barostat.Berendsen(1.0, 5.0)
    e.ensemble_set_coupling([th], [gs.t_ref(0.8)], [ba], [1.0])

    def coupling():
        e.ensemble_get_coupling()
        return th.lambda_, th.psi, ba.myu

    e.ensemble_step(6, 0.004)
    before = coupling()
    e.test_barrier_timeout(hold_block=2, wait_cycles=2_000_000, step=3)
    with pytest.raises(_lib.MdgbError) as err:
        e.ensemble_step(8, 0.004)
    assert err.value.status == 7          # MDGB_ERR_DEVICE_TIMEOUT
    assert coupling() == before
    e.ensemble_step(8, 0.004)
    assert coupling() != before
    e.close()
