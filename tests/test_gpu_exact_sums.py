"""The coupled step's exact sums over runs of tiles: systems whose tiles fill
the warps' runs once, several times and raggedly, and ensembles whose replicas
share blocks and warps, end inside them, or span many.

The first step's lambda and mu must equal the Berendsen formulas
(thermostat.rs:31-34, barostat.rs:29-30) on the temperature and pressure of the
FP64 macro-parameter reduction of the same state, to 1e-14: the sums differ by
FP64 rounding only (a relative 1e-15 of T and P, scaled by dt / tau), cbrt and
sqrt are CUDA's against numpy's."""
from __future__ import annotations

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu

DT, TAU_T, BETA, TAU_P = 0.005, 0.5, 1.0, 5.0

# cells of every replica, in order
LAYOUTS = {
    "one tile a warp, ragged": [(26, 26, 25)],
    "several tiles a warp": [(50, 50, 51)],
    "replicas within blocks": [(2, 2, 2)] * 301 + [(20, 20, 25)] + [(3, 3, 3)] * 302 + [(21, 20, 19)] + [(2, 2, 3)],
    "replicas within warps": [(2, 2, 2)] * 2501 + [(27, 26, 28)] + [(3, 3, 4)] * 1503 + [(30, 30, 31)],
}


@pytest.mark.parametrize("layout", sorted(LAYOUTS))
def test_first_factors_equal_the_fp64_reduction(layout):
    from moldyn_gb300.engine import Engine
    from moldyn_gb300.initializer import Barostat, Thermostat
    cells = LAYOUTS[layout]
    made = {c: gs.fcc(c, jitter=0.02, seed=sum(c), t_star=1.0) for c in set(cells)}
    nrep = len(cells)
    rng = np.random.default_rng(nrep)
    offs = np.cumsum([0] + [len(made[c][0]) for c in cells])
    assert offs[-1] >= 65536
    pos = np.concatenate([made[c][0] for c in cells])
    vel = np.concatenate([made[c][1] * s for c, s in zip(cells, rng.uniform(0.7, 1.4, nrep))])
    vel += rng.uniform(-0.2, 0.2, (nrep, 3)).repeat(np.diff(offs), axis=0)
    T0s = [gs.t_ref(t) for t in rng.uniform(0.6, 1.2, nrep)]
    P0s = list(rng.uniform(0.5, 1.5, nrep))
    ths = [Thermostat.Berendsen(TAU_T) for _ in cells]
    bas = [Barostat.Berendsen(BETA, TAU_P) for _ in cells]
    e = Engine(precision="mixed", threads_per_atom=1)
    e.set_potential(0, 0, 1.0, 1.0)
    types = np.zeros(len(pos), dtype=np.uint16)
    if nrep == 1:
        e.upload(types, pos, vel, [1.0], made[cells[0]][2])
    else:
        e.upload_ensemble(offs, types, pos, vel, [1.0], np.array([made[c][2] for c in cells]))
    e.compute_forces()
    macs = [e.macro(0)] if nrep == 1 else e.macro(0)
    if nrep == 1:
        e.step(1, DT, thermostat=ths[0], target_temperature=T0s[0], barostat=bas[0], target_pressure=P0s[0])
    else:
        e.ensemble_set_coupling(ths, T0s, bas, P0s)
        e.ensemble_step(1, DT)
        e.ensemble_get_coupling()
    e.close()
    lam = np.sqrt([1.0 + DT / TAU_T * (T / m["temperature"] - 1.0) for T, m in zip(T0s, macs)])
    myu = np.cbrt([1.0 + DT * BETA / TAU_P * (m["pressure"] - P) for P, m in zip(P0s, macs)])
    assert np.abs(np.array([t.lambda_ for t in ths]) - lam).max() <= 1e-14
    assert np.abs(np.array([b.myu for b in bas]) - myu).max() <= 1e-14
