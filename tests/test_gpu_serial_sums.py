"""The reference-order reductions against the oracle's serial folds, bit for
bit: the GPU runs the segments of a fold ahead of their turn (128 a round, 8 to
64 terms each) and stitches them together, adding term by term where the
running sum strays too far.  The sizes sit at the edges of a segment, of a
round and of the segment lengths, and the values force every way through --
terms of a few bits spread over many binades (ties, exact cancellation to
zero), all zero, one huge term, and ordinary Maxwellian ones, with and without
zero momentum.
"""
from __future__ import annotations

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu


def _values(kind, shape, rng):
    if kind == "maxwell":
        return rng.standard_normal(shape)
    if kind == "paired":
        v = rng.standard_normal(shape)
        v[len(v) // 2:2 * (len(v) // 2)] = -v[:len(v) // 2]
        return v
    if kind == "bits":    # 1..7 x 2^-30 .. 2^30, either sign
        return rng.integers(-7, 8, shape) * np.exp2(rng.integers(-30, 31, shape))
    if kind == "zero":
        return np.zeros(shape) * rng.choice([1.0, -1.0], shape)
    v = rng.standard_normal(shape) * 1e-3
    v[len(v) // 2] = 1e9
    return v


@pytest.mark.parametrize("kind", ["maxwell", "paired", "bits", "zero", "huge"])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 1024, 1025, 1033, 8191, 8192, 8193, 20011])
def test_folds_equal_the_oracle(n, kind, oracle):
    from moldyn_gb300.engine import Engine
    rng = np.random.default_rng([n, len(kind)])
    box = np.full(3, 40.0)
    pos = rng.random((n, 3)) * box
    vel, pot, tmp = _values(kind, (n, 3), rng), _values(kind, n, rng), _values(kind, n, rng)
    mass = 0.7
    e = Engine(precision="fp64", reference_order=True)
    e.set_potential(0, 0, 1.0, 1.0)
    e.upload(np.zeros(n, dtype=np.uint16), pos, vel, [mass], box)
    e.upload_forces(np.zeros((n, 3)), pot, tmp)
    m = e.macro(0)
    st = oracle.OracleState([n], pos, vel, [mass], box, oracle.pot_table(1, default=(1.0, 1.0)))
    st.potential[:] = pot
    st.temp[:] = tmp
    assert np.array_equal(m["momentum"], st.momentum())
    assert np.array_equal(m["com_velocity"], st.com_velocity())
    assert m["kinetic_energy"] == st.kinetic_energy()
    assert m["potential_energy"] == st.potential_energy()
    assert m["thermal_energy"] == st.thermal_energy()
    assert m["pressure"] == st.pressure()
    e.close()


@pytest.mark.parametrize("n", [17, 513, 1500])
def test_coupled_step_equals_the_oracle(n, oracle):
    """Two Berendsen-thermostat steps through the same folds."""
    from moldyn_gb300.engine import Engine
    from moldyn_gb300.initializer import Thermostat
    pos, vel, box = gs.gas(n, np.full(3, max(9.0, (n / 0.2) ** (1.0 / 3.0))), seed=n, min_dist=0.95)
    e = Engine(precision="fp64", reference_order=True)
    e.set_potential(0, 0, 1.0, 1.0)
    e.upload(np.zeros(n, dtype=np.uint16), pos, vel, [1.0], box)
    e.compute_forces()
    st = oracle.OracleState([n], pos, vel, [1.0], box, oracle.pot_table(1, default=(1.0, 1.0)))
    st.update_force()
    th, oth = Thermostat.Berendsen(0.5), oracle.Thermostat(oracle.BERENDSEN, 0.5, 0.0, 0.0)
    e.step(2, 0.002, thermostat=th, target_temperature=gs.t_ref(1.1))
    st.step(0.002, nsteps=2, thermostat=oth, T0=gs.t_ref(1.1))
    out = e.download()
    assert th.lambda_ == oth.lambda_
    assert np.array_equal(out["pos"], st.pos) and np.array_equal(out["vel"], st.vel)
    e.close()
