"""Whole chunks of small systems in one launch (k_steps) against the same steps
as single launches (an engine that traces phases takes those).

The mixed path and the FP64 path in reference order must agree bit for bit:
the force sums are exact or in list order, the list has the same entries in
the same order, and the reductions are the same.  (The FP64 tree-order pair
terms round differently: 1e-11.)  Sizes sit at the edges of a tile, of the
lanes per atom and of the couplings' limit; two types, brute-mode replicas,
many tiny replicas (one lane an atom), lists longer than the fixed-point words
hold and cells whose candidates do not fit in shared memory.
"""
from __future__ import annotations

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "force", "potential", "temp", "box")


def _coupling(kind, k=1):
    from moldyn_gb300.initializer import Barostat, Thermostat
    if kind == "berendsen":
        return [Thermostat.Berendsen(0.5) for _ in range(k)], [Barostat.Berendsen(1.0, 5.0) for _ in range(k)]
    if kind == "nose_hoover":
        return [Thermostat.NoseHoover(0.5) for _ in range(k)], None
    return None, None


def _run(pos, vel, box, steps, coupling, types=None, pots=((0, 0, 1.0, 1.0),), offsets=None, dt=0.004, **kw):
    from moldyn_gb300.engine import Engine
    outs = []
    for trace in (False, True):
        e = Engine(trace=trace, threads_per_atom=1, **kw)
        for t0, t1, s, ep in pots:
            e.set_potential(t0, t1, s, ep)
        ty = np.zeros(len(pos), dtype=np.uint16) if types is None else types
        mass = [1.0, 2.0][:int(ty.max()) + 1]
        k = 1 if offsets is None else len(offsets) - 1
        th, ba = _coupling(coupling, k)
        T0 = gs.t_ref(0.9)
        if offsets is None:
            e.upload(ty, pos, vel, mass, box)
        else:
            e.upload_ensemble(offsets, ty, pos, vel, mass, box)
            e.ensemble_set_coupling(th, None if th is None else [T0] * k, ba, None if ba is None else [1.0] * k)
        e.compute_forces()
        n0 = e.stats().kernel_launches
        for n in steps:
            if offsets is None:
                e.step(n, dt, thermostat=th and th[0], target_temperature=T0, barostat=ba and ba[0],
                       target_pressure=1.0)
            else:
                e.ensemble_step(n, dt)
        out = e.download()
        if offsets is not None:
            e.ensemble_get_coupling()
        out["coupling"] = np.array([t.lambda_ for t in th or []] + [t.psi for t in th or []] +
                                   [b.myu for b in ba or []])
        st = e.stats()
        outs.append((out, st.kernel_launches - n0, st.rebuilds))
        e.close()
    (a, la, ra), (b, lb, rb) = outs
    assert la < lb, "the small engine took single launches"
    assert ra == rb and ra > 1
    return a, b


@pytest.mark.parametrize("coupling", ["nve", "berendsen", "nose_hoover"])
@pytest.mark.parametrize("n", [127, 128, 129, 2016, 4100, 9000])
def test_mixed(n, coupling):
    pos, vel, box = gs.fcc({9000: (13, 14, 13), 4100: (10, 10, 11)}.get(n, (8, 8, 8)), jitter=0.04, seed=n, t_star=1.2)
    keep = np.random.default_rng(n).permutation(len(pos))[:n]
    a, b = _run(pos[keep], vel[keep], box, (1, 2, 30), coupling, precision="mixed")
    for k in FIELDS + ("coupling",):
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("precision,ref", [("fp64", True), ("fp64", False), ("fp32_naive", False)])
@pytest.mark.parametrize("coupling", ["nve", "berendsen", "nose_hoover"])
def test_other_precisions(precision, ref, coupling):
    pos, vel, box = gs.fcc((7, 8, 9), jitter=0.04, seed=5, t_star=1.2)
    a, b = _run(pos, vel, box, (1, 24), coupling, precision=precision, reference_order=ref)
    for k in FIELDS + ("coupling",):
        if precision == "fp64" and not ref:
            scale = max(1.0, np.abs(b[k]).max(initial=0.0))
            assert np.abs(a[k] - b[k]).max(initial=0.0) <= 1e-11 * scale, k
        else:
            assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("precision,ref", [("mixed", False), ("fp64", True)])
def test_two_types(precision, ref):
    pos, vel, box = gs.fcc((7, 7, 8), jitter=0.04, seed=6, t_star=1.0)
    ids = (np.random.default_rng(1).random(len(pos)) < 0.4).astype(np.uint16)
    pots = ((0, 0, 1.0, 1.0), (0, 1, 0.95, 0.9), (1, 1, 0.9, 0.8))
    for coupling in ("nve", "nose_hoover"):
        a, b = _run(pos, vel, box, (25,), coupling, types=ids, pots=pots, precision=precision, reference_order=ref)
        for k in FIELDS + ("coupling",):
            assert np.array_equal(a[k], b[k]), (coupling, k)


def test_long_lists_and_crowded_cells():
    """416 entries an atom; 27 cells of about 108 atoms each."""
    pos, vel, box = gs.fcc((9, 9, 9), jitter=0.04, seed=8, t_star=3.0)
    a, b = _run(pos, vel, box, (100, 110), "nve", precision="mixed", skin=2.4, dt=0.005)
    for k in FIELDS:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("coupling", ["nve", "berendsen"])
def test_many_replicas(coupling):
    """Brute-mode replicas of 32 atoms beside larger ones: 260 tiles and more,
    one lane an atom, replicas that rebuild alone."""
    rng = np.random.default_rng(3)
    systems = [gs.fcc((2, 2, 2), rho=r, jitter=0.03, seed=i, t_star=1.0) for i, r in
               enumerate(rng.uniform(0.3, 0.9, 256))]
    systems += [gs.fcc((6, 6, 6), jitter=0.03, seed=900, t_star=2.0), gs.fcc((5, 6, 7), rho=0.5, seed=901, jitter=0.03)]
    offs = np.cumsum([0] + [len(s[0]) for s in systems])
    a, b = _run(np.concatenate([s[0] for s in systems]), np.concatenate([s[1] for s in systems]),
                np.array([s[2] for s in systems]), (25,), coupling, offsets=offs, precision="mixed", graph_steps=8)
    for k in FIELDS + ("coupling",):
        assert np.array_equal(a[k], b[k]), k
