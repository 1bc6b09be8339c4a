"""Threads per atom chosen by the engine where some calls run as one launch (NVE
steps) and others as several (coupled steps above 12,288 atoms, forces alone):
the lists change their layout after 32 steps of the other kind, the timing is
made then, and nothing of the state changes with it."""
from __future__ import annotations

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu

DT = 0.003


def _coupling():
    from moldyn_gb300.initializer import Barostat, Thermostat
    return dict(thermostat=Thermostat.Berendsen(0.5), target_temperature=gs.t_ref(0.9),
                barostat=Barostat.Berendsen(1.0, 5.0), target_pressure=1.0)


def _launched(e, f):
    n = e.stats().kernel_launches
    f()
    return e.stats().kernel_launches - n


@pytest.mark.parametrize("graph_steps", [0, 16])
def test_layout_follows_the_calls(graph_steps):
    from moldyn_gb300.engine import Engine
    pos, vel, box = gs.fcc((15, 15, 15), jitter=0.04, seed=31, t_star=1.1)
    engines = []
    for tpa in (0, 1):
        e = Engine(precision="mixed", threads_per_atom=tpa, graph_steps=graph_steps)
        e.set_potential(0, 0, 1.0, 1.0)
        e.upload(np.zeros(len(pos), dtype=np.uint16), pos, vel, [1.0], box)
        e.compute_forces()
        engines.append(e)
    auto, fixed = engines
    th = [_coupling(), _coupling()]

    def both(n, coupled):
        return [_launched(e, lambda: e.step(n, DT, **(th[k] if coupled else {}))) for k, e in enumerate(engines)]

    a, b = both(20, False)
    assert a == b                       # one launch a chunk
    a, b = both(8, True)
    assert a == b                       # a few coupled steps change nothing
    a, b = both(40, True)
    assert a > b                        # the candidates were timed
    a, b = both(20, False)
    assert a > b                        # still in the timed layout: launches
    a, b = both(20, False)
    assert a > b - 1                    # back to one launch a chunk, after a rebuild
    a, b = both(20, False)
    assert a == b
    assert max(auto.stats().class_threads_per_atom) == 1
    n = _launched(auto, lambda: [auto.compute_forces() for _ in range(40)])
    assert n > _launched(fixed, lambda: [fixed.compute_forces() for _ in range(40)])
    x, y = auto.download(), fixed.download()
    d = x["pos"] - y["pos"]
    d -= y["box"] * np.round(d / y["box"])
    # rebuilds at other steps move the FP32 mirrors' roundings (1e-7 of the force)
    assert np.abs(d).max() <= 1e-6 and np.abs(x["box"] - y["box"]).max() <= 1e-8 * y["box"].max()
    assert abs(th[0]["thermostat"].lambda_ - th[1]["thermostat"].lambda_) <= 1e-8
    for e in engines:
        e.close()


def test_uploaded_forces_survive_the_timing():
    """The timing's first rebuild at a new list radius moves the atoms; forces
    uploaded before it go with them."""
    from moldyn_gb300.engine import Engine
    pos, vel, box = gs.fcc((15, 15, 15), jitter=0.04, seed=32, t_star=1.1)
    frc = np.random.default_rng(1).standard_normal(pos.shape)
    types = np.zeros(len(pos), dtype=np.uint16)
    outs = []
    for tpa in (0, 1):
        e = Engine(precision="mixed", threads_per_atom=tpa, trace=True)
        e.set_potential(0, 0, 1.0, 1.0)
        e.upload(types, pos, vel, [1.0], box)
        e.upload_forces(frc)
        e.set_potential_raw(0, 0, 1.0, 1.0, 3.1, 0.0)
        e.step(1, DT)
        outs.append(e.download())
        e.close()
    assert np.array_equal(outs[0]["pos"], outs[1]["pos"])
