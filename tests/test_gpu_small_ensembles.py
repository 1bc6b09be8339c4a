"""Ensembles on both sides of the one-launch kernel's limit of replicas: up to
300 a chunk of steps is one launch, beyond it several, and every replica's
trajectory is the one it has in an ensemble of the other kind -- with cells that
one block clears and scans (60 replicas) and with more (300)."""
from __future__ import annotations

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu


def _run(systems, tpa=1):
    from moldyn_gb300.engine import Engine
    offs = np.cumsum([0] + [len(s[0]) for s in systems])
    e = Engine(precision="mixed", threads_per_atom=tpa)
    e.set_potential(0, 0, 1.0, 1.0)
    e.upload_ensemble(offs, np.zeros(offs[-1], dtype=np.uint16), np.concatenate([s[0] for s in systems]),
                      np.concatenate([s[1] for s in systems]), [1.0], np.array([s[2] for s in systems]))
    e.compute_forces()
    n0 = e.stats().kernel_launches
    e.ensemble_step(20, 0.003)
    n = e.stats().kernel_launches - n0
    out = e.download()
    e.close()
    return n, out


def test_ensembles_beside_the_limit():
    rng = np.random.default_rng(5)
    systems = [gs.fcc((2, 2, 2), rho=r, jitter=0.03, seed=i, t_star=1.0) for i, r in enumerate(rng.uniform(0.3, 0.8, 299))]
    systems.insert(0, gs.fcc((5, 5, 5), jitter=0.03, seed=900, t_star=2.0))
    systems.append(gs.fcc((2, 3, 2), rho=0.4, jitter=0.03, seed=901))
    n_all, all_ = _run(systems)
    assert n_all > 20
    for k in (300, 60):
        n, few = _run(systems[:k])
        assert n == 1
        m = sum(len(s[0]) for s in systems[:k])
        for name in ("pos", "vel", "force", "potential", "temp"):
            assert np.array_equal(all_[name][:m], few[name]), (k, name)


def test_limit_where_threads_per_atom_are_timed():
    """Automatic threads per atom: up to 96 replicas in one launch, the same
    trajectories beyond (the force sums do not depend on the threads)."""
    systems = [gs.fcc((3, 3, 3), rho=0.5, jitter=0.03, seed=i, t_star=1.0) for i in range(97)]
    n_few, few = _run(systems[:96], 0)
    n_all, all_ = _run(systems, 0)
    assert n_few == 1 and n_all > 20
    k = 108 * 96
    for name in ("pos", "vel", "force"):
        assert np.array_equal(all_[name][:k], few[name]), name
