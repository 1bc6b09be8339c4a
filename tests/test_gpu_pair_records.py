"""The FP64 path's pair records (kernels_pairs.cu, from 4,096 atoms on): every
pair computed once, summed on both sides.

Reference order: forces, potential, temp and NVE trajectories keep the
oracle's bits.  Tree order: its pair terms are functions of r^2 with fewer
roundings, summed in list order: within 1e-12 of the force scale, the bar the
one-sided kernel has.  Sizes sit either side of the record threshold and of a
tile; two types (pairs only one side lists), a permuted caller order, an
ensemble with a brute-mode replica, replicas that rebuild alone, and a pair
so close that the kernel leaves it to the library's root and divisions.
"""
from __future__ import annotations

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu


def _engine(ref, **kw):
    from moldyn_gb300.engine import Engine
    return Engine(precision="fp64", reference_order=ref, **kw)


def _system(n, seed, close=False):
    pos, vel, box = gs.fcc((11, 11, 11), jitter=0.05, seed=seed)
    keep = np.random.default_rng(seed).permutation(len(pos))[:n]
    pos, vel = pos[keep], vel[keep]
    if close:   # r^2 = 1e-34
        pos[0] = 0.0
        pos[1] = [1e-17, 0.0, 0.0]
    return pos, vel, box


def _close(out, st, tol=1e-12):
    scale = np.abs(st.force).max()
    assert np.abs(out["force"] - st.force).max() <= tol * scale
    for k, v in (("potential", st.potential), ("temp", st.temp)):
        assert np.abs(out[k] - v).max() <= tol * np.abs(v).max()


@pytest.mark.parametrize("ref", [True, False])
@pytest.mark.parametrize("n,close", [(4095, False), (4096, False), (4097, False), (4224, True), (5323, False)])
def test_forces_and_steps(oracle, ref, n, close):
    pos, vel, box = _system(n, n, close)
    st = oracle.OracleState([n], pos, vel, [1.0], box, oracle.pot_table(1, default=(1.0, 1.0)))
    st.update_force()
    e = _engine(ref)
    e.set_potential(0, 0, 1.0, 1.0)
    e.upload(np.zeros(n, dtype=np.uint16), pos, vel, [1.0], box)
    e.compute_forces()
    out = e.download()
    if ref:
        assert np.array_equal(out["force"], st.force)
        assert np.array_equal(out["potential"], st.potential) and np.array_equal(out["temp"], st.temp)
    else:
        _close(out, st)
    if close:
        e.close()
        return
    e.step(5, 0.004)      # four fused passes, then one that stores everything
    st.step(0.004, nsteps=5)
    out = e.download()
    e.close()
    if ref:
        for k, v in (("pos", st.pos), ("vel", st.vel), ("force", st.force), ("potential", st.potential),
                     ("temp", st.temp)):
            assert np.array_equal(out[k], v), k
    else:
        _close(out, st, 1e-10)


@pytest.mark.parametrize("ref", [True, False])
def test_two_types(oracle, ref):
    n = 4500
    pos, vel, box = _system(n, 7)
    ids = np.sort((np.random.default_rng(8).random(n) < 0.4).astype(np.uint16))
    pairs = {(0, 0): (1.0, 1.0), (0, 1): (0.95, 0.9), (1, 1): (0.9, 0.8)}
    st = oracle.OracleState([int((ids == 0).sum()), int((ids == 1).sum())], pos, vel, [1.0, 2.0], box,
                            oracle.pot_table(2, pairs))
    st.update_force()
    # a caller's order that mixes the types; the k-th atom of a type keeps its place among them
    perm = np.argsort(np.random.default_rng(9).random(n)) if not ref else np.argsort(
        np.concatenate([np.sort(np.random.default_rng(9).random(c)) for c in st.counts]), kind="stable")
    e = _engine(ref)
    for (a, b), (s, ep) in pairs.items():
        e.set_potential(a, b, s, ep)
    e.upload(ids[perm], pos[perm], vel[perm], [1.0, 2.0], box)
    e.compute_forces()
    out = e.download()
    e.close()
    st.force, st.potential, st.temp = st.force[perm], st.potential[perm], st.temp[perm]
    if ref:
        assert np.array_equal(out["force"], st.force)
        assert np.array_equal(out["potential"], st.potential) and np.array_equal(out["temp"], st.temp)
    else:
        _close(out, st)


def test_ensemble_with_a_brute_replica(oracle):
    """Hot and cold replicas (their lists rebuild at different steps) and one
    whose box holds fewer than three cells a side."""
    systems = [gs.fcc((8, 8, 8), jitter=0.03, seed=21, t_star=4.0), gs.fcc((4, 4, 4), jitter=0.03, seed=22),
               gs.fcc((9, 8, 7), rho=0.6, jitter=0.03, seed=23, t_star=0.1),
               gs.fcc((6, 6, 7), jitter=0.03, seed=24, t_star=1.5)]
    offs = np.cumsum([0] + [len(s[0]) for s in systems])
    assert offs[-1] >= 4096
    e = _engine(True)
    e.set_potential(0, 0, 1.0, 1.0)
    e.upload_ensemble(offs, np.zeros(offs[-1], dtype=np.uint16), np.concatenate([s[0] for s in systems]),
                      np.concatenate([s[1] for s in systems]), [1.0], np.array([s[2] for s in systems]))
    e.compute_forces()
    e.ensemble_step(30, 0.004)
    out = e.download()
    e.close()
    for r, (pos, vel, box) in enumerate(systems):
        st = oracle.OracleState([len(pos)], pos, vel, [1.0], box, oracle.pot_table(1, default=(1.0, 1.0)))
        st.update_force()
        st.step(0.004, nsteps=30)
        sl = slice(offs[r], offs[r + 1])
        for k, v in (("pos", st.pos), ("vel", st.vel), ("force", st.force), ("potential", st.potential)):
            assert np.array_equal(out[k][sl], v), (r, k)
