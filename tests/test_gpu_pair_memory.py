"""The FP64 path's pair records and the device's memory: they only save time, so
they leave at least half of the device to others and can be left out.  Which
pass runs shows in the kernels launched: a rebuild and a force pass are seven
with records (step kernel, two of the list, two of the records, terms, sums)
and four without.
"""
from __future__ import annotations

import numpy as np
import pytest

from tests import gpu_systems as gs

pytestmark = pytest.mark.gpu

WITH, WITHOUT = 7, 4


def hold_memory(share):
    """Device memory held until less than `share` of the device is free."""
    torch = pytest.importorskip("torch")
    free, total = torch.cuda.mem_get_info()
    return torch.empty(max(1, free - int(share * total)), dtype=torch.uint8, device="cuda")


def give_back():
    import torch
    torch.cuda.empty_cache()


def launches(e):
    n = e.stats().kernel_launches
    e.set_potential(0, 0, 1.0, 1.0)   # the next pass builds the lists
    e.compute_forces()
    return e.stats().kernel_launches - n


def liquid(cells=(11, 11, 11), seed=3):
    pos, vel, box = gs.fcc(cells, jitter=0.04, seed=seed)
    return np.zeros(len(pos), dtype=np.uint16), pos, vel, [1.0], box


def engine(**kw):
    from moldyn_gb300.engine import Engine
    e = Engine(precision="fp64", threads_per_atom=1, **kw)
    e.set_potential(0, 0, 1.0, 1.0)
    return e


def test_records_leave_half_of_the_device():
    e = engine()
    e.upload(*liquid())
    assert launches(e) == WITH
    e.close()
    held = hold_memory(0.45)
    try:
        e = engine()
        e.upload(*liquid())
        assert launches(e) == WITHOUT
        e.close()
    finally:
        del held
        give_back()


def test_records_can_be_left_out(oracle):
    state = liquid()
    e = engine(pair_records=False, reference_order=True)
    e.upload(*state)
    assert launches(e) == WITHOUT
    st = oracle.OracleState([len(state[0])], state[1], state[2], [1.0], state[4], oracle.pot_table(1, default=(1.0, 1.0)))
    st.update_force()
    assert np.array_equal(e.download()["force"], st.force)
    e.close()


def test_a_longer_list_is_given_the_records_memory():
    """A list that grows frees the records first; they come back for the new one."""
    types, pos, vel, mass, box = liquid()
    e = engine(neighbor_capacity=48)
    e.upload(types, pos, vel, mass, box)     # 77 entries an atom: grows at once
    assert e.stats().neighbor_capacity > 77
    assert launches(e) == WITH
    want = engine()
    want.upload(types, pos, vel, mass, box)
    want.compute_forces()
    a, b = e.download(), want.download()
    for k in ("force", "potential", "temp"):
        assert np.array_equal(a[k], b[k]), k
    e.close()
    want.close()


@pytest.mark.parametrize("how", ["another_upload", "a_longer_list"])
def test_lists_of_several_threads_per_atom_get_no_records(how):
    """Records that found no room at first, threads per atom tuned without them,
    then room: the lists stay in the tuned layout, which the pair kernels do not
    read."""
    from moldyn_gb300.engine import Engine
    types, pos, vel, mass, box = liquid()
    two = types.copy()
    two[::3] = 1
    e = Engine(precision="fp64", trace=True)   # (phases are traced: single launches, tuned at any size)
    for a, b in ((0, 0), (0, 1), (1, 1)):
        e.set_potential(a, b, 1.0, 1.0)
    held = hold_memory(0.45)
    try:
        if how == "another_upload":
            e.upload(two, pos, vel, [1.0, 1.0], box)
        else:
            e.upload(types, pos, vel, mass, box)
        e.compute_forces()
    finally:
        del held
        give_back()
    # (42 blocks of one thread per atom leave most of the chip idle)
    assert max(e.stats().class_threads_per_atom) > 1
    r_cut = 2.5
    if how == "another_upload":
        e.upload(types, pos, vel, mass, box)
    else:
        r_cut = 3.2
        e.set_potential_raw(0, 0, 1.0, 1.0, r_cut, 0.0)
        cap = e.stats().neighbor_capacity
    e.compute_forces()
    if how == "a_longer_list":
        assert e.stats().neighbor_capacity > cap
    want = engine(pair_records=False)
    if r_cut != 2.5:
        want.set_potential_raw(0, 0, 1.0, 1.0, r_cut, 0.0)
    want.upload(types, pos, vel, mass, box)
    want.compute_forces()
    a, b = e.download(), want.download()
    for k in ("force", "potential", "temp"):
        assert np.abs(a[k] - b[k]).max() <= 1e-12 * np.abs(b[k]).max(), k
    e.close()
    want.close()


def test_records_go_with_the_length_of_the_lists():
    """A gas of 1.4 entries an atom has no records; a liquid uploaded into the
    same engine has them, and a gas after it gives them back."""
    gas, dense = gs.fcc((11, 11, 11), rho=0.015, jitter=0.3, seed=4), gs.fcc((11, 11, 11), jitter=0.04, seed=3)
    types = np.zeros(len(gas[0]), dtype=np.uint16)
    e = engine()
    for (pos, vel, box), want in ((gas, WITHOUT), (dense, WITH), (gas, WITHOUT)):
        e.upload(types, pos, vel, [1.0], box)
        assert launches(e) == want
    e.close()
