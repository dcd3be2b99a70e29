"""A batch whose members' parameters change: until bgk_batch_resync the members
keep to the parameters the batch was made or resynced with, in rounds of four
steps as in single steps; after it they take the new ones, and members large
enough go on taking two steps per launch."""
import numpy as np
import pytest

from _cases import BCASE, OMEGA, random_state

pytestmark = pytest.mark.gpu

MEMBERS = [("periodic", (133, 130, 80)), ("channel", (40, 24, 20)), ("inflow", (150, 131, 101))]


def members():
    from bgk3d_gpu_b200.lattice import Lattice
    from test_gpu_lattice import lattice_kwargs
    lats = []
    for q, (case, shape) in enumerate(MEMBERS):
        lat = Lattice(*shape, kind=1, bcase=BCASE[case], omega=OMEGA, **lattice_kwargs(case))
        lat.upload(random_state(*shape, 1, seed=q))
        lats.append(lat)
    return lats


def set_omega(lats, omega):
    for lat in lats:
        assert lat.L.bgk_lattice_set_omega(lat.h, omega) == 0


def same(alone, lats):
    for (case, shape), a, b in zip(MEMBERS, alone, lats):
        assert np.array_equal(a.download(), b.download()), f"{case} {shape}"
        a.close()
        b.close()


@pytest.mark.parametrize("steps", [7, 37])
def test_resync_takes_new_parameters_and_rounds_of_four(steps):
    from bgk3d_gpu_b200.lattice import Batch
    alone, lats = members(), members()
    batch = Batch(lats)
    batch.step(steps)
    for lat in alone:
        for _ in range(steps):
            lat.step(1)
    set_omega(alone + lats, 0.9 * OMEGA)
    batch.resync()
    assert batch.two_step_members == 2
    batch.step(steps)
    for lat in alone:
        for _ in range(steps):
            lat.step(1)
    batch.close()
    same(alone, lats)


@pytest.mark.parametrize("calls", [(7, 37), (1,) * 44])
def test_without_resync_the_parameters_stay(calls):
    from bgk3d_gpu_b200.lattice import Batch
    alone, lats = members(), members()
    batch = Batch(lats)
    batch.step(4)
    set_omega(lats, 0.9 * OMEGA)
    assert batch.two_step_members == 2
    for c in calls:
        batch.step(c)
    set_omega(lats, OMEGA)
    batch.step(5)
    for lat in alone:
        for _ in range(4 + sum(calls) + 5):
            lat.step(1)
    batch.close()
    same(alone, lats)


def test_solo_members_step_with_their_own_parameters():
    """Solo members' plain steps take a new relaxation frequency at once: in rounds of four as one by one."""
    from bgk3d_gpu_b200.lattice import Batch
    out = []
    for calls in ((7,), (1,) * 7):
        lats = members()
        batch = Batch(lats)
        batch.set_solo(1)
        assert batch.two_step_members == 2
        set_omega(lats, 0.9 * OMEGA)
        for c in calls:
            batch.step(c)
        batch.close()
        out.append(lats)
    same(*out)
