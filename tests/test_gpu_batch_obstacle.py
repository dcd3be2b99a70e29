"""Obstacles replaced between the steps of a batch: the batch goes on with the
new ones, in its groups and in its members that take two steps per launch,
although the old masks' memory is freed and may be handed out again at the
same address.  Every member's state is that of the lattice stepped alone, in every
node outside the last obstacle (the nodes that it covers keep what they held in
either of the lattice's two sets of arrays, whose other set is one step back
after a single step and two after two steps per launch)."""
import numpy as np
import pytest

from _cases import BCASE, OMEGA, random_state, sphere_mask

pytestmark = pytest.mark.gpu

MEMBERS = [("periodic", (133, 130, 80)), ("channel", (40, 24, 20)), ("inflow", (150, 131, 101)), ("inflow", (40, 24, 20))]


def sphere(shape, part):
    l, m, n = shape
    return (l / 2, (m + 1) / 2, (n + 1) / 2), (min(m, n) * part / 2) ** 2


def members():
    from bgk3d_gpu_b200.lattice import Lattice
    from test_gpu_lattice import lattice_kwargs
    lats = []
    for q, (case, shape) in enumerate(MEMBERS):
        lat = Lattice(*shape, kind=1, bcase=BCASE[case], omega=OMEGA, **lattice_kwargs(case))
        lat.set_sphere(*sphere(shape, 0.5))
        lat.upload(random_state(*shape, 1, seed=q))
        lats.append(lat)
    return lats


def replace(lats, part, how):
    for lat, (_, shape) in zip(lats, MEMBERS):
        if how == "none":
            lat.set_obstacle(None)
        elif how == "sphere":
            lat.set_sphere(*sphere(shape, part))
        else:
            lat.set_obstacle(sphere_mask(*shape, *sphere(shape, part)))


@pytest.mark.parametrize("retained", [0, 1 << 30])
@pytest.mark.parametrize("resync", [False, True])
@pytest.mark.parametrize("how", ["sphere", "mask", "none"])
def test_obstacles_replaced_between_runs(how, resync, retained):
    """40 steps (graph), smaller obstacles, 40 steps, larger ones again, 5 steps."""
    from bgk3d_gpu_b200.lattice import Batch, set_retained_bytes
    set_retained_bytes(retained)
    try:
        alone, lats = members(), members()
        batch = Batch(lats)
        assert batch.two_step_members == 2
        for steps, part in ((40, 0.2), (40, 0.4), (5, None)):
            batch.step(steps)
            for lat in alone:
                for _ in range(steps):
                    lat.step(1)
            if part is not None:
                replace(alone, part, how)
                replace(lats, part, how)
                if resync:
                    batch.resync()
        for (case, shape), a, b in zip(MEMBERS, alone, lats):
            assert b.L.bgk_lattice_status(b.h) == 0
            same = a.download() == b.download()
            if how != "none":
                same[:, 1:-1, 1:-1, 1:-1] |= sphere_mask(*shape, *sphere(shape, 0.4)) == 1
            assert same.all(), f"{case} {shape}"
        batch.close()
        for lat in alone + lats:
            lat.close()
    finally:
        set_retained_bytes(0)
