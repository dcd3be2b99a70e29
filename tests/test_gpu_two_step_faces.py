"""Two steps per launch with an obstacle one node away from the lattice's faces,
where the rims of the tiles that wrap around a periodic axis have links into
solid nodes, and runs that start at an odd step count: the same bits in every
array cell as single steps (which take the one-step sweep)."""
import functools

import numpy as np
import pytest

from _cases import BCASE, OMEGA, random_state

pytestmark = pytest.mark.gpu

SHAPES = {"periodic": (133, 130, 80), "channel": (101, 170, 100), "inflow": (150, 131, 101), "driven": (199, 150, 95)}
# where the obstacle's box lies along x, y, z: -1 starts at node 2, +1 ends at the last node but one, 0 inside
PLACES = [(-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1),
          (-1, -1, 0), (1, 1, 0), (-1, 1, -1), (1, -1, 1), (1, 1, 1), (-1, -1, -1)]


def solids_at(shape, place, seed=4):
    """Random solid nodes in a box of 12 x 9 x 7 nodes; its corners are solid."""
    rng = np.random.default_rng(seed)
    at = []
    for ext, size, p in zip(shape, (12, 9, 7), place):
        lo = {-1: 2, 0: ext // 2, 1: ext - size}[p]
        at.append(slice(lo - 1, lo - 1 + size))
    obs = np.zeros(shape[::-1], np.int32)
    box = rng.random((7, 9, 12)) < 0.5
    box[::6, ::8, ::11] = True
    obs[at[2], at[1], at[0]] = box
    return obs


@functools.lru_cache(maxsize=2)
def state(shape, kind):
    return random_state(*shape, kind, seed=shape[0] + kind)


def run(shape, kind, case, calls, obs=None, fast=False):
    from bgk3d_gpu_b200.lattice import Lattice
    from test_gpu_lattice import lattice_kwargs
    lat = Lattice(*shape, kind=kind, bcase=BCASE[case], omega=OMEGA, fast=fast, **lattice_kwargs(case))
    if obs is not None:
        lat.set_obstacle(obs)
    assert lat.uses_two_steps or kind == 4
    lat.upload(state(shape, kind))
    for c in calls:
        lat.step(c)
    out = lat.download()
    lat.close()
    return out


def differing(a, b):
    a, b = (x.view(np.uint64 if x.itemsize == 8 else np.uint32) for x in (a, b))
    return int((a != b).sum())


@pytest.mark.parametrize("case", ["periodic", "channel", "inflow", "driven"])
@pytest.mark.parametrize("place", PLACES)
def test_obstacle_one_node_from_the_faces(case, place):
    shape = SHAPES[case]
    obs = solids_at(shape, place)
    assert differing(run(shape, 1, case, (8,), obs), run(shape, 1, case, (1,) * 8, obs)) == 0


@pytest.mark.parametrize("case", ["periodic", "channel", "inflow"])
@pytest.mark.parametrize("kind,fast", [(0, False), (4, False), (1, True)])
@pytest.mark.parametrize("place", [(1, 1, 1), (-1, -1, -1)])
def test_obstacle_at_the_corners_every_kind(case, kind, fast, place):
    shape = SHAPES[case]
    obs = solids_at(shape, place)
    assert differing(run(shape, kind, case, (4,), obs, fast), run(shape, kind, case, (1,) * 4, obs, fast)) == 0


@pytest.mark.parametrize("case", ["periodic", "inflow"])
def test_batch_members_with_obstacles_at_the_faces(case):
    from bgk3d_gpu_b200.lattice import Batch, Lattice
    from test_gpu_lattice import lattice_kwargs
    shape = SHAPES[case]
    lats, want = [], []
    for place in [(0, 1, 0), (1, -1, 0)]:
        obs = solids_at(shape, place)
        lat = Lattice(*shape, kind=1, bcase=BCASE[case], omega=OMEGA, **lattice_kwargs(case))
        lat.set_obstacle(obs)
        lat.upload(random_state(*shape, 1, seed=shape[0] + 1))
        lats.append(lat)
        want.append(run(shape, 1, case, (1,) * 21, obs))
    batch = Batch(lats)
    batch.step(21)
    for lat, w in zip(lats, want):
        assert differing(lat.download(), w) == 0
    batch.close()
    for lat in lats:
        lat.close()


@pytest.mark.parametrize("case", ["periodic", "channel", "inflow", "driven"])
@pytest.mark.parametrize("calls", [(1, 8), (3, 4, 2), (1, 35)])
def test_runs_that_start_at_an_odd_step_count(case, calls):
    shape = SHAPES[case]
    obs = solids_at(shape, (0, 0, 0)) if case == "inflow" else None
    assert differing(run(shape, 1, case, calls, obs), run(shape, 1, case, (1,) * sum(calls), obs)) == 0


@pytest.mark.parametrize("case", ["periodic", "channel", "inflow", "driven"])
@pytest.mark.parametrize("shape", [(1000, 900, 1), (900, 1, 1100), (1, 200, 170), (2, 170, 200), (640, 900, 2), (3, 190, 180)])
def test_lattices_of_one_to_three_nodes_along_an_axis(case, shape):
    assert differing(run(shape, 1, case, (4, 5), None), run(shape, 1, case, (1,) * 9, None)) == 0
