"""Two steps per launch (bgk_lattice_step on AB lattices of the 4- and 8-byte
kinds that outgrow L2) against single steps, which take the one-step sweep:
the same bits in every array cell, halo and solid nodes included.  The sizes
lie above the dispatch's line; their rows, columns and planes leave ragged
tiles and chunks on every side."""
import numpy as np
import pytest

from _cases import BCASE, OMEGA, random_state

pytestmark = pytest.mark.gpu

# case -> extents: ragged tiles; rows narrower than a tile (both x faces in it)
SHAPES = {"periodic": [(133, 97, 49), (7, 150, 103)], "driven": [(199, 83, 61), (9, 211, 150)],
          "channel": [(101, 131, 67), (33, 140, 130)], "channel_const": [(161, 90, 75)],
          "inflow": [(150, 131, 101), (34, 260, 161)]}


def scattered_solids(l, m, n, seed):
    """Solid nodes scattered over a box inside the lattice: every combination of solid links."""
    rng = np.random.default_rng(seed)
    obs = np.zeros((n, m, l), np.int32)
    k, j, i = (slice(s // 4, max(s // 2, s // 4 + 2)) for s in (n, m, l))
    obs[k, j, i] = rng.random(obs[k, j, i].shape) < 0.3
    return obs


def both(l, m, n, kind, case, steps, fast=False, obs=None):
    from bgk3d_gpu_b200.lattice import Lattice
    from test_gpu_lattice import lattice_kwargs
    st0 = random_state(l, m, n, kind, seed=l + kind)
    out = []
    for at_once in (True, False):
        lat = Lattice(l, m, n, kind=kind, bcase=BCASE[case], omega=OMEGA, fast=fast, **lattice_kwargs(case))
        if obs is not None:
            lat.set_obstacle(obs)
        lat.upload(st0)
        if at_once:
            lat.step(steps)
        else:
            for _ in range(steps):
                lat.step(1)
        out.append((lat.download(), lat.moments(), lat.steps))
        lat.close()
    return out


def assert_same(out, what):
    (a, ma, sa), (b, mb, sb) = out
    assert sa == sb
    assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), f"{what}: {(a != b).sum()} values differ"
    assert np.array_equal(ma, mb)


@pytest.mark.parametrize("kind", [0, 1, 4])
@pytest.mark.parametrize("case,shape", [(c, s) for c, ss in SHAPES.items() for s in ss])
def test_two_steps_per_launch_are_single_steps(case, shape, kind):
    assert_same(both(*shape, kind, case, steps=7), f"{case} {shape} kind={kind}")


@pytest.mark.parametrize("case", ["periodic", "driven", "channel", "inflow"])
@pytest.mark.parametrize("kind,fast", [(0, False), (1, False), (1, True)])
def test_two_steps_per_launch_with_solid_nodes(case, kind, fast):
    l, m, n = SHAPES[case][0]
    assert_same(both(l, m, n, kind, case, steps=6, fast=fast, obs=scattered_solids(l, m, n, 5)), f"{case} kind={kind} fast={fast}")


@pytest.mark.parametrize("case", ["periodic", "inflow"])
def test_graph_of_two_step_launches(case):
    """37 steps: a single step to an even count does not occur, two graph replays and a remainder of five."""
    assert_same(both(*SHAPES[case][0], 1, case, steps=37, fast=True), case)


@pytest.mark.parametrize("steps", [5, 23])
def test_batch_members_that_take_two_steps_per_launch(steps):
    """A batch of members above and below the dispatch's line, stepped plainly
    (5: a round of four and one) and through its graph (23: two replays, a
    round and three), against every lattice stepped alone by single steps."""
    from bgk3d_gpu_b200.lattice import Batch, Lattice
    from test_gpu_lattice import lattice_kwargs
    specs = [("periodic", (133, 97, 49)), ("channel", (20, 18, 16)), ("driven", (199, 83, 61)), ("channel", (101, 131, 67)),
             ("inflow", (150, 131, 101)), ("periodic", (24, 20, 22))]
    lats = {True: [], False: []}
    for q, (case, (l, m, n)) in enumerate(specs):
        st0 = random_state(l, m, n, 1, seed=q)
        for alone in (True, False):
            lat = Lattice(l, m, n, kind=1, bcase=BCASE[case], omega=OMEGA, **lattice_kwargs(case))
            if case == "inflow":
                lat.set_obstacle(scattered_solids(l, m, n, 9))
            lat.upload(st0)
            lats[alone].append(lat)
    batch = Batch(lats[False])
    batch.step(steps)
    for lat in lats[True]:
        for _ in range(steps):
            lat.step(1)
    for (case, shape), a, b in zip(specs, lats[True], lats[False]):
        assert a.steps == b.steps
        assert np.array_equal(a.download(), b.download()), f"{case} {shape}"
    batch.close()
    for lat in lats[True] + lats[False]:
        lat.close()


def test_batch_member_changed_after_the_batch_was_made():
    """Groups keep to the parameters their members had when the batch was made;
    a member that would take four steps at a time does the same, whether the
    steps run in rounds of four or one by one."""
    from bgk3d_gpu_b200.lattice import Batch, Lattice
    l, m, n = 133, 97, 49
    st0 = random_state(l, m, n, 1, seed=3)
    out = []
    for calls in ((7,), (1,) * 7):
        lats = [Lattice(l, m, n, kind=1, bcase=BCASE["periodic"], omega=OMEGA) for _ in range(2)]
        for lat in lats:
            lat.upload(st0)
        batch = Batch(lats)
        lats[0].L.bgk_lattice_set_omega(lats[0].h, OMEGA * 0.9)
        for c in calls:
            batch.step(c)
        out.append([lat.download() for lat in lats])
        batch.close()
        for lat in lats:
            lat.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert np.array_equal(out[0][0], out[0][1])
