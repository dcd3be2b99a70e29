"""Which calls take two steps per launch, and that the launches end without a
wait that gave up: the tests that compare such runs with single steps say
nothing where both take single steps."""
import numpy as np
import pytest

from _cases import BCASE, OMEGA, random_state, sphere_mask

pytestmark = pytest.mark.gpu

# above the lines of the dispatch, with and without an obstacle
LARGE = {"periodic": (133, 130, 80), "channel": (101, 170, 100), "driven": (199, 150, 95), "inflow": (150, 131, 101)}


def lattice(shape, case, kind=1, sphere=False, state=None, fast=False):
    from bgk3d_gpu_b200.lattice import Lattice
    from test_gpu_lattice import lattice_kwargs
    lat = Lattice(*shape, kind=kind, bcase=BCASE[case], omega=OMEGA, fast=fast, **lattice_kwargs(case))
    if sphere:
        l, m, n = shape
        lat.set_obstacle(sphere_mask(l, m, n, (l / 3, (m + 1) / 2, (n + 1) / 2), min(m, n) / 6))
    if state is not None:
        lat.upload(state)
    return lat


def status(lat):
    return lat.L.bgk_lattice_status(lat.h)


@pytest.mark.parametrize("sphere", [False, True])
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("case", sorted(LARGE))
def test_large_lattices_take_two_steps_per_launch(case, kind, sphere):
    """... and their states are those of single steps, bit for bit."""
    shape = LARGE[case]
    st0 = random_state(*shape, kind, seed=7)
    a, b = (lattice(shape, case, kind, sphere, st0) for _ in range(2))
    assert a.uses_two_steps
    a.step(5)
    for _ in range(5):
        b.step(1)
    assert status(a) == 0
    assert np.array_equal(a.download().view(np.uint8), b.download().view(np.uint8))
    a.close()
    b.close()


@pytest.mark.parametrize("case", sorted(LARGE))
def test_small_in_place_and_16_bit_lattices_take_single_steps(case):
    from bgk3d_gpu_b200.lattice import Lattice
    for kind, shape, pattern in [(1, (40, 40, 40), "ab"), (1, LARGE[case], "aa"), (2, LARGE[case], "ab"), (3, LARGE[case], "ab")]:
        lat = Lattice(*shape, kind=kind, bcase=BCASE[case], omega=OMEGA, pattern=pattern, scale=256.0 if kind == 2 else 1.0)
        assert not lat.uses_two_steps
        lat.close()


def test_switches_that_turn_two_steps_off():
    from bgk3d_gpu_b200._lib import lib
    lat = lattice(LARGE["periodic"], "periodic")
    assert lat.uses_two_steps
    lat.set_zhalo(1)
    assert not lat.uses_two_steps
    lat.set_zhalo(0)
    prev = lib().bgk_set_tma_kernels(1)
    try:
        assert lat.uses_two_steps != bool(lib().bgk_lattice_uses_tma(lat.h))
    finally:
        lib().bgk_set_tma_kernels(prev)
    lat.close()


def test_batches_count_their_two_step_members():
    from bgk3d_gpu_b200.lattice import Batch
    lats = [lattice(LARGE["periodic"], "periodic"), lattice((24, 20, 22), "channel"), lattice(LARGE["inflow"], "inflow", sphere=True)]
    batch = Batch(lats)
    assert batch.two_step_members == 2
    batch.step(20)
    assert [status(lat) for lat in lats] == [0, 0, 0]
    batch.set_config(2, 4)                       # the tile-queue form takes single steps
    assert batch.two_step_members == 0
    batch.close()
    for lat in lats:
        lat.close()


# shapes on both sides of the lines: (kind, case, shape, sphere, two steps per launch); each pair of
# neighbours differs in what the rule looks at
LINES = [
    (0, "periodic", (20, 95, 95), False, False), (0, "periodic", (38, 95, 95), False, True),       # nodes fill L2 or not
    (0, "driven", (24, 105, 100), False, False), (0, "driven", (128, 80, 80), False, True),
    (1, "driven", (96, 90, 90), False, False), (1, "driven", (100, 90, 80), False, True),           # rows end inside a sector
    (1, "driven", (128, 128, 128), True, False), (1, "driven", (128, 128, 128), False, True),      # obstacle
    (1, "channel", (104, 100, 78), True, False), (1, "channel", (101, 131, 67), True, True),
    (1, "periodic", (104, 90, 70), True, False), (1, "periodic", (104, 100, 120), True, True),
    (0, "driven", (128, 80, 80), True, False), (0, "driven", (128, 128, 128), True, True),
    (0, "driven", (34, 120, 120), True, True),                                                      # idle lanes
    (4, "periodic", (128, 128, 128), False, False), (4, "periodic", (40, 150, 110), False, True),   # mixed precision
    (4, "driven", (128, 200, 200), False, False), (4, "channel", (33, 140, 130), False, True),
    (4, "periodic", (40, 150, 110), True, False), (4, "inflow", (128, 130, 130), False, False),
    (4, "inflow", (34, 260, 161), False, True),
]


@pytest.mark.parametrize("kind,case,shape,sphere,two", LINES)
def test_lines_of_the_dispatch(kind, case, shape, sphere, two):
    """The route, and the same state as by single steps."""
    st0 = random_state(*shape, kind, seed=11)
    a, b = (lattice(shape, case, kind, sphere, st0) for _ in range(2))
    assert a.uses_two_steps == two
    a.step(6)
    for _ in range(6):
        b.step(1)
    assert status(a) == 0
    assert np.array_equal(a.download().view(np.uint8), b.download().view(np.uint8))
    if sphere:                                   # without it, what the open lattice takes
        a.set_obstacle(None)
        c = lattice(shape, case, kind)
        assert a.uses_two_steps == c.uses_two_steps
        c.close()
    a.close()
    b.close()


@pytest.mark.parametrize("kind,case,shape,part,fill,two", [
    (1, "driven", (128, 100, 90), 1.0, 0.3, True),       # porous: fluid nodes all over the box
    (1, "driven", (128, 100, 90), 0.4, 0.3, False),      # a body: below the line for obstacles
    (0, "periodic", (100, 70, 70), 0.8, 0.2, True), (0, "periodic", (128, 100, 90), 0.8, 1.0, False),   # a block
    (0, "inflow", (128, 90, 90), 0.8, 0.3, True), (4, "channel", (128, 100, 90), 1.0, 0.3, False),
])
def test_obstacles_by_their_share_of_the_lattice(kind, case, shape, part, fill, two):
    """Solid nodes at random in a part of every extent: the route, and the same fluid state as by single steps."""
    l, m, n = shape
    rng = np.random.default_rng(2)
    obs = np.zeros((n, m, l), np.int32)
    at = tuple(slice(1 + (e - 2 - int((e - 2) * part)) // 2, 1 + (e - 2 - int((e - 2) * part)) // 2 + int((e - 2) * part)) for e in (n, m, l))
    obs[at] = rng.random(obs[at].shape) < fill
    st0 = random_state(*shape, kind, seed=13)
    lats = [lattice(shape, case, kind, state=st0) for _ in range(2)]
    for lat in lats:
        lat.set_obstacle(obs)
        assert lat.uses_two_steps == two
    lats[0].step(6)
    for _ in range(6):
        lats[1].step(1)
    assert status(lats[0]) == 0
    a, b = (lat.download().view(np.uint8) for lat in lats)
    assert np.array_equal(a, b)
    for lat in lats:
        lat.close()


@pytest.mark.parametrize("kind,sphere", [(0, False), (1, False), (4, False), (0, True), (1, True), (4, True)])
def test_group_members_take_two_steps_earlier_than_lattices_alone(kind, sphere):
    """Members between the two lines: in rounds of four in a batch's groups, by
    single steps alone and as solo members; the same states, mixed precision
    with an obstacle included (inflow only)."""
    from bgk3d_gpu_b200.lattice import Batch
    specs = {0: [("driven", (72, 72, 72)), ("periodic", (20, 95, 95)), ("channel", (20, 95, 95))],
             1: [("driven", (96, 90, 90)), ("periodic", (20, 160, 110)), ("inflow", (128, 120, 110))],
             4: [("driven", (128, 90, 90)), ("periodic", (128, 80, 80)), ("inflow", (128, 120, 110))]}[kind]
    st = [random_state(*shape, kind, seed=17 + q) for q, (_, shape) in enumerate(specs)]
    alone, lats = ([lattice(shape, case, kind, sphere, s) for (case, shape), s in zip(specs, st)] for _ in range(2))
    batch = Batch(lats)
    members = batch.two_step_members
    assert members == (1 if kind == 4 and sphere else 3)
    assert sum(lat.uses_two_steps for lat in lats) < members
    batch.step(21)
    batch.set_solo(1)
    assert batch.two_step_members == sum(lat.uses_two_steps for lat in lats)
    batch.step(5)
    for a, b in zip(alone, lats):
        for _ in range(26):
            a.step(1)
        assert status(b) == 0
        assert np.array_equal(a.download().view(np.uint8), b.download().view(np.uint8))
    batch.close()
    for lat in alone + lats:
        lat.close()
