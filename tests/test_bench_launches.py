"""bench.py's count of its launches follows the route the lattice takes, not its
pattern alone: a lattice without the array for two-step launches takes one step
per launch."""
import pytest


@pytest.mark.parametrize("start,steps,two,want", [
    (0, 100, False, 100), (0, 100, True, 50), (1, 100, True, 1 + 2 * 24 + 3), (3, 8, True, 4), (0, 7, True, 5), (5, 31, True, 17),
])
def test_launches_of_a_run(start, steps, two, want):
    import bench
    assert bench.step_launches(start, steps, two) == want
