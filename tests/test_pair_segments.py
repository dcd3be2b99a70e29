"""The rows of the 16-bit pair kernels cut into segments of 32, 16 or 8 lanes,
checked on the CPU: row_lanes and pair_geometry (csrc/host_args.cuh) and the
lane arithmetic of the kernels (lane_segment, csrc/sweep_ab.cuh) restated.
Every pair of every row belongs to exactly one lane, the lanes of a segment to
one row, and cutting never takes more warps."""
import pytest


def row_lanes(pairs, fifth):
    best, lanes = 5, (pairs + 31) // 32 * 32
    for gs in (4, 3):
        w = 1 << gs
        n = (pairs + w - 1) // w * w
        if n * 10 <= lanes * (8 if fifth else 9):
            best, lanes = gs, n
    return best


@pytest.mark.parametrize("fifth", [False, True])
@pytest.mark.parametrize("m,n", [(1, 1), (5, 3), (7, 2)])
def test_every_pair_has_one_lane(m, n, fifth):
    for pairs in range(1, 140):
        gs = row_lanes(pairs, fifth)
        nseg, rows = (pairs + (1 << gs) - 1) >> gs, m * n
        warps = (nseg * rows + (32 >> gs) - 1) // (32 >> gs)
        assert warps <= (pairs + 31) // 32 * rows
        seen = {}
        for t in range(warps * 32):
            gw, lane = divmod(t, 32)
            sg = (gw << (5 - gs)) + (lane >> gs)
            row, seg = divmod(sg, nseg)
            i0 = 2 * ((seg << gs) + (lane & ((1 << gs) - 1))) + 1
            if row < rows and i0 < 2 * pairs:
                assert (row, i0) not in seen
                seen[(row, i0)] = t
                if lane & ((1 << gs) - 1):          # the lane below holds the pair to the left
                    assert seen[(row, i0 - 2)] == t - 1
        assert len(seen) == pairs * rows
