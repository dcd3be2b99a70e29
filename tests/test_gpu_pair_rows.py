"""Rows that the 16-bit pair kernels cut into segments of 16 or 8 lanes, so that
a warp holds pieces of several rows: bit-identical to the one-node kernels.
Row lengths around the segments' edges, rows whose last segment is partial,
lattices whose last warp is, and (inflow, obstacles, the driven cavity's
in-place step, which are cut only from a certain size) larger ones."""
import numpy as np
import pytest

from _cases import BCASE, CASE_PARAMS, OMEGA, SCALE, interior, random_state, sphere_mask

pytestmark = pytest.mark.gpu

SMALL = [(14, 7, 5), (16, 5, 3), (18, 5, 7), (30, 3, 5), (32, 5, 3), (34, 5, 3), (48, 7, 3), (72, 5, 5), (80, 3, 3),
         (82, 5, 3), (130, 3, 5), (144, 3, 3)]
LARGE = [(72, 53, 51), (144, 37, 41)]       # more than 148 x 28 whole warps, a quarter or more of the lanes idle


def _run(kind, case, shape, fast, pattern, on, steps, obs):
    from bgk3d_gpu_b200._lib import lib
    from bgk3d_gpu_b200.lattice import Lattice
    l, m, n = shape
    p = CASE_PARAMS[case]
    prev = lib().bgk_set_pair_kernels(1 if on else 0)
    try:
        lat = Lattice(l, m, n, kind=kind, bcase=BCASE[case], omega=OMEGA, scale=SCALE[kind], fast=fast,
                      pattern=pattern, lid_force=p.get("lid_force", 0.0), u_inflow=p.get("u_inflow", 0.0),
                      force_mode=p.get("force_mode", 0), force=p.get("force", (0.0, 0.0, 0.0)))
        if obs is not None:
            lat.set_obstacle(obs)
        lat.upload(random_state(l, m, n, kind, seed=l + m, scale=SCALE[kind]))
        lat.step(steps)
        out = interior(lat.download(), l, m, n)
        lat.close()
    finally:
        lib().bgk_set_pair_kernels(prev)
    return out


@pytest.mark.parametrize("pattern", ["ab", "aa"])
@pytest.mark.parametrize("case", ["driven", "periodic", "channel", "inflow"])
@pytest.mark.parametrize("kind,fast", [(2, True), (3, False)])
@pytest.mark.parametrize("sphere", [False, True])
def test_cut_rows_equal_one_node_kernels(pattern, case, kind, fast, sphere):
    for shape in ([] if sphere else SMALL) + LARGE:
        l, m, n = shape
        obs = sphere_mask(l, m, n, (l / 2, (m + 1) / 2, (n + 1) / 2), min(m, n) / 5) if sphere else None
        a = _run(kind, case, shape, fast, pattern, True, 6, obs)
        b = _run(kind, case, shape, fast, pattern, False, 6, obs)
        same = (a == b) if obs is None else (a == b) | (np.broadcast_to(obs, a.shape) != 0)
        assert same.all(), (shape, np.argwhere(~same)[:5].tolist())
