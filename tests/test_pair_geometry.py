"""The launch geometry of the 16-bit pair kernels and the tiles of the two-step
sweep, taken from the compiled rules themselves (row_lanes and pair_geometry of
csrc/host_args.cuh, t2_tiles of csrc/sweep_t2.cuh in a host program): every pair
of every row belongs to exactly one lane, whose segment lies in one row, cutting
never takes more warps, and the tiles cover every node once within the ring."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "host_args.cuh"
#include "sweep_t2.cuh"
using namespace bgk;
int main() {
    SweepArgs<__half, float> A{};
    const int sides[] = {2, 14, 16, 18, 30, 34, 40, 48, 62, 64, 66, 72, 80, 96, 98, 100, 128, 130, 144, 200, 256, 258};
    const int rows[][2] = {{1, 1}, {7, 5}, {53, 51}, {96, 96}};
    for (int l : sides)
        for (auto& r : rows)
            for (int bc : {BC_DRIVEN, BC_PERIODIC, BC_INFLOW})
                for (int f = 0; f < 4; ++f)
                    for (int nsm : {148, 20}) {
                        A.l = l; A.m = r[0]; A.n = r[1]; A.bcase = bc;
                        const long long w = pair_geometry(A, f & 1, f & 2, nsm);
                        std::printf("P %d %d %d %d %d %d %d %d %d %lld\n", l, r[0], r[1], bc, f, nsm, A.gs, A.lmask, A.nseg, w);
                    }
    for (int l : {1, 7, 16, 17, 33, 100, 199, 256})
        for (int m : {1, 5, 8, 9, 83, 131})
            for (int n : {1, 2, 61, 128})
                for (int wide : {0, 1})
                    for (int slots : {40, 296}) {
                        const int txmax = wide ? T2Cfg<float>::TX : T2Cfg<double>::TX;
                        const int H = wide ? T2Lay<float, float, BC_PERIODIC, false>::H : T2Lay<double, double, BC_PERIODIC, false>::H;
                        const T2Tiles g = t2_tiles(l, m, n, txmax, H, slots, wide ? 0.0 : 0.58, 0.5);
                        std::printf("T %d %d %d %d %d %d %d %d %d %d %d\n", l, m, n, txmax, H, slots, g.tx, g.ty, g.ntx, g.nty, g.zc);
                    }
}
"""


@pytest.fixture(scope="module")
def printed(tmp_path_factory):
    d = tmp_path_factory.mktemp("geometry")
    src, exe = d / "geometry.cu", d / "geometry"
    src.write_text(PROGRAM)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "bgk3d_gpu_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    return [(x[0], [int(v) for v in x[1:].split()]) for x in out if x]


def test_every_pair_has_one_lane(printed):
    seen_gs = set()
    for l, m, n, bc, f, nsm, gs, lmask, nseg, warps in (v for k, v in printed if k == "P"):
        pairs, lanes = l // 2, 1 << gs
        assert gs in (3, 4, 5) and lmask == lanes - 1
        assert (nseg - 1) * lanes < pairs <= nseg * lanes          # a segment's lanes lie in one row
        assert (warps - 1) * (32 >> gs) < nseg * m * n <= warps * (32 >> gs)
        assert warps <= (pairs + 31) // 32 * m * n
        whole = (pairs + 31) // 32 * m * n <= nsm * 28             # whole warps that all run at a time
        if whole and (f or bc == 3):
            assert gs == 5
        seen_gs.add(gs)
        if warps > 400:
            continue
        seen = set()
        for t in range(warps * 32):                                 # the kernels' lane arithmetic
            gw, lane = divmod(t, 32)
            row, seg = divmod((gw << (5 - gs)) + (lane >> gs), nseg)
            i0 = 2 * ((seg << gs) + (lane & lmask)) + 1
            if row < m * n and i0 < l:
                assert (row, i0) not in seen
                seen.add((row, i0))
        assert len(seen) == pairs * m * n
    assert seen_gs == {3, 4, 5}


def test_tiles_cover_the_lattice(printed):
    for l, m, n, txmax, H, slots, tx, ty, ntx, nty, zc in (v for k, v in printed if k == "T"):
        assert 1 <= tx <= txmax and 1 <= ty <= H - 2               # a tile and its rim fit the ring
        assert (ntx - 1) * tx < l <= ntx * tx
        assert (nty - 1) * ty < m <= nty * ty
        assert 1 <= zc <= n
