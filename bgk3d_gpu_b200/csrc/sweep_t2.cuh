// Two time steps in one pass over memory, two-lattice (A -> B) pattern of the
// 4- and 8-byte kinds on library-owned lattices.
//
// The one-step sweep of these kinds runs at the copy bandwidth of HBM (FP32
// 0.95, FP64 1.0 of measured at 256^3), so it can only get faster by moving
// the populations less often.  Here a block owns a tile of tx x ty columns and
// marches along z: per plane it advances the tile and a rim of one node by the
// first step into a ring of planes in shared memory, and the tile one plane
// behind by the second step from the ring into b.  Per two updates a node is
// read once and written once, plus the rims, which neighbouring blocks read at
// about the same time (DRAM reads 1.03x the algorithmic bytes at 256x256x128).
// The state in between is rounded to storage precision, so the results are bit
// for bit those of two one-step launches, every face and obstacle included.
//
// What bounds it now is instruction issue (FP32 256x256x128: 486
// thread-instructions per update, rims included, 75 % of the issue slots, DRAM at
// half its rate).  What the layout rests on, each measured at 256^3:
//  * a thread reads the 19 values of the next plane straight into registers
//    before its second step, so that the loads are in flight while it works;
//    rows staged through shared memory instead, by bulk copies or tensor boxes,
//    ran 34-44 GLUPS against 57 (the copies' issue and a plane's exposed
//    latency);
//  * the ring keeps only the planes the second step pulls from: three of the
//    populations with c_z = +1, two with 0, one with -1 (two where links bounce
//    back).  Most of the 256 KB stays L1, whose size bounds the loads in
//    flight: a ring over all of shared memory ran at 27 GLUPS;
//  * two blocks per SM, so that one works while the other waits: 57 against 51
//    for one block of twice the size.  FP32 11 warps (76-80 registers) 59.0, 13
//    warps 57.4, 16 warps (at most 64) 52.6; FP64 6 warps (146-160 registers)
//    31.0, 5 warps x 3 blocks 30.4, 8 warps 28.0;
//  * split barriers: a warp arrives when its plane is stored or read and waits
//    only before it needs the others' (59.0 -> 59.6 FP32, 48.3 -> 56.6 FP32
//    inflow, whose edge warps work longest).
// One FP32 pair per thread (packed arithmetic) left too few warps: 27-44.
// Library lattices, before -> after: 256^3 FP32 periodic 40.3 -> 55.3 GLUPS,
// driven 39.1 -> 52.3, channel 38.8 -> 50.2, inflow with a sphere 36.9 -> 44.2;
// FP64 periodic 21.7 -> 29.1, driven 21.5 -> 28.5; 128^3 FP32 periodic 38.7 ->
// 49.9, driven 38.0 -> 44.8, FP64 driven 20.6 -> 26.2.
#pragma once
#include <cmath>
#include <type_traits>
#include "sweep_ab.cuh"

namespace bgk {

// Block shape per compute type: warps of a block, resident blocks per SM, widest tile.
template <class C> struct T2Cfg { static constexpr int WARPS = 11, BLOCKS = 2, TX = 32; };
template <> struct T2Cfg<double> { static constexpr int WARPS = 6, BLOCKS = 2, TX = 16; };

// Tiles of one launch: tx x ty nodes (edge tiles smaller), chunks of zc planes.
struct T2Tiles {
    int tx, ty, ntx, nty, zc;
};
// Kernel arguments: src[d] = a[d] moved by -c_d, so that a node's own element
// offset finds the value it pulls.
template <class S, class C> struct T2Args {
    SweepArgs<S, C> s;
    const S* src[19];
    int* err;                // set when a wait inside a block gives up
    const uint32_t* links;   // with an obstacle: t2_links_kernel's table
    T2Tiles g;
};

__host__ __device__ constexpr int t2_class(int d) { return cz_of(d) == 1 ? 0 : (cz_of(d) == 0 ? 1 : 2); }
__host__ __device__ constexpr int t2_index(int d) {   // number of lower populations of d's class
    int n = 0;
    for (int e = 0; e < d; ++e) n += t2_class(e) == t2_class(d) ? 1 : 0;
    return n;
}

// Populations with c_axis = sign, as bits.
__host__ __device__ constexpr uint32_t t2_mask(int axis, int sign) {
    uint32_t b = 0;
    for (int d = 0; d < 18; ++d)
        if ((axis == 0 ? cx_of(d) : (axis == 1 ? cy_of(d) : cz_of(d))) == sign) b |= 1u << d;
    return b;
}

// The ring of planes of the state in between, in shared memory: row stride W;
// RP / RZ / RM planes of the populations with c_z = +1 / 0 / -1.
template <class S, class C, int BC, bool OBS> struct T2Lay {
    typedef Faces<BC> F;
    static constexpr bool BOUNCE = F::WX || F::WY || F::WZ || OBS;
    static constexpr int THREADS = 32 * T2Cfg<C>::WARPS, TX = T2Cfg<C>::TX, W = TX + 2;
    static constexpr int RP = 3, RZ = 2, RM = BOUNCE ? 2 : 1;
    static constexpr int SLOTS = 5 * RP + 9 * RZ + 5 * RM;
    static constexpr int H = THREADS / W;                // rows of the largest tile and its rim
    static constexpr int NPL = H * W;
    static constexpr int OZ = 5 * RP * NPL, OM = OZ + 9 * RZ * NPL;
    static constexpr int BYTES = SLOTS * NPL * (int)sizeof(S);
};

// How much longer than the others a block at a face or an obstacle takes (a
// part of a block's time), which the last blocks to run show: with it FP32
// driven 128^3 runs in two chunks instead of one, 102.9 -> 96.1 us per launch.
template <int BC> constexpr double t2_uneven(bool obs) {
    return (BC == BC_PERIODIC ? 0.0 : 0.08) + (obs ? 0.5 : 0.0);
}

// The tiles of an l x m x n lattice (rows: of the largest tile and its rim;
// slots: blocks that run at a time).  The widest and highest tile was the
// fastest at every size tried (less of a plane is rim), so only the chunk
// length is chosen: short chunks repeat more planes (two per chunk) and fill
// more often, long ones leave slots idle at the end.  The cost counts nodes,
// 250 per plane and 500 per block for what does not depend on them, and runs
// of blocks with a part `idle` of the idle share of the last one (FP32 0.5,
// whose blocks end more unevenly, FP64 0.85).  Against all chunk
// lengths at nine sizes from 80^3 to 256^3 (FP32 and FP64, periodic and
// driven): 0.7 % (FP32) and 0.1 % (FP64) off the fastest on average, 3.6 % at most.
inline T2Tiles t2_tiles(int l, int m, int n, int txmax, int rows, int slots, double uneven, double idle) {
    T2Tiles g;
    g.ntx = (l + txmax - 1) / txmax;
    g.tx = (l + g.ntx - 1) / g.ntx;
    g.nty = (m + rows - 3) / (rows - 2);
    g.ty = (m + g.nty - 1) / g.nty;
    g.nty = (m + g.ty - 1) / g.ty;
    const long long tiles = (long long)g.ntx * g.nty;
    const double n1 = (g.tx + 2) * (g.ty + 2) + 250.0, n2 = g.tx * g.ty + 250.0;
    double cost = 0;
    g.zc = 0;
    for (long long nz = 1; nz <= n && (nz == 1 || (nz - 1) * tiles < 10LL * slots); ++nz) {
        const int zc = (int)((n + nz - 1) / nz);
        const double w = (double)(tiles * ((n + zc - 1) / zc)) / slots, up = std::ceil(w);
        const double c = (w <= 1.0 ? 1.0 + uneven : w + idle * (up - w) + uneven) * ((zc + 2) * n1 + zc * n2 + 500.0);
        if (g.zc == 0 || c < cost) { cost = c; g.zc = zc; }
    }
    return g;
}

// Loads (at a byte offset) that stay where they are written, ahead of the work that hides them.
__device__ __forceinline__ float t2_ld(const float* p, uint32_t off) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(reinterpret_cast<const char*>(p) + off));
    return v;
}
__device__ __forceinline__ double t2_ld(const double* p, uint32_t off) {
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(reinterpret_cast<const char*>(p) + off));
    return v;
}

// Split barriers of a block in shared memory (one arrival per warp): a warp
// arrives when it is done and waits only where it needs the others.
__device__ __forceinline__ void t2_arrive(uint32_t bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// (err is set when a wait gives up; the kernel then runs to its end)
__device__ __forceinline__ void t2_wait(uint32_t bar, uint32_t parity, int* err) {
    uint32_t ok = 0;
    for (int it = 0; it < (1 << 20) && !ok; ++it)
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    if (!ok) *err = 1;
}

// The table of solid links over the obstacle's box grown by one node (i
// fastest): obstacle_links of every node, made once per obstacle, so that a
// sweep reads one word per node near it instead of 19 mask entries.
static __global__ void t2_links_kernel(const SweepArgs<float, float> P, uint32_t* out) {
    const int bx = P.imax - P.imin + 3, by = P.jmax - P.jmin + 3, bz = P.kmax - P.kmin + 3;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)bx * by * bz) return;
    out[t] = obstacle_links(P, P.imin - 1 + (int)(t % bx), P.jmin - 1 + (int)((t / bx) % by), P.kmin - 1 + (int)(t / ((long long)bx * by)));
}

template <class S, class C, int BC, int CM, bool OBS>
__global__ void __launch_bounds__(32 * T2Cfg<C>::WARPS, T2Cfg<C>::BLOCKS) sweep_t2_kernel(const __grid_constant__ T2Args<S, C> Q) {
    typedef Faces<BC> F;
    typedef T2Lay<S, C, BC, OBS> R;
    const SweepArgs<S, C>& P = Q.s;
    const T2Tiles& G = Q.g;
    constexpr int NPL = R::NPL, W = R::W;
    extern __shared__ __align__(16) unsigned char t2_raw[];
    __shared__ unsigned long long t2_bars[2];
    const uint32_t done = (uint32_t)__cvta_generic_to_shared(t2_bars), freed = done + 8;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(done), "n"(T2Cfg<C>::WARPS) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(freed), "n"(T2Cfg<C>::WARPS) : "memory");
    }
    __syncthreads();
    S* const sm = reinterpret_cast<S*>(t2_raw);

    const int tiles = G.ntx * G.nty;
    const int zchunk = (int)blockIdx.x / tiles, tile = (int)blockIdx.x - zchunk * tiles;
    const int tj = tile / G.ntx, ti = tile - tj * G.ntx;
    const int i0 = ti * G.tx + 1, j0 = tj * G.ty + 1;
    const int tx = min(G.tx, P.l - i0 + 1), ty = min(G.ty, P.m - j0 + 1), rows = ty + 2;
    const int kb = zchunk * G.zc + 1, ke = min(kb + G.zc - 1, P.n);
    const int nx = (int)P.nx, nxy = (int)P.nxy;
    const int tid = (int)threadIdx.x;
    // planes of the state in between: kb - 1 .. ke + 1, inside the lattice where z does not wrap
    const int qa = F::PZ ? kb - 1 : max(kb - 1, 1), qb = F::PZ ? ke + 1 : min(ke + 1, P.n);
    auto wrap_z = [&](int k) { return F::PZ ? (k < 1 ? k + P.n : (k > P.n ? k - P.n : k)) : k; };

    // first step: this thread's node of the tile and its rim (s1: its place in
    // a plane of the ring, c1: its byte offset in plane 0); second step: its
    // node of the tile (s2, o2).  A thread without a node repeats the tile's
    // first one.  at: the faces the nodes lie on (bits 0..3: i = 1, i = l, j = 1,
    // j = m of the first step's node, 4..7 of the second's); w1, w2: the links
    // that bounce back at x and y walls.
    constexpr uint32_t ES = sizeof(S);
    int s1, s2;
    uint32_t c1, o2, at, w1, w2;
    auto face_bits = [&](int i, int j) { return (i == 1 ? 1u : 0u) | (i == P.l ? 2u : 0u) | (j == 1 ? 4u : 0u) | (j == P.m ? 8u : 0u); };
    auto wall_links = [&](uint32_t f) {
        return (F::WX ? ((f & 1u) ? t2_mask(0, 1) : 0u) | ((f & 2u) ? t2_mask(0, -1) : 0u) : 0u) |
               (F::WY ? ((f & 4u) ? t2_mask(1, 1) : 0u) | ((f & 8u) ? t2_mask(1, -1) : 0u) : 0u);
    };
    {
        const int y = tid / (tx + 2), x = tid - y * (tx + 2);
        int i = i0 - 1 + x, j = j0 - 1 + y;
        bool ok = y < rows;
        if (F::PX) i = i < 1 ? i + P.l : (i > P.l ? i - P.l : i); else ok = ok && i >= 1 && i <= P.l;
        if (F::PY) j = j < 1 ? j + P.m : (j > P.m ? j - P.m : j); else ok = ok && j >= 1 && j <= P.m;
        if (!ok) { i = i0; j = j0; }
        s1 = ok ? y * W + x : W + 1;
        c1 = (uint32_t)(nx * j + i) * ES;
        at = face_bits(i, j);
        w1 = wall_links(at);
        const int y2 = tid / tx, x2 = tid - y2 * tx;
        const bool ok2 = y2 < ty;
        i = i0 + (ok2 ? x2 : 0);
        j = j0 + (ok2 ? y2 : 0);
        s2 = (j - j0 + 1) * W + i - i0 + 1;
        o2 = (uint32_t)(nx * j + i) * ES;
        at |= face_bits(i, j) << 4;
        w2 = wall_links(at >> 4);
    }
    const uint32_t cz1 = (uint32_t)nxy * ES;
    const bool warp2 = (tid & ~31) < tx * ty;
    // the tile with its rim reaches x / y faces that wrap, bounce back or carry the inflow and outflow
    const bool xface = i0 <= 2 || i0 + tx >= P.l, yface = j0 <= 2 || j0 + ty >= P.m;
    const bool wraps = (F::PX && xface) || (F::PY && yface), walls = (F::WX && xface) || (F::WY && yface);
    // nodes of the tile or its rim may have links into solid nodes; a rim that
    // wraps is the node at the axis' other end
    auto near = [](bool wrapping, int lo, int hi, int ext, int bmin, int bmax) {
        return (lo <= bmax + 1 && hi >= bmin - 1) || (wrapping && ((lo < 1 && bmax + 1 >= ext) || (hi > ext && bmin - 1 <= 1)));
    };
    const bool near_ij = OBS && P.obs != nullptr && near(F::PX, i0 - 1, i0 + tx, P.l, P.imin, P.imax) &&
                         near(F::PY, j0 - 1, j0 + ty, P.m, P.jmin, P.jmax);
    // plane k of the tile has links that may bounce back
    auto bouncing = [&](int k) {
        return R::BOUNCE && (walls || (F::WZ && (k == 1 || k == P.n)) || (OBS && near_ij && k >= P.kmin - 1 && k <= P.kmax + 1));
    };
    const float inv = P.inv_scale;
    // links that bounce back at a z wall
    auto z_links = [&](int k) { return F::WZ ? (k == 1 ? t2_mask(2, 1) : 0u) | (k == P.n ? t2_mask(2, -1) : 0u) : 0u; };
    // links into solid nodes (bit 31: a solid node) of the node at place p of
    // plane k, from the table over the obstacle's box grown by one node
    auto solid_links = [&](int p, int k) -> uint32_t {
        if (!OBS || !near_ij || k < P.kmin - 1 || k > P.kmax + 1) return 0;
        int i = i0 - 1 + p % W, j = j0 - 1 + p / W;
        if (F::PX) i = i < 1 ? i + P.l : (i > P.l ? i - P.l : i);
        if (F::PY) j = j < 1 ? j + P.m : (j > P.m ? j - P.m : j);
        i -= P.imin - 1; j -= P.jmin - 1;
        const int bx = P.imax - P.imin + 3, by = P.jmax - P.jmin + 3;
        if (i < 0 || i >= bx || j < 0 || j >= by) return 0;
        return __ldg(Q.links + (size_t)(k - P.kmin + 1) * (size_t)(bx * by) + (size_t)(bx * j + i));
    };
    // what a face does to a pulled value beyond the bounce: the lid, the inflow
    auto faced = [&](int d, C v, bool first_column, int k) -> C {
        if (BC == BC_DRIVEN && (d == 1 || d == 10) && k == P.n) v = roundtrip<S, C>(d == 1 ? v + P.lid_force : v - P.lid_force);
        if (BC == BC_INFLOW && cx_of(d) == 1 && first_column) v = Conv<S, C>::raw(P.inflow_s[d]);
        return v;
    };

    S x[19];                 // the values plane q pulls, loaded while the plane before is worked on
    uint32_t sl1 = 0;         // its links that bounce back (bit 31: solid node)
    uint32_t next1 = OBS ? solid_links(s1, wrap_z(qa)) : 0u;   // the solid ones of the plane to be pulled next
    auto pull_as = [&](int zq, auto wc, auto gc) {
        constexpr bool WRAP = decltype(wc)::value, GEN = decltype(gc)::value;
        const uint32_t c = c1 + cz1 * (uint32_t)zq;
        const uint32_t xm = (at & 1u) ? (uint32_t)P.l * ES : 0u, xp = (at & 2u) ? 0u - (uint32_t)P.l * ES : 0u;
        const uint32_t ym = (at & 4u) ? (uint32_t)(P.m * nx) * ES : 0u, yp = (at & 8u) ? 0u - (uint32_t)(P.m * nx) * ES : 0u;
        const uint32_t zm = (F::PZ && zq == 1) ? (uint32_t)P.n * cz1 : 0u, zp = (F::PZ && zq == P.n) ? 0u - (uint32_t)P.n * cz1 : 0u;
        sl1 = GEN ? w1 | z_links(zq) | next1 : 0u;
#pragma unroll
        for (int d = 0; d < 19; ++d) {
            const int cx = cx_of(d), cy = cy_of(d), cz = cz_of(d);
            uint32_t off = c;
            if (WRAP && F::PX && cx) off += cx == 1 ? xm : xp;
            if (WRAP && F::PY && cy) off += cy == 1 ? ym : yp;
            if (WRAP && F::PZ && cz) off += cz == 1 ? zm : zp;
            if (GEN && R::BOUNCE && d < 18) {
                const bool b = (sl1 >> d) & 1u;
                x[d] = t2_ld(b ? P.a[opp_of(d)] : Q.src[d], WRAP ? (b ? c : off) : c);
            } else {
                x[d] = t2_ld(Q.src[d], off);
            }
        }
    };
    auto pull = [&](int q) {
        const int zq = wrap_z(q);
        const bool w = wraps || (F::PZ && (zq == 1 || zq == P.n));
        if (bouncing(zq)) {
            pull_as(zq, std::integral_constant<bool, F::PX || F::PY || F::PZ>{}, std::true_type{});
        } else if ((F::PX || F::PY || F::PZ) && w) {
            pull_as(zq, std::true_type{}, std::false_type{});
        } else {
            pull_as(zq, std::false_type{}, std::false_type{});
        }
    };
    pull(qa);
    if (OBS && qa < qb) next1 = solid_links(s1, wrap_z(qa + 1));
    int rp = 0, rz = 0, rm = 0;      // ring position of the plane being written
    uint32_t par = 0;
    for (int q = qa; q <= ke + 1; ++q) {
        const uint32_t now2 = OBS ? solid_links(s2, q - 1) : 0u;     // of the node of the second step
        if (q <= qb) {
            const int zq = wrap_z(q);
            S* const wP = sm + rp * 5 * NPL + s1;
            S* const wZ = sm + R::OZ + rz * 9 * NPL + s1;
            S* const wM = sm + R::OM + rm * 5 * NPL + s1;
            auto put = [&](int d) { return (cz_of(d) == 1 ? wP : (cz_of(d) == 0 ? wZ : wM)) + t2_index(d) * NPL; };
            C v[19];
#pragma unroll
            for (int d = 0; d < 19; ++d) v[d] = Conv<S, C>::raw(x[d]);
            const bool solid = OBS && (sl1 & 0x80000000u);
            if ((BC == BC_DRIVEN && zq == P.n) || (BC == BC_INFLOW && xface)) {
#pragma unroll
                for (int d = 0; d < 18; ++d) v[d] = faced(d, v[d], at & 1u, zq);
            }
            auto xs = [&](int d) { return v[d]; };
            auto ys = [&](int d, C y) {
                if (d == 0 && q > qa) t2_wait(freed, par ^ 1u, Q.err);     // (its first store) the ring's oldest planes are free
                const S w = Conv<S, C>::pack(y);
                if (!OBS || !solid) *put(d) = w;
                if (BC == BC_INFLOW) v[d] = Conv<S, C>::raw(w);      // (population d has been read)
            };
            if constexpr (cm_fast(CM)) bgk_collide_fast_f<C, C, cm_generic(CM), Scaled<S>::value>(xs, xs, ys, P.fc, inv);
            else bgk_collide_f<C, C, cm_generic(CM), Scaled<S>::value>(xs, xs, ys, P.col, inv);
            if (BC == BC_INFLOW && i0 + tx > P.l && (at & 2u) && !solid) {
                // the tile holds the nodes i = l: the outflow plane of the state in between in its column l + 1
                C eq[5];
                outflow_eq<C, Scaled<S>::value>(v, P.inflow_cte1, P.col, inv, eq);
#pragma unroll
                for (int e = 0; e < 5; ++e) put(9 + e)[1] = Conv<S, C>::pack(eq[e]);
            }
        }
        t2_arrive(done);
        if (q < qb) pull(q + 1);
        if (OBS && q + 1 < qb) next1 = solid_links(s1, wrap_z(q + 2));
        t2_wait(done, par, Q.err);     // plane q of the state in between is complete
        const int k = q - 1;
        if (k >= kb && warp2) {
            // ring positions of planes k - 1, k, k + 1 (plane k + 1 was just written)
            const S* const fP = sm + (rp == 2 ? 0 : rp + 1) * 5 * NPL + s2;      // c_z = +1 of plane k - 1
            const S* const fZ = sm + R::OZ + (rz ^ 1) * 9 * NPL + s2;            // c_z =  0 of plane k
            const S* const fM = sm + R::OM + rm * 5 * NPL + s2;                  // c_z = -1 of plane k + 1
            C y[19];
#pragma unroll
            for (int d = 0; d < 19; ++d) {
                const int cx = cx_of(d), cy = cy_of(d), cz = cz_of(d);
                y[d] = Conv<S, C>::raw((cz == 1 ? fP : (cz == 0 ? fZ : fM))[t2_index(d) * NPL - cx - W * cy]);
            }
            bool solid = false;
            if (bouncing(k)) {
                const S* const oP = sm + (rp == 0 ? 2 : rp - 1) * 5 * NPL + s2;      // own plane, for bounced links
                const S* const oM = sm + R::OM + (rm ^ 1) * 5 * NPL + s2;
                const uint32_t sl = w2 | z_links(k) | now2;
                solid = (sl & 0x80000000u) != 0;
#pragma unroll
                for (int d = 0; d < 18; ++d) {
                    const int cz = cz_of(d);
                    if ((sl >> d) & 1u) y[d] = Conv<S, C>::raw((cz == 1 ? oM : (cz == 0 ? fZ : oP))[t2_index(opp_of(d)) * NPL]);
                }
            }
            if ((BC == BC_DRIVEN && k == P.n) || (BC == BC_INFLOW && xface)) {
#pragma unroll
                for (int d = 0; d < 18; ++d) y[d] = faced(d, y[d], at & 16u, k);
            }
            const uint32_t to = o2 + cz1 * (uint32_t)k;
            auto out = [&](int d) { return reinterpret_cast<S*>(reinterpret_cast<char*>(P.b[d]) + to); };
            auto xs = [&](int d) { return y[d]; };
            auto ys = [&](int d, C v) {
                const S w = Conv<S, C>::pack(v);
                if (!OBS || !solid) *out(d) = w;
                if (BC == BC_INFLOW) y[d] = Conv<S, C>::raw(w);
            };
            if constexpr (cm_fast(CM)) bgk_collide_fast_f<C, C, cm_generic(CM), Scaled<S>::value>(xs, xs, ys, P.fc, inv);
            else bgk_collide_f<C, C, cm_generic(CM), Scaled<S>::value>(xs, xs, ys, P.col, inv);
            if (BC == BC_INFLOW && i0 + tx > P.l && (at & 32u) && !solid) {
                // the next state's outflow plane
                C eq[5];
                outflow_eq<C, Scaled<S>::value>(y, P.inflow_cte1, P.col, inv, eq);
#pragma unroll
                for (int e = 0; e < 5; ++e) out(9 + e)[1] = Conv<S, C>::pack(eq[e]);
            }
        }
        t2_arrive(freed);
        par ^= 1u;
        rp = rp == 2 ? 0 : rp + 1;
        rz ^= 1;
        rm = R::RM == 2 ? rm ^ 1 : 0;
    }
}

}  // namespace bgk
