// Line-march stage kernels of the fast FP64 form.
//
// One block per SM: eight or twelve consumer warps (line_shape) and a producer
// thread whose warpgroup gives its registers up.  The producer streams the planes
// of U[tn] (the tile with the stencil's or the viscous halo) and of U[to] (the
// tile alone) into rings of shared-memory slots by TMA, one copy per variable,
// each variable at a fixed stride.  Y and Z sweeps: a consumer thread walks one
// grid line along the sweep axis; X sweeps march along y with a lane per node
// (stage_line_x).
//
// What bounds it: the FP64 pipe and the issue slots beside it.  Measured on
// B200: a scheduler issues an FP64 operation in two cycles (three for an FMA of
// three different registers, none of them shared with the operation before),
// and every other instruction takes about 0.75 of a cycle more.  A viscous
// WENO5 interface takes 651 FP64 and about 350 other instructions; at those
// costs a stage of TGV 128^3 cannot take less than about 100 us, and it takes
// 134 us on Y and Z and 148 us on X (187 and 198 us in the kernels before, 816
// FP64 instructions an interface and seven consumer warps on four schedulers;
// DRAM 310 MB, 35% of the copy bandwidth).
//  * WENO works on first differences (fast::weno5_departure).
//  * A node's velocity, total enthalpy, temperature and sqrt(rho) are computed
//    once with one reciprocal square root (1/rho = r^2, sqrt(rho) = rho r) and
//    carried to the next interface; the interface's sound speed and its
//    reciprocal come from one reciprocal square root too.  Both are refined
//    from the hardware's approximation by one third-order step, without the
//    branches of sqrt() and division, so that an interface is one basic block.
//  * The stencil is read from shared memory each time it is needed instead of
//    being held in registers: no window to shift, no spills.
//  * U[to] arrives with the planes instead of by loads inside the march, and
//    the node types are loaded a plane ahead.
// Measured and left out, on eight warps at 134 us: the loop unrolled twice (138
// us), the next interface's state computed beside the reconstruction (154 us), the
// acoustic field that runs downwind reconstructed on one side only (143 us: 5%
// fewer FP64 operations, but longer chains).
//
// The lines of a launch are cut as in the plane march (plane_next_item), by
// one compiled kernel for both forms, so that the results do not depend on
// how a launch is cut.
#pragma once

#include "sweep_plane.cuh"

namespace acfd {
namespace ACFD_NS {

namespace line {

// 1/sqrt(x) for positive normal x, from the hardware's approximation y by one step
// of the third-order iteration of Householder's family (A. S. Householder, The
// Numerical Treatment of a Single Nonlinear Equation, 1970): the binomial series
// of y (1 - e)^(-1/2), e = 1 - x y^2, up to e^2.  The instruction works in the
// 1.11.20 format, its result's lower 32 bits are zero: |d| < 2^-20 relative.  With
// e = -2 d the step leaves 5/16 |e|^3 < 2^-58, below the roundings: of x y into e
// (2^-54 in the result) and of the result (2^-53), 1.5 x 2^-53 in all
// (tests/test_gpu_line_roots.py).
__device__ __forceinline__ double rsqrt3(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-__dmul_rn(x, y), y, 1.0);
    return fma(fma(0.375, e, 0.5), __dmul_rn(y, e), y);
}

// 1/x for normal x and 1/x, the same way: the geometric series of y / (1 - e),
// e = 1 - x y (one rounding, of |e| < 2^-20), up to e^2; it leaves |e|^3 < 2^-60
// beside the result's rounding, 1.01 x 2^-53 in all.
__device__ __forceinline__ double rcp3(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// a node in the kernel's frame: velocities along x (or the first transverse
// axis), the march axis and the second transverse axis, total enthalpy,
// sqrt(rho), temperature
struct Node {
    double u, v, w, H, s, T;
};

// constants of the model and the mesh, formed once per thread (as operands from
// the kernel's parameters they made the viscous stage 5% slower)
struct Gas {
    double gamma, gm1, hgm1, cvinv;
    double refT, mu, heat;   // reference temperature, refMu 1.458e-6, gamma cv / 0.71
    double dds, q0, q2;      // 1/d along the sweep axis, 1/(4 d) along the transverse axes
    int roe, llf;
};

// s: the sweep axis, t0 and t2 the transverse axes of the kernel's frame
__device__ __forceinline__ Gas gas_of(const ModelParams &mp, const Grid &g, int t0, int s, int t2)
{
    Gas k;
    k.gamma = mp.gamma;
    k.gm1 = mp.gamma - 1.0;
    k.hgm1 = 0.5 * k.gm1;
    k.cvinv = 1.0 / mp.cv;
    k.refT = mp.refT;
    k.mu = mp.refMu * 1.458e-6;
    k.heat = mp.gamma * mp.cv / 0.71;
    k.dds = g.dd[s];
    k.q0 = 0.25 * g.dd[t0];
    k.q2 = 0.25 * g.dd[t2];
    k.roe = mp.jacobMean != 0;
    k.llf = mp.fluxSplit == 0;
    return k;
}

// Every operation is written out (no contraction left to the compiler): the
// node left of a segment's first interface takes these values in the
// segment's preamble, while the segment before it carries them from its march.
__device__ __forceinline__ Node node_of_state(const Gas &k, const double (&U)[5])
{
    Node n;
    const double r = rsqrt3(U[0]);
    const double ir = __dmul_rn(r, r);
    n.s = __dmul_rn(U[0], r);
    n.u = __dmul_rn(U[1], ir);
    n.v = __dmul_rn(U[2], ir);
    n.w = __dmul_rn(U[3], ir);
    const double e = __dmul_rn(U[4], ir);
    const double vv = fma(n.w, n.w, fma(n.v, n.v, __dmul_rn(n.u, n.u)));
    n.H = fma(k.gamma, e, -__dmul_rn(k.hgm1, vv));
    n.T = __dmul_rn(fma(-0.5, vv, e), k.cvinv);
    return n;
}

// central differences of the transverse velocity t and of the march velocity
// across a node, from the states at its two neighbours: one reciprocal of the
// product of their densities
__device__ __forceinline__ void across(double rp, double tp, double sp, double rm, double tm, double sm, double D[2])
{
    const double ir = rcp3(__dmul_rn(rp, rm));
    D[0] = __dmul_rn(fma(tp, rm, -__dmul_rn(tm, rp)), ir);
    D[1] = __dmul_rn(fma(sp, rm, -__dmul_rn(sm, rp)), ir);
}

// Roe (or arithmetic) state of an interface and the factors of its projection
struct Face {
    double V0, V1, V2, H, c, q, d, b;
    double lp[3], ln[3];  // split eigenvalues of V1 - c, V1, V1 + c
};

__device__ __forceinline__ Face face_of(const Gas &k, const Node &L, const Node &R)
{
    Face f;
    const double t = k.roe ? R.s * rcp3(L.s + R.s) : 0.5;
    f.V0 = fma(t, R.u - L.u, L.u);
    f.V1 = fma(t, R.v - L.v, L.v);
    f.V2 = fma(t, R.w - L.w, L.w);
    f.H = fma(t, R.H - L.H, L.H);
    f.q = 0.5 * fma(f.V2, f.V2, fma(f.V1, f.V1, f.V0 * f.V0));
    const double c2 = k.gm1 * (f.H - f.q);
    const double r = rsqrt3(c2);
    f.c = c2 * r;
    f.d = 0.5 * r;
    f.b = k.hgm1 * (r * r);
    const double lam[3] = {f.V1 - f.c, f.V1, f.V1 + f.c};
    if (k.llf) {
        const double ls = fabs(f.V1) + f.c;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            f.lp[i] = 0.5 * (lam[i] + ls);
            f.ln[i] = 0.5 * (lam[i] - ls);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double l2 = fma(lam[i], lam[i], 1.0e-6);
            const double sr = l2 * rsqrt3(l2);
            f.lp[i] = 0.5 * (lam[i] + sr);
            f.ln[i] = 0.5 * (lam[i] - sr);
        }
    }
    return f;
}

// WENO3 in first differences: the candidates are W[1] + {e_0, e_1} / 2 (+
// side) and W[2] - {e_2, e_1} / 2 (- side), the indicators the e^2
__device__ __forceinline__ double weno3_departure(double e0, double e1, double e2, double lp, double ln)
{
    const double eps = 1.0e-6;
    const double lp2 = lp * lp, ln2 = ln * ln;
    const double t0 = e0 * e0, t1 = e1 * e1, t2 = e2 * e2;
    double p0 = fma(lp2, t0, eps), p1 = fma(lp2, t1, eps);
    double m0 = fma(ln2, t2, eps), m1 = fma(ln2, t1, eps);
    p0 *= p0;
    p1 *= p1;
    m0 *= m0;
    m1 *= m1;
    // weights (1/3)/p0 and (2/3)/p1, both times 3 p0 p1
    const double Np = p1 * e0 + 2.0 * p0 * e1, Sp = p1 + 2.0 * p0;
    const double Nn = m1 * e2 + 2.0 * m0 * e1, Sn = m1 + 2.0 * m0;
    return 0.5 * (lp * Np * Sn - ln * Nn * Sp) * rcp3(Sp * Sn);
}

// Convective flux of an interface.  src(m, v): variable v of stencil node m
// (the interface lies between nodes NP/2-1 and NP/2), read from shared memory
// each time it is needed: the stencil of the five fields (30 values) is not
// held in registers, which leaves room for a third warp per scheduler.
template <int NP, class Src>
__device__ __forceinline__ void convective(const Face &f, const Src &src, double F[5])
{
    constexpr int M = NP - 1, c0 = NP / 2 - 1;  // difference c0 lies across the interface
    // projections A = q U0 - V.U + U4 and B = V_s U0 - U_s of the differences
    // of neighbouring nodes, and of the central values of the two sides
    // (WENO5: W[2] + e_1/2 and W[3] - e_3/2; WENO3: W[1] and W[2])
    double A[M], B[M], Ac[2], Bc[2];
    {
        // a variable at a time: neighbouring operations share the coefficient
        // (an FP64 FMA with three different registers takes three cycles of the
        // pipe, with one of them shared two)
        double a[NP], b[NP];
#pragma unroll
        for (int m = 0; m < NP; ++m) a[m] = src(m, 4);
#pragma unroll
        for (int m = 0; m < NP; ++m) {
            b[m] = src(m, 0);
            a[m] = fma(f.q, b[m], a[m]);
        }
#pragma unroll
        for (int m = 0; m < NP; ++m) a[m] = fma(-f.V0, src(m, 1), a[m]);
#pragma unroll
        for (int m = 0; m < NP; ++m) {
            const double us = src(m, 2);
            a[m] = fma(-f.V1, us, a[m]);
            b[m] = fma(f.V1, b[m], -us);
        }
#pragma unroll
        for (int m = 0; m < NP; ++m) a[m] = fma(-f.V2, src(m, 3), a[m]);
#pragma unroll
        for (int m = 0; m < M; ++m) {
            A[m] = a[m + 1] - a[m];
            B[m] = b[m + 1] - b[m];
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            Ac[q] = a[c0 + q];
            Bc[q] = b[c0 + q];
        }
    }
    auto central = [&](double (&c)[2], const double (&e)[M]) {
        if constexpr (NP == 6) {
            c[0] = fma(0.5, e[1], c[0]);
            c[1] = fma(-0.5, e[3], c[1]);
        }
    };
    central(Ac, A);
    central(Bc, B);
    auto side = [&](const double (&C)[M], double cp, double cn, double lp, double ln) {
        double dep;
        if constexpr (NP == 6) {
            dep = fast::weno5_departure<double>(C[0], C[1], C[2], C[3], C[4], lp, ln);
        } else {
            dep = weno3_departure(C[0], C[1], C[2], lp, ln);
        }
        return fma(lp, cp, fma(ln, cn, dep));
    };
    double G[5];
    {
        double C[M];
        const double dm = -f.d;
#pragma unroll
        for (int m = 0; m < M; ++m) C[m] = fma(f.d, B[m], f.b * A[m]);
        G[0] = side(C, fma(f.d, Bc[0], f.b * Ac[0]), fma(f.d, Bc[1], f.b * Ac[1]), f.lp[0], f.ln[0]);
#pragma unroll
        for (int m = 0; m < M; ++m) C[m] = fma(dm, B[m], f.b * A[m]);
        G[4] = side(C, fma(dm, Bc[0], f.b * Ac[0]), fma(dm, Bc[1], f.b * Ac[1]), f.lp[2], f.ln[2]);
    }
    const double b2 = -2.0 * f.b;
#pragma unroll
    for (int r = 1; r < 4; ++r) {
        const int v = r == 2 ? 0 : r;
        const double kr = r == 2 ? b2 : b2 * (r == 1 ? f.V0 : f.V2);
        double C[M], c[2], y0;
#pragma unroll
        for (int m = 0; m < NP; ++m) {
            const double y = src(m, v);
            if (m > 0) C[m - 1] = y - y0;
            if (m == c0 || m == c0 + 1) c[m - c0] = y;
            y0 = y;
        }
        central(c, C);
#pragma unroll
        for (int m = 0; m < M; ++m) C[m] = fma(kr, A[m], C[m]);
        G[r] = side(C, fma(kr, Ac[0], c[0]), fma(kr, Ac[1], c[1]), f.lp[1], f.ln[1]);
    }
    // F = R G by columns
    const double a = G[0] + G[4], z = G[4] - G[0];
    F[0] = a + G[2];
    F[1] = fma(f.V0, a, G[1]);
    F[2] = fma(f.V1, F[0], f.c * z);
    F[3] = fma(f.V2, a, G[3]);
    F[4] = fma(f.H, a, fma(f.V1 * f.c, z, fma(fma(f.V1, f.V1, -f.q), G[2], fma(f.V0, G[1], f.V2 * G[3]))));
}

// central viscous flux of an interface (x, march and second transverse
// momentum, energy)
__device__ __forceinline__ void viscous_part(const Gas &k, const Node &c, const Node &n, const double (&Dc)[2][2],
                                             const double (&Dn)[2][2], double Fv[4])
{
    const double g0s = (n.u - c.u) * k.dds, gss = (n.v - c.v) * k.dds, g2s = (n.w - c.w) * k.dds;
    const double g00 = (Dc[0][0] + Dn[0][0]) * k.q0, gs0 = (Dc[0][1] + Dn[0][1]) * k.q0;
    const double g22 = (Dc[1][0] + Dn[1][0]) * k.q2, gs2 = (Dc[1][1] + Dn[1][1]) * k.q2;
    const double Ts = 0.5 * (c.T + n.T) * k.refT;
    // T^1.5 as T^2 / sqrt(T) (the added constant keeps T = 0 at zero)
    const double mu = k.mu * (Ts * Ts) * rsqrt3(Ts + 1.0e-200) * rcp3(Ts + 110.4);
    const double div = gss + g00 + g22;
    const double ts = mu * fma(-2.0 / 3.0, div, 2.0 * gss);
    const double t0 = mu * (gs0 + g0s), t2 = mu * (gs2 + g2s);
    Fv[0] = t0;
    Fv[1] = ts;
    Fv[2] = t2;
    const double w = fma(t0, c.u + n.u, fma(ts, c.v + n.v, t2 * (c.w + n.w)));
    Fv[3] = fma(k.heat * mu, (n.T - c.T) * k.dds, 0.5 * w);
}

// rsqrt3 and rcp3 of count values (acfd_line_roots)
__global__ void roots(const double *x, double *rsqrt, double *rcp, int count)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= count) return;
    rsqrt[q] = rsqrt3(x[q]);
    rcp[q] = rcp3(x[q]);
}

}  // namespace line

template <int NP, bool VISC>
__global__ void __launch_bounds__(line_threads(line_shape(false, VISC)), 1)
stage_line(Grid g, ModelParams mp, StageArgs a, LineTile lt, const __grid_constant__ CUtensorMap map,
           const __grid_constant__ CUtensorMap omap)
{
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int S = 1, T2 = 2;
    constexpr int H = NP / 2;
    constexpr int hv = VISC ? 1 : 0;
    constexpr LineShape shape = line_shape(false, VISC);
    constexpr int NS = line_slots(false, NP, VISC), NO = shape.oslots;
    constexpr int PE = shape.plane, OE = shape.oplane;  // elements of a variable in a slot
    constexpr unsigned kAll = 0xffffffffu;
    const PlaneTile &pt = lt.pt;
    double *ring = reinterpret_cast<double *>(smem);
    double *oring = ring + (size_t)NS * 5 * PE;
    uint64_t *full = reinterpret_cast<uint64_t *>(oring + (size_t)NO * 5 * OE);
    uint64_t *empty = full + NS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int q = 0; q < NS; ++q) {
            tma::mbar_init(full + q, 1);
            tma::mbar_init(empty + q, shape.warps);
        }
    }
    __syncthreads();
    pdl_wait();

    const int Ls = g.hi[S] - g.lo[S];
    const long long tiles = (long long)pt.ntx * pt.ntc;
    const int blk = (int)blockIdx.x;
    long long r0 = 0, r1 = 1;
    if (pt.share) {
        plane_share(pt, Ls, tiles, blk, r0, r1);
        if (r1 <= r0) return;
    }
    auto next_item = [&](long long &w, int &x0, int &c0, int &p0, int &p1) {
        long long T;
        const bool more = pt.share ? plane_next_item<true>(pt, Ls, tiles, blk, r1, w, T, p0, p1)
                                   : plane_next_item<false>(pt, Ls, tiles, blk, r1, w, T, p0, p1);
        if (!more) return false;
        p0 += g.lo[S];
        p1 += g.lo[S];
        x0 = g.lo[0] + (int)(T % pt.ntx) * pt.WX;
        c0 = g.lo[T2] + (int)(T / pt.ntx) * pt.NR;
        return true;
    };
    const bool same_o = (a.Uo == a.Un);
    const bool use_o = !same_o && !a.accumulate;  // U[to] read at the node
    // variable v of the kernel's frame is variable vg(v) of the state
    const int o2 = pt.swap ? 3 : 2, o3 = pt.swap ? 2 : 3;
    auto vg = [&](int v) { return v == 2 ? o2 : (v == 3 ? o3 : v); };

    if (warp >= shape.warps) {
        // the producer's warpgroup gives its registers to the consumers
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(shape.producer_regs));
        // producer: plane q of the block's sequence into slot q % NS, its
        // variables in the kernel's order; with the plane of node p+H the
        // tile of U[to] of node p, which the same iteration updates.  A slot
        // is free again when the iteration that read it last is done, and by
        // then the tile of U[to] NO planes before this one is done with too
        // (NS <= 2 H - 1 + NO).
        if (warp == shape.warps && lane == 0) {
            int q = 0, issued = 0, slot = 0, oslot = 0;
            unsigned phase = 1;  // parity of the empty barrier's phase before
            bool ok = true;
            long long w = r0;
            int x0, c0, p0, p1;
            while (ok && next_item(w, x0, c0, p0, p1)) {
                const int xs = (x0 - hv) & ~1, cs = c0 - hv, xo = x0 & ~1;
                const int NQ = p1 - p0 + 2 * H;  // planes p0-H .. p1+H-1
                for (int ql = 0; ql < NQ; ++ql, ++q) {
                    if (q >= NS && !tma::mbar_wait_bounded(empty + slot, phase, a.status, 5, a.wait_limit)) {
                        ok = false;
                        break;
                    }
                    const int pos = p0 - H + ql, po = pos - H;
                    const bool o = use_o && po >= p0;
                    tma::mbar_expect_tx(full + slot, (pt.BXp * pt.BC + (o ? lt.OX * pt.NR : 0)) * 5 * 8);
#pragma unroll
                    for (int v = 0; v < 5; ++v) {
                        double *dst = ring + (size_t)(slot * 5 + v) * PE;
                        tma::load_5d(dst, &map, xs, pt.swap ? cs : pos, pt.swap ? pos : cs, vg(v), a.tn, full + slot);
                    }
                    if (o) {
#pragma unroll
                        for (int v = 0; v < 5; ++v) {
                            double *dst = oring + (size_t)(oslot * 5 + v) * OE;
                            tma::load_5d(dst, &omap, xo, pt.swap ? c0 : po, pt.swap ? po : c0, vg(v), a.to,
                                         full + slot);
                        }
                        if (++oslot == NO) oslot = 0;
                    }
                    issued = q + 1;
                    if (++slot == NS) {
                        slot = 0;
                        phase ^= 1;
                    }
                }
            }
            // the block must not end with copies in flight
            for (int qq = issued - NS > 0 ? issued - NS : 0; qq < issued; ++qq) {
                tma::mbar_wait_bounded(full + qq % NS, (qq / NS) & 1, a.status, 5, kPlaneWaitLimit);
            }
        }
        return;
    }

    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(shape.consumer_regs));
    const line::Gas k = line::gas_of(mp, g, 0, S, T2);
    const long long nn = g.nn;
    const long long st = pt.st;  // node stride along the line
    const double rdt = (a.dt_scale * a.dt[0]) * g.dd[S];
    const int rl = (int)threadIdx.x / pt.WX, xl = (int)threadIdx.x - rl * pt.WX;
    const uint32_t ring0 = tma::smem_addr(ring);
    auto lds = [](uint32_t addr) {
        double x;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x) : "r"(addr));
        return x;
    };
    int front = 0, par = 0;  // slot of the front plane and the phase of its full barrier
    int oslot = 0;
    long long wi = r0;
    int x0, c0, p0, p1;
    while (next_item(wi, x0, c0, p0, p1)) {
        const int xs = (x0 - hv) & ~1;
        const int i = x0 + xl, c = c0 + rl;
        const bool active = (rl < pt.NR) && (i < g.hi[0]) && (c < g.hi[T2]);
        // element of (i, c) in a plane and in a tile of U[to] (inactive
        // threads: the tile's first node)
        const int e0 = active ? (rl + hv) * pt.BXp + (i - xs) : hv * pt.BXp + (x0 - xs);
        const int eo = active ? rl * lt.OX + (i - (x0 & ~1)) : 0;
        auto wait = [&]() {
            const bool ok = tma::mbar_wait_bounded(full + front, par, a.status, 5, a.wait_limit);
            return (bool)__all_sync(kAll, ok);
        };
        auto advance = [&]() {
            if (++front == NS) {
                front = 0;
                par ^= 1;
            }
        };
        // the slot `back` planes behind the front one
        auto behind = [&](int back) { return front >= back ? front - back : front - back + NS; };
        auto release = [&](int slot) {
            __syncwarp();
            if (lane == 0) tma::mbar_arrive(empty + slot);
        };
        // the state of the node at address A, and its differences across
        auto node_at = [&](uint32_t A) {
            const double u[5] = {lds(A), lds(A + PE * 8), lds(A + 2 * PE * 8), lds(A + 3 * PE * 8), lds(A + 4 * PE * 8)};
            return line::node_of_state(k, u);
        };
        auto differences = [&](uint32_t A, double (&D)[2][2]) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const uint32_t es = q == 0 ? 8 : pt.BXp * 8, tv = (q == 0 ? 1 : 3) * PE * 8, sv = 2 * PE * 8;
                const uint32_t P = A + es, N = A - es;
                line::across(lds(P), lds(P + tv), lds(P + sv), lds(N), lds(N + tv), lds(N + sv), D[q]);
            }
        };
        // preamble: the planes before the front one of the first interface
        // (nodes p0-H .. p0+H-2), and node p0-1
        bool failed = false;
#pragma unroll 1
        for (int q = 0; q < 2 * H - 1; ++q) {
            if (!failed && !wait()) failed = true;
            advance();
        }
        line::Node nc;
        double Dc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
        uint32_t P[NP];  // address of this thread's element of the planes p-H+1 .. p+H
#pragma unroll
        for (int m = 0; m < NP - 1; ++m) P[m + 1] = ring0 + (behind(NP - 1 - m) * (5 * PE) + e0) * 8;
        nc = node_at(P[H]);
        if (VISC) differences(P[H], Dc);
        int did = 1;  // type of the node updated next, loaded one plane ahead
        double Fl[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        long long id = (long long)c * pt.rs + i + (long long)(p0 - 1) * st;
#pragma unroll 1
        for (int p = p0 - 1; p < p1; ++p, id += st) {
            const int did_p = did;
            if (active && p + 1 < p1) did = a.did[id + st];
            if (failed || !wait()) {
                failed = true;
                break;
            }
#pragma unroll
            for (int m = 0; m < NP - 1; ++m) P[m] = P[m + 1];
            P[NP - 1] = ring0 + (front * (5 * PE) + e0) * 8;
            auto src = [&](int m, int v) { return lds(P[m] + v * PE * 8); };
            double F[5];
            {
                line::Node nx;
                double Dn[2][2], Fv[4];
                nx = node_at(P[H]);
                if (VISC) differences(P[H], Dn);
                const line::Face f = line::face_of(k, nc, nx);
                if (VISC) line::viscous_part(k, nc, nx, Dc, Dn, Fv);
                line::convective<NP>(f, src, F);
                if (VISC) {
#pragma unroll
                    for (int v = 0; v < 4; ++v) F[v + 1] -= Fv[v];
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        Dc[q][0] = Dn[q][0];
                        Dc[q][1] = Dn[q][1];
                    }
                }
                nc = nx;
            }
            if (p >= p0 && active && did_p == 0) {
                const double *O = oring + oslot * (5 * OE) + eo;
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    const double phi = Fl[v] - F[v];
                    double *um = a.Um + vg(v) * nn + id;
                    if (a.accumulate) {
                        *um = __ldcg(um) + a.coeB * rdt * phi;
                    } else {
                        const double un = src(H - 1, v), uo = same_o ? un : O[v * OE];
                        *um = fma(a.coeB, fma(rdt, phi, un), a.coeA * uo);
                    }
                }
            }
            if (use_o && p >= p0 && ++oslot == NO) oslot = 0;
            release(behind(NP - 1));  // plane p-H+1 was read for the last time
            advance();
#pragma unroll
            for (int v = 0; v < 5; ++v) Fl[v] = F[v];
        }
        if (failed) return;
        // the planes left (p1-H+1 .. p1+H-1): free their slots for the next item
#pragma unroll
        for (int q = NP - 1; q >= 1; --q) release(behind(q));
    }
}

// ---------------------------------------------------------------------------
// X sweep: the block marches along y over a tile of WX nodes along x by NR
// z-rows, the stencil along x read from the plane.  A lane owns a node and
// the interface on its right: the state of the node on the right and the
// transverse differences there come from the next lane, the flux on the left
// from the lane before, by shuffles, so that no barrier joins the warps.  The
// nodes x0-1 .. x0+WX of every row of the tile follow one another in the warps,
// each warp's first and last lane repeating a node of its neighbours: 30
// nodes a warp.
// ---------------------------------------------------------------------------
template <int NP, bool VISC>
__global__ void __launch_bounds__(line_threads(line_shape(true, VISC)), 1)
stage_line_x(Grid g, ModelParams mp, StageArgs a, LineTile lt, const __grid_constant__ CUtensorMap map,
             const __grid_constant__ CUtensorMap omap)
{
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int H = NP / 2;
    constexpr int hv = VISC ? 1 : 0;
    constexpr LineShape shape = line_shape(true, VISC);
    constexpr int NS = line_slots(true, NP, VISC), NO = shape.oslots;
    constexpr int PE = shape.plane, OE = shape.oplane;
    constexpr unsigned kAll = 0xffffffffu;
    const PlaneTile &pt = lt.pt;
    double *ring = reinterpret_cast<double *>(smem);
    double *oring = ring + (size_t)NS * 5 * PE;
    uint64_t *full = reinterpret_cast<uint64_t *>(oring + (size_t)NO * 5 * OE);
    uint64_t *empty = full + NS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int q = 0; q < NS; ++q) {
            tma::mbar_init(full + q, 1);
            tma::mbar_init(empty + q, shape.warps);
        }
    }
    __syncthreads();
    pdl_wait();

    const long long tiles = (long long)pt.ntx * pt.ntc;
    const int blk = (int)blockIdx.x;
    long long r0 = 0, r1 = 1;
    if (pt.share) {
        plane_share(pt, g.hi[1] - g.lo[1], tiles, blk, r0, r1);
        if (r1 <= r0) return;
    }
    auto next_item = [&](long long &w, int &x0, int &c0, int &j0, int &j1) {
        return pt.share ? plane_x_item<true>(g, pt, tiles, blk, r1, w, x0, c0, j0, j1)
                        : plane_x_item<false>(g, pt, tiles, blk, r1, w, x0, c0, j0, j1);
    };
    const bool same_o = (a.Uo == a.Un);
    const bool use_o = !same_o && !a.accumulate;
    // the kernel's frame: rho, y momentum, x momentum (the sweep's), z momentum, energy
    auto vg = [](int v) { return v == 1 ? 2 : (v == 2 ? 1 : v); };

    if (warp >= shape.warps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(shape.producer_regs));
        // producer: with the plane of row j+hv the tile of U[to] of row j
        // (NS <= 2 hv + NO: see stage_line)
        if (warp == shape.warps && lane == 0) {
            int q = 0, issued = 0, slot = 0, oslot = 0;
            unsigned phase = 1;
            bool ok = true;
            long long w = r0;
            int x0, c0, j0, j1;
            while (ok && next_item(w, x0, c0, j0, j1)) {
                const int xs = (x0 - 3) & ~1, cs = c0 - hv, xo = x0 & ~1;
                const int NQ = j1 - j0 + 2 * hv;  // rows j0-hv .. j1-1+hv
                for (int ql = 0; ql < NQ; ++ql, ++q) {
                    if (q >= NS && !tma::mbar_wait_bounded(empty + slot, phase, a.status, 5, a.wait_limit)) {
                        ok = false;
                        break;
                    }
                    const int row = j0 - hv + ql, ro = row - hv;
                    const bool o = use_o && ro >= j0;
                    tma::mbar_expect_tx(full + slot, (pt.BXp * pt.BC + (o ? lt.OX * pt.NR : 0)) * 5 * 8);
#pragma unroll
                    for (int v = 0; v < 5; ++v) {
                        tma::load_5d(ring + (size_t)(slot * 5 + v) * PE, &map, xs, row, cs, vg(v), a.tn, full + slot);
                    }
                    if (o) {
#pragma unroll
                        for (int v = 0; v < 5; ++v) {
                            tma::load_5d(oring + (size_t)(oslot * 5 + v) * OE, &omap, xo, ro, c0, vg(v), a.to,
                                         full + slot);
                        }
                        if (++oslot == NO) oslot = 0;
                    }
                    issued = q + 1;
                    if (++slot == NS) {
                        slot = 0;
                        phase ^= 1;
                    }
                }
            }
            for (int qq = issued - NS > 0 ? issued - NS : 0; qq < issued; ++qq) {
                tma::mbar_wait_bounded(full + qq % NS, (qq / NS) & 1, a.status, 5, kPlaneWaitLimit);
            }
        }
        return;
    }

    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(shape.consumer_regs));
    const line::Gas k = line::gas_of(mp, g, 1, 0, 2);
    const long long nn = g.nn;
    const double rdt = (a.dt_scale * a.dt[0]) * g.dd[0];
    // entry of this lane in the tile's rows of WX + 2 nodes
    const int entry = warp * 30 + lane;
    const int rl = entry / (pt.WX + 2), xl = entry - rl * (pt.WX + 2) - 1;  // node x0 + xl

    const uint32_t ring0 = tma::smem_addr(ring);
    auto lds = [](uint32_t addr) {
        double x;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x) : "r"(addr));
        return x;
    };
    int front = 0, par = 0, oslot = 0;
    long long wi = r0;
    int x0, c0, j0, j1;
    while (next_item(wi, x0, c0, j0, j1)) {
        const int xs = (x0 - 3) & ~1;
        const int i = x0 + xl, c = c0 + rl;
        const bool row_ok = rl < pt.NR && c < g.hi[2];
        // a node of the row (the last tile's rows end at the node after the
        // last computed one); the others compute on the tile's first node
        const bool active = row_ok && i <= g.hi[0];
        const bool upd = active && xl >= 0 && xl < pt.WX && i < g.hi[0] && lane > 0 && lane < 31;
        const int e0 = active ? (rl + hv) * pt.BXp + (i - xs) : hv * pt.BXp + (x0 - xs);
        const int eo = upd ? rl * lt.OX + (i - (x0 & ~1)) : 0;
        auto wait = [&]() {
            const bool ok = tma::mbar_wait_bounded(full + front, par, a.status, 5, a.wait_limit);
            return (bool)__all_sync(kAll, ok);
        };
        auto advance = [&]() {
            if (++front == NS) {
                front = 0;
                par ^= 1;
            }
        };
        auto behind = [&](int back) { return front >= back ? front - back : front - back + NS; };
        auto at = [&](int slot) { return ring0 + (slot * (5 * PE) + e0) * 8; };
        auto release = [&](int slot) {
            __syncwarp();
            if (lane == 0) tma::mbar_arrive(empty + slot);
        };
        auto across = [&](uint32_t P, uint32_t N, int tvar, double D[2]) {
            const uint32_t tv = tvar * PE * 8, sv = 2 * PE * 8;
            line::across(lds(P), lds(P + tv), lds(P + sv), lds(N), lds(N + tv), lds(N + sv), D);
        };
        bool failed = false;
#pragma unroll
        for (int q = 0; q < 2 * hv; ++q) {  // rows j0-1 and j0 (viscous)
            if (!failed && !wait()) failed = true;
            advance();
        }
        long long id = ((long long)c * g.n[1] + j0) * g.pitch + i;
        int did = upd ? a.did[id] : 1;
#pragma unroll 1
        for (int j = j0; j < j1; ++j, id += g.pitch) {
            const int did_j = did;
            if (upd && j + 1 < j1) did = a.did[id + g.pitch];
            if (failed || !wait()) {
                failed = true;
                break;
            }
            const uint32_t A = at(behind(hv));
            auto src = [&](int m, int v) { return lds(A + (m - (H - 1)) * 8 + v * PE * 8); };
            double F[5];
            {
                line::Node nc, nx;
                {
                    const double u[5] = {lds(A), lds(A + PE * 8), lds(A + 2 * PE * 8), lds(A + 3 * PE * 8),
                                         lds(A + 4 * PE * 8)};
                    nc = line::node_of_state(k, u);
                }
                nx.u = __shfl_down_sync(kAll, nc.u, 1);
                nx.v = __shfl_down_sync(kAll, nc.v, 1);
                nx.w = __shfl_down_sync(kAll, nc.w, 1);
                nx.H = __shfl_down_sync(kAll, nc.H, 1);
                nx.s = __shfl_down_sync(kAll, nc.s, 1);
                const line::Face f = line::face_of(k, nc, nx);
                double Fv[4];
                if (VISC) {
                    double Dc[2][2], Dn[2][2];
                    across(at(front), at(behind(2)), 1, Dc[0]);
                    across(A + pt.BXp * 8, A - pt.BXp * 8, 3, Dc[1]);
                    nx.T = __shfl_down_sync(kAll, nc.T, 1);
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        Dn[q][0] = __shfl_down_sync(kAll, Dc[q][0], 1);
                        Dn[q][1] = __shfl_down_sync(kAll, Dc[q][1], 1);
                    }
                    line::viscous_part(k, nc, nx, Dc, Dn, Fv);
                }
                line::convective<NP>(f, src, F);
                if (VISC) {
#pragma unroll
                    for (int v = 0; v < 4; ++v) F[v + 1] -= Fv[v];
                }
            }
            const double *O = oring + oslot * (5 * OE) + eo;
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                const double phi = __shfl_up_sync(kAll, F[v], 1) - F[v];
                if (upd && did_j == 0) {
                    double *um = a.Um + vg(v) * nn + id;
                    if (a.accumulate) {
                        *um = __ldcg(um) + a.coeB * rdt * phi;
                    } else {
                        const double un = src(H - 1, v), uo = same_o ? un : O[v * OE];
                        *um = fma(a.coeB, fma(rdt, phi, un), a.coeA * uo);
                    }
                }
            }
            if (use_o && ++oslot == NO) oslot = 0;
            release(behind(2 * hv));  // row j-1 (viscous) or j was read for the last time
            advance();
        }
        if (failed) return;
        // rows j1-1 and j1 (viscous): free their slots for the next item
#pragma unroll
        for (int q = 2 * hv; q >= 1; --q) release(behind(q));
    }
}

template <int NP, bool VISC, bool XS>
static int launch_line_one(const Grid &g, const ModelParams &m, const StageArgs &a, const LineTile &lt,
                           const CUtensorMap &map, const CUtensorMap &omap, cudaStream_t st)
{
    static bool configured[64] = {false};
    constexpr int smem = line_smem_bytes(XS, NP, VISC), threads = line_threads(line_shape(XS, VISC));
    auto kernel = XS ? stage_line_x<NP, VISC> : stage_line<NP, VISC>;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(stage_line)");
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    cudaError_t e = launch_k(kernel, dim3((unsigned)lt.pt.nblk), dim3(threads), smem, st, g, m, a, lt, map, omap);
    return e == cudaSuccess ? ACFD_OK : cuda_status(e, "stage_line launch");
}

template <bool XS>
static int launch_line_s(const Grid &g, const ModelParams &m, const StageArgs &a, bool viscous, const LineTile &lt,
                         const CUtensorMap &map, const CUtensorMap &omap, cudaStream_t st)
{
    if (m.sScheme == 1) {
        return viscous ? launch_line_one<6, true, XS>(g, m, a, lt, map, omap, st)
                       : launch_line_one<6, false, XS>(g, m, a, lt, map, omap, st);
    }
    return viscous ? launch_line_one<4, true, XS>(g, m, a, lt, map, omap, st)
                   : launch_line_one<4, false, XS>(g, m, a, lt, map, omap, st);
}

// `map` and `omap`: the state with boxes (BXp, 1, BC) and (OX, 1, NR) for
// s = 0 and 1, (BXp, BC, 1) and (OX, NR, 1) for s = 2, one variable, one level
static int launch_line_impl(const Grid &g, const ModelParams &m, const StageArgs &a, int s, bool viscous,
                            const LineTile &lt0, const CUtensorMap &map, const CUtensorMap &omap, cudaStream_t st)
{
    if (g.hi[0] <= g.lo[0] || g.hi[1] <= g.lo[1] || g.hi[2] <= g.lo[2]) {
        return ACFD_OK;
    }
    if (s == 0) return launch_line_s<true>(g, m, a, viscous, lt0, map, omap, st);
    LineTile lt = lt0;
    Grid gk = g;
    const long long sy = (long long)g.pitch, sz = (long long)g.pitch * g.n[1];
    lt.pt.swap = s == 2;
    lt.pt.st = s == 1 ? sy : sz;
    lt.pt.rs = s == 1 ? sz : sy;
    if (s == 2) {
        // the Z sweep as a Y sweep of the grid with axes 1 and 2 exchanged
        std::swap(gk.n[1], gk.n[2]);
        std::swap(gk.lo[1], gk.lo[2]);
        std::swap(gk.hi[1], gk.hi[2]);
        std::swap(gk.dd[1], gk.dd[2]);
    }
    return launch_line_s<false>(gk, m, a, viscous, lt, map, omap, st);
}

}  // namespace ACFD_NS
}  // namespace acfd
