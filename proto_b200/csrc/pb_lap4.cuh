// The 4th-order flux-form Laplacian as a z march, shared by BoxOp_Laplace::operator() on a box and the
// FAS solver's sweeps, residuals and restrictions.
//
// A cell's value is t = 0 + sum_d [cp F(upper face) - cp F(lower face)], F(face) = g0 a + g1 b + g2 c +
// g3 d over the four cells around the face (DiffCellToFace(d, Lo, 4) scaled by 1/h), cp = 1/h; the
// operator is t times the flux scale. Per cell that is 62 rounded operations and 13 loads if every
// cell works alone, and FP64 issue bounds it (HBM needs 16 bytes a cell). A thread here takes two rows
// (y, y+1) of one x and marches z, so that it can share, with every operation rounded as before:
//   * g3 = -g0 and g2 = -g1 exactly, and the three directions have the same coefficients, so a cell
//     enters all its fluxes through two products, A = g0 v and B = g1 v: F = A(a) + B(b) - B(c) - A(d);
//   * a face's product cp F serves the cell below it and, subtracted, the cell above (the divergence's
//     coefficients are +cp and -cp); the z faces are carried from plane to plane, the y face between
//     the two rows is computed once;
//   * the leading "0 +" of a flux only decides the sign of a zero, which the final 0 + t removes.
// That leaves 38 operations and 7 loads a cell (22 operations that the two rows share and 27 for each; the z
// window keeps values, and their products are formed again as they are needed: three operations a cell for
// 28 registers). With two resident blocks per SM
// only four warps share a scheduler, so no load may be waited for: a plane's neighbours, and what the
// epilogue needs, are loaded one plane ahead. All loads are 8 bytes wide from L1-resident rows, so odd
// sizes and any alignment run the same code. Two cells beyond the range are
// readable in x and y; in z either too (a box), or the planes wrap (a periodic level, which then needs no
// images in z).
#pragma once
#include <type_traits>

#include "pb_internal.cuh"
#include "pb_star.cuh"

namespace pb {

struct FasCoef {
    double g[4];     // DiffCellToFace(d, Lo, 4) * 1/dx, offsets -2, -1, 0, +1 along d
    double cp;       // divergence 1.0*Shift(+e) - 1.0*Shift(0), * 1/dx: +cp and -cp
};

// one field as the march sees it: address of cell (0, 0, 0) of the range, pitches, cell counts
struct Lap4Geom {
    const double* u;
    long long sy, sz;
    int nx, ny, nz;
    int zd;            // planes per thread
    int bx;            // blocks along x
};

constexpr int kLap4Lanes = 32;

// c of a periodic axis of n cells, wrapped into [0, n)
__device__ __forceinline__ int lap4_wrap(int c, int n)
{
    while (c < 0) c += n;
    while (c >= n) c -= n;
    return c;
}

// what one plane's step reads besides the z window: rows y-2, y-1, y+2, y+3 and the x neighbours of rows
// y and y+1
struct Lap4Taps {
    double ya, yb, yd, ye;
    double xm2[2], xm1[2], xp1[2], xp2[2];
};

// t of the two rows from the taps and their z windows w[row][z-1 .. z+2] (as planes m, c, p, q); Pz: the
// lower z faces' products, replaced by the upper ones'
__device__ __forceinline__ void lap4_cells(const Lap4Taps& n, const double (&wm)[2], const double (&wc)[2],
                                           const double (&wp)[2], const double (&wq)[2], double (&Pz)[2],
                                           const FasCoef& k, double (&t)[2])
{
    const double g0 = k.g[0], g1 = k.g[1], cp = k.cp;
    const double B0 = dmul(g1, wc[0]), B1 = dmul(g1, wc[1]);
    // y faces: below row 0, between the rows, above row 1
    const double Bb = dmul(g1, n.yb), Bd = dmul(g1, n.yd);
    const double Py0 = dmul(cp, dsub(dsub(dadd(dmul(g0, n.ya), Bb), B0), dmul(g0, wc[1])));
    const double Py1 = dmul(cp, dsub(dsub(dadd(dmul(g0, n.yb), B0), B1), dmul(g0, n.yd)));
    const double Py2 = dmul(cp, dsub(dsub(dadd(dmul(g0, wc[0]), B1), Bd), dmul(g0, n.ye)));
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const double Bc = r ? B1 : B0, Bm = dmul(g1, n.xm1[r]), Bp = dmul(g1, n.xp1[r]);
        const double Px0 = dmul(cp, dsub(dsub(dadd(dmul(g0, n.xm2[r]), Bm), Bc), dmul(g0, n.xp1[r])));
        const double Px1 = dmul(cp, dsub(dsub(dadd(dmul(g0, n.xm1[r]), Bc), Bp), dmul(g0, n.xp2[r])));
        const double Pz1 = dmul(cp, dsub(dsub(dadd(dmul(g0, wm[r]), Bc), dmul(g1, wp[r])), dmul(g0, wq[r])));
        double d = dsub(Px1, Px0);
        d = dadd(d, r ? Py2 : Py1);
        d = dsub(d, r ? Py1 : Py0);
        d = dadd(d, Pz1);
        d = dsub(d, Pz[r]);
        Pz[r] = Pz1;
        t[r] = dadd(0.0, d);
    }
}

// t of a cell by itself, from its values at -2, -1, +1, +2 along each axis
__device__ __forceinline__ double lap4_cell(const double (&v)[3][4], double c, const FasCoef& k)
{
    double div = 0.0;
    const double B = dmul(k.g[1], c);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double m2 = v[d][0], m1 = v[d][1], p1 = v[d][2], p2 = v[d][3];
        const double Fp = dmul(k.cp, dsub(dsub(dadd(dmul(k.g[0], m1), B), dmul(k.g[1], p1)), dmul(k.g[0], p2)));
        const double Fm = dmul(k.cp, dsub(dsub(dadd(dmul(k.g[0], m2), dmul(k.g[1], m1)), B), dmul(k.g[0], p1)));
        div = d == 0 ? Fp : dadd(div, Fp);
        div = dsub(div, Fm);
    }
    return dadd(0.0, div);
}

// The epilogue: cursor(x, y, z0, act0, act1) once per thread (its addresses at the chunk's first plane);
// per plane pre(cursor, ahead, p0, p1) loads what it needs of both cells, `ahead` planes above the cursor,
// cells(cursor, z, t0, t1, c0, c1, p0, p1) takes the rows' t and centre values (every thread of the block
// calls it, idle ones too) and moves the cursor up; end() once.
template <bool WRAPZ, class Epi>
__global__ void __launch_bounds__(256, 2) k_lap4(const Lap4Geom g, const FasCoef k, Epi epi)
{
    const int by = blockIdx.x / g.bx;                      // blocks of a plane, x fastest
    const int xr = (blockIdx.x - by * g.bx) * kLap4Lanes + threadIdx.x;
    const int y = 2 * (by * blockDim.y + threadIdx.y);
    const int z0 = blockIdx.y * g.zd, z1 = min(z0 + g.zd, g.nz);
    const bool act0 = xr < g.nx && y < g.ny, act1 = xr < g.nx && y + 1 < g.ny;
    // idle threads follow a cell of the range (their loads stay in bounds, nothing is stored)
    const int x = min(xr, g.nx - 1), yc = min(y, g.ny - 1);
    // offsets of rows y+1 and y+3; row y+3 may lie past the readable rows when row y+1 is past the range:
    // row y+2 stands in
    const long long e1 = g.sy, ee = (yc + 3 <= g.ny + 1 ? 3 : 2) * g.sy;
    const double* const q0 = g.u + x + g.sy * yc;
    auto plane = [&](int z) { return q0 + g.sz * (WRAPZ ? lap4_wrap(z, g.nz) : z); };
    auto taps = [&](Lap4Taps& n, const double* q) {
        n.ya = __ldg(q - 2 * e1);
        n.yb = __ldg(q - e1);
        n.yd = __ldg(q + 2 * e1);
        n.ye = __ldg(q + ee);
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const double* c = q + (r ? e1 : 0);
            n.xm2[r] = __ldg(c - 2);
            n.xm1[r] = __ldg(c - 1);
            n.xp1[r] = __ldg(c + 1);
            n.xp2[r] = __ldg(c + 2);
        }
    };
    typename Epi::Cursor cur = epi.cursor(x, yc, z0, act0, act1);
    // window slots of planes z-1 .. z+2 at phase PH: PH .. PH+3 (mod 4); taps and epilogue loads in PH & 1
    double w[4][2], Pz[2], pre[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    Lap4Taps nb[2];
    {
        const double* qm2 = plane(z0 - 2);
        const double* qs[4] = {plane(z0 - 1), plane(z0), plane(z0 + 1), plane(z0 + 2)};
        double m2[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            m2[r] = __ldg(qm2 + (r ? e1 : 0));
#pragma unroll
            for (int s = 0; s < 4; s++) w[s][r] = __ldg(qs[s] + (r ? e1 : 0));
        }
        taps(nb[0], qs[1]);
        epi.pre(cur, 0, pre[0][0], pre[0][1]);
#pragma unroll
        for (int r = 0; r < 2; r++)
            Pz[r] = dmul(k.cp, dsub(dsub(dadd(dmul(k.g[0], m2[r]), dmul(k.g[1], w[0][r])), dmul(k.g[1], w[1][r])),
                                    dmul(k.g[0], w[2][r])));
    }
    // planes z+1 and z+3, moved up once a step (around the end of a periodic axis)
    int zn = WRAPZ ? lap4_wrap(z0 + 1, g.nz) : 0, zf = WRAPZ ? lap4_wrap(z0 + 3, g.nz) : 0;
    const double* qn = q0 + g.sz * (WRAPZ ? zn : z0 + 1);
    const double* qf = q0 + g.sz * (WRAPZ ? zf : z0 + 3);
    const long long around = g.sz * g.nz;
    auto step = [&](auto PHc, int z) {
        constexpr int PH = decltype(PHc)::value;
        constexpr int M = PH, C = (PH + 1) & 3, P = (PH + 2) & 3, Q = (PH + 3) & 3, NOW = PH & 1, NEXT = 1 - NOW;
        double far[2] = {0.0, 0.0};
        if (z + 1 < z1) {
#pragma unroll
            for (int r = 0; r < 2; r++) far[r] = __ldg(qf + (r ? e1 : 0));
            taps(nb[NEXT], qn);
            epi.pre(cur, 1, pre[NEXT][0], pre[NEXT][1]);
            qn += g.sz;
            qf += g.sz;
            if constexpr (WRAPZ) {
                if (++zn == g.nz) {
                    zn = 0;
                    qn -= around;
                }
                if (++zf == g.nz) {
                    zf = 0;
                    qf -= around;
                }
            }
        }
        double t[2];
        lap4_cells(nb[NOW], w[M], w[C], w[P], w[Q], Pz, k, t);
        epi.cells(cur, z, t[0], t[1], w[C][0], w[C][1], pre[NOW][0], pre[NOW][1]);
#pragma unroll
        for (int r = 0; r < 2; r++) w[M][r] = far[r];      // plane z+3, the next step's z+2
    };
    for (int z = z0; z < z1; z += 4) {
        step(std::integral_constant<int, 0>{}, z);
        if (z + 1 >= z1) break;
        step(std::integral_constant<int, 1>{}, z + 1);
        if (z + 2 >= z1) break;
        step(std::integral_constant<int, 2>{}, z + 2);
        if (z + 3 >= z1) break;
        step(std::integral_constant<int, 3>{}, z + 3);
    }
    epi.end();
}

// Launch shape: blocks of 32 x 8 threads (32 x 4 where those leave SMs idle), two resident per SM, and
// the even z chunk that makes waves x (planes + 3) smallest: a chunk starts with four planes of loads
// and products beyond its own, worth about three planes.
template <bool WRAPZ, class Epi>
int launch_lap4(Lap4Geom g, const FasCoef& k, const Epi& epi, int sms, cudaStream_t st)
{
    const long long gx = (g.nx + kLap4Lanes - 1) / kLap4Lanes;
    int rows = 8;
    auto plane = [&] { return gx * ((g.ny + 2LL * rows - 1) / (2 * rows)); };
    if (plane() * ((g.nz + 1) / 2) < sms) rows = 4;
    const long long slots = (long long)sms * (rows == 8 ? 2 : 4);
    long long best = -1;
    for (int zd = 2; zd <= 64; zd += 2) {
        const long long blocks = plane() * ((g.nz + (long long)zd - 1) / zd);
        const long long cost = (blocks + slots - 1) / slots * (zd + 3);
        if (best < 0 || cost < best) {
            best = cost;
            g.zd = zd;
        }
    }
    while ((g.nz + (long long)g.zd - 1) / g.zd > 65535) g.zd *= 2;
    g.bx = (int)gx;
    k_lap4<WRAPZ, Epi><<<dim3((unsigned)plane(), (unsigned)((g.nz + (long long)g.zd - 1) / g.zd)), dim3(kLap4Lanes, rows), 0, st>>>(g, k, epi);
    PB_LAUNCH_CHECK();
    return PB_OK;
}

} // namespace pb
