// The gamma-law stage as a row march (gam.cu includes this file into namespace
// gam, after the zone functions). The reference evaluates every quantity of a
// neighbour inside each zone's update (cbdgam_2d.c:499-682): the x and y slopes of five
// zones, four sound speeds, five scale heights and strain tensors, and all
// four faces. The kernel is a row march like the isothermal one's
// (cbd_stencil.cuh): a CTA of BJ threads owns a strip of BJ columns and walks
// down a segment of rows with one barrier per row; thread t holds column
// c0 + t. Per row it computes
//  * the slopes, p / Sigma, sound speed, strain and scale height of each zone
//    once (row r + 1, kept in registers for the own column and put into shared
//    memory for the neighbours in y);
//  * each face's reconstructed states and their fluxes once. The two zones of
//    a face take different fluxes from them, because each uses the sound
//    speed, and for the viscous flux the scale height, of the neighbour across
//    the face (cbdgam_2d.c:608-647), so the upwinding is done twice.
// Every value is computed by the same operations in the same order as in the
// reference, so the sharing changes no bit. Divisions by a constant (dx, dy,
// gamma - 1) or by one value several times (the HLLE denominator, Sigma in the
// primitive recovery, a face's geometry) use a reciprocal rounded to nearest
// and a Markstein correction, which returns the correctly rounded quotient.
//
// What bounds it is the latency of a row's chain of dependent FP64 operations
// at 12 warps per SM (168 registers; at 128 it spills 170 bytes and runs 8 %
// slower): FP64 pipe 57 % busy, issue 0.56 per cycle, DRAM a fifth of its peak.
// Against the tiles of gam_tile.cuh it executes 756 instead of 835 FP64
// instructions per zone in a reader stage (1041 against 1113 in a writer):
// 2048^2 0.867 -> 0.752 ms per step, 1024^2 227 -> 206 us.
#pragma once

// cbdgam_2d.c:411-434 on one face for two sound speeds: f1 with cs1, f2 with cs2
template <int DIR>
__device__ __forceinline__ void hlle_pair(const Consts &k, const double *pl, const double *pr, double cs1, double cs2,
                                          double *f1, double *f2)
{
    double ul[NF], ur[NF];
    p2c_fast(k, pl, ul);
    p2c_fast(k, pr, ur);
    const double vl = DIR == 0 ? pl[1] : pl[2], vr = DIR == 0 ? pr[1] : pr[2];
    // the pressure enters the normal momentum (adding the reference's
    // `pressure * 0` to the other component changes no value)
    double fl[NF] = {vl * ul[0], vl * ul[1], vl * ul[2], vl * (ul[3] + pl[3])};
    double fr[NF] = {vr * ur[0], vr * ur[1], vr * ur[2], vr * (ur[3] + pr[3])};
    fl[1 + DIR] += pl[3];
    fr[1 + DIR] += pr[3];
    // rounding is monotonic: min(vl - cs, vr - cs) is min(vl, vr) - cs
    const bool left_less = vl < vr;
    const double lo = left_less ? vl : vr, hi = left_less ? vr : vl;
#pragma unroll
    for (int v = 0; v < 2; ++v) {
        const double cs = v == 0 ? cs1 : cs2;
        const double sm = lo - cs, sp = hi + cs;
        const double am = __double2hiint(sm) < 0 ? sm : 0.0;
        const double ap = __double2hiint(sp) < 0 ? 0.0 : sp;
        const double den = ap - am, y = recip_rn(den);
        double *f = v == 0 ? f1 : f2;
#pragma unroll
        for (int q = 0; q < NF; ++q)
            f[q] = div_by(fl[q] * ap - fr[q] * am - (ul[q] - ur[q]) * ap * am, den, y);
    }
}

// Shared memory of the march. Values that are read together lie in pairs, so
// that a warp reads or writes them with 16-byte accesses.
template <int BJ>
struct MarchSmem {
    double2 prim[5][2][BJ + 4];  // ring of primitive rows, columns c0-2 .. c0+BJ+1: (Sigma, vx), (vy, p)
    double2 zone[2][4][BJ + 2];  // by row parity, columns c0-1 .. c0+BJ: y-slopes (2 pairs), (cs, sqrt(p / Sigma)),
                                 // strain (xy, yy)
    double2 north[2][3][BJ + 1]; // by row parity: the flux through face f as the north face of zone f - 1 (2
                                 // pairs), the stress products of the zone beyond
    double un[2][NF][BJ];        // by row parity, each thread's own zones: u_n's source
    double cache[2][5][BJ];      // by row parity, each thread's own: a reader's values for the next row's iteration
    double warp_max[BJ / 32];
};

// One RK stage: CTA (x, y) marches strip x, segment y of `rows` rows.
// primitive_n supplies u_n (cons of it, rebuilt in the kernel) or un_all does
// (the reference's conserved_rk array). With ws_max set, the largest
// wavespeed of the written zones is max-ed into it (non-negative doubles
// order as their bit patterns do). ROLE (ROLE_*) is what the stage does with
// the face cache `fc`; WIDE as in thermal.
//
// Ring slot of row i: (i - r0 + 2) mod 5. Iteration r reads rows r .. r + 2;
// row r + 4 is fetched after its barrier into the slot of row r - 1, and each
// thread has waited for its copies of row r + 3 before the barrier. zone[]
// of row r + 1 and north[] of row r alternate between two buffers by row
// parity, so that a warp ahead of the others writes beside what they read.
template <int BJ, int MINB, int ROLE, bool WIDE>
__global__ void __launch_bounds__(BJ, MINB) stage_kernel(const Consts k, const Stage st, const int rows,
                                                         const double *prd, const double *pn, const double *un_all,
                                                         double *pwr, unsigned long long *ws_max, double *fc)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MarchSmem<BJ> &sm = *reinterpret_cast<MarchSmem<BJ> *>(smem_raw);
    cbd::chain_begin();
    const int t = threadIdx.x;
    if (st.ws_clear && blockIdx.x == 0 && blockIdx.y == 0 && t == 0)
        *st.ws_clear = 0.0;
    const int ni = k.ni, nj = k.nj;
    const int c0 = blockIdx.x * BJ, r0 = blockIdx.y * rows;
    const int W = min(BJ, nj - c0), r1 = min(r0 + rows, ni);
    const int j = c0 + t, jc = min(j, nj - 1);
    const bool active = t < W;
    // a warp whose columns all lie beyond the strip's last face computes
    // nothing; the other lanes past the strip compute on what the ring holds
    const bool busy = (t & ~31) <= W;
    const bool viscous = k.alpha > 0.0, heights = viscous && !st.massless;
    CacheView cv = {};
    if (ROLE != ROLE_NONE) {
        cv = cache_view(k, fc);
        if (ROLE == ROLE_WRITER && blockIdx.x == 0 && blockIdx.y == 0 && t < CACHE_KEY)
            fc[t] = cache_key_value(k, st.m, t);
    }
    auto fetch_row = [&](int slot, int i) {
        const double *src = prd + at(i, c0 - 2, nj);
        for (int c = t; c < W + 4; c += BJ) {
            double *lo = &sm.prim[slot][0][c].x, *hi = &sm.prim[slot][1][c].x;
            cbd::async_copy8(lo, src + NF * c);
            cbd::async_copy8(lo + 1, src + NF * c + 1);
            cbd::async_copy8(hi, src + NF * c + 2);
            cbd::async_copy8(hi + 1, src + NF * c + 3);
        }
    };
    auto load_zone = [&](int slot, int c, double *z) {
        const double2 a = sm.prim[slot][0][c], b = sm.prim[slot][1][c];
        z[0] = a.x;
        z[1] = a.y;
        z[2] = b.x;
        z[3] = b.y;
    };
    // Slopes, p / Sigma, sound speed and strain of ring column c at row r + 1,
    // given the zones of rows r, r + 1, r + 2 there; the neighbours' share into
    // shared memory.
    struct Zone {
        double gx[NF], T, cs, sq, sxx, sxy, syy;
    };
    auto zone_values = [&](int slot, int par, int c, const double *zl, const double *zc, const double *zr, Zone &v) {
        double a[NF], b[NF], gy[NF];
        load_zone(slot, c - 1, a);
        load_zone(slot, c + 1, b);
#pragma unroll
        for (int q = 0; q < NF; ++q) {
            v.gx[q] = slope(zl[q], zc[q], zr[q], k.theta);
            gy[q] = slope(a[q], zc[q], b[q], k.theta);
        }
        const Thermal th = thermal<WIDE>(zc[3], zc[0], k.gamma);
        v.T = th.T;
        v.cs = th.cs;
        v.sq = th.sq;
        // strain (cbdgam_2d.c:278-294): (4/3 gx_vx) / dx - (2/3 gy_vy) / dy, ...
        v.sxx = div_by(4.0 / 3.0 * v.gx[1], k.dx, k.inv_dx) - div_by(2.0 / 3.0 * gy[2], k.dy, k.inv_dy);
        v.sxy = div_by(v.gx[2], k.dx, k.inv_dx) + div_by(gy[1], k.dy, k.inv_dy);
        v.syy = div_by(-2.0 / 3.0 * v.gx[1], k.dx, k.inv_dx) + div_by(4.0 / 3.0 * gy[2], k.dy, k.inv_dy);
        sm.zone[par][0][c - 1] = make_double2(gy[0], gy[1]);
        sm.zone[par][1][c - 1] = make_double2(gy[2], gy[3]);
        sm.zone[par][2][c - 1] = make_double2(v.cs, v.sq);
        sm.zone[par][3][c - 1] = make_double2(v.sxy, v.syy);
    };
    // y-face f of row r (between ring columns f + 1 and f + 2) with geometry w:
    // its flux as the south face of zone f with the stress products of the zone
    // before it, and into shared memory the same as the north face of zone f - 1.
    // zr: the zone on the plus side.
    auto y_face = [&](int slot, int par, int f, const double *zr, double w, double *south, double *products,
                      double *zl) {
        load_zone(slot, f + 1, zl);
        const double2 l0 = sm.zone[par][0][f], l1 = sm.zone[par][1][f], l2 = sm.zone[par][2][f];
        const double2 n0 = sm.zone[par][0][f + 1], n1 = sm.zone[par][1][f + 1], n2 = sm.zone[par][2][f + 1];
        const double lo[NF] = {fma(0.5, l0.x, zl[0]), fma(0.5, l0.y, zl[1]), fma(0.5, l1.x, zl[2]),
                               fma(0.5, l1.y, zl[3])};
        const double hi[NF] = {fma(-0.5, n0.x, zr[0]), fma(-0.5, n0.y, zr[1]), fma(-0.5, n1.x, zr[2]),
                               fma(-0.5, n1.y, zr[3])};
        double north[NF], np0 = 0.0, np1 = 0.0;
        hlle_pair<1>(k, lo, hi, l2.x, n2.x, south, north);
        if (viscous) {
            const double2 l3 = sm.zone[par][3][f], n3 = sm.zone[par][3][f + 1];
            double hs = 1.0, hn = 1.0;
            if (heights) {
                const double y = recip_rn(w);
                hs = div_by(l2.y, w, y);
                hn = div_by(n2.y, w, y);
            }
            const double ns = k.alpha * hs * l2.x * zl[0], nn = k.alpha * hn * n2.x * zr[0];
            products[0] = ns * l3.x;
            products[1] = ns * l3.y;
            np0 = nn * n3.x;
            np1 = nn * n3.y;
        }
        sm.north[par][0][f] = make_double2(north[0], north[1]);
        sm.north[par][1][f] = make_double2(north[2], north[3]);
        sm.north[par][2][f] = make_double2(np0, np1);
    };
    // lanes with the strip's extra work, in warps of their own: the two halo
    // columns' zone values, the last y-face
    constexpr int HALO_LANE = 32, FACE_LANE = BJ >= 128 ? 64 : 0;

    // the own column's values at row r: zone, x-slope, p / Sigma, sound speed and
    // its root, height geometry and height, strain (xx, xy), the zone's stress
    // times its viscosity (xx, xy, yy), and the flux through its west face
    double z0[NF] = {}, gx0[NF] = {}, T0 = 0.0, cs0 = 0.0, sq0 = 0.0, wc0 = 1.0, hc0 = 1.0, sxx0 = 0.0, sxy0 = 0.0;
    double v0[3] = {}, fw[NF] = {};
    double ws = 0.0;
    double rd = (double)(r0 - 2);  // row r as a double
    const double yc = k.yl + (j + 0.5) * k.dy;

    // what iteration r reads besides the rows, for this thread alone: u_n's
    // source zone, and a reader's face geometry, height geometry of row r + 1
    // and gravity factors of row r (loads at their use left the march waiting
    // for HBM a seventh of its time)
    const double *un_src = st.un_from_primitive ? pn : un_all;
    auto fetch_own = [&](int r) {
        if (!busy)
            return;
        const int p = r & 1;
        if (r >= r0 && r < r1) {
            const double *src = un_src + at(r, jc, nj);
#pragma unroll
            for (int q = 0; q < NF; ++q)
                cbd::async_copy8(&sm.un[p][q][t], src + q);
        }
        if (ROLE == ROLE_READER) {
            if (heights && r >= r0 - 1 && r < r1)
                cbd::async_copy8(&sm.cache[p][0][t], cv.xf + (size_t)(r + 1) * nj + jc);
            if (r + 1 >= r0 && r + 1 < r1)
                cbd::async_copy8(&sm.cache[p][1][t], cv.zp + 2 * ((size_t)(r + 1) * nj + jc));
            if (r >= r0 && r < r1) {
                if (heights)
                    cbd::async_copy8(&sm.cache[p][2][t], cv.yf + (size_t)r * (nj + 1) + min(j, nj));
                cbd::async_copy8(&sm.cache[p][3][t], cv.zp + 2 * ((size_t)r * nj + jc) + 1);
                cbd::async_copy8(&sm.cache[p][4][t], cv.zg2 + (size_t)r * nj + jc);
            }
        }
    };

    fetch_row(0, r0 - 2);
    fetch_row(1, r0 - 1);
    fetch_row(2, r0);
    cbd::async_commit();
    cbd::async_wait<0>();
    __syncthreads();
    if (r0 + 1 <= r1 + 1)
        fetch_row(3, r0 + 1);
    fetch_own(r0 - 1);
    cbd::async_commit();
    int s0 = 0;

#pragma unroll 1
    for (int r = r0 - 2; r < r1; ++r, rd += 1.0) {
        const int s1 = s0 == 4 ? 0 : s0 + 1, s2 = s1 == 4 ? 0 : s1 + 1;
        const int p1 = (r + 1) & 1, p0 = r & 1;
        double z1[NF] = {}, wc1 = 1.0, hc1 = 1.0, v1[3] = {}, fe[NF] = {}, fw1[NF] = {}, fs[NF] = {};
        Zone n = {};
        if (busy) {
            double wx = 0.0, wy = 0.0;
            if (ROLE == ROLE_READER) {
                wx = sm.cache[p0][0][t];
                wc1 = sm.cache[p0][1][t];
                wy = sm.cache[p0][2][t];
            }

            // (1) zone values at row r + 1, own column
            double z2[NF];
            if (r == r0 - 2)
                load_zone(s0, t + 2, z0);
            load_zone(s1, t + 2, z1);
            load_zone(s2, t + 2, z2);
            zone_values(s1, p1, t + 2, z0, z1, z2, n);
            if (r + 1 >= r0 && r + 1 < r1 && !st.massless) {
                if (ROLE != ROLE_READER)
                    wc1 = root_w2(st.m, k.xl + (rd + 1.5) * k.dx, yc);
                hc1 = div_rn(n.sq, wc1);
            }
            const double nu1 = k.alpha * hc1 * n.cs * z1[0];
            v1[0] = nu1 * n.sxx;
            v1[1] = nu1 * n.sxy;
            v1[2] = nu1 * n.syy;

            // (2) the x-face between rows r and r + 1: the east flux of zone r,
            // the west flux of zone r + 1
            if (r >= r0 - 1) {
                double lo[NF], hi[NF];
#pragma unroll
                for (int q = 0; q < NF; ++q) {
                    // p +- g / 2, and f - S / 2 below, are single FMAs: halving a
                    // normal number is exact, so the fused operation rounds as
                    // the reference's multiply then add
                    lo[q] = fma(0.5, gx0[q], z0[q]);
                    hi[q] = fma(-0.5, n.gx[q], z1[q]);
                }
                hlle_pair<0>(k, lo, hi, n.cs, cs0, fe, fw1);
                if (viscous) {
                    double he = 1.0, hw = 1.0;
                    if (heights) {
                        if (ROLE != ROLE_READER) {
                            wx = root_w2(st.m, k.xl + (rd + 1.0) * k.dx, yc);
                            // face r + 1 is stored by the tile above it, except the grid's first
                            if (ROLE == ROLE_WRITER && active && (r >= r0 || r0 == 0))
                                cv.xf[(size_t)(r + 1) * nj + j] = wx;
                        }
                        const double y = recip_rn(wx);
                        he = div_by(n.sq, wx, y);
                        hw = div_by(sq0, wx, y);
                    }
                    const double ne = k.alpha * he * n.cs * z1[0], nw = k.alpha * hw * cs0 * z0[0];
                    const double e0 = ne * n.sxx, e1 = ne * n.sxy, w0 = nw * sxx0, w1 = nw * sxy0;
                    fe[1] = fma(-0.5, v0[0] + e0, fe[1]);
                    fe[2] = fma(-0.5, v0[1] + e1, fe[2]);
                    fe[3] = fma(-0.5, v0[0] * z0[1] + e0 * z1[1], fe[3]);
                    fe[3] = fma(-0.5, v0[1] * z0[2] + e1 * z1[2], fe[3]);
                    fw1[1] = fma(-0.5, w0 + v1[0], fw1[1]);
                    fw1[2] = fma(-0.5, w1 + v1[1], fw1[2]);
                    fw1[3] = fma(-0.5, w0 * z0[1] + v1[0] * z1[1], fw1[3]);
                    fw1[3] = fma(-0.5, w1 * z0[2] + v1[1] * z1[2], fw1[3]);
                }
            }

            // (3) the y-face of row r at the own column's minus side
            if (r >= r0) {
                if (ROLE != ROLE_READER && heights) {
                    wy = root_w2(st.m, k.xl + (rd + 0.5) * k.dx, k.yl + (j + 0.0) * k.dy);
                    if (ROLE == ROLE_WRITER && active)
                        cv.yf[(size_t)r * (nj + 1) + j] = wy;
                }
                double products[2] = {0.0, 0.0}, zl[NF];
                y_face(s0, p0, t, z0, wy, fs, products, zl);
                if (viscous) {
                    fs[1] = fma(-0.5, products[0] + v0[1], fs[1]);
                    fs[2] = fma(-0.5, products[1] + v0[2], fs[2]);
                    fs[3] = fma(-0.5, products[0] * zl[1] + v0[1] * z0[1], fs[3]);
                    fs[3] = fma(-0.5, products[1] * zl[2] + v0[2] * z0[2], fs[3]);
                }
            }
        }
        if (t == HALO_LANE || t == HALO_LANE + 1) {
            const int c = t == HALO_LANE ? 1 : W + 2;
            double zl[NF], zc[NF], zr[NF];
            Zone h;
            load_zone(s0, c, zl);
            load_zone(s1, c, zc);
            load_zone(s2, c, zr);
            zone_values(s1, p1, c, zl, zc, zr, h);
        }
        if (t == FACE_LANE && r >= r0) {
            double w = 0.0, south[NF], products[2], zl[NF], zr[NF];
            if (heights) {
                if (ROLE == ROLE_READER) {
                    w = cv.yf[(size_t)r * (nj + 1) + c0 + W];
                } else {
                    w = root_w2(st.m, k.xl + (rd + 0.5) * k.dx, k.yl + (c0 + W + 0.0) * k.dy);
                    // stored by the next strip, except the last
                    if (ROLE == ROLE_WRITER && c0 + W == nj)
                        cv.yf[(size_t)r * (nj + 1) + nj] = w;
                }
            }
            load_zone(s0, W + 2, zr);
            y_face(s0, p0, W, zr, w, south, products, zl);
        }
        // row r + 3 has landed for this thread, after the barrier for all; the
        // slot of row r - 1 is free for row r + 4
        cbd::async_wait<0>();
        __syncthreads();
        if (r + 4 <= r1 + 1)
            fetch_row(s2 >= 3 ? s2 - 3 : s2 + 2, r + 4);
        cbd::async_commit();

        // (4) update zone (r, j)
        if (active && r >= r0) {
            const double dt = st.dt, xc = k.xl + (rd + 0.5) * k.dx;
            const double2 n0 = sm.north[p0][0][t + 1], n1 = sm.north[p0][1][t + 1];
            double fn[NF] = {n0.x, n0.y, n1.x, n1.y};
            if (viscous) {
                const double2 np = sm.north[p0][2][t + 1];
                const double vx = sm.prim[s0][0][t + 3].y, vy = sm.prim[s0][1][t + 3].x;
                fn[1] = fma(-0.5, v0[1] + np.x, fn[1]);
                fn[2] = fma(-0.5, v0[2] + np.y, fn[2]);
                fn[3] = fma(-0.5, v0[1] * z0[1] + np.x * vx, fn[3]);
                fn[3] = fma(-0.5, v0[2] * z0[2] + np.y * vy, fn[3]);
            }
            double un[NF], gz[2] = {0.0, 0.0};
#pragma unroll
            for (int q = 0; q < NF; ++q)
                un[q] = sm.un[p0][q][t];
            if (ROLE == ROLE_READER) {
                gz[0] = sm.cache[p0][3][t];
                gz[1] = sm.cache[p0][4][t];
            }
            if (st.un_from_primitive) {
                // u_n enters as (1 - a) u + a u_n even when a = 0, as in the reference
                const double pz[NF] = {un[0], un[1], un[2], un[3]};
                p2c_fast(k, pz, un);
            }
            double u[NF];
            p2c_fast(k, z0, u);
            buffer_source(k, st, xc, yc, dt, u);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                double du[NF];
                const bool cached_g = ROLE == ROLE_READER && k.constant_softening;
                mass_source<true, false>(st.m[m], xc, yc, dt, z0, T0, hc0, k.constant_softening, k.gm1, k.inv_gm1,
                                         du, cached_g ? &gz[m] : nullptr, ROLE == ROLE_WRITER ? &gz[m] : nullptr);
#pragma unroll
                for (int q = 0; q < NF; ++q)
                    u[q] += du[q];
            }
            if (ROLE == ROLE_WRITER) {
                const size_t zc = (size_t)r * nj + j;
                *reinterpret_cast<double2 *>(cv.zp + 2 * zc) = make_double2(wc0, gz[0]);
                cv.zg2[zc] = gz[1];
            }
            cooling_fast(k, dt, z0, T0, u);
#pragma unroll
            for (int q = 0; q < NF; ++q) {
                u[q] -= (div_by(fe[q] - fw[q], k.dx, k.inv_dx) + div_by(fn[q] - fs[q], k.dy, k.inv_dy)) * dt;
                u[q] = (1.0 - st.a) * u[q] + st.a * un[q];
            }
            double out[NF];
            c2p_fast(k, u, out);
            // the zone and, on the edges, its zero-gradient guard images
            const bool edge = st.write_guards && (r == 0 || r == ni - 1 || j == 0 || j == nj - 1);
            if (!edge) {
                double *dst = pwr + at(r, j, nj);
#pragma unroll
                for (int q = 0; q < NF; ++q)
                    dst[q] = out[q];
            } else {
                const int ilo = r == 0 ? -NG : r, ihi = r == ni - 1 ? ni + 1 : r;
                const int jlo = j == 0 ? -NG : j, jhi = j == nj - 1 ? nj + 1 : j;
                for (int ii = ilo; ii <= ihi; ++ii)
                    for (int jj = jlo; jj <= jhi; ++jj) {
                        double *dst = pwr + at(ii, jj, nj);
#pragma unroll
                        for (int q = 0; q < NF; ++q)
                            dst[q] = out[q];
                    }
            }
            if (ws_max)
                ws = max_nan(ws, zone_wavespeed(out, k.gamma));
        }
        // into the buffers this iteration has read; landed by the next barrier
        fetch_own(r + 2);
        cbd::async_commit();
#pragma unroll
        for (int q = 0; q < NF; ++q) {
            z0[q] = z1[q];
            gx0[q] = n.gx[q];
            fw[q] = fw1[q];
        }
        T0 = n.T;
        cs0 = n.cs;
        sq0 = n.sq;
        wc0 = wc1;
        hc0 = hc1;
        sxx0 = n.sxx;
        sxy0 = n.sxy;
        v0[0] = v1[0];
        v0[1] = v1[1];
        v0[2] = v1[2];
        s0 = s1;
    }
    cbd::chain_end();
    if (ws_max) {  // uniform over the block
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            ws = max_nan(ws, __shfl_xor_sync(0xffffffffu, ws, o));
        if ((t & 31) == 0)
            sm.warp_max[t >> 5] = ws;
        __syncthreads();
        if (t == 0) {
            double m = sm.warp_max[0];
            for (int w = 1; w < BJ / 32; ++w)
                m = max_nan(m, sm.warp_max[w]);
            atomicMax(ws_max, (unsigned long long)__double_as_longlong(m));
        }
    }
}
