// The gamma-law stage in tiles, for grids of middle size (gam.cu includes this
// file into namespace gam, after the zone functions). A CTA of 256 threads over
// a tile of 16 x 32 zones, two rows of zones per thread: a first phase computes
// the per-zone quantities that every neighbouring update needs (slopes, p /
// Sigma, sound speed, strain) and the scale heights' face geometry into shared
// memory, a second the zone updates, each zone its four faces. A zone's chain
// of dependent operations is walked twice per CTA here, against once per row in
// the march, which makes up for the arithmetic that the march shares wherever
// the march's segments are short or leave slots idle (march_suits has the
// measured line).
#pragma once

constexpr int TI = 16, TJ = 32;  // CTA tile (rows i, columns j)
constexpr int RPT = 2;            // tile rows per thread: zone rows ty and ty + TI / RPT
constexpr int NT = TI * TJ / RPT; // threads per CTA, a (TJ, TI / RPT) block
constexpr int HI = TI + 2 * NG, HJ = TJ + 2 * NG;
constexpr int TILE_MIN_BLOCKS = 2;  // resident CTAs per SM the stage kernel is built for

constexpr int ZI = TI + 2, ZJ = TJ + 2;  // zones with shared quantities: the tile and a ring of one
// per-zone quantities: x and y slopes, p / Sigma, sound speed, sqrt(p / Sigma), strain xx, xy, yy
enum { Q_GX = 0, Q_GY = 4, Q_T = 8, Q_CS = 9, Q_SQ = 10, Q_SXX = 11, Q_SXY = 12, Q_SYY = 13, NZQ = 14 };

struct TileSmem {
    double prim[NF][HI][HJ];
    double z[NZQ][ZI][ZJ];
    double fx[TI + 1][TJ];  // sqrt(sum_m M_m r^-3) at the x-faces (x_l of zone i0 + a, y_c of zone j0 + b)
    double fy[TI][TJ + 1];  // the same at the y-faces (x_c of zone i0 + a, y_l of zone j0 + b)
    double warp_max[NT / 32];
};

// cbdgam_2d.c:411-434 given the neighbour's sound speed cs = sqrt(cs2)
template <int DIR>
__device__ __forceinline__ void hlle_fast(const Consts &k, const double *pl, const double *pr, double cs, double *f)
{
    double ul[NF], ur[NF];
    p2c_fast(k, pl, ul);
    p2c_fast(k, pr, ur);
    const double vl = DIR == 0 ? pl[1] : pl[2], vr = DIR == 0 ? pr[1] : pr[2];
    const double fl[NF] = {vl * ul[0], vl * ul[1] + pl[3] * (double)(DIR == 0), vl * ul[2] + pl[3] * (double)(DIR == 1),
                           vl * (ul[3] + pl[3])};
    const double fr[NF] = {vr * ur[0], vr * ur[1] + pr[3] * (double)(DIR == 0), vr * ur[2] + pr[3] * (double)(DIR == 1),
                           vr * (ur[3] + pr[3])};
    // rounding is monotonic: min(vl - cs, vr - cs) is min(vl, vr) - cs
    const bool left_less = vl < vr;
    const double sm = (left_less ? vl : vr) - cs, sp = (left_less ? vr : vl) + cs;
    const double am = __double2hiint(sm) < 0 ? sm : 0.0;
    const double ap = __double2hiint(sp) < 0 ? 0.0 : sp;
    const double den = ap - am, y = recip_rn(den);
#pragma unroll
    for (int q = 0; q < NF; ++q)
        f[q] = div_by(fl[q] * ap - fr[q] * am - (ul[q] - ur[q]) * ap * am, den, y);
}

// Phase 1: the per-zone quantities of zone (i0 - 1 + a, j0 - 1 + b) and the
// face geometry of the tile.
template <int ROLE, bool WIDE>
__device__ __forceinline__ void tile_phase1(const Consts &k, const Stage &st, TileSmem &sm, int i0, int j0, int tid,
                                             const CacheView &cv)
{
    // one pool of work items for the whole CTA: the zones of the tile and its
    // ring, then (with viscosity) the x-faces and the y-faces, so that the
    // last pass over the pool is the only partly idle one
    constexpr int NZI = ZI * ZJ, NFX = (TI + 1) * TJ, NFY = TI * (TJ + 1);
    const bool faces = k.alpha > 0.0 && !st.massless;
    const int total = NZI + (faces ? NFX + NFY : 0);
    const double theta = k.theta;
    for (int s = tid; s < total; s += NT) {
        if (s >= NZI + NFX) {
            const int f = s - NZI - NFX, a = f / (TJ + 1), b = f % (TJ + 1);
            const int i = i0 + a, j = j0 + b;
            const bool in = i < k.ni && j <= k.nj;
            double w = 0.0;
            if (ROLE == ROLE_READER) {
                if (in)
                    w = cv.yf[(size_t)i * (k.nj + 1) + j];
            } else {
                w = root_w2(st.m, k.xl + (i + 0.5) * k.dx, k.yl + (j + 0.0) * k.dy);
                // a tile's last face column is stored by the next tile, except the last
                if (ROLE == ROLE_WRITER && in && (b < TJ || j == k.nj))
                    cv.yf[(size_t)i * (k.nj + 1) + j] = w;
            }
            sm.fy[a][b] = w;
            continue;
        }
        if (s >= NZI) {
            const int f = s - NZI, a = f / TJ, b = f % TJ;
            const int i = i0 + a, j = j0 + b;
            const bool in = i <= k.ni && j < k.nj;
            double w = 0.0;
            if (ROLE == ROLE_READER) {
                if (in)
                    w = cv.xf[(size_t)i * k.nj + j];
            } else {
                w = root_w2(st.m, k.xl + (i + 0.0) * k.dx, k.yl + (j + 0.5) * k.dy);
                // a tile's last face row is stored by the next tile, except the last
                if (ROLE == ROLE_WRITER && in && (a < TI || i == k.ni))
                    cv.xf[(size_t)i * k.nj + j] = w;
            }
            sm.fx[a][b] = w;
            continue;
        }
        const int a = s / ZJ, b = s % ZJ;
        if (i0 - 1 + a > k.ni || j0 - 1 + b > k.nj)
            continue;  // beyond the guard zones of the last tile: never read
        double gx[NF], gy[NF];
#pragma unroll
        for (int q = 0; q < NF; ++q) {
            gx[q] = slope(sm.prim[q][a][b + 1], sm.prim[q][a + 1][b + 1], sm.prim[q][a + 2][b + 1], theta);
            gy[q] = slope(sm.prim[q][a + 1][b], sm.prim[q][a + 1][b + 1], sm.prim[q][a + 1][b + 2], theta);
            sm.z[Q_GX + q][a][b] = gx[q];
            sm.z[Q_GY + q][a][b] = gy[q];
        }
        const Thermal th = thermal<WIDE>(sm.prim[3][a + 1][b + 1], sm.prim[0][a + 1][b + 1], k.gamma);
        sm.z[Q_T][a][b] = th.T;
        sm.z[Q_CS][a][b] = th.cs;
        sm.z[Q_SQ][a][b] = th.sq;
        // strain (cbdgam_2d.c:278-294): (4/3 gx_vx) / dx - (2/3 gy_vy) / dy, ...
        sm.z[Q_SXX][a][b] = div_by(4.0 / 3.0 * gx[1], k.dx, k.inv_dx) - div_by(2.0 / 3.0 * gy[2], k.dy, k.inv_dy);
        sm.z[Q_SXY][a][b] = div_by(gx[2], k.dx, k.inv_dx) + div_by(gy[1], k.dy, k.inv_dy);
        sm.z[Q_SYY][a][b] = div_by(-2.0 / 3.0 * gx[1], k.dx, k.inv_dx) + div_by(4.0 / 3.0 * gy[2], k.dy, k.inv_dy);
    }
}

// Phase 2: zone (i, j) = (i0 + ty, j0 + tx); returns its new primitives.
template <int ROLE>
__device__ __forceinline__ void tile_phase2(const Consts &k, const Stage &st, const TileSmem &sm, int ty, int tx,
                                             const double *un, double *out, const CacheView &cv)
{
    const int i = blockIdx.y * TI + ty, j = blockIdx.x * TJ + tx;
    const double dt = st.dt;
    const double xc = k.xl + (i + 0.5) * k.dx, yc = k.yl + (j + 0.5) * k.dy;
    // primitives and per-zone quantities of the zone and its four neighbours
    auto P = [&](int di, int dj, int q) { return sm.prim[q][ty + NG + di][tx + NG + dj]; };
    auto Z = [&](int di, int dj, int q) { return sm.z[q][ty + 1 + di][tx + 1 + dj]; };
    double c[NF];
#pragma unroll
    for (int q = 0; q < NF; ++q)
        c[q] = P(0, 0, q);

    // p +- g / 2 and f - S / 2 below are single FMAs: halving a normal number
    // is exact, so the fused operation rounds as the reference's multiply
    // then add
    double fw[NF], fe[NF], fs[NF], fn[NF];
    {
        double lo[NF], hi[NF];
#pragma unroll
        for (int q = 0; q < NF; ++q) {
            lo[q] = fma(0.5, Z(-1, 0, Q_GX + q), P(-1, 0, q));
            hi[q] = fma(-0.5, Z(0, 0, Q_GX + q), c[q]);
        }
        hlle_fast<0>(k, lo, hi, Z(-1, 0, Q_CS), fw);
#pragma unroll
        for (int q = 0; q < NF; ++q) {
            lo[q] = fma(0.5, Z(0, 0, Q_GX + q), c[q]);
            hi[q] = fma(-0.5, Z(1, 0, Q_GX + q), P(1, 0, q));
        }
        hlle_fast<0>(k, lo, hi, Z(1, 0, Q_CS), fe);
#pragma unroll
        for (int q = 0; q < NF; ++q) {
            lo[q] = fma(0.5, Z(0, -1, Q_GY + q), P(0, -1, q));
            hi[q] = fma(-0.5, Z(0, 0, Q_GY + q), c[q]);
        }
        hlle_fast<1>(k, lo, hi, Z(0, -1, Q_CS), fs);
#pragma unroll
        for (int q = 0; q < NF; ++q) {
            lo[q] = fma(0.5, Z(0, 0, Q_GY + q), c[q]);
            hi[q] = fma(-0.5, Z(0, 1, Q_GY + q), P(0, 1, q));
        }
        hlle_fast<1>(k, lo, hi, Z(0, 1, Q_CS), fn);
    }

    const size_t zc = (size_t)i * k.nj + j;
    double wc = 1.0, gz[2] = {0.0, 0.0};
    if (ROLE == ROLE_READER) {
        const double2 v = *reinterpret_cast<const double2 *>(cv.zp + 2 * zc);
        wc = v.x;
        gz[0] = v.y;
        gz[1] = cv.zg2[zc];
    } else if (!st.massless) {
        wc = root_w2(st.m, xc, yc);
    }
    const double hc = st.massless ? 1.0 : div_rn(Z(0, 0, Q_SQ), wc);

    if (k.alpha > 0.0) {
        const double hw = st.massless ? 1.0 : div_rn(Z(-1, 0, Q_SQ), sm.fx[ty][tx]);
        const double he = st.massless ? 1.0 : div_rn(Z(1, 0, Q_SQ), sm.fx[ty + 1][tx]);
        const double hs = st.massless ? 1.0 : div_rn(Z(0, -1, Q_SQ), sm.fy[ty][tx]);
        const double hn = st.massless ? 1.0 : div_rn(Z(0, 1, Q_SQ), sm.fy[ty][tx + 1]);
        const double nuc = k.alpha * hc * Z(0, 0, Q_CS);
        const double nuw = k.alpha * hw * Z(-1, 0, Q_CS), nue = k.alpha * he * Z(1, 0, Q_CS);
        const double nus = k.alpha * hs * Z(0, -1, Q_CS), nun = k.alpha * hn * Z(0, 1, Q_CS);
        const double w0 = P(-1, 0, 0), e0 = P(1, 0, 0), s0 = P(0, -1, 0), n0 = P(0, 1, 0);
        // strain tensors (xx, xy, yx = xy, yy) of the zone and its neighbours
        const double tc0 = Z(0, 0, Q_SXX), tc1 = Z(0, 0, Q_SXY), tc3 = Z(0, 0, Q_SYY);
        const double tw0 = Z(-1, 0, Q_SXX), tw1 = Z(-1, 0, Q_SXY);
        const double te0 = Z(1, 0, Q_SXX), te1 = Z(1, 0, Q_SXY);
        const double ts2 = Z(0, -1, Q_SXY), ts3 = Z(0, -1, Q_SYY);
        const double tn2 = Z(0, 1, Q_SXY), tn3 = Z(0, 1, Q_SYY);
        const double tc2 = tc1;

        fw[1] = fma(-0.5, nuw * w0 * tw0 + nuc * c[0] * tc0, fw[1]);
        fw[2] = fma(-0.5, nuw * w0 * tw1 + nuc * c[0] * tc1, fw[2]);
        fe[1] = fma(-0.5, nuc * c[0] * tc0 + nue * e0 * te0, fe[1]);
        fe[2] = fma(-0.5, nuc * c[0] * tc1 + nue * e0 * te1, fe[2]);
        fs[1] = fma(-0.5, nus * s0 * ts2 + nuc * c[0] * tc2, fs[1]);
        fs[2] = fma(-0.5, nus * s0 * ts3 + nuc * c[0] * tc3, fs[2]);
        fn[1] = fma(-0.5, nuc * c[0] * tc2 + nun * n0 * tn2, fn[1]);
        fn[2] = fma(-0.5, nuc * c[0] * tc3 + nun * n0 * tn3, fn[2]);

        fw[3] = fma(-0.5, nuw * w0 * tw0 * P(-1, 0, 1) + nuc * c[0] * tc0 * c[1], fw[3]);
        fe[3] = fma(-0.5, nuc * c[0] * tc0 * c[1] + nue * e0 * te0 * P(1, 0, 1), fe[3]);
        fw[3] = fma(-0.5, nuw * w0 * tw1 * P(-1, 0, 2) + nuc * c[0] * tc1 * c[2], fw[3]);
        fe[3] = fma(-0.5, nuc * c[0] * tc1 * c[2] + nue * e0 * te1 * P(1, 0, 2), fe[3]);
        fs[3] = fma(-0.5, nus * s0 * ts2 * P(0, -1, 1) + nuc * c[0] * tc2 * c[1], fs[3]);
        fn[3] = fma(-0.5, nuc * c[0] * tc2 * c[1] + nun * n0 * tn2 * P(0, 1, 1), fn[3]);
        fs[3] = fma(-0.5, nus * s0 * ts3 * P(0, -1, 2) + nuc * c[0] * tc3 * c[2], fs[3]);
        fn[3] = fma(-0.5, nuc * c[0] * tc3 * c[2] + nun * n0 * tn3 * P(0, 1, 2), fn[3]);
    }

    const double T = Z(0, 0, Q_T);
    double u[NF];
    p2c_fast(k, c, u);
    buffer_source(k, st, xc, yc, dt, u);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        double du[NF];
        const bool cached_g = ROLE == ROLE_READER && k.constant_softening;
        mass_source<true, false>(st.m[m], xc, yc, dt, c, T, hc, k.constant_softening, k.gm1, k.inv_gm1, du,
                    cached_g ? &gz[m] : nullptr, ROLE == ROLE_WRITER ? &gz[m] : nullptr);
#pragma unroll
        for (int q = 0; q < NF; ++q)
            u[q] += du[q];
    }
    if (ROLE == ROLE_WRITER) {
        *reinterpret_cast<double2 *>(cv.zp + 2 * zc) = make_double2(wc, gz[0]);
        cv.zg2[zc] = gz[1];
    }
    cooling_fast(k, dt, c, T, u);
#pragma unroll
    for (int q = 0; q < NF; ++q) {
        u[q] -= (div_by(fe[q] - fw[q], k.dx, k.inv_dx) + div_by(fn[q] - fs[q], k.dy, k.inv_dy)) * dt;
        u[q] = (1.0 - st.a) * u[q] + st.a * un[q];
    }
    c2p_fast(k, u, out);
}

// One RK stage. primitive_n supplies u_n (cons of it, rebuilt in the kernel)
// or un_all does (the reference's conserved_rk array). With ws_max set, the
// largest wavespeed of the written zones is max-ed into it (non-negative
// doubles order as their bit patterns do).
// ROLE (ROLE_*) is what the stage does with the face cache `fc`; WIDE as in thermal.
template <int ROLE, bool WIDE>
__global__ void __launch_bounds__(NT, TILE_MIN_BLOCKS) tile_kernel(Consts k, Stage st,
                                                                          const double *prd,
                                                                          const double *pn,
                                                                          const double *un_all,
                                                                          double *pwr, unsigned long long *ws_max,
                                                                          double *fc)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TileSmem &sm = *reinterpret_cast<TileSmem *>(smem_raw);
    cbd::chain_begin();
    const int i0 = blockIdx.y * TI, j0 = blockIdx.x * TJ;
    const int ni = k.ni, nj = k.nj;
    const int tid = threadIdx.y * TJ + threadIdx.x;
    if (st.ws_clear && blockIdx.x == 0 && blockIdx.y == 0 && tid == 0)
        *st.ws_clear = 0.0;
    for (int s = tid; s < HI * HJ; s += NT) {
        const int ii = i0 - NG + s / HJ, jj = j0 - NG + s % HJ;
        if (ii <= ni + 1 && jj <= nj + 1) {
            const double *src = prd + at(ii, jj, nj);
#pragma unroll
            for (int q = 0; q < NF; ++q)
                sm.prim[q][s / HJ][s % HJ] = src[q];
        }
    }
    __syncthreads();
    CacheView cv = {};
    if (ROLE != ROLE_NONE) {
        cv = cache_view(k, fc);
        if (ROLE == ROLE_WRITER && blockIdx.x == 0 && blockIdx.y == 0 && tid < CACHE_KEY)
            fc[tid] = cache_key_value(k, st.m, tid);
    }
    tile_phase1<ROLE, WIDE>(k, st, sm, i0, j0, tid, cv);
    __syncthreads();
    double ws = 0.0;
#pragma unroll 1
    for (int h = 0; h < RPT; ++h) {
        const int ty = threadIdx.y + h * (TI / RPT);
        const int i = i0 + ty, j = j0 + threadIdx.x;
        if (i >= ni || j >= nj)
            continue;
        // u_n enters as (1 - a) u + a u_n even when a = 0, as in the reference
        double un[NF];
        if (st.un_from_primitive) {
            double pn_z[NF];
#pragma unroll
            for (int q = 0; q < NF; ++q)
                pn_z[q] = pn[at(i, j, nj) + q];
            p2c_fast(k, pn_z, un);
        } else {
#pragma unroll
            for (int q = 0; q < NF; ++q)
                un[q] = un_all[at(i, j, nj) + q];
        }
        double out[NF];
        tile_phase2<ROLE>(k, st, sm, ty, threadIdx.x, un, out, cv);
        // the zone and, on the edges, its zero-gradient guard images
        const int ilo = (st.write_guards && i == 0) ? -NG : i, ihi = (st.write_guards && i == ni - 1) ? ni + 1 : i;
        const int jlo = (st.write_guards && j == 0) ? -NG : j, jhi = (st.write_guards && j == nj - 1) ? nj + 1 : j;
        for (int ii = ilo; ii <= ihi; ++ii)
            for (int jj = jlo; jj <= jhi; ++jj) {
                double *dst = pwr + at(ii, jj, nj);
#pragma unroll
                for (int q = 0; q < NF; ++q)
                    dst[q] = out[q];
            }
        if (ws_max)
            ws = max_nan(ws, zone_wavespeed(out, k.gamma));
    }
    cbd::chain_end();
    if (ws_max) {  // uniform over the block
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            ws = max_nan(ws, __shfl_xor_sync(0xffffffffu, ws, o));
        if ((tid & 31) == 0)
            sm.warp_max[tid >> 5] = ws;
        __syncthreads();
        if (tid == 0) {
            double m = sm.warp_max[0];
            for (int w = 1; w < NT / 32; ++w)
                m = max_nan(m, sm.warp_max[w]);
            atomicMax(ws_max, (unsigned long long)__double_as_longlong(m));
        }
    }
}
