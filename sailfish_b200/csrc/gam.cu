// The gamma-law circumbinary-disk stage (cbdgam_2d): the reference's
// energy-equation sibling of cbdiso_2d (sailfish/solvers/cbdgam_2d.c), with
// four fields (sigma, vx, vy, pressure), alpha viscosity with the disk's
// scale height, softening that may follow the scale height, cooling, a
// pressure floor and a Mach ceiling.
//
// Built with -fmad=false: every +, -, *, / and sqrt gives the IEEE result the
// reference's CPU build computes, in the reference's order, and every power
// and exponential is correctly rounded (cr_math.cuh), so results differ from
// the reference only where glibc's pow / exp are not (about one call in a
// thousand for the non-integer exponents).
//
// One launch per RK stage: a row march (gam_march.cuh), or 16 x 32 tiles on
// grids of middle size (gam_tile.cuh).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>

#include "async.cuh"
#include "cbdiso_b200.h"
#include "chain.cuh"
#include "cr_math.cuh"
#include "zone_walk.cuh"

namespace cbd {
cudaStream_t drop_in_stream();  // capi.cu: the stream set by cbdiso_b200_set_stream
int segment_rows(int ni, int strips, int bj, int slots);  // capi.cu: rows per CTA of a march
}

namespace gam {

constexpr int NF = 4;
constexpr int NG = 2;

struct Mass {
    double x, y, vx, vy, mass, soft, rate, radius;
    int model;
};

struct Consts {
    int ni, nj;
    double xl, yl, dx, dy;
    double theta, gamma, alpha, cooling, mach_ceiling, vmax, rho_floor, p_floor;
    int constant_softening;
    int buffer_on;
    // the buffer: Sigma, internal energy and onset radius of its target, the span
    // of its ramp, a squared radius surely inside the onset, reciprocals
    double buf_sigma, buf_energy, buf_onset, buf_span, buf_lo2, inv_buf_sigma, inv_buf_span;
    double mach_m2;       // pow(mach_ceiling, -2.0), glibc's on the host
    double inv_dx, inv_dy, gm1, inv_gm1, inv_gamma;  // RN(1 / dx), ..., gamma - 1, RN(1 / (gamma - 1)), RN(1 / gamma)
};

struct Stage {
    Mass m[2];
    double buf_mass, a, dt;
    double buf_k;  // driving rate times the orbital frequency at the onset radius
    int massless;  // both masses have zero mass: every scale height is 1
    int write_guards;
    int un_from_primitive;  // u_n = cons(primitive_n) in-kernel (else: a conserved array)
    double *ws_clear;  // zeroed by the stage (or null): the maximum that a later stage of the step maxes into
};

// Powers and the exponential are correctly rounded (cr_math.cuh): in a
// near-vacuum zone an ulp in the energy update is amplified by the
// cancellation between total and kinetic energy, so matching glibc's
// correctly rounded results matters here.
using crm::cube_rn;
using crm::exp_rn;
using crm::fourth_rn;
using crm::inv_pow15_rn;
using crm::inv_square_rn;
using crm::pow_m13_rn;
using crm::recip_rn;
using crm::sqrt_rn;

__device__ __forceinline__ double lesser(double a, double b) { return a < b ? a : b; }
__device__ __forceinline__ double greater(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ double sign_of(double x) { return copysign(1.0, x); }
__device__ __forceinline__ size_t at(int i, int j, int nj) { return ((size_t)(i + NG) * (nj + 2 * NG) + (j + NG)) * NF; }

// cbdgam_2d.c:27-33: 0.25 |sgn a + sgn b| (sgn a + sgn c) min(|a|, |b|, |c|),
// up to the sign of a zero: theta min(|dl|, |dr|) is min(|a|, |c|) because
// rounding is monotonic, and where dl and dr are nonzero with one sign yr - yl
// has it too.
__device__ __forceinline__ double slope(double yl, double y0, double yr, double theta)
{
    const double dl = y0 - yl, dr = yr - y0;
    const double m = lesser(0.5 * fabs(yr - yl), theta * lesser(fabs(dl), fabs(dr)));
    return (__double2hiint(dl) ^ __double2hiint(dr)) < 0 ? 0.0 : copysign(m, dl);
}

template <class V>
__device__ __forceinline__ double cs2_of(double gamma, const V &p) { return p[3] / p[0] * gamma; }

// a / b rounded to nearest from y = RN(1 / b): the remainder a - q b of
// q = RN(a y) is exact under FMA and one correction rounds to RN(a / b)
__device__ __forceinline__ double div_by(double a, double b, double y)
{
    const double q = a * y;
    return fma(fma(-q, b, a), y, q);
}

__device__ __forceinline__ double div_rn(double a, double b) { return div_by(a, b, recip_rn(b)); }

// T = p / Sigma, the sound speed sqrt(T gamma) (cbdgam_2d.c:231-236) and sqrt(T)
struct Thermal {
    double T, cs, sq;
};

// for any pressure and density, by CUDA's operators; out of line, where its
// callers go only for arguments that the straight-line ones do not cover
__device__ __noinline__ Thermal thermal_any(double pres, double sigma, double gamma)
{
    Thermal r;
    r.T = pres / sigma;
    r.cs = sqrt(r.T * gamma);
    r.sq = sqrt(r.T);
    return r;
}

__device__ __forceinline__ bool thermal_in_range(double pres, double T)
{
    return crm::mid_range(pres) & crm::mid_range(T);
}

// WIDE: any pressure and density (stage_wide says when a stage needs that)
template <bool WIDE>
__device__ __forceinline__ Thermal thermal(double pres, double sigma, double gamma)
{
    Thermal r;
    r.T = div_rn(pres, sigma);
    r.cs = sqrt_rn(r.T * gamma);
    r.sq = sqrt_rn(r.T);
    if (WIDE && !thermal_in_range(pres, r.T))
        r = thermal_any(pres, sigma, gamma);
    return r;
}

// cbdgam_2d.c:238-276
__device__ __forceinline__ void buffer_source(const Consts &k, const Stage &st, double x, double y, double dt,
                                              double *u)
{
    const double r2 = x * x + y * y;
    if (!k.buffer_on || !(r2 > k.buf_lo2))
        return;
    const double rc = sqrt_rn(r2);
    if (rc > k.buf_onset) {
        const double yr = recip_rn(rc);
        const double pf = k.buf_sigma * sqrt_rn(div_by(st.buf_mass, rc, yr));
        const double px = pf * div_by(-y, rc, yr), py = pf * div_by(x, rc, yr);
        const double ek = div_by(0.5 * (px * px + py * py), k.buf_sigma, k.inv_buf_sigma);
        const double target[NF] = {k.buf_sigma, px, py, k.buf_energy + ek};
        // a ramp of no width, or one that starts at the origin, has an infinite
        // rate, as in the reference
        const double ramp = st.buf_k * (rc - k.buf_onset), steep = ramp * k.inv_buf_span;
        const double rate = isinf(steep) ? steep : div_by(ramp, k.buf_span, k.inv_buf_span);
#pragma unroll
        for (int q = 0; q < NF; ++q)
            u[q] -= (u[q] - target[q]) * rate * dt;
    }
}

// cbdgam_2d.c:347-362
template <class V>
__device__ __forceinline__ void prim_to_cons(const V &p, double *u, double gamma)
{
    const double rho = p[0], vx = p[1], vy = p[2], pres = p[3];
    u[0] = rho;
    u[1] = vx * rho;
    u[2] = vy * rho;
    u[3] = pres / (gamma - 1.0) + 0.5 * rho * (vx * vx + vy * vy);
}

// cbdgam_2d.c:401-409 for a sound speed
template <class V>
__device__ __forceinline__ double max_wavespeed(const V &p, double cs)
{
    const double ax = greater(fabs(p[1] - cs), fabs(p[1] + cs));
    const double ay = greater(fabs(p[2] - cs), fabs(p[2] + cs));
    return greater(ax, ay);
}

// the same of a zone with any pressure and density
__device__ __forceinline__ double zone_wavespeed(const double *p, double gamma)
{
    const double T = div_rn(p[3], p[0]);
    double cs = sqrt_rn(T * gamma);
    if (!thermal_in_range(p[3], T))
        cs = thermal_any(p[3], p[0], gamma).cs;
    return max_wavespeed(p, cs);
}

// sqrt(w2) of the scale height (cbdgam_2d.c:75-106) at (x, y)
__device__ __forceinline__ double root_w2(const Mass *m, double x, double y)
{
    double w2 = 0.0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (m[k].mass > 0.0) {
            const double dx = x - m[k].x, dy = y - m[k].y;
            w2 += m[k].mass * crm::inv_cube_of_sqrt_rn(dx * dx + dy * dy + 1e-12);
        }
    }
    return sqrt_rn(w2);
}

// cbdgam_2d.c:347-362 with the constant divisor gamma - 1
template <class V>
__device__ __forceinline__ void p2c_fast(const Consts &k, const V &p, double *u)
{
    const double rho = p[0], vx = p[1], vy = p[2], pres = p[3];
    u[0] = rho;
    u[1] = vx * rho;
    u[2] = vy * rho;
    u[3] = div_by(pres, k.gm1, k.inv_gm1) + 0.5 * rho * (vx * vx + vy * vy);
}

template <bool ANY>
__device__ __forceinline__ double gravity_factor(double s2)
{
    return ANY ? inv_pow15_rn(s2) : crm::pow_m15_rn(s2);
}

// cbdgam_2d.c:108-203: gravity, sink and their work on the gas for one mass,
// given T = p / Sigma, the disk height h and gamma - 1 with its reciprocal.
// FAR takes the short form beyond the sink's reach, where the stages lose
// nothing by it: a term that is zero times a non-finite value adds a NaN to a
// conserved value that already is one. ANY: any r^2 + softening^2 and T.
template <bool FAR, bool ANY, class V>
__device__ __forceinline__ void mass_source(const Mass &m, double x, double y, double dt, const V &p, double T,
                                            double h, int constant_softening, double gm1, double inv_gm1, double *du,
                                            const double *g_in = nullptr, double *g_out = nullptr)
{
    const double sigma = p[0];
    const double dx = x - m.x, dy = y - m.y;
    const double r2 = dx * dx + dy * dy;
    // Beyond four sink radii (with a margin far above the square root's
    // rounding) the sink rate is zero and the softening, if it follows the
    // disk height, is half of it: only gravity's terms are left, the others
    // being exact zeros for a finite state.
    const double far2 = 16.0 * (m.radius * m.radius);
    if (FAR && r2 > far2 * (1.0 + 1e-10)) {
        const double soft = constant_softening ? m.soft : 0.5 * h;
        const double g = g_in ? *g_in : gravity_factor<ANY>(r2 + soft * soft);
        if (g_out)
            *g_out = g;
        const double fnum = m.model >= 1 && m.model <= 3 ? sigma * m.mass * g : 0.0;
        const double fx = -fnum * dx, fy = -fnum * dy;
        du[0] = 0.0;
        du[1] = dt * fx;
        du[2] = dt * fy;
        du[3] = dt * (fx * p[1] + fy * p[2]);
        return;
    }
    const double eps = ANY ? T / gm1 : div_by(T, gm1, inv_gm1);
    const double dr = sqrt_rn(r2);
    const double rs = m.radius;
    double soft;
    if (constant_softening) {
        soft = m.soft;
    } else if (dr > rs) {
        soft = 0.5 * h;
    } else {
        const double q = dr / rs;
        const double w = (1.0 - q * q) * (1.0 - q * q);  // pow(., 2.0) is the correctly rounded square
        soft = w * rs + (1.0 - w) * 0.5 * h;
    }
    const double rate = (dr < 4.0 * rs) ? m.rate * exp_rn(-fourth_rn(dr / rs)) : 0.0;
    // the gravity factor: from the face cache (constant softening), or computed
    const double g = g_in ? *g_in : gravity_factor<ANY>(r2 + soft * soft);
    if (g_out)
        *g_out = g;
    const double fnum = sigma * m.mass * g;
    const double fx = -fnum * dx, fy = -fnum * dy;
    const double mdot = sigma * rate * -1.0;
    const double vx = p[1], vy = p[2];
    if (m.model == 1) {
        du[0] = dt * mdot;
        du[1] = dt * mdot * p[1] + dt * fx;
        du[2] = dt * mdot * p[2] + dt * fy;
        du[3] = dt * (mdot * eps + 0.5 * mdot * (vx * vx + vy * vy)) + dt * (fx * vx + fy * vy);
    } else if (m.model == 2) {
        const double den = dr + 1e-12, yd = recip_rn(den);
        const double ex = div_by(dx, den, yd), ey = div_by(dy, den, yd);
        const double dvr = (vx - m.vx) * ex + (vy - m.vy) * ey;
        const double wx = dvr * ex + m.vx, wy = dvr * ey + m.vy;
        du[0] = dt * mdot;
        du[1] = dt * mdot * wx + dt * fx;
        du[2] = dt * mdot * wy + dt * fy;
        du[3] = dt * (mdot * eps + 0.5 * mdot * (wx * wx + wy * wy)) + dt * (fx * vx + fy * vy);
    } else if (m.model == 3) {
        du[0] = dt * mdot;
        du[1] = dt * fx;
        du[2] = dt * fy;
        du[3] = dt * (fx * vx + fy * vy);
    } else {
        du[0] = du[1] = du[2] = du[3] = 0.0;
    }
}

// 2^-298 <= |x| < 2^298, by the exponent field: within 1e-90 to 1e90
__device__ __forceinline__ bool power_range(double x)
{
    return ((unsigned)__double2hiint(x) & 0x7fffffffu) - 0x2d500000u < 0x25400000u;
}

// cooling's factor for any argument, out of line
__device__ __noinline__ double cooling_factor(double cooling, double sigma, double eps, double dt)
{
    return pow_m13_rn(1.0 + 3.0 * cooling * inv_square_rn(sigma) * cube_rn(eps) * dt);
}

// cbdgam_2d.c:298-317 with T = p / Sigma given
template <class V>
__device__ __forceinline__ void cooling_fast(const Consts &k, double dt, const V &p, double T, double *u)
{
    const double sigma = p[0];
    const double eps = div_by(T, k.gm1, k.inv_gm1);
    // without cooling the power's argument is exactly 1 and so is the power
    // (for finite Sigma^-2 eps^3, which the floors keep)
    double cooled = eps;
    if (k.cooling != 0.0) {
        const double x = 1.0 + 3.0 * k.cooling * crm::inv_square_in(sigma) * crm::cube_in(eps) * dt;
        double w = crm::pow_m13_in(x);
        // outside the powers' safe ranges, 1e-90 to 1e90 in magnitude and 1 to
        // 1e90, or thereabouts (by the exponent fields)
        if (!(power_range(sigma) && power_range(eps) && (unsigned)(__double2hiint(x) - 0x3ff00000) < 0x12a00000u))
            w = cooling_factor(k.cooling, sigma, eps, dt);
        cooled *= w;
    }
    const double ek = 0.5 * (p[1] * p[1] + p[2] * p[2]);
    cooled = greater(cooled, div_by(div_by(2.0 * ek, k.gamma, k.inv_gamma), k.gm1, k.inv_gm1) * k.mach_m2);
    u[3] += sigma * (cooled - eps);
}

// cbdgam_2d.c:319-345 with one reciprocal of Sigma
__device__ __forceinline__ void c2p_fast(const Consts &k, const double *u, double *p)
{
    const double y = recip_rn(u[0]);
    double pres = greater(k.p_floor, (u[3] - div_by(0.5 * (u[1] * u[1] + u[2] * u[2]), u[0], y)) * k.gm1);
    double vx = sign_of(u[1]) * lesser(fabs(div_by(u[1], u[0], y)), k.vmax);
    double vy = sign_of(u[2]) * lesser(fabs(div_by(u[2], u[0], y)), k.vmax);
    double rho = u[0];
    if (u[0] < k.rho_floor) {
        rho = k.rho_floor;
        vx = 0.0;
        vy = 0.0;
        pres = k.p_floor;
    }
    p[0] = rho;
    p[1] = vx;
    p[2] = vy;
    p[3] = pres;
}

// a maximum that keeps a NaN operand, so that a NaN wavespeed reaches the host
__device__ __forceinline__ double max_nan(double a, double b) { return (a > b || a != a) ? a : b; }

// ---------------------------------------------------------------------------
// Face cache. The scale heights' geometry sqrt(sum_m M_m r^-3) at every x- and
// y-face and zone centre, and (with constant softening) the gravity factors
// (r^2 + s^2)^-1.5 of both masses at every zone, depend only on the mesh and
// the point masses. RK2's second stage runs at t0 + dt, which is the next
// step's start time in all but about 1 step in 5000 (cbdgam_2d.py's time
// update), so the host makes that stage a writer when its masses equal the
// end-of-step masses (it stores the values with a key of their inputs) and
// the next step's first stage a reader (it loads them, after a fill kernel
// that recomputes them when the key does not match). The same bits either
// way; each role is its own kernel.
//
// Layout (doubles): a 32-double header holding the key, then the zones'
// (sqrt(w2), g_1) pairs ni x nj, the zones' g_2 ni x nj, the x-faces
// (ni + 1) x nj ([i][j]: between rows i - 1 and i) and the y-faces
// ni x (nj + 1) ([i][j]: between columns j - 1 and j).
// ---------------------------------------------------------------------------

enum { ROLE_NONE = 0, ROLE_WRITER = 1, ROLE_READER = 2 };
constexpr int CACHE_HEADER = 32;
constexpr int CACHE_KEY = 16;

struct CacheView {
    double *zp, *zg2, *xf, *yf;
};

__host__ __device__ inline size_t cache_doubles(int ni, int nj)
{
    return CACHE_HEADER + 3 * (size_t)ni * nj + (size_t)(ni + 1) * nj + (size_t)ni * (nj + 1);
}

__device__ __forceinline__ CacheView cache_view(const Consts &k, double *fc)
{
    CacheView v;
    v.zp = fc + CACHE_HEADER;
    v.zg2 = v.zp + 2 * (size_t)k.ni * k.nj;
    v.xf = v.zg2 + (size_t)k.ni * k.nj;
    v.yf = v.xf + (size_t)(k.ni + 1) * k.nj;
    return v;
}

// the key: a format tag, then every input of the cached values
__device__ __forceinline__ double cache_key_value(const Consts &k, const Mass *m, int v)
{
    switch (v) {
    case 0: return 20260102.5;
    case 1: return (double)k.ni;
    case 2: return (double)k.nj;
    case 3: return k.xl;
    case 4: return k.yl;
    case 5: return k.dx;
    case 6: return k.dy;
    case 7: return (double)k.constant_softening;
    default: {
        const Mass &q = m[(v - 8) >> 2];
        switch ((v - 8) & 3) {
        case 0: return q.x;
        case 1: return q.y;
        case 2: return q.mass;
        default: return q.soft;
        }
    }
    }
}

#include "gam_march.cuh"
#include "gam_tile.cuh"

// Makes the face cache valid for a reader stage: when the key does not match
// the stage's masses, marks it invalid (no later key check passes on what
// follows) and computes every value for those masses with the stage kernel's
// own expressions. CTAs take rows i = blockIdx.x, blockIdx.x + gridDim.x, ...
__global__ void __launch_bounds__(128) cache_fill_kernel(Consts k, Stage st, double *fc)
{
    cbd::chain_begin();
    const int v = threadIdx.x;
    if (__syncthreads_and(v >= CACHE_KEY ||
                          __double_as_longlong(fc[v]) == __double_as_longlong(cache_key_value(k, st.m, v))))
        return;
    if (v == 0)
        fc[0] = 0.0;  // every block compares before its own write, and any order of the others' reads is a mismatch
    const CacheView cv = cache_view(k, fc);
    const int ni = k.ni, nj = k.nj;
    for (int i = blockIdx.x; i <= ni; i += gridDim.x) {
        for (int j = threadIdx.x; j <= nj; j += blockDim.x) {
            if (j < nj)
                cv.xf[(size_t)i * nj + j] = root_w2(st.m, k.xl + (i + 0.0) * k.dx, k.yl + (j + 0.5) * k.dy);
            if (i < ni)
                cv.yf[(size_t)i * (nj + 1) + j] = root_w2(st.m, k.xl + (i + 0.5) * k.dx, k.yl + (j + 0.0) * k.dy);
            if (i < ni && j < nj) {
                const double xc = k.xl + (i + 0.5) * k.dx, yc = k.yl + (j + 0.5) * k.dy;
                double g[2];
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const double dx = xc - st.m[p].x, dy = yc - st.m[p].y;
                    const double r2 = dx * dx + dy * dy;
                    g[p] = crm::pow_m15_rn(r2 + st.m[p].soft * st.m[p].soft);
                }
                const size_t z = (size_t)i * nj + j;
                *reinterpret_cast<double2 *>(cv.zp + 2 * z) = make_double2(root_w2(st.m, xc, yc), g[0]);
                cv.zg2[z] = g[1];
            }
        }
    }
}

__global__ void p2c_kernel(int ni, int nj, double gamma, const double *prim, double *cons)
{
    const long n = (long)ni * nj;
    const long step = (long)gridDim.x * blockDim.x, z0 = blockIdx.x * (long)blockDim.x + threadIdx.x;
    cbd::ZoneWalk w(z0, step, nj);
    for (long z = z0; z < n; z += step, w.next()) {
        const int i = w.i, j = w.j;
        prim_to_cons(prim + at(i, j, nj), cons + at(i, j, nj), gamma);
    }
}

__global__ void wavespeed_kernel(int ni, int nj, double gamma, const double *prim, double *ws)
{
    const long n = (long)ni * nj;
    const long step = (long)gridDim.x * blockDim.x, z0 = blockIdx.x * (long)blockDim.x + threadIdx.x;
    cbd::ZoneWalk w(z0, step, nj);
    for (long z = z0; z < n; z += step, w.next()) {
        const int i = w.i, j = w.j;
        const double *p = prim + at(i, j, nj);
        ws[(size_t)(i + NG) * (nj + 2 * NG) + (j + NG)] = max_wavespeed(p, sqrt(cs2_of(gamma, p)));
    }
}

// whether the straight-line operations cover a zone, given T = p / Sigma
__device__ __forceinline__ bool zone_in_range(const double *p, double T)
{
    const int vx = __double2hiint(p[1]) & 0x7ff00000, vy = __double2hiint(p[2]) & 0x7ff00000;
    return thermal_in_range(p[3], T) & (max(vx, vy) != 0x7ff00000);
}

struct SourceArgs {
    int ni, nj;
    double xl, yl, dx, dy;
    Mass m[2];
    int which, constant_softening, massless;
    double gm1, inv_gm1;
};

// one zone's source terms; ANY as in mass_source, with the height by CUDA's operators
template <bool ANY>
__device__ __forceinline__ void zone_source(const SourceArgs &a, int i, int j, const double *p, double T, double *rate)
{
    const double xc = a.xl + (i + 0.5) * a.dx, yc = a.yl + (j + 0.5) * a.dy;
    double h = 1.0;  // cbdgam_2d.c:75-106
    if (!a.massless) {
        const double w = root_w2(a.m, xc, yc);
        h = ANY ? sqrt(T) / w : div_rn(sqrt_rn(T), w);
    }
    mass_source<!ANY, ANY>(a.m[a.which - 1], xc, yc, 1.0, p, T, h, a.constant_softening, a.gm1, a.inv_gm1, rate);
}

__device__ __noinline__ void any_zone_source(const SourceArgs &a, int i, int j, const double *p, double *rate)
{
    zone_source<true>(a, i, j, p, p[3] / p[0], rate);
}

__global__ void source_kernel(const __grid_constant__ SourceArgs a, const double *prim, double *rate)
{
    const long n = (long)a.ni * a.nj;
    const long step = (long)gridDim.x * blockDim.x, z0 = blockIdx.x * (long)blockDim.x + threadIdx.x;
    cbd::ZoneWalk w(z0, step, a.nj);
    for (long z = z0; z < n; z += step, w.next()) {
        const double *p = prim + at(w.i, w.j, a.nj);
        double *r = rate + at(w.i, w.j, a.nj);
        const double T = div_rn(p[3], p[0]);
        if (zone_in_range(p, T))
            zone_source<false>(a, w.i, w.j, p, T, r);
        else
            any_zone_source(a, w.i, w.j, p, r);
    }
}

// zero-gradient guard images of a state (the reference's outflow set_bc)
__global__ void guards_kernel(int ni, int nj, double *a)
{
    const long wi = ni + 2 * NG, wj = nj + 2 * NG;
    const long step = (long)gridDim.x * blockDim.x, z0 = blockIdx.x * (long)blockDim.x + threadIdx.x;
    cbd::ZoneWalk w(z0, step, (int)wj);
    for (long z = z0; z < wi * wj; z += step, w.next()) {
        const int ii = w.i - NG, jj = w.j - NG;
        if (ii >= 0 && ii < ni && jj >= 0 && jj < nj)
            continue;
        const int ci = ii < 0 ? 0 : (ii >= ni ? ni - 1 : ii);
        const int cj = jj < 0 ? 0 : (jj >= nj ? nj - 1 : jj);
#pragma unroll
        for (int q = 0; q < NF; ++q)
            a[at(ii, jj, nj) + q] = a[at(ci, cj, nj) + q];
    }
}

// ---------------------------------------------------------------------------
// reductions: the CFL wavespeed maximum and the diagnostic sums
// ---------------------------------------------------------------------------

constexpr int RED_THREADS = 256;
constexpr int MAX_DIAG = 4;
constexpr int RED_VALUES = 1 + 2 * MAX_DIAG;

struct Diag {
    int quantity, which_mass, gravity, accretion, has_cut;
    double r0, r1;
};

struct RedArgs {
    Consts k;
    Mass m[2];
    Diag d[MAX_DIAG];
    int nd;
};

// a mass's source rates (dt = 1) for a diagnostic: the accretion rates
// (masses zero) when its accretion flag is set, else the gravity rates
// (sink rates zero), as the reference's reductions pass mass * gravity and
// sink_rate * accretion (cbdgam_2d.py:104-139, 346-349, 397-402); the first
// three, rate[3] is not used. ANY: a zone of any values, whose non-finite ones
// show, else one that zone_in_range has passed.
template <bool ANY>
__device__ __forceinline__ void diag_rates(const RedArgs &r, const Diag &d, int which, double xc, double yc,
                                           const double *p, double *rate)
{
    Mass m = r.m[which - 1];
    const double T = ANY ? p[3] / p[0] : div_rn(p[3], p[0]);
    double h = 1.0;
    if (d.accretion) {
        // without masses every height is 1; beyond the sink's reach the rates
        // of finite values are zeros
        const double dx = xc - m.x, dy = yc - m.y;
        if (!ANY && dx * dx + dy * dy > 16.0 * (m.radius * m.radius) * (1.0 + 1e-10)) {
            rate[0] = rate[1] = rate[2] = 0.0;
            return;
        }
        m.mass = m.mass * 0.0;
    } else {
        m.rate = m.rate * 0.0;
        // the height enters through a softening that follows it (cbdgam_2d.c:75-106)
        const bool massless = r.m[0].mass == 0.0 && r.m[1].mass == 0.0;
        if (!r.k.constant_softening && !massless) {
            const double w = root_w2(r.m, xc, yc);
            h = ANY ? sqrt(T) / w : div_rn(sqrt_rn(T), w);
        }
    }
    mass_source<!ANY, ANY>(m, xc, yc, 1.0, p, T, h, r.k.constant_softening, r.k.gm1, r.k.inv_gm1, rate);
}

template <bool ANY>
__device__ __forceinline__ void diag_value(const RedArgs &r, const Diag &d, double x, double y, const double *p,
                                           double *re, double *im)
{
    const bool polar = d.quantity == CBD_Q_SIGMA_M1 || d.quantity == CBD_Q_ECCENTRICITY_VECTOR;
    const double rr = polar || d.has_cut ? sqrt(x * x + y * y) : 0.0;
    const double cut = d.has_cut ? (double)((d.r0 < rr) * (rr < d.r1)) : 1.0;
    *im = 0.0;
    if (d.quantity == CBD_Q_SIGMA_M1) {
        const double s = p[0] * cut;
        *re = s * (x / rr);
        *im = s * (y / rr);
        return;
    }
    if (d.quantity == CBD_Q_ECCENTRICITY_VECTOR) {
        const double s = p[0] * cut, vx = p[1] * cut, vy = p[2] * cut;
        const double vv = vx * vx + vy * vy, vr = vx * x + vy * y;
        *re = s * ((vv * x - vr * vx) / 1.0 - x / rr);
        *im = s * ((vv * y - vr * vy) / 1.0 - y / rr);
        return;
    }
    double f[3] = {0.0, 0.0, 0.0};
    for (int which = 1; which <= 2; ++which) {
        if (d.which_mass != 3 && d.which_mass != which)
            continue;
        double rate[NF];
        diag_rates<ANY>(r, d, which, x, y, p, rate);
        for (int q = 0; q < 3; ++q)
            f[q] += rate[q];
    }
    if (d.quantity == CBD_Q_MDOT)
        *re = f[0] * cut;
    else  // torque
        *re = x * (f[2] * cut) - y * (f[1] * cut);
}

// The values of a thread's zones z0, z0 + step, ... into v; false when one of
// them needs ANY.
template <bool ANY>
__device__ __forceinline__ bool add_zones(const RedArgs &r, const double *prim, long z0, long step, double *v)
{
    const Consts &k = r.k;
    const long n = (long)k.ni * k.nj;
    bool ok = true;
    for (int q = 0; q < RED_VALUES; ++q)
        v[q] = 0.0;
    cbd::ZoneWalk w(z0, step, k.nj);
    for (long z = z0; z < n; z += step, w.next()) {
        const int i = w.i, j = w.j;
        const double *p = prim + at(i, j, k.nj);
        const double T = ANY ? p[3] / p[0] : div_rn(p[3], p[0]);
        v[0] = max_nan(v[0], max_wavespeed(p, ANY ? sqrt(T * k.gamma) : sqrt_rn(T * k.gamma)));
        ok &= zone_in_range(p, T);
        const double x = k.xl + (i + 0.5) * k.dx, y = k.yl + (j + 0.5) * k.dy;
        for (int d = 0; d < r.nd; ++d) {
            double re, im;
            diag_value<ANY>(r, r.d[d], x, y, p, &re, &im);
            v[1 + 2 * d] += re;
            v[2 + 2 * d] += im;
        }
    }
    return ok;
}

__device__ __noinline__ void add_any_zones(const RedArgs &r, const double *prim, long z0, long step, double *v)
{
    add_zones<true>(r, prim, z0, step, v);
}

// Per-block partial sums in a fixed tree order; the wavespeed maximum. A
// thread that met a value outside the straight-line operations' range (a flag
// kept beside the sums; tested zone by zone it cost 5 %) takes its zones again.
__global__ void __launch_bounds__(RED_THREADS) reduce_kernel(const __grid_constant__ RedArgs r, const double *prim,
                                                             double *partials)
{
    __shared__ double sm[RED_VALUES][RED_THREADS];
    cbd::chain_begin();
    double v[RED_VALUES];
    const long step = (long)gridDim.x * RED_THREADS, z0 = blockIdx.x * (long)RED_THREADS + threadIdx.x;
    if (!add_zones<false>(r, prim, z0, step, v))
        add_any_zones(r, prim, z0, step, v);
    for (int q = 0; q < RED_VALUES; ++q)
        sm[q][threadIdx.x] = v[q];
    __syncthreads();
    for (int w = RED_THREADS / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            sm[0][threadIdx.x] = max_nan(sm[0][threadIdx.x], sm[0][threadIdx.x + w]);
            for (int q = 1; q < RED_VALUES; ++q)
                sm[q][threadIdx.x] += sm[q][threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x < RED_VALUES)
        partials[(size_t)blockIdx.x * RED_VALUES + threadIdx.x] = sm[threadIdx.x][0];
}

// The blocks' partials to the result, a warp per value: lane l takes the blocks
// l, l + 32, ... in order, then a fixed shuffle tree (one thread per value over
// all blocks took 13 us, most of it the chain of comparisons and additions).
__global__ void __launch_bounds__(32 * RED_VALUES) finish_kernel(const double *partials, int nblocks, double *result)
{
    cbd::chain_begin();
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double s = 0.0;
#pragma unroll 4
    for (int b = lane; b < nblocks; b += 32) {
        const double x = partials[(size_t)b * RED_VALUES + q];
        s = q == 0 ? max_nan(s, x) : s + x;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_down_sync(0xffffffffu, s, o);
        s = q == 0 ? max_nan(s, x) : s + x;
    }
    if (lane == 0)
        result[q] = s;
}

// RN(x^-3), the hook's alone (the kernels cube a root: inv_cube_of_sqrt_rn): x^3
// as a double-double p + e, whose reciprocal's first approximation q = RN(1 / p)
// leaves the exact residual 1 - q p, and one correction rounds once
__device__ __forceinline__ double inv_cube_rn(double x)
{
    if (!crm::in_range(fabs(x)))
        return pow(x, -3.0);
    const double h = x * x, l = fma(x, x, -h);
    const double p = h * x, e = fma(h, x, -p) + l * x;
    const double q = 1.0 / p;
    return q + q * (fma(-q, p, 1.0) - q * e);
}

// the correctly rounded helpers on device arrays (a test hook)
__global__ void eval_powers_kernel(long n, const double *x, double *out)
{
    for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
        const double v = x[t];
        double *o = out + 8 * t;
        o[0] = cube_rn(v);
        o[1] = inv_square_rn(v);
        o[2] = inv_cube_rn(v);
        o[3] = fourth_rn(v);
        o[4] = inv_pow15_rn(v);
        o[5] = pow_m13_rn(1.0 + v);
        o[6] = exp_rn(-v);
        o[7] = crm::inv_cube_of_sqrt_rn(v * v + 1e-12);
    }
}

constexpr int RED_BLOCKS = 592;  // 4 per SM on a B200; fixed so the summation order is too

double g_theta = 1.5;  // the drop-in kernels' PLM theta (the reference fixes 1.5)

bool grid_ok(const cbdgam_grid_t *g)
{
    return g && g->ni > 0 && g->nj > 0 && g->xr > g->xl && g->yr > g->yl && g->gamma_law_index != 1.0;
}

Consts consts_of(const cbdgam_grid_t *g)
{
    Consts k;
    std::memset(&k, 0, sizeof(k));
    k.ni = g->ni;
    k.nj = g->nj;
    k.xl = g->xl;
    k.yl = g->yl;
    k.dx = (g->xr - g->xl) / g->ni;
    k.dy = (g->yr - g->yl) / g->nj;
    k.theta = g->plm_theta;
    k.gamma = g->gamma_law_index;
    k.alpha = g->alpha;
    k.cooling = g->cooling_coefficient;
    k.mach_ceiling = g->mach_ceiling;
    k.vmax = g->velocity_ceiling;
    k.rho_floor = g->density_floor;
    k.p_floor = g->pressure_floor;
    k.constant_softening = g->constant_softening;
    k.buffer_on = g->buffer_is_enabled;
    k.buf_sigma = g->buffer_surface_density;
    k.buf_energy = g->buffer_surface_pressure / (k.gamma - 1.0);
    k.buf_onset = g->buffer_outer_radius - g->buffer_onset_width;
    k.buf_span = g->buffer_outer_radius - k.buf_onset;
    k.buf_lo2 = k.buf_onset > 0.0 ? k.buf_onset * k.buf_onset * (1.0 - 1e-10) : -1.0;
    k.inv_buf_sigma = 1.0 / k.buf_sigma;
    k.inv_buf_span = 1.0 / k.buf_span;
    k.mach_m2 = std::pow(g->mach_ceiling, -2.0);
    k.inv_dx = 1.0 / k.dx;
    k.inv_dy = 1.0 / k.dy;
    k.gm1 = k.gamma - 1.0;
    k.inv_gm1 = 1.0 / k.gm1;
    k.inv_gamma = 1.0 / k.gamma;
    return k;
}

// cbdgam_2d.c:266-267 on the host, with the C library's pow
double buffer_k(double driving_rate, double central_mass, double outer_radius, double onset_width)
{
    return driving_rate * std::sqrt(central_mass * std::pow(outer_radius - onset_width, -3.0));
}

Mass mass_of(const cbd_mass_t &m)
{
    return Mass{m.x, m.y, m.vx, m.vy, m.mass, m.softening_length, m.sink_rate, m.sink_radius, m.sink_model};
}

Mass mass_args(double x, double y, double vx, double vy, double mass, double soft, double rate, double radius,
               int model)
{
    return Mass{x, y, vx, vy, mass, soft, rate, radius, model};
}

int status_of(cudaError_t e) { return e == cudaSuccess ? CBD_OK : CBD_ERR_CUDA; }

// raises a kernel's dynamic shared memory limit, a per-device attribute, once
int prepare_kernel(const void *kernel, int smem, bool (&ready)[64])
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
        return CBD_ERR_CUDA;
    if (!ready[dev]) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return CBD_ERR_CUDA;
        ready[dev] = true;
    }
    return CBD_OK;
}

// the reader stage's fill pass
int launch_fill(const Consts &k, const Stage &st, double *fc, cudaStream_t s)
{
    const int rows = k.ni + 1 < 148 * 4 ? k.ni + 1 : 148 * 4;
    return status_of(cbd::launch_chained(cache_fill_kernel, rows, 128, 0, s, k, st, fc));
}

template <int BJ, int MINB, int ROLE, bool WIDE>
int launch_march(const Consts &k, const Stage &st, const double *prd, const double *pn, const double *un,
                 double *pwr, double *ws_max, double *fc, cudaStream_t s)
{
    static bool ready[64] = {};
    const int smem = (int)sizeof(MarchSmem<BJ>);
    int rc = prepare_kernel(reinterpret_cast<const void *>(stage_kernel<BJ, MINB, ROLE, WIDE>), smem, ready);
    if (rc == CBD_OK && ROLE == ROLE_READER)
        rc = launch_fill(k, st, fc, s);
    if (rc != CBD_OK)
        return rc;
    const int strips = (k.nj + BJ - 1) / BJ;
    const int rows = cbd::segment_rows(k.ni, strips, BJ, 148 * MINB);
    return status_of(cbd::launch_chained(stage_kernel<BJ, MINB, ROLE, WIDE>, dim3(strips, (k.ni + rows - 1) / rows), BJ, smem,
                                         s, k, st, rows, prd, pn, un, pwr,
                                         reinterpret_cast<unsigned long long *>(ws_max), fc));
}

template <int ROLE, bool WIDE>
int launch_tiles(const Consts &k, const Stage &st, const double *prd, const double *pn, const double *un,
                 double *pwr, double *ws_max, double *fc, cudaStream_t s)
{
    static bool ready[64] = {};
    int rc = prepare_kernel(reinterpret_cast<const void *>(tile_kernel<ROLE, WIDE>), (int)sizeof(TileSmem), ready);
    if (rc == CBD_OK && ROLE == ROLE_READER)
        rc = launch_fill(k, st, fc, s);
    if (rc != CBD_OK)
        return rc;
    const dim3 grid((k.nj + TJ - 1) / TJ, (k.ni + TI - 1) / TI), block(TJ, TI / RPT);
    return status_of(cbd::launch_chained(tile_kernel<ROLE, WIDE>, grid, block, sizeof(TileSmem), s, k, st, prd, pn, un, pwr,
                                         reinterpret_cast<unsigned long long *>(ws_max), fc));
}

// The march where its CTAs hold one row each and all fit at once (the latency
// of one zone's update is what counts there), and on large grids, where its
// segments are long; the tiles between. Measured, us per step, tiles / march:
// 64^2 30 / 20, 130^2 29 / 23, 200^2 30 / 26, 256^2 30 / 32, 384^2 38 / 50, 512^2
// 66 / 69, 704^2 111 / 126, 900^2 175 / 188, 1000^2 227 / 216, 1280^2 358 / 323,
// 2048^2 870 / 760 (with cooling 238 / 228, 377 / 345, 920 / 818).
//
// A last strip of few columns takes up the march's slots like a full one, so on
// a large grid its strips may hold at most 8 % more columns than the tiles'
// 32-column ones: 13000 x 130 428 / 591 (strips of 256 against 160 columns),
// 13000 x 200 600 / 654, 8000 x 260 478 / 555, 8000 x 300 528 / 559, 4096 x 385
// 358 / 445, 1153^2 294 / 300, 1700 x 1025 373 / 377 (1.09); 1281^2 356 / 342
// (1.07), 1024 x 1800 396 / 399 (1.05), 2600 x 640 346 / 348, 13000 x 256 681 /
// 649, 26000 x 100 675 / 651, 300 x 8000 517 / 470. Its 64-column strips serve
// small grids only: 26000 x 60 350 / 367, 26000 x 96 519 / 704.
// Strips of 128 columns at 3 CTAs per SM, narrow grids in 64 columns.
constexpr int MARCH_CTAS = 3;

bool march_suits(int ni, int nj)
{
    const long strips = (nj + 127) / 128, zones = (long)ni * nj;
    if (strips * ni <= 148 * MARCH_CTAS * (nj <= 96 ? 2 : 1))
        return true;
    const long tile_columns = (nj + TJ - 1) / TJ * TJ;
    return zones >= 960L * 960 && nj > 96 && strips * 128 <= 1.08 * tile_columns;
}

// columns of a CTA of the stage kernel
int stage_columns(int ni, int nj) { return !march_suits(ni, nj) ? TJ : (nj <= 96 ? 64 : 128); }

template <int ROLE, bool WIDE>
int launch_form(const Consts &k, const Stage &st, const double *prd, const double *pn, const double *un,
                double *pwr, double *ws_max, double *fc, cudaStream_t s)
{
    switch (stage_columns(k.ni, k.nj)) {
    case TJ:
        return launch_tiles<ROLE, WIDE>(k, st, prd, pn, un, pwr, ws_max, fc, s);
    case 64:
        return launch_march<64, 2 * MARCH_CTAS, ROLE, WIDE>(k, st, prd, pn, un, pwr, ws_max, fc, s);
    default:
        return launch_march<128, MARCH_CTAS, ROLE, WIDE>(k, st, prd, pn, un, pwr, ws_max, fc, s);
    }
}

// Whether a stage may meet temperatures outside the range of the straight-line
// roots. The test splits the march's longest chain: 2048^2 743 -> 761 us per
// step, 1153^2 (tiles) 290 -> 291. With a pressure floor above 1e-90 only
// densities above 1e198, or an initial state below the floor whose sound speed
// (below 1e-144) moves nothing, could have one; without such a floor a cold gas
// can.
bool stage_wide(const Consts &k) { return !(k.p_floor > 1e-90); }

template <int ROLE>
int launch_role(const Consts &k, const Stage &st, const double *prd, const double *pn, const double *un,
                double *pwr, double *ws_max, double *fc, cudaStream_t s)
{
    return stage_wide(k) ? launch_form<ROLE, true>(k, st, prd, pn, un, pwr, ws_max, fc, s)
                         : launch_form<ROLE, false>(k, st, prd, pn, un, pwr, ws_max, fc, s);
}

int launch_stage(const Consts &k, const Stage &st, const double *prd, const double *pn, const double *un,
                 double *pwr, double *ws_max, cudaStream_t s, double *fc = nullptr, int role = ROLE_NONE)
{
    Stage s2 = st;
    s2.massless = st.m[0].mass == 0.0 && st.m[1].mass == 0.0;
    switch (role) {
    case ROLE_WRITER:
        return launch_role<ROLE_WRITER>(k, s2, prd, pn, un, pwr, ws_max, fc, s);
    case ROLE_READER:
        return launch_role<ROLE_READER>(k, s2, prd, pn, un, pwr, ws_max, fc, s);
    default:
        return launch_role<ROLE_NONE>(k, s2, prd, pn, un, pwr, ws_max, nullptr, s);
    }
}

int blocks_for(long n, int t)
{
    const long b = (n + t - 1) / t;
    return (int)(b < 2048 ? (b > 0 ? b : 1) : 2048);
}

}  // namespace gam

using namespace gam;

extern "C" {

int cbdgam_b200_eval_powers(long n, const double *x, double *out, void *stream)
{
    if (n < 0 || (n > 0 && (!x || !out)))
        return CBD_ERR_ARGUMENT;
    if (n == 0)
        return CBD_OK;
    eval_powers_kernel<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(n, x, out);
    return status_of(cudaGetLastError());
}

void cbdgam_b200_disk_primitive(long n, const double *x, const double *y, double softening_length,
                                double initial_sigma, double initial_pressure, double *primitive)
{
    // host code: the C library's sqrt / pow / exp, as Python's math and float
    // power call them, in the setup's operation order
    for (long k = 0; k < n; ++k) {
        const double xk = x[k], yk = y[k];
        const double r = std::sqrt(xk * xk + yk * yk);
        const double rs = std::sqrt(xk * xk + yk * yk + softening_length * softening_length);
        const double rmax = 1e-12 > r ? 1e-12 : r;
        const double phx = -yk / rmax, phy = +xk / rmax;
        const double taper = 0.0001 + 0.9999 * std::exp(-std::pow(1.0 / rs, 30.0));
        double *p = primitive + 4 * k;
        p[0] = initial_sigma * std::pow(rs, -3.0 / 5.0) * taper;
        p[1] = std::sqrt(1.0 / rs) * phx;
        p[2] = std::sqrt(1.0 / rs) * phy;
        p[3] = initial_pressure * std::pow(rs, -3.0 / 2.0) * taper;
    }
}

void cbdgam_b200_abi_sizes(size_t out[2])
{
    out[0] = sizeof(cbdgam_grid_t);
    out[1] = sizeof(cbdgam_stage_t);
}

int cbdgam_b200_set_plm_theta(double theta)
{
    if (!(theta >= 1.0 && theta <= 2.0))
        return CBD_ERR_ARGUMENT;
    g_theta = theta;
    return CBD_OK;
}

int cbdgam_2d_advance_rk(int ni, int nj, double xl, double xr, double yl, double yr, double *conserved_rk,
                         double *primitive_rd, double *primitive_wr, double gamma_law_index,
                         double buffer_surface_density, double buffer_surface_pressure, double buffer_central_mass,
                         double buffer_driving_rate, double buffer_outer_radius, double buffer_onset_width,
                         int buffer_is_enabled, double x1, double y1, double vx1, double vy1, double mass1,
                         double softening_length1, double sink_rate1, double sink_radius1, int sink_model1, double x2,
                         double y2, double vx2, double vy2, double mass2, double softening_length2,
                         double sink_rate2, double sink_radius2, int sink_model2, double alpha, double a, double dt,
                         double velocity_ceiling, double cooling_coefficient, double mach_ceiling,
                         double density_floor, double pressure_floor, int constant_softening)
{
    if (ni <= 0 || nj <= 0 || !conserved_rk || !primitive_rd || !primitive_wr)
        return CBD_ERR_ARGUMENT;
    cbdgam_grid_t g;
    std::memset(&g, 0, sizeof(g));
    g.ni = ni;
    g.nj = nj;
    g.xl = xl;
    g.xr = xr;
    g.yl = yl;
    g.yr = yr;
    g.plm_theta = g_theta;
    g.gamma_law_index = gamma_law_index;
    g.alpha = alpha;
    g.cooling_coefficient = cooling_coefficient;
    g.mach_ceiling = mach_ceiling;
    g.velocity_ceiling = velocity_ceiling;
    g.density_floor = density_floor;
    g.pressure_floor = pressure_floor;
    g.constant_softening = constant_softening;
    g.buffer_is_enabled = buffer_is_enabled;
    g.buffer_surface_density = buffer_surface_density;
    g.buffer_surface_pressure = buffer_surface_pressure;
    g.buffer_driving_rate = buffer_driving_rate;
    g.buffer_outer_radius = buffer_outer_radius;
    g.buffer_onset_width = buffer_onset_width;
    Stage st;
    std::memset(&st, 0, sizeof(st));
    st.m[0] = mass_args(x1, y1, vx1, vy1, mass1, softening_length1, sink_rate1, sink_radius1, sink_model1);
    st.m[1] = mass_args(x2, y2, vx2, vy2, mass2, softening_length2, sink_rate2, sink_radius2, sink_model2);
    st.buf_mass = buffer_central_mass;
    st.buf_k = buffer_k(buffer_driving_rate, buffer_central_mass, buffer_outer_radius, buffer_onset_width);
    st.a = a;
    st.dt = dt;
    st.write_guards = 0;
    st.un_from_primitive = 0;
    return launch_stage(consts_of(&g), st, primitive_rd, nullptr, conserved_rk, primitive_wr, nullptr,
                        cbd::drop_in_stream());
}

int cbdgam_2d_wavespeed(int ni, int nj, double *primitive, double *wavespeed, double gamma_law_index)
{
    if (ni <= 0 || nj <= 0 || !primitive || !wavespeed)
        return CBD_ERR_ARGUMENT;
    wavespeed_kernel<<<blocks_for((long)ni * nj, 256), 256, 0,
                       cbd::drop_in_stream()>>>(ni, nj, gamma_law_index,
                                                                                   primitive, wavespeed);
    return status_of(cudaGetLastError());
}

int cbdgam_2d_primitive_to_conserved(int ni, int nj, double *primitive, double *conserved, double gamma_law_index)
{
    if (ni <= 0 || nj <= 0 || !primitive || !conserved)
        return CBD_ERR_ARGUMENT;
    p2c_kernel<<<blocks_for((long)ni * nj, 256), 256, 0, cbd::drop_in_stream()>>>(
        ni, nj, gamma_law_index, primitive, conserved);
    return status_of(cudaGetLastError());
}

int cbdgam_2d_point_mass_source_term(int ni, int nj, double xl, double xr, double yl, double yr, double x1,
                                     double y1, double vx1, double vy1, double mass1, double softening_length1,
                                     double sink_rate1, double sink_radius1, int sink_model1, double x2, double y2,
                                     double vx2, double vy2, double mass2, double softening_length2,
                                     double sink_rate2, double sink_radius2, int sink_model2, int which_mass,
                                     double *primitive, double *cons_rate, int constant_softening,
                                     double gamma_law_index)
{
    if (ni <= 0 || nj <= 0 || !primitive || !cons_rate || (which_mass != 1 && which_mass != 2))
        return CBD_ERR_ARGUMENT;
    SourceArgs a;
    a.ni = ni;
    a.nj = nj;
    a.xl = xl;
    a.yl = yl;
    a.dx = (xr - xl) / ni;
    a.dy = (yr - yl) / nj;
    a.m[0] = mass_args(x1, y1, vx1, vy1, mass1, softening_length1, sink_rate1, sink_radius1, sink_model1);
    a.m[1] = mass_args(x2, y2, vx2, vy2, mass2, softening_length2, sink_rate2, sink_radius2, sink_model2);
    a.which = which_mass;
    a.constant_softening = constant_softening;
    a.massless = mass1 == 0.0 && mass2 == 0.0;
    a.gm1 = gamma_law_index - 1.0;
    a.inv_gm1 = 1.0 / a.gm1;
    source_kernel<<<blocks_for((long)ni * nj, 256), 256, 0, cbd::drop_in_stream()>>>(a, primitive, cons_rate);
    return status_of(cudaGetLastError());
}

}  // extern "C"

namespace {

bool cache_ok(const double *face_cache, int role)
{
    // the zone pairs are moved as 16-byte vectors
    return face_cache && (reinterpret_cast<uintptr_t>(face_cache) & 15) == 0 && role >= ROLE_NONE &&
           role <= ROLE_READER;
}

int advance_stage(const cbdgam_grid_t *grid, const cbdgam_stage_t *stage, const double *primitive_rd,
                  const double *primitive_n, double *primitive_wr, double *wavespeed_max, double *face_cache,
                  int role, void *stream, double *wavespeed_clear = nullptr)
{
    if (!grid_ok(grid) || !stage || !primitive_rd || !primitive_wr || primitive_wr == primitive_rd)
        return CBD_ERR_ARGUMENT;
    if (!primitive_n) {
        if (stage->a != 0.0)
            return CBD_ERR_ARGUMENT;
        primitive_n = primitive_rd;  // the first stage's u_n is the state it reads
    }
    Stage st;
    std::memset(&st, 0, sizeof(st));
    st.m[0] = mass_of(stage->mass[0]);
    st.m[1] = mass_of(stage->mass[1]);
    st.buf_mass = stage->buffer_central_mass;
    st.buf_k = buffer_k(grid->buffer_driving_rate, stage->buffer_central_mass, grid->buffer_outer_radius,
                        grid->buffer_onset_width);
    st.a = stage->a;
    st.dt = stage->dt;
    st.write_guards = 1;
    st.un_from_primitive = 1;
    st.ws_clear = wavespeed_clear;
    return launch_stage(consts_of(grid), st, primitive_rd, primitive_n, nullptr, primitive_wr, wavespeed_max,
                        static_cast<cudaStream_t>(stream), face_cache, role);
}

}  // namespace

extern "C" {

int cbdgam_b200_advance_stage(const cbdgam_grid_t *grid, const cbdgam_stage_t *stage, const double *primitive_rd,
                              const double *primitive_n, double *primitive_wr, double *wavespeed_max, void *stream)
{
    return advance_stage(grid, stage, primitive_rd, primitive_n, primitive_wr, wavespeed_max, nullptr, ROLE_NONE,
                         stream);
}

size_t cbdgam_b200_face_cache_bytes(const cbdgam_grid_t *grid)
{
    if (!grid_ok(grid))
        return 0;
    return cache_doubles(grid->ni, grid->nj) * sizeof(double);
}

int cbdgam_b200_advance_stage_cached(const cbdgam_grid_t *grid, const cbdgam_stage_t *stage,
                                     const double *primitive_rd, const double *primitive_n, double *primitive_wr,
                                     double *wavespeed_max, double *face_cache, int role, void *stream)
{
    if (!cache_ok(face_cache, role))
        return CBD_ERR_ARGUMENT;
    return advance_stage(grid, stage, primitive_rd, primitive_n, primitive_wr, wavespeed_max, face_cache, role,
                         stream);
}

int cbdgam_b200_advance_first_stage(const cbdgam_grid_t *grid, const cbdgam_stage_t *stage,
                                    const double *primitive_rd, double *primitive_wr, double *wavespeed_clear,
                                    double *face_cache, int role, void *stream)
{
    if (!wavespeed_clear || (role != ROLE_NONE && !cache_ok(face_cache, role)))
        return CBD_ERR_ARGUMENT;
    return advance_stage(grid, stage, primitive_rd, nullptr, primitive_wr, nullptr, face_cache, role, stream,
                         wavespeed_clear);
}

int cbdgam_b200_stage_columns(const cbdgam_grid_t *grid)
{
    return grid_ok(grid) ? stage_columns(grid->ni, grid->nj) : 0;
}

int cbdgam_b200_fill_guards(const cbdgam_grid_t *grid, double *primitive, void *stream)
{
    if (!grid_ok(grid) || !primitive)
        return CBD_ERR_ARGUMENT;
    const long n = (long)(grid->ni + 4) * (grid->nj + 4);
    guards_kernel<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(grid->ni, grid->nj,
                                                                                      primitive);
    return status_of(cudaGetLastError());
}

size_t cbdgam_b200_scratch_bytes(const cbdgam_grid_t *grid)
{
    if (!grid_ok(grid))
        return 0;
    return (size_t)RED_BLOCKS * RED_VALUES * sizeof(double);
}

int cbdgam_b200_reduce(const cbdgam_grid_t *grid, const cbd_mass_t *masses, const cbd_diag_t *diags, int num_diags,
                       const double *primitive, double *scratch, double *result, void *stream)
{
    if (!grid_ok(grid) || !masses || !primitive || !scratch || !result || num_diags < 0 ||
        num_diags > MAX_DIAG || (num_diags > 0 && !diags))
        return CBD_ERR_ARGUMENT;
    RedArgs r;
    std::memset(&r, 0, sizeof(r));
    r.k = consts_of(grid);
    r.m[0] = mass_of(masses[0]);
    r.m[1] = mass_of(masses[1]);
    for (int d = 0; d < num_diags; ++d) {
        const cbd_diag_t &src = diags[d];
        if (src.quantity != CBD_Q_MDOT && src.quantity != CBD_Q_TORQUE && src.quantity != CBD_Q_SIGMA_M1 &&
            src.quantity != CBD_Q_ECCENTRICITY_VECTOR)
            return CBD_ERR_ARGUMENT;
        const bool rates = src.quantity == CBD_Q_MDOT || src.quantity == CBD_Q_TORQUE;
        if (rates && ((!src.accretion && !src.gravity) || src.which_mass < 1 || src.which_mass > 3))
            return CBD_ERR_ARGUMENT;
        r.d[d] = Diag{src.quantity, src.which_mass, src.gravity, src.accretion, src.has_cut, src.r0, src.r1};
    }
    r.nd = num_diags;
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    const cudaError_t e = cbd::launch_chained(reduce_kernel, RED_BLOCKS, RED_THREADS, 0, s, r, primitive, scratch);
    if (e != cudaSuccess)
        return status_of(e);
    return status_of(cbd::launch_chained(finish_kernel, 1, 32 * RED_VALUES, 0, s, scratch, RED_BLOCKS, result));
}

}  // extern "C"
