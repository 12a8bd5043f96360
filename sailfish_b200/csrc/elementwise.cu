// Zone-wise kernels: the three smaller drop-in kernels of the reference
// (cbdiso_2d.c:606-722), the guard-zone fill, and the standalone reduction of
// the CFL wavespeed and diagnostics. Built with -fmad=false so their
// arithmetic matches the reference's CPU build operation for operation.
#include "cbd_internal.h"
#include "elementwise.h"
#include "zone_walk.cuh"

namespace cbd {

namespace {

__device__ __forceinline__ size_t zoff(int i, int j, int nj)
{
    return ((size_t)(i + NG) * (size_t)(nj + 2 * NG) + (size_t)(j + NG)) * NQ;
}

// A zone's three values to `dst`, a warp's 32 consecutive zones together where
// they lie in one row: through `sm` (the warp's own 96 doubles), so that each
// store writes whole sectors. The conversion is bound by its stores: zone by
// zone, 8 of every 24 bytes at a time, 512^2 4.7 us, 1000^2 13.3, 2048^2 49,
// 4096^2 192 (4.2 TB/s); together 2.9, 6.8, 32 and 124 (6.5 TB/s). The source
// term reads the sectors that it writes, and gains nothing by it (1511^2 22.0
// -> 24.1 us, 2048^2 47 -> 49).
__device__ __forceinline__ void store_zone(double *dst, const double *v, double *sm, long z, long n, int j, int nj)
{
    const int lane = threadIdx.x & 31;
    const long last = z - lane + 31;
    if (j >= lane && j - lane + 31 < nj && last < n) {
#pragma unroll
        for (int q = 0; q < 3; ++q)
            sm[3 * lane + q] = v[q];
        __syncwarp();
        double *base = dst - 3 * lane;
#pragma unroll
        for (int q = 0; q < 3; ++q)
            base[32 * q + lane] = sm[32 * q + lane];
        __syncwarp();
    } else {
#pragma unroll
        for (int q = 0; q < 3; ++q)
            dst[q] = v[q];
    }
}

// Threads map to zones with j (the contiguous axis) fastest.
__global__ void __launch_bounds__(256) p2c_kernel(int ni, int nj, const double *p, double *u)
{
    __shared__ double stage[8][96];
    chain_begin();
    const long n = (long)ni * nj;
    const long step = (long)gridDim.x * blockDim.x, z0 = blockIdx.x * (long)blockDim.x + threadIdx.x;
    ZoneWalk w(z0, step, nj);
    for (long z = z0; z < n; z += step, w.next()) {
        const int i = w.i, j = w.j;
        const size_t o = zoff(i, j, nj);
        const double rho = p[o];
        const double v[3] = {rho, p[o + 1] * rho, p[o + 2] * rho};
        store_zone(u + o, v, stage[threadIdx.x >> 5], z, n, j, nj);
    }
}

__global__ void source_kernel(int ni, int nj, double xl, double yl, double dx, double dy, MassDev m,
                              const double *p, double *rate)
{
    chain_begin();
    const long n = (long)ni * nj;
    const long step = (long)gridDim.x * blockDim.x, z0 = blockIdx.x * (long)blockDim.x + threadIdx.x;
    ZoneWalk w(z0, step, nj);
    for (long z = z0; z < n; z += step, w.next()) {
        const int i = w.i, j = w.j;
        const size_t o = zoff(i, j, nj);
        const double xc = xl + (i + 0.5) * dx;
        const double yc = yl + (j + 0.5) * dy;
        double du[3] = {rate[o], rate[o + 1], rate[o + 2]};
        mass_source<false>(m, xc, yc, 1.0, p + o, du);
        rate[o] = du[0];
        rate[o + 1] = du[1];
        rate[o + 2] = du[2];
    }
}

// ANY: a sound speed whose square may lie outside the straight-line root's range
template <bool ANY>
__global__ void wavespeed_kernel(int ni, int nj, Consts k, MassDev m0, MassDev m1, const double *p, double *ws)
{
    chain_begin();
    const long n = (long)ni * nj;
    MassDev m[2] = {m0, m1};
    const long step = (long)gridDim.x * blockDim.x, z0 = blockIdx.x * (long)blockDim.x + threadIdx.x;
    ZoneWalk w(z0, step, nj);
    for (long z = z0; z < n; z += step, w.next()) {
        const int i = w.i, j = w.j;
        const double xc = k.xl + (i + 0.5) * k.dx;
        const double yc = k.yl + (j + 0.5) * k.dy;
        const double c2 = sound_speed2<false>(k, m, xc, yc);
        ws[(size_t)(i + NG) * (nj + 2 * NG) + (j + NG)] =
            signal_speed(p + zoff(i, j, nj), ANY ? sqrt(c2) : crm::sqrt_rn(c2));
    }
}

__global__ void fill_guards_kernel(int ni, int nj, double *p)
{
    const long wi = ni + 2 * NG, wj = nj + 2 * NG;
    const long step = (long)gridDim.x * blockDim.x, z0 = blockIdx.x * (long)blockDim.x + threadIdx.x;
    ZoneWalk w(z0, step, (int)wj);
    for (long z = z0; z < wi * wj; z += step, w.next()) {
        const int ii = w.i - NG, jj = w.j - NG;
        if (ii >= 0 && ii < ni && jj >= 0 && jj < nj)
            continue;
        const int ci = ii < 0 ? 0 : (ii >= ni ? ni - 1 : ii);
        const int cj = jj < 0 ? 0 : (jj >= nj ? nj - 1 : jj);
        const size_t src = zoff(ci, cj, nj), dst = zoff(ii, jj, nj);
        p[dst] = p[src];
        p[dst + 1] = p[src + 1];
        p[dst + 2] = p[src + 2];
    }
}

template <int BJ>
__global__ void __launch_bounds__(BJ) reduce_kernel(const Consts k, const StageDev st, const double *p,
                                                    double *scratch, double *out0, double *out_rest)
{
    __shared__ double sred[PARTIAL_STRIDE * (BJ / 32)];
    chain_begin();
    double acc[PARTIAL_STRIDE];
#pragma unroll
    for (int v = 0; v < PARTIAL_STRIDE; ++v)
        acc[v] = 0.0;
    const long n = (long)k.ni * k.nj;
    const long step = (long)gridDim.x * BJ, z0 = blockIdx.x * (long)BJ + threadIdx.x;
    ZoneWalk w(z0, step, k.nj);
    for (long z = z0; z < n; z += step, w.next()) {
        const int i = w.i, j = w.j;
        const double *pc = p + zoff(i, j, k.nj);
        const double pz[3] = {pc[0], pc[1], pc[2]};
        const double xc = k.xl + (i + 0.5) * k.dx;
        const double yc = k.yl + (j + 0.5) * k.dy;
        accumulate_zone<false>(k, st.e, xc, yc, pz, acc);
    }
    double red[PARTIAL_STRIDE];
    block_reduce<BJ>(acc, sred, red);
    grid_finish<BJ>(red, 1 + 2 * k.num_diag, scratch, out0, out_rest, sred);
}

// Evaluates the stencil's correctly rounded arithmetic on arrays, so tests
// can compare it with IEEE division and high-precision powers:
// out[4i] = a / b, out[4i+1] = a^-1.5, out[4i+2] = a^4, out[4i+3] = the
// limited slope of (a, b, a + b) with theta = 1.5.
__global__ void primitives_kernel(long n, const double *a, const double *b, double *out)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        out[4 * i] = div_rn<false>(a[i], b[i]);
        out[4 * i + 1] = pow_m15_rn(a[i]);
        out[4 * i + 2] = pow4_rn(a[i]);
        out[4 * i + 3] = limited_slope(a[i], b[i], a[i] + b[i], 1.5);
    }
}

// quotients and roots without CUDA's slow paths: a / b, sqrt |b|, a / sqrt |b|
__global__ void roots_kernel(long n, const double *a, const double *b, double *out)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        out[3 * i] = div_rn<false>(a[i], b[i]);
        out[3 * i + 1] = crm::sqrt_rn(fabs(b[i]));
        out[3 * i + 2] = crm::over_sqrt_rn(a[i], fabs(b[i]));
    }
}

inline int blocks_for(long n, int bs, int cap)
{
    long b = (n + bs - 1) / bs;
    if (b < 1)
        b = 1;
    return (int)(b < cap ? b : cap);
}

// Blocks of 256 threads for a pass over n zones: two waves of them, the rest in
// further rounds, which keeps the arrays' sectors close in time while they fit
// the L2; a zone or two per thread where they do not. Measured, conversion /
// source / wavespeed, us, 16 and 64 blocks per SM: 1511^2 16.8 / 22.0 / 15.6
// and 18.4 / 23.6 / 18.4, 2048^2 33.9 / 47.2 / 28.4 and 31.6 / 45.1 / 28.7,
// 4096^2 136 / 184 / 103 and 123 / 178 / 97.
int zone_blocks(long n)
{
    return blocks_for(n, 256, n < 2048L * 2048 ? 148 * 16 : 148 * 64);
}

}  // namespace

cudaError_t launch_p2c(int ni, int nj, const double *p, double *u, cudaStream_t s)
{
    return launch_chained(p2c_kernel, zone_blocks((long)ni * nj), 256, 0, s, ni, nj, p, u);
}

cudaError_t launch_source(int ni, int nj, double xl, double yl, double dx, double dy, const MassDev &m,
                          const double *p, double *rate, cudaStream_t s)
{
    return launch_chained(source_kernel, zone_blocks((long)ni * nj), 256, 0, s, ni, nj, xl, yl, dx, dy, m,
                          p, rate);
}

cudaError_t launch_wavespeed(const Consts &k, const MassDev &m0, const MassDev &m1, const double *p, double *ws,
                             cudaStream_t s)
{
    // a constant cs^2 is the caller's; the masses' potentials are numbers of
    // ordinary size unless Mach^2 is not (tested zone by zone: 27.7 -> 28.8 us at
    // 2048^2)
    const bool any = k.eos == 1   ? k.cs2 != 0.0 && !(k.cs2 >= 0x1p-960 && k.cs2 < 0x1p960)
                     : k.eos == 2 ? !(k.mach2 > 1e-100 && k.mach2 < 1e100)
                                  : false;
    return launch_chained(any ? wavespeed_kernel<true> : wavespeed_kernel<false>, zone_blocks((long)k.ni * k.nj), 256,
                          0, s, k.ni, k.nj, k, m0, m1, p, ws);
}

cudaError_t launch_fill_guards(int ni, int nj, double *p, cudaStream_t s)
{
    const long n = (long)(ni + 2 * NG) * (nj + 2 * NG);
    fill_guards_kernel<<<blocks_for(n, 256, 148 * 16), 256, 0, s>>>(ni, nj, p);
    return cudaGetLastError();
}

cudaError_t launch_primitives(long n, const double *a, const double *b, double *out, cudaStream_t s)
{
    primitives_kernel<<<blocks_for(n, 256, 148 * 16), 256, 0, s>>>(n, a, b, out);
    return cudaGetLastError();
}

cudaError_t launch_roots(long n, const double *a, const double *b, double *out, cudaStream_t s)
{
    roots_kernel<<<blocks_for(n, 256, 148 * 16), 256, 0, s>>>(n, a, b, out);
    return cudaGetLastError();
}

int reduce_ctas(int ni, int nj)
{
    return blocks_for((long)ni * nj, 256, 148 * 8);
}

cudaError_t launch_reduce(const Consts &k, const StageDev &st, const double *p, double *scratch, double *out0,
                          double *out_rest, cudaStream_t s)
{
    return launch_chained(reduce_kernel<256>, reduce_ctas(k.ni, k.nj), 256, 0, s, k, st, p, scratch, out0, out_rest);
}

}  // namespace cbd
