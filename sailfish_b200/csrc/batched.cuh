// Many grids ("disks") of different sizes and physics advanced by one
// persistent launch per RK stage. The work is the list of all tiles
// (disk, strip, segment), largest disks first; each CTA takes the next tile
// from an atomic counter, loads that disk's constants and stage record into
// shared memory and marches the tile with the same code as the single-grid
// kernel. Per-tile epilogue partials are reduced per disk afterwards, in tile
// order, by one CTA per disk.
#pragma once

#include "cbd_stencil.cuh"

namespace cbd {

struct DiskDev {
    Consts k;            // the disk's kernel constants (k.rows_per_cta = tile rows)
    long long offset;    // offset of the disk's state, in doubles, in the batch buffers
    int strip_width;     // tile columns (<= the kernel's thread count)
    int strips;
    int segments;
    int unit_begin;      // index of the disk's first tile in the batch's tile list
    long long cache_offset;  // offset of the disk's face cache in BatchArgs::fcache, in doubles; -1: none
};

struct BatchArgs {
    const DiskDev *disks;
    int num_disks;
    int total_units;
    const double *prd;
    const double *un;    // u_n source (primitive_n), or null for a = 0 stages
    double *pwr;
    const StageDev *records;  // records[disk * num_stages + stage]
    int num_stages;
    int stage;
    int epilogue;        // the step's last stage: 1, or 2 when every disk's diagnostics are source
                         // rates without a radial cut (Consts::rates_only; the launch then takes the
                         // kernel compiled for those)
    int _pad;
    double *partials;    // [total_units][PARTIAL_STRIDE]
    unsigned int *counters;  // [0] next tile, [1] CTAs finished; both return to zero at the end
    double *fcache;      // face-cache arena (disk d's cache at disks[d].cache_offset), or null
};

// the disk that tile u belongs to
__device__ __forceinline__ int disk_of_unit(const BatchArgs &a, int u)
{
    int lo = 0, hi = a.num_disks - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (a.disks[mid].unit_begin <= u)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// disk d's constants and stage record into shared memory, a word per thread
template <int BJ>
__device__ __forceinline__ void load_disk(const BatchArgs &a, int d, Consts &k, StageDev &st)
{
    const double *src = reinterpret_cast<const double *>(&a.disks[d].k);
    double *dst = reinterpret_cast<double *>(&k);
    for (int w = threadIdx.x; w < (int)(sizeof(Consts) / sizeof(double)); w += BJ)
        dst[w] = src[w];
    load_record<BJ>(st, st, &a.records[(size_t)d * a.num_stages + a.stage]);
}

// ROLE (ROLE_*) is what the launch does with each disk's face cache: a writer
// stores into the caches of the disks that have one; a reader requires one
// for every disk (the batch's fill kernel ran before it), skips the tiles of
// a disk without one, and the disk's first tile records the key.
template <int BJ, int MINB, int PREC, int ROLE = ROLE_NONE>
__global__ void __launch_bounds__(BJ, MINB) batched_stage_kernel(const BatchArgs a)
{
    constexpr bool FAST = PREC == CBD_PRECISION_FAST;
    __shared__ Consts k;
    __shared__ StageDev st;
    __shared__ int s_unit, s_disk;
    const int t = threadIdx.x;
    chain_begin();

    for (;;) {
        if (t == 0) {
            const int u = (int)atomicAdd(&a.counters[0], 1u);
            s_unit = u;
            if (u < a.total_units)
                s_disk = disk_of_unit(a, u);
        }
        __syncthreads();
        const int u = s_unit;
        if (u >= a.total_units)
            break;
        const DiskDev &D = a.disks[s_disk];
        load_disk<BJ>(a, s_disk, k, st);
        __syncthreads();
        if (t == 0) {
            k.un_kind = a.un ? 1 : 0;
            k.write_guards = 1;
        }
        __syncthreads();
        const int local = u - D.unit_begin;
        const int strip = local % D.strips;
        const int seg = local / D.strips;
        StageArgs sa;
        sa.prd = a.prd + D.offset;
        sa.un = a.un ? a.un + D.offset : nullptr;
        sa.pwr = a.pwr + D.offset;
        sa.stage_dev = nullptr;
        sa.scratch = nullptr;
        sa.result = nullptr;
        const bool cached = ROLE != ROLE_NONE && a.fcache && D.cache_offset >= 0;
        sa.fcache = cached ? a.fcache + D.cache_offset : nullptr;
        const int c0 = strip * D.strip_width, r0 = seg * k.rows_per_cta;
        if (st.halt) {
            // the disk's stepper stopped: no march
        } else if (ROLE == ROLE_WRITER) {
            // the same answer in every thread; the block with the disk's first tile writes the key
            const bool store = cached && cache_write_check<PREC>(k, st, sa.fcache, u == D.unit_begin);
            march_tile<BJ, FAST, CACHE_WRITE>(k, st, sa, c0, D.strip_width, r0, store);
        } else if (ROLE == ROLE_READER) {
            if (cached) {
                march_tile<BJ, FAST, CACHE_READ>(k, st, sa, c0, D.strip_width, r0);
                // the fill kernel ran before this launch; no tile reads the key
                if (u == D.unit_begin)
                    cache_write_key<PREC>(k, st, sa.fcache);
            }
        } else {
            march_tile<BJ, FAST, CACHE_NONE>(k, st, sa, c0, D.strip_width, r0);
        }
        __syncthreads();
    }
    if (t == 0) {
        __threadfence();
        const unsigned int done = atomicAdd(&a.counters[1], 1u);
        if (done == gridDim.x - 1) {
            a.counters[0] = 0u;
            a.counters[1] = 0u;
            __threadfence();
        }
    }
}

// The face caches of every disk valid for a reader stage (see
// face_cache_fill_kernel): CTA (d, b) compares disk d's key and, when it does
// not match the disk's stage masses, fills the disk's tiles b, b + gridDim.y,
// ... (One comparison per tile, by one thread, took 37 us for 1864 tiles of 24
// disks.)
template <int BJ, int PREC>
__global__ void __launch_bounds__(BJ, FILL_WARPS_PER_SM * 32 / BJ) batched_fill_kernel(const BatchArgs a)
{
    __shared__ Consts k;
    __shared__ StageDev st;
    chain_begin();
    const DiskDev &D = a.disks[blockIdx.x];
    if (D.cache_offset < 0)
        return;
    load_disk<BJ>(a, blockIdx.x, k, st);
    __syncthreads();
    double *fc = a.fcache + D.cache_offset;
    if (cache_key_matches<PREC>(k, st, fc) || st.halt)
        return;
    for (int u = blockIdx.y; u < D.strips * D.segments; u += gridDim.y)
        face_cache_fill_tile<BJ, PREC == CBD_PRECISION_FAST>(k, st.m, fc, (u % D.strips) * D.strip_width,
                                                             D.strip_width, (u / D.strips) * k.rows_per_cta,
                                                             k.rows_per_cta);
}

// The epilogue of every disk's tiles after the step's last stage: CTA u
// reduces tile u exactly as the single grid's epilogue kernel does and leaves
// its partials for batched_finalize. CACHED: the stage before was a writer,
// whose gravity factors serve when its masses are the end-of-step masses.
template <int BJ, int PREC, bool RATES>
__global__ void __launch_bounds__(BJ, epi_warps(RATES) * 32 / BJ)
    batched_epilogue_kernel(const BatchArgs a, const bool cached)
{
    constexpr bool FAST = PREC == CBD_PRECISION_FAST;
    __shared__ Consts k;
    __shared__ StageDev st;
    __shared__ double sred[PARTIAL_STRIDE * (BJ / 32)];
    __shared__ int s_disk;
    const int u = blockIdx.x, t = threadIdx.x;
    chain_begin();
    if (t == 0)
        s_disk = disk_of_unit(a, u);
    __syncthreads();
    load_disk<BJ>(a, s_disk, k, st);
    __syncthreads();
    const DiskDev &D = a.disks[s_disk];
    double acc[PARTIAL_STRIDE];
#pragma unroll
    for (int v = 0; v < PARTIAL_STRIDE; ++v)
        acc[v] = 0.0;
    // a disk whose stepper stopped: zero partials
    if (!st.halt) {
        const int local = u - D.unit_begin;
        const double *grav = nullptr;
        if (cached && a.fcache && D.cache_offset >= 0 && same_cached_inputs(st))
            grav = cache_arrays(a.fcache + D.cache_offset, k.ni, k.nj).grav;
        epilogue_tile<BJ, FAST, RATES>(k, st, a.pwr + D.offset, grav, (local % D.strips) * D.strip_width, D.strip_width,
                                   (local / D.strips) * k.rows_per_cta, acc);
    }
    double red[PARTIAL_STRIDE];
    block_reduce<BJ, RATES>(acc, sred, red);
    // a disk whose diagnostics the rates-only kernel cannot evaluate (a wrong
    // epilogue form from the caller): NaN sums, not wrong ones
    if (RATES && !k.rates_only) {
#pragma unroll
        for (int v = 1; v < PARTIAL_STRIDE; ++v)
            red[v] = __longlong_as_double(0x7ff8000000000000LL);
    }
    if (t == 0) {
#pragma unroll
        for (int v = 0; v < PARTIAL_STRIDE; ++v)
            a.partials[(size_t)u * PARTIAL_STRIDE + v] = red[v];
    }
}

cudaError_t launch_batched_exact(const BatchArgs &a, int ctas, int role, cudaStream_t s);
cudaError_t launch_batched_fma(const BatchArgs &a, int ctas, int role, cudaStream_t s);
cudaError_t launch_batched_fast(const BatchArgs &a, int ctas, int role, cudaStream_t s);

// One batched stage launch at precision PREC with a face-cache role; the
// reader is preceded by the fill kernel, about 6 CTAs per SM of it.
template <int PREC>
cudaError_t launch_batched(const BatchArgs &a, int ctas, int role, cudaStream_t s)
{
    cudaError_t e = cudaSuccess;
    switch (role) {
    case ROLE_WRITER:
        e = launch_chained(batched_stage_kernel<128, 6, PREC, ROLE_WRITER>, ctas, 128, 0, s, a);
        break;
    case ROLE_READER:
        e = launch_chained(batched_fill_kernel<128, PREC>,
                           dim3(a.num_disks, (148 * 6 + a.num_disks - 1) / a.num_disks), 128, 0, s, a);
        if (e == cudaSuccess)
            e = launch_chained(batched_stage_kernel<128, 6, PREC, ROLE_READER>, ctas, 128, 0, s, a);
        break;
    default:
        e = launch_chained(batched_stage_kernel<128, 6, PREC, ROLE_NONE>, ctas, 128, 0, s, a);
        break;
    }
    if (e != cudaSuccess || !a.epilogue)
        return e;
    if (a.epilogue == 2)
        return launch_chained(batched_epilogue_kernel<128, PREC, true>, a.total_units, 128, 0, s, a,
                              role == ROLE_WRITER);
    return launch_chained(batched_epilogue_kernel<128, PREC, false>, a.total_units, 128, 0, s, a, role == ROLE_WRITER);
}

}  // namespace cbd
