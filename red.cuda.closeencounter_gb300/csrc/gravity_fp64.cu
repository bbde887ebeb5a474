// gravity_fp64.cu -- FP64 direct-summation gravity with collision / close-encounter
// screening, bit-identical to the reference's FP64 path.
//
// Reference: kernel_pp_disk::calc_grav_accel (pp_disk.cu:217-296) and its CPU twin
// pp_disk::cpu_calc_grav_accel_SI (pp_disk.cu:404-572).  For every sink i the reference
// adds the source terms m_j (r_j - r_i) / (|r_j - r_i| * |r_j - r_i|^2) one after the
// other in ascending j.  This file is compiled with -fmad=false and keeps that operation
// order, so the accelerations equal the CPU path's bit for bit.
//
// GB300 design.  GB300 retires about two FP64 lanes per SM and clock, so the FP64 pipe
// bounds this file.  The square root and the division of each pair term, about half of its
// FP64 instructions in hardware form, are computed exactly (correctly rounded, the same
// bits) with integer arithmetic on the other pipes (exact_fp64.h); the FP64 pipe keeps the
// additions and multiplications.  The pair terms do not depend on the order, so they are formed
// side by side, and the sums are added in ascending j: a CTA per row (grav_fp64_rows, the sum by
// segments, row_sum.h) for rows of many sources in blocks of few pairs, and for the rows that
// gravity_cert.cu, which takes the large blocks, leaves over; the row-serial kernel (thread per
// sink) for blocks with few sources per sink (planetesimals x 3 massive bodies); and the
// pair-parallel kernel (S x J terms into shared memory, 3 S threads add them) for blocks of many
// sinks with a hundred sources or so, and the astrocentric frame.
#include <atomic>
#include <string>
#include <type_traits>

#include "../../include/redgb.h"
#include "common.cuh"
#include "exact_fp64.h"
#include "kernels.h"
#include "pair_fp64.cuh"
#include "row_sum.h"

namespace redgb {

int set_error(int code, const std::string& msg);

// ---------------------------------------------------------------------------------------
// Pair-parallel kernel: CTA = S sinks, source tiles of J = 1024 / S, for blocks of many sinks with a
// hundred sources or so (fp64_block_form, plan_tools.h) and the astrocentric frame (ASTRO) of the
// reference's CPU path -- there each sink starts from the star's pull
// and, for every source it interacts with, adds the direct term and then subtracts the
// source's indirect term (pp_disk.cu:413-454), in source order.
// RG_PAIRPAR_RESIDENT (kernels.h): resident CTAs per SM the register budget is cut for (the
// pair term's integer square root and division hold many values; more resident warps hide
// their latency)

// S sinks x STRIDE threads per CTA, four pair terms per thread and tile (J = 4 STRIDE sources).
// S sets the number of CTAs, ceil(sinks / S): the tuner picks the S whose grid fills the last
// wave of resident CTAs best, since every CTA of a block runs the same sources and so takes the
// same time.  In the barycentric frame the plan takes the S of the least waves x steps (PairparSinks):
// an evaluation of 65 massive bodies and 5000 / 20 000 test particles 23 / 57 us, their rows a CTA each
// 85 / 295 us, certified 68 / 97 us; an RKF7(8) attempt of 64 / 256 disks of 103 / 73 bodies 529 / 963
// us, in rows 1625 / 4095 us.
template <int S, int STRIDE, bool ASTRO>
__global__ void __launch_bounds__(S * STRIDE, RG_PAIRPAR_RESIDENT) grav_fp64_pairpar(GravArgs g)
{
    constexpr int NT = S * STRIDE;
    constexpr int JPT = 4;           // terms per thread per tile
    constexpr int J = JPT * STRIDE;  // sources per tile
    __shared__ double tx[J * S], ty[J * S], tz[J * S];
    __shared__ double sx[J], sy[J], sz[J], sm[J], sR[J], srho[J];
    __shared__ double sind[3][ASTRO ? J : 1];  // the sources' indirect terms
    __shared__ int sid[J];

    const Tile tile = g.tiles[blockIdx.x];
    if (g.sys_active && !g.sys_active[tile.sys]) return;
    const int t = threadIdx.x;
    const int s = t % S;
    const int q0 = t / S;
    const int i = tile.sink_begin + s;
    const bool sink_ok = i < tile.sink_end;
    double xi = 0, yi = 0, zi = 0, Ri = 0, mi = 0, rhoi = 0;
    bool active = false;
    if (sink_ok) {
        xi = g.px[i]; yi = g.py[i]; zi = g.pz[i];
        Ri = g.radius[i]; mi = g.mass[i];
        rhoi = g.hill ? g.rho[i] : 0.0;
        active = 0 < g.id[i];
    }
    const int bc = t / S;  // phase-B component (0, 1, 2) for t < 3 S
    const double* Tb = bc == 0 ? tx : (bc == 1 ? ty : tz);
    double acc = 0.0;
    if (ASTRO && t < 3 * S && sink_ok) acc = g.astro[bc * g.astro_stride + i];

    for (int j0 = tile.src_begin; j0 < tile.src_end; j0 += J) {
        const int nj = min(J, tile.src_end - j0);
        for (int q = t; q < nj; q += NT) {
            const int j = j0 + q;
            sx[q] = g.px[j]; sy[q] = g.py[j]; sz[q] = g.pz[j];
            sm[q] = g.mass[j]; sR[q] = g.radius[j]; sid[q] = g.id[j];
            srho[q] = g.hill ? g.rho[j] : 0.0;
            if (ASTRO) {
                sind[0][q] = g.astro[3 * g.astro_stride + j];
                sind[1][q] = g.astro[4 * g.astro_stride + j];
                sind[2][q] = g.astro[5 * g.astro_stride + j];
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < JPT; k++) {
            const int q = q0 + k * STRIDE;
            const int j = j0 + q;
            PairOut o{0.0, 0.0, 0.0};
            if (active && q < nj && j != i && 0 <= sid[q])
                pair_term(g, tile, i, j, xi, yi, zi, Ri, mi, rhoi, sx[q], sy[q], sz[q], sm[q], sR[q], srho[q], o);
            tx[q * S + s] = o.tx;
            ty[q * S + s] = o.ty;
            tz[q * S + s] = o.tz;
        }
        __syncthreads();
        if (ASTRO) {
            if (t < 3 * S && active) {
                const double* Ib = sind[bc < 3 ? bc : 0];
                for (int q = 0; q < nj; q++)
                    if (j0 + q != i && 0 <= sid[q]) {
                        acc = acc + Tb[q * S + s];
                        acc = acc - Ib[q];
                    }
            }
        } else if (t < 3 * S) {
            for (int q = 0; q < nj; q++) acc = acc + Tb[q * S + s];
        }
        __syncthreads();
    }
    if (t < 3 * S && sink_ok) {
        double* out = bc == 0 ? g.ax : (bc == 1 ? g.ay : g.az);
        out[i] = acc;
    }
}

// ---------------------------------------------------------------------------------------
// Row-serial kernel: one thread per sink, sources staged through shared memory.
__global__ void __launch_bounds__(128) grav_fp64_rowseq(GravArgs g)
{
    constexpr int NT = 128;
    __shared__ double sx[NT], sy[NT], sz[NT], sm[NT], sR[NT], srho[NT];
    __shared__ int sid[NT];
    const Tile tile = g.tiles[blockIdx.x];
    if (g.sys_active && !g.sys_active[tile.sys]) return;
    const int t = threadIdx.x;
    const int i = tile.sink_begin + t;
    const bool sink_ok = i < tile.sink_end;
    double xi = 0, yi = 0, zi = 0, Ri = 0, mi = 0, rhoi = 0;
    bool active = false;
    if (sink_ok) {
        xi = g.px[i]; yi = g.py[i]; zi = g.pz[i];
        Ri = g.radius[i]; mi = g.mass[i];
        rhoi = g.hill ? g.rho[i] : 0.0;
        active = 0 < g.id[i];
    }
    double ax = 0.0, ay = 0.0, az = 0.0;
    for (int j0 = tile.src_begin; j0 < tile.src_end; j0 += NT) {
        const int nj = min(NT, tile.src_end - j0);
        if (t < nj) {
            const int j = j0 + t;
            sx[t] = g.px[j]; sy[t] = g.py[j]; sz[t] = g.pz[j];
            sm[t] = g.mass[j]; sR[t] = g.radius[j]; sid[t] = g.id[j];
            srho[t] = g.hill ? g.rho[j] : 0.0;
        }
        __syncthreads();
        if (active) {
            for (int q = 0; q < nj; q++) {
                const int j = j0 + q;
                if (j == i || 0 > sid[q]) continue;
                PairOut o;
                pair_term(g, tile, i, j, xi, yi, zi, Ri, mi, rhoi, sx[q], sy[q], sz[q], sm[q], sR[q], srho[q], o);
                ax = ax + o.tx;
                ay = ay + o.ty;
                az = az + o.tz;
            }
        }
        __syncthreads();
    }
    if (sink_ok) {
        g.ax[i] = ax;
        g.ay[i] = ay;
        g.az[i] = az;
    }
}

// Distance of every body from its disk's body 0 (the star), for the Hill test:
// sqrt(SQR(x_i - x_0) + SQR(y_i - y_0) + SQR(z_i - z_0)).
__global__ void star_distance(const double* __restrict__ x, const double* __restrict__ y,
                              const double* __restrict__ z, const int* __restrict__ base_of, int n,
                              double* __restrict__ rho)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int b = base_of ? base_of[i] : 0;
    const double dx = x[i] - x[b], dy = y[i] - y[b], dz = z[i] - z[b];
    rho[i] = rn_sqrt(dx * dx + dy * dy + dz * dz);  // sqrt.rn's bits, off the FP64 pipe
}

// ---------------------------------------------------------------------------------------
// Row path: rows whose sums need every bit of their terms -- blocks with a handful of sinks and
// many sources (the star and giants of a planetesimal disk), and the rows gravity_cert.cu leaves
// over.  One CTA per row: six or eight warps compute the exact terms of a chunk of sources into shared
// memory while three groups of two, one per component, add the chunk before it in ascending source
// order (group_row_sum, row_sum.h).
//
// Bound: a chunk's 1152 pairs, 36 warps x (12 FP64 operations x 16 cycles of the SM's FP64 pipe and
// the integer square root and division), about 12 k cycles; the sums take as long beside them,
// also where they hover (one warp a component: up to 30 k cycles a chunk for a coplanar system's z
// row).
//
// A listed row (LIST) has other rows beside it on its SM, three CTAs with a summing warp per component
// (warp_row_sum): a force evaluation of the dense ring, 11 000 listed rows, 131.5 ms, with the two
// CTAs that the groups leave room for 135.2 ms.  Few rows have an SM each: 64 disks in FP64 131 ms
// with single warps, 117 ms with groups beside eight warps for the terms, 114 ms beside six, which
// leave more issue slots to the sums' first warps (four: 126 ms).
//
// TERMS, the warps for the terms: six (self-interacting blocks of 300 / 500 / 1000 / 1480 bodies: 14.4
// / 22.8 / 56 / 101 us, with eight 14.9 / 25.0 / 62 / 110 us), except where eight form a row's only
// chunk at once and six do not (400 bodies: 18.3 against 20.8 us).
constexpr int ROW_CHUNK = 1152;
static_assert(ROW_CHUNK >= 32 * ROW_SEG_MAX, "codes of a chunk");

template <bool LIST, int TERMS>
struct RowShape {
    static constexpr int SUM_WARPS = LIST ? 1 : 2;  // per component
    static constexpr int WARPS = 3 * SUM_WARPS + TERMS;  // (all of them form the first chunk's terms)
    static constexpr int CTAS = LIST ? 3 : 2;  // per SM
    static constexpr int LANES = 32 * SUM_WARPS;
    static constexpr int PITCH = LANES * (ROW_CHUNK / LANES | 1);
};

struct NoRules {};
template <bool LIST, int TERMS>
struct RowSmem {
    double term[2][3][RowShape<LIST, TERMS>::PITCH];
    uint32_t codes[3][ROW_CHUNK];
    std::conditional_t<LIST, NoRules, GroupRowSmem<640, RowShape<LIST, TERMS>::SUM_WARPS>> sum[3];
};

// the event tests of a listed row's body with the sources from sink_end on (a pair's tests are its later
// body's), by a CTA: for the few rows with a pair that may pass
__device__ __forceinline__ void row_events(const GravArgs& g, const Tile* row)
{
    const Tile tile = *row;
    const int i = tile.sink_begin;
    if (!(0 < g.id[i])) return;
    const double xi = g.px[i], yi = g.py[i], zi = g.pz[i], cut = __int_as_float(tile.part & ~7);
    for (int j = tile.sink_end + (int)threadIdx.x; j < min(i, tile.src_end); j += blockDim.x) {
        const double dx = g.px[j] - xi, dy = g.py[j] - yi, dz = g.pz[j] - zi;
        PairOut o;
        if (!(dx * dx + dy * dy + dz * dz >= cut) && 0 <= g.id[j])
            pair_term(g, tile, i, j, xi, yi, zi, g.radius[i], g.mass[i], g.hill ? g.rho[i] : 0.0, g.px[j], g.py[j],
                      g.pz[j], g.mass[j], g.radius[j], g.hill ? g.rho[j] : 0.0, o);
    }
}

// LIST: the rows *n_list of `list` (part: components to add; sink_end: the event tests of sources from
// there on are the row's too)
template <bool LIST, int TERMS>
__global__ void __launch_bounds__(32 * RowShape<LIST, TERMS>::WARPS, RowShape<LIST, TERMS>::CTAS)
    grav_fp64_rows(const __grid_constant__ GravArgs g, const Tile* list, const unsigned int* n_list)
{
    extern __shared__ __align__(16) unsigned char row_smem[];
    using Shape = RowShape<LIST, TERMS>;
    constexpr int LANES = Shape::LANES;
    RowSmem<LIST, TERMS>& M = *reinterpret_cast<RowSmem<LIST, TERMS>*>(row_smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_rows = LIST ? (int)*n_list : g.n_tiles;
    const int comp = warp / Shape::SUM_WARPS;  // of a sum warp: 0, 1, 2
    [[maybe_unused]] const RowGroup grp{1 + min(comp, 3), LANES, (int)threadIdx.x - LANES * comp};
    for (int row = blockIdx.x; row < n_rows; row += gridDim.x) {
        const Tile tile = LIST ? list[row] : g.tiles[row];
        if (g.sys_active && !g.sys_active[tile.sys]) continue;
        const int comps = LIST ? tile.part & 7 : 7;
        const int i = tile.sink_begin;
        const bool active = 0 < g.id[i];
        const double xi = g.px[i], yi = g.py[i], zi = g.pz[i];
        const double Ri = LIST ? 0.0 : g.radius[i], mi = LIST ? 0.0 : g.mass[i], rhoi = !LIST && g.hill ? g.rho[i] : 0.0;
        double acc = 0.0;
        const int n = tile.src_end - tile.src_begin;
        const int chunks = (n + ROW_CHUNK - 1) / ROW_CHUNK;
        const bool adds = comp < 3 && (comps >> comp & 1);
        // a listed row's event tests: the upper word of the r^2 that none passes, -1 where it has none to make
        [[maybe_unused]] const int cut = LIST && tile.sink_end < min(i, tile.src_end) && (g.record || g.hill)
                                             ? __double2hiint((double)__int_as_float(tile.part & ~7))
                                             : -1;
        [[maybe_unused]] bool candidate = false;
        for (int c = 0; c <= chunks; c++) {
            if (c < chunks && (c == 0 || comp >= 3)) {  // terms of chunk c (the first one: by every warp)
                const int q0 = c * ROW_CHUNK, m = min(ROW_CHUNK, n - q0);
                const int seg = (m + LANES - 1) / LANES, pitch = seg | 1;
                const int w0 = c == 0 ? 0 : 3 * Shape::SUM_WARPS, nw = Shape::WARPS - w0;
                for (int q = (warp - w0) * 32 + lane; q < m; q += 32 * nw) {
                    const int j = tile.src_begin + q0 + q;
                    const double xj = g.px[j], yj = g.py[j], zj = g.pz[j], mj = g.mass[j];
                    PairOut o{0.0, 0.0, 0.0, 1e300};
                    if (active && j != i && 0 <= g.id[j])
                        pair_term<!LIST>(g, tile, i, j, xi, yi, zi, Ri, mi, rhoi, xj, yj, zj, mj, LIST ? 0.0 : g.radius[j],
                                         !LIST && g.hill ? g.rho[j] : 0.0, o);
                    if (LIST) candidate = candidate | (__double2hiint(o.r2) <= cut);
                    const int at = q / seg * pitch + q % seg;
                    M.term[c & 1][0][at] = o.tx;
                    M.term[c & 1][1][at] = o.ty;
                    M.term[c & 1][2][at] = o.tz;
                }
            }
            if (c > 0 && adds) {
                const int m = min(ROW_CHUNK, n - (c - 1) * ROW_CHUNK);
                const int seg = (m + LANES - 1) / LANES;
                const double* const T = M.term[(c - 1) & 1][comp];
                if constexpr (LIST)
                    acc = warp_row_sum(acc, T, seg, seg | 1, m, M.codes[comp]);
                else
                    acc = group_row_sum(grp, acc, T, seg, seg | 1, m, M.codes[comp], M.sum[comp]);
            }
            __syncthreads();
        }
        if (adds && (int)threadIdx.x == LANES * comp) (comp == 0 ? g.ax : comp == 1 ? g.ay : g.az)[i] = acc;
        if (LIST && cut >= 0 && __syncthreads_or(candidate)) row_events(g, list + row);
    }
}

// The astrocentric frame's per-body terms (pp_disk.cu:413-420 and 447-454) for bodies
// [1, n): the star's pull on body i, -mu / (r2 sqrt(r2)) r_i with mu = m_star + m_i, and the
// indirect term m_i / (r2 sqrt(r2)) r_i, r2 = |r_i|^2, each component evaluated as the
// reference writes it (division first, then the product).  Body 0 (the star) gets zeros.
__global__ void astro_terms_kernel(const double* __restrict__ x, const double* __restrict__ y,
                                   const double* __restrict__ z, const double* __restrict__ mass, int n,
                                   double m_star, double* __restrict__ out, long long stride)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double sx = 0.0, sy = 0.0, sz = 0.0, ix = 0.0, iy = 0.0, iz = 0.0;
    if (i > 0) {
        const double xi = x[i], yi = y[i], zi = z[i], m = mass[i];
        const double r2 = xi * xi + yi * yi + zi * zi;
        const double den = r2 * rn_sqrt(r2);
        const double mu = m_star + m;
        const double ws = -mu / den;
        const double wi = rn_div(m, den);
        sx = ws * xi; sy = ws * yi; sz = ws * zi;
        ix = wi * xi; iy = wi * yi; iz = wi * zi;
    }
    out[i] = sx;
    out[stride + i] = sy;
    out[2 * stride + i] = sz;
    out[3 * stride + i] = ix;
    out[4 * stride + i] = iy;
    out[5 * stride + i] = iz;
}

// ---------------------------------------------------------------------------------------
// Host launchers
int launch_grav_fp64_pairpar(const GravArgs& g, int S, cudaStream_t st)
{
    if (g.n_tiles <= 0) return 0;
    auto launch = [&](auto kernel) { kernel<<<g.n_tiles, 256, 0, st>>>(g); };
    switch (S) {
    case 4:
        if (g.astro) return set_error(RG_ERR_ARG, "pair-parallel sinks per CTA: 8, 16 or 32 in the astrocentric frame");
        launch(grav_fp64_pairpar<4, 64, false>);
        break;
    case 8: launch(g.astro ? grav_fp64_pairpar<8, 32, true> : grav_fp64_pairpar<8, 32, false>); break;
    case 16: launch(g.astro ? grav_fp64_pairpar<16, 16, true> : grav_fp64_pairpar<16, 16, false>); break;
    case 32: launch(g.astro ? grav_fp64_pairpar<32, 8, true> : grav_fp64_pairpar<32, 8, false>); break;
    default: return set_error(RG_ERR_ARG, "pair-parallel sinks per CTA: 4, 8, 16 or 32");
    }
    RG_CUDA_CHECK(cudaGetLastError());
    return 0;
}

int launch_astro_terms(const double* x, const double* y, const double* z, const double* mass, int n, double m_star,
                       double* out, long long stride, cudaStream_t st)
{
    if (n <= 0) return 0;
    astro_terms_kernel<<<(n + 255) / 256, 256, 0, st>>>(x, y, z, mass, n, m_star, out, stride);
    RG_CUDA_CHECK(cudaGetLastError());
    return 0;
}

int launch_grav_fp64_rowseq(const GravArgs& g, cudaStream_t st)
{
    if (g.n_tiles <= 0) return 0;
    grav_fp64_rowseq<<<g.n_tiles, 128, 0, st>>>(g);
    RG_CUDA_CHECK(cudaGetLastError());
    return 0;
}

// the row kernels' shared memory: a per-device attribute, set once per device (setting it again
// from another thread is harmless)
static int row_attributes()
{
    static std::atomic<bool> attr_set[64];
    int dev = 0;
    RG_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
        auto set = [](auto kernel, size_t bytes) {
            return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        };
        RG_CUDA_CHECK(set(grav_fp64_rows<true, 8>, sizeof(RowSmem<true, 8>)));
        RG_CUDA_CHECK(set(grav_fp64_rows<false, 6>, sizeof(RowSmem<false, 6>)));
        RG_CUDA_CHECK(set(grav_fp64_rows<false, 8>, sizeof(RowSmem<false, 8>)));
        if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
    }
    return 0;
}

int launch_grav_fp64_rows(const GravArgs& g, int max_src, cudaStream_t st)
{
    if (g.n_tiles <= 0) return 0;
    if (const int rc = row_attributes()) return rc;
    using Six = RowShape<false, 6>;
    using Eight = RowShape<false, 8>;
    if (max_src > 32 * Six::WARPS && max_src <= 32 * Eight::WARPS)
        grav_fp64_rows<false, 8><<<g.n_tiles, 32 * Eight::WARPS, sizeof(RowSmem<false, 8>), st>>>(g, nullptr, nullptr);
    else
        grav_fp64_rows<false, 6><<<g.n_tiles, 32 * Six::WARPS, sizeof(RowSmem<false, 6>), st>>>(g, nullptr, nullptr);
    RG_CUDA_CHECK(cudaGetLastError());
    return 0;
}

int launch_grav_fp64_list(const GravArgs& g, const CertRows& cr, cudaStream_t st)
{
    if (const int rc = row_attributes()) return rc;
    // as many CTAs as are resident; the list's length is known on the device
    using Shape = RowShape<true, 8>;
    grav_fp64_rows<true, 8><<<Shape::CTAS * NUM_SMS_HINT, 32 * Shape::WARPS, sizeof(RowSmem<true, 8>), st>>>(g, cr.list, cr.n_list);
    RG_CUDA_CHECK(cudaGetLastError());
    return 0;
}

int launch_star_distance(const double* x, const double* y, const double* z, const int* base_of, int n, double* rho,
                         cudaStream_t st)
{
    if (n <= 0) return 0;
    star_distance<<<(n + 255) / 256, 256, 0, st>>>(x, y, z, base_of, n, rho);
    RG_CUDA_CHECK(cudaGetLastError());
    return 0;
}

}  // namespace redgb
