// swarm_fp64.cu -- the FP64 form of a planetesimal disk's cluster step (swarm.cuh), bit-exact with the
// reference's order of operations: pair terms as in pair_fp64.cuh, a pair's square root taken once
// for its two rows; the heavy rows' terms go to the CTA that owns the row and component, in source
// order, and all its warps add them up (cta_row_sum, row_sum.h).
//
// Measured, an attempt with the host's launch and wait (at first separate kernels with serial sums,
// then with segmented ones): 64 light bodies 140 us (238), 1024 189 us (731, 420), 3072 363 us
// (1634).  An evaluation of 1027 bodies is 26 k cycles: the pairs 4.6 k, the light bodies' next stage
// sums 3.5 k (FP64 pipe), the slowest row's sum 15.5 k (a coplanar system's z row, some 250 offset
// codes applied one after the other), the heavy bodies' stage sums 1.5 k.
#include <algorithm>

#include "pair_fp64.cuh"
#include "row_sum.h"
#include "swarm.cuh"

namespace redgb {

namespace {

using namespace swarm;

struct Fp64Form {
    const Smem& M;
    const Place& w;
    cg::cluster_group& cluster;
    double* own;      // [heavy][component][light]: the light bodies' terms
    double* row;      // the terms of the heavy rows (3 h + component) this CTA owns, one after the other
    uint32_t* codes;
    CtaRowSmem* sum;

    __host__ __device__ static size_t row_doubles(int slice)  // (8 CTAs of 32: two rows each)
    {
        const size_t one = HEAVY + (size_t)CTAS * slice, two = 2 * (HEAVY + 256);
        return one > two ? one : two;
    }
    __host__ __device__ static size_t code_words(int slice)
    {
        const size_t n = HEAVY + (size_t)CTAS * slice, least = 32 * ROW_SEG_MAX;
        return (n > least ? n : least) / 2 * 2;
    }
    __host__ __device__ static size_t bytes(int slice)
    {
        return 8 * ((size_t)3 * HEAVY * slice) + 8 * row_doubles(slice) + 4 * code_words(slice) + sizeof(CtaRowSmem);
    }
    __device__ Fp64Form(const Smem& m, const Place& p, cg::cluster_group& c) : M(m), w(p), cluster(c)
    {
        own = reinterpret_cast<double*>(M.form);
        row = own + 3 * HEAVY * w.slice;
        codes = reinterpret_cast<uint32_t*>(row + row_doubles(w.slice));
        sum = reinterpret_cast<CtaRowSmem*>(codes + code_words(w.slice));
    }
    __device__ void body(int, double, double, int) {}
    __device__ void position(int, int, double) {}
    __device__ void pairs(GravArgs& g, int)
    {
        const int ns = M.ns, nh = w.nh;
        const Tile tile{0, 0, 0, nh, 0, 0, 1, 0};  // numbers of this CTA's slots; body 0 (the star) is slot 0
#pragma unroll 1
        for (int q = w.warp; q <= w.chunks; q += w.nw) {
            const bool heavy = q == w.chunks;  // the last warp's pairs: heavy x heavy
            const int h = heavy ? w.lane % nh : q / w.pieces;
            const int l = (q % w.pieces) * 32 + w.lane;
            const int s = heavy ? w.lane / nh : HEAVY + l;  // the sink's slot; h is the source's
            const bool there = heavy ? w.lane < nh * nh && s != h : l < w.nl;
            double tx = 0.0, ty = 0.0, tz = 0.0, ux = 0.0, uy = 0.0, uz = 0.0;
            const bool sink = there && 0 < M.id[s] && 0 <= M.id[h];
            const bool rev = !heavy && there && 0 <= M.id[s] && 0 < M.id[h];
            if (sink || rev) {
                const double xi = M.pos[s], yi = M.pos[ns + s], zi = M.pos[2 * ns + s];
                const double xj = M.pos[h], yj = M.pos[ns + h], zj = M.pos[2 * ns + h];
                const double mi = M.mass[s], mj = M.mass[h];
                const double dx = xj - xi, dy = yj - yi, dz = zj - zi;
                const double r2 = dx * dx + dy * dy + dz * dz;
                const double d = rn_sqrt(r2), den = d * r2;
                if (sink) {
                    const double f = rn_div(mj, den);
                    tx = f * dx;
                    ty = f * dy;
                    tz = f * dz;
                    if (!heavy || w.rank == 0) {
                        g.i_shift = heavy ? 0 : w.shift;
                        pair_events(g, tile, s, h, xi, yi, zi, M.radius[s], mi, M.rho[s], xj, yj, zj, mj, M.radius[h],
                                    M.rho[h], d);
                    }
                }
                if (rev) {
                    const double f = -rn_div(mi, den);
                    ux = f * dx;
                    uy = f * dy;
                    uz = f * dz;
                }
            }
            if (heavy) {  // a source of the row s
                if (w.lane < nh * nh)
                    for (int c = 0; c < 3; c++) {
                        const int rr = 3 * s + c;
                        if (rr % w.n_cta == w.rank) row[rr / w.n_cta * w.n + h] = c == 0 ? tx : c == 1 ? ty : tz;
                    }
            } else if (l < w.nl) {
                own[(h * 3 + 0) * w.slice + l] = tx;
                own[(h * 3 + 1) * w.slice + l] = ty;
                own[(h * 3 + 2) * w.slice + l] = tz;
                for (int c = 0; c < 3; c++) {
                    const int rr = 3 * h + c;
                    *cluster.map_shared_rank(row + rr / w.n_cta * w.n + w.b0 + l, rr % w.n_cta) = c == 0 ? ux : c == 1 ? uy : uz;
                }
            }
        }
    }
    __device__ void light_sums(int r)
    {
        for (int e = w.t; e < 3 * w.nl; e += w.nt) {
            const int c = e / w.nl, l = e % w.nl;
            double acc = 0.0;
            for (int h = 0; h < w.nh; h++) acc = acc + own[(h * 3 + c) * w.slice + l];
            M.k[(r * 6 + 3 + c) * M.ns + HEAVY + l] = acc;
        }
    }
    // the rows this CTA owns, into every CTA's stage vector
    __device__ void heavy_rows(int r)
    {
        for (int rr = w.rank; rr < 3 * w.nh; rr += w.n_cta) {
            const double v = cta_row_sum(row + rr / w.n_cta * w.n, w.n, codes, *sum);
            if (w.t < w.n_cta) *cluster.map_shared_rank(M.k + (r * 6 + 3 + rr % 3) * M.ns + rr / 3, w.t) = v;
        }
        cluster_arrive();
        cluster_wait();
    }
};

}  // namespace

__global__ void __launch_bounds__(THREADS) swarm_rkf78_fp64_kernel(SmallStepArgs a, int slice)
{
    extern __shared__ __align__(16) unsigned char swarm_fp64_smem[];
    attempt<Fp64Form>(a, slice, swarm_fp64_smem);
}

bool swarm_fp64_fits(int n_heavy, int n_light) { return fits<Fp64Form>(swarm_rkf78_fp64_kernel, n_heavy, n_light); }

int launch_swarm_rkf78_fp64(const SmallStepArgs& a, cudaStream_t st)
{
    return launch<Fp64Form>(swarm_rkf78_fp64_kernel, a, st);
}

}  // namespace redgb
