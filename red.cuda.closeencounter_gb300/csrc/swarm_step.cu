// swarm_step.cu -- the mixed-precision form of a planetesimal disk's cluster step (swarm.cuh) and
// its launchers: double-float pair terms and compensated sums as in grav_df_sym, whose segments are
// these slices (swarm_slice), event decisions in FP64: the separate kernels' bits.  Each CTA writes
// its light bodies' part of the heavy rows into every CTA's shared memory, and each adds them up.
//
// Measured, an attempt with the host's launch and wait (before: separate kernels from a graph): 64
// light bodies 69 us (237), 1024 88 us (247), 2000 107 us (245), 3072 140 us (247).  The limit is
// the slice whose vectors fit the shared memory with room for the terms (172 of 227 KB); the FP64
// pipe of 16 SMs, 36 warps of stage sums an SM at 3072 bodies, would reach the separate kernels'
// time at about twice that.
#include <algorithm>
#include <atomic>

#include "pair_df.cuh"
#include "swarm.cuh"

namespace redgb {

namespace {

using namespace swarm;

struct MixedForm {
    const Smem& M;
    const Place& w;
    cg::cluster_group& cluster;
    float2 *split, *massf;    // split positions (3 rows) and masses
    float2* own;              // [heavy][component][light]: the light bodies' terms
    DF (*red)[3];             // per pair warp: its light bodies' sum for the heavy row
    DF (*hh)[HEAVY][3];       // [sink][source]: the heavy pairs
    double* part;             // [2][CTA][heavy x component]
    float* rf;

    __host__ __device__ static size_t bytes(int slice)
    {
        const size_t ns = slice + HEAVY, chunks = (size_t)HEAVY * slice / 32;
        return 8 * (2 * CTAS * 3 * HEAVY) + 8 * (4 * ns) + 8 * ((size_t)3 * HEAVY * slice) + 24 * chunks +
               24 * HEAVY * HEAVY + 4 * ns;
    }
    __device__ MixedForm(const Smem& m, const Place& p, cg::cluster_group& c) : M(m), w(p), cluster(c)
    {
        part = reinterpret_cast<double*>(M.form);
        float2* f = reinterpret_cast<float2*>(part + 2 * CTAS * 3 * HEAVY);
        split = f, f += 3 * M.ns;
        massf = f, f += M.ns;
        own = f, f += 3 * HEAVY * w.slice;
        red = reinterpret_cast<DF(*)[3]>(f), f += 3 * (HEAVY * w.slice / 32);
        hh = reinterpret_cast<DF(*)[HEAVY][3]>(f), f += 3 * HEAVY * HEAVY;
        rf = reinterpret_cast<float*>(f);
    }
    __device__ void body(int s, double m, double R, int id)
    {
        float lo;
        split_bits(R, rf[s], lo);
        float2 mf = make_float2(0.0f, 0.0f);
        if (id >= 0) split_bits(m, mf.x, mf.y);
        massf[s] = mf;
    }
    __device__ void position(int row, int s, double v)
    {
        float2& f = split[row * M.ns + s];
        split_coord(v, f.x, f.y);
    }
    __device__ SplitPos record(int s) const
    {
        SplitPos p;
        const float2 x = split[s], y = split[M.ns + s], z = split[2 * M.ns + s], m = massf[s];
        p.xy = make_float4(x.x, x.y, y.x, y.y);
        p.zm = make_float4(z.x, z.y, m.x, m.y);
        return p;
    }
    // the light bodies' terms and this CTA's part of the heavy rows
    __device__ void pairs(GravArgs& g, int)
    {
        const int ns = M.ns, nh = w.nh;
        const Tile tile{0, 0, 0, nh, 0, 0, 1, 0};  // numbers of this CTA's slots; body 0 (the star) is slot 0
        g.rf = rf;
        const SplitPos p0 = record(0);
        const float inv3M = g.hill ? 1.0f / (3.0f * p0.zm.z) : 0.0f;
        const float frad = g.f_rad_f;
#pragma unroll 1
        for (int q = w.warp; q <= w.chunks; q += w.nw) {
            const bool heavy = q == w.chunks;  // the last warp's pairs: heavy x heavy
            const int h = heavy ? w.lane % nh : q / w.pieces;
            const int l = (q % w.pieces) * 32 + w.lane;
            const int s = heavy ? (w.lane / nh) : HEAVY + l;  // the sink's slot; h is the source's
            const bool there = heavy ? w.lane < nh * nh && s != h : l < w.nl;
            DF tx{0.0f, 0.0f}, ty{0.0f, 0.0f}, tz{0.0f, 0.0f}, ux = tx, uy = tx, uz = tx;
            const bool src_ok = there && 0 <= M.id[s];  // as a source; 0 < id: as a sink
            const bool own_ok = there && 0 < M.id[s] && 0 <= M.id[h], rev = !heavy && src_ok && 0 < M.id[h];
            if (own_ok || rev) {
                const SplitPos pi = record(s), ph = record(h);
                const float2 mh = massf[h], mi = massf[s];
                DF dx = df_diff(ph.xy.x, ph.xy.y, pi.xy.x, pi.xy.y);
                DF dy = df_diff(ph.xy.z, ph.xy.w, pi.xy.z, pi.xy.w);
                DF dz = df_diff(ph.zm.x, ph.zm.y, pi.zm.x, pi.zm.y);
                DF r2 = df_add_same_sign(df_add_same_sign(df_mul(dx, dx), df_mul(dy, dy)), df_mul(dz, dz));
                const float close = heavy ? close_r2(pi) : fmaxf(close_r2(pi), close_r2(ph));
                if (r2.hi < close) {  // the FP64 displacement (df_term_fp64)
                    dx = split_df(M.pos[h] - M.pos[s]);
                    dy = split_df(M.pos[ns + h] - M.pos[ns + s]);
                    dz = split_df(M.pos[2 * ns + h] - M.pos[2 * ns + s]);
                    r2 = df_add_same_sign(df_add_same_sign(df_mul(dx, dx), df_mul(dy, dy)), df_mul(dz, dz));
                }
                if (!(r2.hi < 1.0e30f)) r2 = DF{1.0e30f, 0.0f};  // a merged body parked at 1e20 AU
                const float y0 = rsqrt_approx(r2.hi);
                const DF p = df_mul(r2, df_two_prod(y0, y0));
                const float hf = (1.0f - p.hi) - p.lo;
                const DF y = df_fast_sum(y0, 0.5f * y0 * hf);
                const DF y3 = df_mul(df_mul(y, y), y);
                if (own_ok) {
                    const DF wt = df_mul(y3, DF{mh.x, mh.y});
                    tx = df_mul(wt, dx);
                    ty = df_mul(wt, dy);
                    tz = df_mul(wt, dz);
                    if ((g.record || g.hill) && (!heavy || w.rank == 0)) {
                        g.i_shift = heavy ? 0 : w.shift;
                        df_screen(g, tile, s, h, r2.hi, rf[s], rf[h], g.hill ? star_dist_f(pi, p0) : 0.0f,
                                  g.hill ? star_dist_f(ph, p0) : 0.0f, mi.x, mh.x, inv3M, frad);
                    }
                }
                if (rev) {
                    const DF wt = df_mul(y3, DF{mi.x, mi.y});
                    ux = df_mul(wt, dx);
                    uy = df_mul(wt, dy);
                    uz = df_mul(wt, dz);
                }
            }
            if (heavy) {
                if (w.lane < nh * nh) {
                    hh[s][h][0] = tx;
                    hh[s][h][1] = ty;
                    hh[s][h][2] = tz;
                }
            } else {
                own[(h * 3 + 0) * w.slice + l] = make_float2(tx.hi, tx.lo);
                own[(h * 3 + 1) * w.slice + l] = make_float2(ty.hi, ty.lo);
                own[(h * 3 + 2) * w.slice + l] = make_float2(tz.hi, tz.lo);
                Acc2 v[3] = {{-ux.hi, -ux.lo}, {-uy.hi, -uy.lo}, {-uz.hi, -uz.lo}};
#pragma unroll
                for (int off = 16; off > 0; off >>= 1)
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const Acc2 o{__shfl_xor_sync(0xffffffffu, v[c].s, off), __shfl_xor_sync(0xffffffffu, v[c].c, off)};
                        v[c] = two_sum_merge(v[c], o);
                    }
                if (w.lane == 0)
                    for (int c = 0; c < 3; c++) red[q][c] = df_two_sum(v[c].s, v[c].c);
            }
        }
    }
    // this CTA's part of the heavy rows into every CTA's part[r & 1], and the light bodies' accelerations
    __device__ void light_sums(int r)
    {
        const int ns = M.ns, nh = w.nh;
        if (w.t < 3 * nh) {
            const int h = w.t / 3, c = w.t % 3;
            DF v = red[h * w.pieces][c];
            for (int p = 1; p < w.pieces; p++) v = df_add(v, red[h * w.pieces + p][c]);
            const double d = df_to_double(v);
            double* const at = part + ((r & 1) * CTAS + w.rank) * 3 * HEAVY + w.t;
            for (int q = 0; q < w.n_cta; q++) *cluster.map_shared_rank(at, q) = d;
        }
        for (int e = w.nt - 1 - w.t; e < 3 * w.nl; e += w.nt) {  // (the first warp has the parts)
            const int c = e / w.nl, l = e % w.nl;
            Acc2 o{0.0f, 0.0f};
            for (int h = 0; h < nh; h++) {
                const float2 f = own[(h * 3 + c) * w.slice + l];
                acc_df(o, DF{f.x, f.y});
            }
            M.k[(r * 6 + 3 + c) * ns + HEAVY + l] = f2d_bits(o.s) + f2d_bits(o.c);
        }
    }
    // the heavy rows, by the first warp
    __device__ void heavy_rows(int r)
    {
        const int ns = M.ns, nh = w.nh;
        if (w.warp != 0) return;
        if (w.t < 3 * nh) {
            const int h = w.t / 3, c = w.t % 3;
            Acc2 o{0.0f, 0.0f};
            for (int q = 0; q < nh; q++) acc_df(o, hh[h][q][c]);
            double v = f2d_bits(o.s) + f2d_bits(o.c);
            const double* const P = part + (r & 1) * CTAS * 3 * HEAVY + w.t;
            for (int q = 0; q < w.n_cta; q++) v += P[q * 3 * HEAVY];
            M.k[(r * 6 + 3 + c) * ns + h] = v;
        }
        __syncwarp();
    }
};

}  // namespace

__global__ void __launch_bounds__(THREADS) swarm_rkf78_kernel(SmallStepArgs a, int slice)
{
    extern __shared__ __align__(16) unsigned char swarm_smem[];
    attempt<MixedForm>(a, slice, swarm_smem);
}

Shape swarm::shape(int n_heavy, int n_light)
{
    Shape s;
    s.ctas = n_light <= 32 * 8 ? 8 : CTAS;
    s.slice = swarm_slice(n_light);
    // a warp per pair chunk and one for the heavy pairs, as far as there are
    s.threads = std::min(THREADS, std::max(256, 32 * (n_heavy * s.slice / 32 + 1)));
    return s;
}

// light bodies of a CTA: a sixteenth, in whole warps; up to 256 bodies an eighth (CTAs of 32)
int swarm_slice(int n_light)
{
    const int ctas = n_light <= 32 * 8 ? 8 : CTAS;
    return std::max(1, (n_light + 32 * ctas - 1) / (32 * ctas)) * 32;
}

bool swarm_step_fits(int n_heavy, int n_light) { return fits<MixedForm>(swarm_rkf78_kernel, n_heavy, n_light); }

int launch_swarm_rkf78(const SmallStepArgs& a, cudaStream_t st) { return launch<MixedForm>(swarm_rkf78_kernel, a, st); }

}  // namespace redgb
