// swarm_step.cu -- one attempt of an RKF7(8) step of a planetesimal disk (a star and up to three
// giants, light bodies that feel them and pull on them) in one kernel of one thread-block cluster,
// mixed precision.
//
// Such a step of a thousand bodies is all latency: 13 evaluations of three short kernels each (stage
// sums, split positions, grav_df_sym on four of the 152 SMs), 19 us an evaluation.  Here 16 CTAs
// keep the state and the stage vectors in shared memory for the whole attempt, a slice of the light
// bodies each, and the heavy bodies in every CTA.  What crosses CTAs is the heavy rows' partial
// sums: each CTA writes its own into all others' shared memory, and one cluster barrier per
// evaluation covers them; the light bodies' next stage sums run between its two halves, so the
// FP64 pipe's time (64 cycles a warp instruction) hides the barrier.  The pairs are dealt out with
// a warp per heavy body and 32 light ones, so that a light body's heavy pairs run side by side.
//
// The arithmetic is the separate kernels': FP64 state, stage sums (stages.cu) and error norm, the
// double-float pair terms and compensated sums of grav_df_sym, whose segments are these slices
// (swarm_slice), and event decisions in FP64: the same bits (this unit contracts FP32 multiply-adds
// as the mixed kernels' does; FP64 operations are written rounded one by one).
//
// Measured, an attempt with the host's launch and wait (before: separate kernels from a graph): 64
// light bodies 69 us (237), 1024 88 us (247), 2000 107 us (245), 3072 140 us (247).  The limit is
// the slice whose vectors fit the shared memory with room for the terms (172 of 227 KB); the FP64
// pipe of 16 SMs, 36 warps of stage sums an SM at 3072 bodies, would reach the separate kernels'
// time at about twice that.
#include <algorithm>
#include <atomic>

#include <cooperative_groups.h>

#include "../../include/redgb.h"
#include "common.cuh"
#include "exact_fp64.h"
#include "kernels.h"
#include "pair_df.cuh"

namespace redgb {

namespace {

namespace cg = cooperative_groups;

constexpr int HEAVY = DF_SYM_MAX_HEAVY;       // slots 0 .. HEAVY - 1: the heavy bodies; then the CTA's light ones
constexpr int SWARM_CTAS = 16;                // of the largest cluster
constexpr int SWARM_SLICE = 192;              // most light bodies of a CTA
constexpr int SWARM_THREADS = 512;
static_assert(SWARM_MAX_LIGHT == SWARM_CTAS * SWARM_SLICE, "limit of the plan");

// the CTA's shared memory for slices of `slice` light bodies (a multiple of 32)
struct SwarmSmem {
    double *y, *k, *pos, *mass, *radius, *rho;  // rows of `ns` slots: y 6, k 13 x 6, pos 3
    float2 *split, *massf;                      // split positions (3 rows) and masses
    float* rf;
    int* id;
    float2* own;                                // [heavy][component][light]: the light bodies' terms
    DF (*red)[3];                               // per pair warp: its light bodies' sum for the heavy row
    DF (*hh)[HEAVY][3];                         // [sink][source]: the heavy pairs
    double* part;                               // [2][CTA][heavy x component]
    unsigned long long* max_bits;               // [CTA]
    unsigned int* n_eject;                      // [CTA]
    int ns;

    __host__ __device__ static size_t bytes(int slice)
    {
        const size_t ns = slice + HEAVY, chunks = (size_t)HEAVY * slice / 32;
        return 8 * (90 * ns) + 8 * (4 * ns) + 4 * (2 * ns) + 8 * ((size_t)3 * HEAVY * slice) + 24 * chunks +
               24 * HEAVY * HEAVY + 8 * (2 * SWARM_CTAS * 3 * HEAVY) + 16 * SWARM_CTAS;
    }
    __device__ SwarmSmem(unsigned char* base, int slice)
    {
        ns = slice + HEAVY;
        double* d = reinterpret_cast<double*>(base);
        y = d, d += 6 * ns;
        k = d, d += 78 * ns;
        pos = d, d += 3 * ns;
        mass = d, d += ns;
        radius = d, d += ns;
        rho = d, d += ns;
        part = d, d += 2 * SWARM_CTAS * 3 * HEAVY;
        max_bits = reinterpret_cast<unsigned long long*>(d), d += SWARM_CTAS;
        float2* f = reinterpret_cast<float2*>(d);
        split = f, f += 3 * ns;
        massf = f, f += ns;
        own = f, f += 3 * HEAVY * slice;
        red = reinterpret_cast<DF(*)[3]>(f), f += 3 * (HEAVY * slice / 32);
        hh = reinterpret_cast<DF(*)[HEAVY][3]>(f), f += 3 * HEAVY * HEAVY;
        rf = reinterpret_cast<float*>(f);
        id = reinterpret_cast<int*>(rf + ns);
        n_eject = reinterpret_cast<unsigned int*>(id + ns);
    }
    __device__ SplitPos record(int s) const
    {
        SplitPos p;
        const float2 x = split[s], yy = split[ns + s], z = split[2 * ns + s], m = massf[s];
        p.xy = make_float4(x.x, x.y, yy.x, yy.y);
        p.zm = make_float4(z.x, z.y, m.x, m.y);
        return p;
    }
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

}  // namespace

__global__ void __launch_bounds__(SWARM_THREADS) swarm_rkf78_kernel(SmallStepArgs a, int slice)
{
    extern __shared__ __align__(16) unsigned char swarm_smem[];
    SwarmSmem M(swarm_smem, slice);
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), n_cta = (int)cluster.num_blocks();
    const int t = threadIdx.x, nt = blockDim.x, lane = t & 31, warp = t >> 5, nw = nt >> 5;
    const int ns = M.ns, nh = a.n_si;
    const int b0 = nh + rank * slice;                                   // the slice's first body
    const int nl = max(0, min(slice, a.n_massive - b0));                // its light bodies
    const int pieces = slice / 32, chunks = nh * pieces;                // pair warps per heavy body, and of all
    auto body_of = [&](int s) { return s < HEAVY ? s : b0 + s - HEAVY; };
    auto valid = [&](int s) { return s < HEAVY ? s < nh : s - HEAVY < nl; };
    GravArgs g = a.g;
    const bool record = g.record != 0, hill = g.hill != 0;
    g.px = M.pos;
    g.py = M.pos + ns;
    g.pz = M.pos + 2 * ns;
    g.mass = M.mass;
    g.radius = M.radius;
    g.id = M.id;
    g.rho = M.rho;
    g.rf = M.rf;
    const Tile tile{0, 0, 0, nh, 0, 0, 1, 0};  // numbers of this CTA's slots; body 0 (the star) is slot 0
    const int shift = b0 - HEAVY;              // of a light slot to its body

    if (rank == 0 && t == 0) {
        *g.ev.count = 0u;
        if (a.first) *g.hv.count = 0u;
        __threadfence();
    }
    __shared__ unsigned long long s_max;
    __shared__ unsigned int s_eject;
    if (t == 0) {
        s_max = 0ull;
        s_eject = 0u;
    }
    for (int s = t; s < ns; s += nt) {
        const bool ok = valid(s);
        const int b = ok ? body_of(s) : 0;
        const double m = ok ? a.g.mass[b] : 0.0, R = ok ? a.g.radius[b] : 0.0;
        const int id = ok ? a.g.id[b] : -1;
        M.mass[s] = m;
        M.radius[s] = R;
        M.id[s] = id;
        float lo;
        split_bits(R, M.rf[s], lo);
        float2 mf = make_float2(0.0f, 0.0f);
        if (id >= 0) split_bits(m, mf.x, mf.y);
        M.massf[s] = mf;
        M.rho[s] = 0.0;
    }
    for (int e = t; e < 6 * ns; e += nt) {
        const int row = e / ns, s = e % ns;
        const bool ok = valid(s);
        const size_t at = (size_t)row * a.stride + (ok ? body_of(s) : 0);
        const double v = ok ? a.y[at] : 0.0;
        M.y[e] = v;
        if (!a.first) M.k[e] = ok ? a.k0[at] : 0.0;
        if (a.first) {  // stage 0: (v, a(y))
            if (row >= 3) M.k[e - 3 * ns] = v;
            if (row < 3) {
                M.pos[e] = v;
                split_coord(v, M.split[e].x, M.split[e].y);
            }
        }
    }
    cluster_arrive();
    cluster_wait();
    if (a.first && hill) {
        for (int s = t; s < ns; s += nt) {
            const double dx = M.y[s] - M.y[0], dy = M.y[ns + s] - M.y[ns], dz = M.y[2 * ns + s] - M.y[2 * ns];
            if (valid(s))
                M.rho[s] = rn_sqrt(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
        }
        __syncthreads();
    }

    // element (row, s) of stage r's positions and velocities
    auto stage_element = [&](int r, int row, int s) {
        const double* const k = M.k + row * ns + s;
        double sum = __dmul_rn(a.a[r][0], k[a.stage[r][0] * 6 * ns]);
        for (int q = 1; q < a.nterm[r]; q++) sum = __dadd_rn(sum, __dmul_rn(a.a[r][q], k[a.stage[r][q] * 6 * ns]));
        const double out = __dadd_rn(M.y[row * ns + s], __dmul_rn(a.dt, sum));
        if (row < 3) {
            M.pos[row * ns + s] = out;
            split_coord(out, M.split[row * ns + s].x, M.split[row * ns + s].y);
        } else {
            M.k[(r * 6 + row - 3) * ns + s] = out;
        }
    };
    // element (row, s) of y_{n+1}
    auto next_element = [&](int row, int s) {
        auto k = [&](int q) { return M.k[(q * 6 + row) * ns + s]; };
        double sum = __dadd_rn(__dmul_rn(a.b[0], k(0)), __dmul_rn(a.b[1], k(5)));
        sum = __dadd_rn(sum, __dmul_rn(a.b[2], __dadd_rn(k(6), k(7))));
        sum = __dadd_rn(sum, __dmul_rn(a.b[3], __dadd_rn(k(8), k(9))));
        sum = __dadd_rn(sum, __dmul_rn(a.b[4], k(10)));
        const double out = __dadd_rn(M.y[row * ns + s], __dmul_rn(a.dt, sum));
        a.y_out[(size_t)row * a.stride + body_of(s)] = out;
        if (row < 3) M.pos[row * ns + s] = out;
    };
    // the ejection / hit-star screen (stages.cu) of a body at its y_{n+1}
    auto eject_screen = [&](int s) {
        const int b = body_of(s);
        if (!(0 < M.id[s] && a.type[b] != RG_BODY_STAR)) return;
        const double x = M.pos[s], y = M.pos[ns + s], z = M.pos[2 * ns + s];
        const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
        if ((0.0 < a.thr_ej && a.thr_ej2 < r2) || (0.0 < a.thr_hit && a.thr_hit2 > r2)) atomicAdd(&s_eject, 1u);
    };
    // the pairs of stage r's positions: the light bodies' terms and this CTA's part of the heavy rows
    auto pairs = [&](int r) {
        g.vx = r > 0 ? M.k + r * 6 * ns : M.y + 3 * ns;
        g.vy = g.vx + ns;
        g.vz = g.vx + 2 * ns;
        g.record = record && r > 0;  // events of stage 0 are dropped (int_rungekutta8.cu:730-733)
        g.hill = hill && r == 0;
        g.seq = (r > 0 ? a.attempt << 8 : 0u) | (unsigned)r;
        const SplitPos p0 = M.record(0);
        const float inv3M = g.hill ? 1.0f / (3.0f * p0.zm.z) : 0.0f;
        const float frad = g.f_rad_f;
#pragma unroll 1
        for (int q = warp; q <= chunks; q += nw) {
            const bool heavy = q == chunks;  // the last warp's pairs: heavy x heavy
            const int h = heavy ? lane % nh : q / pieces;
            const int l = (q % pieces) * 32 + lane;
            const int s = heavy ? (lane / nh) : HEAVY + l;  // the sink's slot; h is the source's
            const bool there = heavy ? lane < nh * nh && s != h : l < nl;
            DF tx{0.0f, 0.0f}, ty{0.0f, 0.0f}, tz{0.0f, 0.0f}, ux = tx, uy = tx, uz = tx;
            const bool src_ok = there && 0 <= M.id[s];  // as a source; 0 < id: as a sink
            const bool own = there && 0 < M.id[s] && 0 <= M.id[h], rev = !heavy && src_ok && 0 < M.id[h];
            if (own || rev) {
                const SplitPos pi = M.record(s), ph = M.record(h);
                const float2 mh = M.massf[h], mi = M.massf[s];
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
                if (own) {
                    const DF w = df_mul(y3, DF{mh.x, mh.y});
                    tx = df_mul(w, dx);
                    ty = df_mul(w, dy);
                    tz = df_mul(w, dz);
                    if ((g.record || g.hill) && (!heavy || rank == 0)) {
                        g.i_shift = heavy ? 0 : shift;
                        df_screen(g, tile, s, h, r2.hi, M.rf[s], M.rf[h], g.hill ? star_dist_f(pi, p0) : 0.0f,
                                  g.hill ? star_dist_f(ph, p0) : 0.0f, mi.x, mh.x, inv3M, frad);
                    }
                }
                if (rev) {
                    const DF w = df_mul(y3, DF{mi.x, mi.y});
                    ux = df_mul(w, dx);
                    uy = df_mul(w, dy);
                    uz = df_mul(w, dz);
                }
            }
            if (heavy) {
                if (lane < nh * nh) {
                    M.hh[s][h][0] = tx;
                    M.hh[s][h][1] = ty;
                    M.hh[s][h][2] = tz;
                }
            } else {
                M.own[(h * 3 + 0) * slice + l] = make_float2(tx.hi, tx.lo);
                M.own[(h * 3 + 1) * slice + l] = make_float2(ty.hi, ty.lo);
                M.own[(h * 3 + 2) * slice + l] = make_float2(tz.hi, tz.lo);
                Acc2 v[3] = {{-ux.hi, -ux.lo}, {-uy.hi, -uy.lo}, {-uz.hi, -uz.lo}};
#pragma unroll
                for (int off = 16; off > 0; off >>= 1)
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const Acc2 o{__shfl_xor_sync(0xffffffffu, v[c].s, off), __shfl_xor_sync(0xffffffffu, v[c].c, off)};
                        v[c] = two_sum_merge(v[c], o);
                    }
                if (lane == 0)
                    for (int c = 0; c < 3; c++) M.red[q][c] = df_two_sum(v[c].s, v[c].c);
            }
        }
    };
    // after the pairs: this CTA's part of the heavy rows into every CTA's part[r & 1], and the
    // light bodies' accelerations
    auto sums = [&](int r) {
        if (t < 3 * nh) {
            const int h = t / 3, c = t % 3;
            DF v = M.red[h * pieces][c];
            for (int p = 1; p < pieces; p++) v = df_add(v, M.red[h * pieces + p][c]);
            const double d = df_to_double(v);
            double* const at = M.part + ((r & 1) * SWARM_CTAS + rank) * 3 * HEAVY + t;
            for (int q = 0; q < n_cta; q++) *cluster.map_shared_rank(at, q) = d;
        }
        for (int e = nt - 1 - t; e < 3 * nl; e += nt) {  // (the first warp has the parts)
            const int c = e / nl, l = e % nl;
            Acc2 o{0.0f, 0.0f};
            for (int h = 0; h < nh; h++) {
                const float2 f = M.own[(h * 3 + c) * slice + l];
                acc_df(o, DF{f.x, f.y});
            }
            M.k[(r * 6 + 3 + c) * ns + HEAVY + l] = f2d_bits(o.s) + f2d_bits(o.c);
        }
    };
    // after the barrier: the heavy rows, by the first warp
    auto heavy_rows = [&](int r) {
        if (t < 3 * nh) {
            const int h = t / 3, c = t % 3;
            Acc2 o{0.0f, 0.0f};
            for (int q = 0; q < nh; q++) acc_df(o, M.hh[h][q][c]);
            double v = f2d_bits(o.s) + f2d_bits(o.c);
            const double* const P = M.part + (r & 1) * SWARM_CTAS * 3 * HEAVY + t;
            for (int q = 0; q < n_cta; q++) v += P[q * 3 * HEAVY];
            M.k[(r * 6 + 3 + c) * ns + h] = v;
        }
        __syncwarp();
    };

    if (!a.first) {
        __syncthreads();
        for (int e = t; e < 6 * ns; e += nt) stage_element(1, e / ns, e % ns);
        __syncthreads();
    }
    for (int r = a.first ? 0 : 1; r < 13; r++) {
        pairs(r);
        __syncthreads();
        sums(r);
        cluster_arrive();
        __syncthreads();
        // the light bodies' part of what follows, while the others arrive
        if (r == 10) {
            for (int e = t; e < 6 * nl; e += nt) next_element(e / nl, HEAVY + e % nl);
            __syncthreads();
            for (int l = t; l < nl; l += nt) eject_screen(HEAVY + l);
            __syncthreads();
        }
        const bool more = r < 12 && (r != 10 || a.adaptive);
        if (more)
            for (int e = t; e < 6 * nl; e += nt) stage_element(r + 1, e / nl, HEAVY + e % nl);
        cluster_wait();
        if (warp == 0) {
            heavy_rows(r);
            if (r == 10 && rank == 0) {
                if (lane < 6 * nh) next_element(lane / nh, lane % nh);
                __syncwarp();
                if (lane < nh) eject_screen(lane);
                __syncwarp();
            }
            if (more && lane < 6 * nh) stage_element(r + 1, lane / nh, lane % nh);
        }
        if (!more) break;
        __syncthreads();
        if (r == 0)
            for (int e = t; e < 6 * ns; e += nt)
                if (valid(e % ns) && (rank == 0 || e % ns >= HEAVY))
                    a.k0[(size_t)(e / ns) * a.stride + body_of(e % ns)] = M.k[e];
    }
    __syncthreads();
    if (a.adaptive) {
        for (int e = t; e < 6 * ns; e += nt) {
            const int row = e / ns, s = e % ns;
            if (!valid(s) || body_of(s) >= a.n_err || (s < HEAVY && rank != 0)) continue;
            auto k = [&](int q) { return M.k[(q * 6 + row) * ns + s]; };
            const double v = k(0) + k(10) - k(11) - k(12);
            if (0.0 < v) atomicMax(&s_max, (unsigned long long)__double_as_longlong(v));
        }
        __syncthreads();
    }
    if (t == 0) {
        *cluster.map_shared_rank(M.max_bits + rank, 0) = s_max;
        *cluster.map_shared_rank(M.n_eject + rank, 0) = s_eject;
        __threadfence();  // the event counts
    }
    cluster_arrive();
    cluster_wait();
    if (rank == 0 && t == 0) {  // what the host needs, straight into its pinned memory
        unsigned long long m = 0ull;
        unsigned int ej = 0u;
        for (int q = 0; q < n_cta; q++) {
            m = max(m, M.max_bits[q]);
            ej += M.n_eject[q];
        }
        a.out->max_bits = m;
        a.out->n_event = atomicAdd(g.ev.count, 0u);
        a.out->n_hill = atomicAdd(g.hv.count, 0u);
        a.out->n_eject = ej;
    }
}

namespace {

struct SwarmShape {
    int ctas, slice, threads;
};

SwarmShape swarm_shape(int n_heavy, int n_light)
{
    SwarmShape s;
    s.ctas = n_light <= 32 * 8 ? 8 : SWARM_CTAS;
    s.slice = swarm_slice(n_light);
    // a warp per pair chunk and one for the heavy pairs, as far as there are
    s.threads = std::min(SWARM_THREADS, std::max(256, 32 * (n_heavy * s.slice / 32 + 1)));
    return s;
}

void swarm_config(const SwarmShape& s, cudaStream_t st, cudaLaunchAttribute* attr, cudaLaunchConfig_t* cfg)
{
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)s.ctas;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg->gridDim = dim3((unsigned)s.ctas);
    cfg->blockDim = dim3((unsigned)s.threads);
    cfg->dynamicSmemBytes = SwarmSmem::bytes(s.slice);
    cfg->stream = st;
    cfg->attrs = attr;
    cfg->numAttrs = 1;
}

}  // namespace

// light bodies of a CTA: a sixteenth, in whole warps; up to 256 bodies an eighth (CTAs of 32)
int swarm_slice(int n_light)
{
    const int ctas = n_light <= 32 * 8 ? 8 : SWARM_CTAS;
    return std::max(1, (n_light + 32 * ctas - 1) / (32 * ctas)) * 32;
}

// whether the device takes such a cluster (asked once per device and cluster size, for the largest slice)
bool swarm_step_fits(int n_heavy, int n_light)
{
    if (n_heavy < 1 || n_heavy > HEAVY || n_light < 1 || n_light > SWARM_MAX_LIGHT) return false;
    static std::atomic<int> known[64][2];  // 0: not asked, 1: yes, 2: no
    SwarmShape s = swarm_shape(n_heavy, n_light);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    std::atomic<int>& answer = known[dev][s.ctas == SWARM_CTAS];
    if (answer.load(std::memory_order_acquire) == 0) {
        s.slice = SWARM_SLICE;
        s.threads = SWARM_THREADS;
        cudaLaunchAttribute attr{};
        cudaLaunchConfig_t cfg{};
        swarm_config(s, nullptr, &attr, &cfg);
        int clusters = 0;
        const bool ok =
            cudaFuncSetAttribute(swarm_rkf78_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)SwarmSmem::bytes(SWARM_SLICE)) == cudaSuccess &&
            cudaFuncSetAttribute(swarm_rkf78_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&clusters, swarm_rkf78_kernel, &cfg) == cudaSuccess && clusters > 0;
        if (!ok) cudaGetLastError();
        answer.store(ok ? 1 : 2, std::memory_order_release);
    }
    return answer.load(std::memory_order_acquire) == 1;
}

int launch_swarm_rkf78(const SmallStepArgs& a, cudaStream_t st)
{
    const SwarmShape s = swarm_shape(a.n_si, a.n_massive - a.n_si);
    cudaLaunchAttribute attr{};
    cudaLaunchConfig_t cfg{};
    swarm_config(s, st, &attr, &cfg);
    RG_CUDA_CHECK(cudaLaunchKernelEx(&cfg, swarm_rkf78_kernel, a, s.slice));
    RG_CUDA_CHECK(cudaGetLastError());
    return 0;
}

}  // namespace redgb
