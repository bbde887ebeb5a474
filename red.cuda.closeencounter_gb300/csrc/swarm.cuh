// swarm.cuh -- one attempt of an RKF7(8) step of a planetesimal disk (a star and up to three giants,
// light bodies that feel them and pull on them) in one kernel of one thread-block cluster; the two
// precisions' forms of an evaluation are in swarm_step.cu and swarm_fp64.cu.
//
// Such a step of a thousand bodies is all latency: 13 evaluations of two or three short kernels
// each on a few of the 152 SMs.  Here 16 CTAs keep the state and the stage vectors in shared memory
// for the whole attempt, a slice of the light bodies each, and the heavy bodies in every CTA.  What
// crosses CTAs is the heavy rows, by stores into the others' shared memory and a cluster barrier;
// the light bodies' next stage sums run between the barrier's two halves, so the FP64 pipe's time
// (64 cycles a warp instruction) hides it.  The pairs are dealt out with a warp per heavy body and
// 32 light ones, so that a light body's heavy pairs run side by side.
//
// The arithmetic is the separate kernels', with FP64 operations written rounded one by one (the
// mixed form's unit contracts FP32 multiply-adds).
#pragma once

#include <cooperative_groups.h>

#include <atomic>

#include "../../include/redgb.h"
#include "common.cuh"
#include "dfloat.cuh"
#include "exact_fp64.h"
#include "kernels.h"

namespace redgb {
namespace swarm {

namespace cg = cooperative_groups;

constexpr int HEAVY = DF_SYM_MAX_HEAVY;  // slots 0 .. HEAVY - 1: the heavy bodies; then the CTA's light ones
constexpr int CTAS = 16;                 // of the largest cluster
constexpr int SLICE = 192;               // most light bodies of a CTA
constexpr int THREADS = 512;
static_assert(SWARM_MAX_LIGHT == CTAS * SLICE, "limit of the plan");

struct Shape {
    int ctas, slice, threads;
};
Shape shape(int n_heavy, int n_light);

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// A CTA's shared memory for a slice (a multiple of 32 light bodies): rows of `ns` slots
struct Smem {
    double *y, *k, *pos, *mass, *radius, *rho;  // y 6 rows, k 13 x 6, pos 3
    unsigned long long* max_bits;               // [CTA]
    unsigned int* n_eject;                      // [CTA]
    int* id;
    int ns;
    unsigned char* form;  // what the form adds, on a 16-byte boundary

    __host__ __device__ static size_t bytes(int slice)
    {
        const size_t ns = slice + HEAVY;  // a multiple of 4
        return 8 * 90 * ns + 8 * CTAS + 4 * CTAS + 4 * ns;
    }
    __device__ Smem(unsigned char* base, int slice)
    {
        ns = slice + HEAVY;
        double* d = reinterpret_cast<double*>(base);
        y = d, d += 6 * ns;
        k = d, d += 78 * ns;
        pos = d, d += 3 * ns;
        mass = d, d += ns;
        radius = d, d += ns;
        rho = d, d += ns;
        max_bits = reinterpret_cast<unsigned long long*>(d), d += CTAS;
        n_eject = reinterpret_cast<unsigned int*>(d);
        id = reinterpret_cast<int*>(n_eject + CTAS);
        form = reinterpret_cast<unsigned char*>(id + ns);
    }
};
static_assert((SLICE + HEAVY) % 4 == 0 && HEAVY % 4 == 0, "alignment of the form's part");

// where a thread stands and what its CTA holds
struct Place {
    int rank, n_cta, t, nt, lane, warp, nw;
    int n, nh;              // bodies, heavy ones
    int b0, nl, slice;      // the slice's first body, its light bodies and their most
    int shift;              // of a light slot to its body
    int pieces, chunks;     // pair warps per heavy body, and of all
};

// Form: body(s, ok, mass, radius, id) at the start; position(row, s, value) for every new position;
// pairs(g, r) the pairs of stage r; light_sums(r) after them, before the cluster barrier;
// heavy_rows(r) after it, by every thread, the rows valid for the CTA's first warp
template <class Form>
__device__ __forceinline__ void attempt(const SmallStepArgs& a, int slice, unsigned char* smem)
{
    Smem M(smem, slice);
    cg::cluster_group cluster = cg::this_cluster();
    Place w;
    w.rank = (int)cluster.block_rank();
    w.n_cta = (int)cluster.num_blocks();
    w.t = threadIdx.x;
    w.nt = blockDim.x;
    w.lane = w.t & 31;
    w.warp = w.t >> 5;
    w.nw = w.nt >> 5;
    w.n = a.n_massive;
    w.nh = a.n_si;
    w.slice = slice;
    w.b0 = w.nh + w.rank * slice;
    w.nl = max(0, min(slice, a.n_massive - w.b0));
    w.shift = w.b0 - HEAVY;
    w.pieces = slice / 32;
    w.chunks = w.nh * w.pieces;
    const int ns = M.ns, rank = w.rank, n_cta = w.n_cta, t = w.t, nt = w.nt, lane = w.lane, warp = w.warp, nh = w.nh;
    const int b0 = w.b0, nl = w.nl;
    Form form(M, w, cluster);
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
        form.body(s, m, R, id);
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
                form.position(row, s, v);
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
            form.position(row, s, out);
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
    // stage r's event options, positions and velocities
    auto stage_args = [&](int r) {
        g.vx = r > 0 ? M.k + r * 6 * ns : M.y + 3 * ns;
        g.vy = g.vx + ns;
        g.vz = g.vx + 2 * ns;
        g.record = record && r > 0;  // events of stage 0 are dropped (int_rungekutta8.cu:730-733)
        g.hill = hill && r == 0;
        g.seq = (r > 0 ? a.attempt << 8 : 0u) | (unsigned)r;
    };

    if (!a.first) {
        __syncthreads();
        for (int e = t; e < 6 * ns; e += nt) stage_element(1, e / ns, e % ns);
        __syncthreads();
    }
    for (int r = a.first ? 0 : 1; r < 13; r++) {
        stage_args(r);
        form.pairs(g, r);
        __syncthreads();
        form.light_sums(r);
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
        form.heavy_rows(r);
        if (warp == 0) {
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
            const double v = __dadd_rn(__dadd_rn(__dadd_rn(k(0), k(10)), -k(11)), -k(12));
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

// ---- the launch
using Kernel = void (*)(SmallStepArgs, int);

template <class Form>
void config(const Shape& s, cudaStream_t st, cudaLaunchAttribute* attr, cudaLaunchConfig_t* cfg)
{
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)s.ctas;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg->gridDim = dim3((unsigned)s.ctas);
    cfg->blockDim = dim3((unsigned)s.threads);
    cfg->dynamicSmemBytes = Smem::bytes(s.slice) + Form::bytes(s.slice);
    cfg->stream = st;
    cfg->attrs = attr;
    cfg->numAttrs = 1;
}

// whether the device takes such a cluster (asked once per device and cluster size, for the largest slice)
template <class Form>
bool fits(Kernel kernel, int n_heavy, int n_light)
{
    if (n_heavy < 1 || n_heavy > HEAVY || n_light < 1 || n_light > SWARM_MAX_LIGHT) return false;
    static std::atomic<int> known[64][2];  // 0: not asked, 1: yes, 2: no
    Shape s = shape(n_heavy, n_light);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    std::atomic<int>& answer = known[dev][s.ctas == CTAS];
    if (answer.load(std::memory_order_acquire) == 0) {
        s.slice = SLICE;
        s.threads = THREADS;
        cudaLaunchAttribute attr{};
        cudaLaunchConfig_t cfg{};
        config<Form>(s, nullptr, &attr, &cfg);
        int clusters = 0;
        const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)cfg.dynamicSmemBytes) == cudaSuccess &&
                        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0;
        if (!ok) cudaGetLastError();
        answer.store(ok ? 1 : 2, std::memory_order_release);
    }
    return answer.load(std::memory_order_acquire) == 1;
}

template <class Form>
int launch(Kernel kernel, const SmallStepArgs& a, cudaStream_t st)
{
    const Shape s = shape(a.n_si, a.n_massive - a.n_si);
    cudaLaunchAttribute attr{};
    cudaLaunchConfig_t cfg{};
    config<Form>(s, st, &attr, &cfg);
    RG_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, a, s.slice));
    RG_CUDA_CHECK(cudaGetLastError());
    return 0;
}

}  // namespace swarm
}  // namespace redgb
