// small_step.cu -- one attempt of an RKF7(8) step of a small system (at most 32 bodies: a star and
// its planets) in one kernel of one CTA.
//
// Such a step is all latency: 13 force evaluations, each a pair term (about 2 000 cycles) and one
// FP64 addition per source (71 cycles each), and 13 stage sums of up to 18 dependent FP64
// operations.  As separate kernels each evaluation paid two launches and the thread-per-sink
// kernel's serial pairs (15.7 us for nine bodies).  Here the state, the stage vectors and the
// terms stay in shared memory; pairs, sums and state elements are each dealt out densely over
// the threads, because a warp's FP64 instruction costs its SM sub-partition 64 cycles however
// few lanes are active (a warp per body took 75 us per attempt of nine bodies, this form
// 38; a step 281 us before, 45 now, with the host's launch and wait).  The arithmetic is the
// other kernels': pair_term, the sums in ascending source order, the stage sums of stages.cu.
#include <algorithm>
#include <atomic>

#include "../../include/redgb.h"
#include "common.cuh"
#include "kernels.h"
#include "pair_fp64.cuh"

namespace redgb {

namespace {

struct SmallSmem {
    double y[6][SMALL_MAX];
    double k[13][6][SMALL_MAX];
    double pos[3][SMALL_MAX];              // stage positions
    double term[3][SMALL_MAX][SMALL_MAX];  // [component][source][sink]
    double rho[SMALL_MAX];
    unsigned long long max_bits;
    unsigned int n_eject;
};

}  // namespace

__global__ void __launch_bounds__(SMALL_MAX * SMALL_MAX) small_rkf78_kernel(SmallStepArgs a)
{
    extern __shared__ __align__(16) unsigned char small_smem[];
    SmallSmem& M = *reinterpret_cast<SmallSmem*>(small_smem);
    const int t = threadIdx.x, n = a.n;
    // this thread's pair (sink pi, source pj), state element (row er of body ei) and sum
    // (component sc of body si)
    const int pi = t / n, pj = t % n, er = t / n, ei = t % n, sc = t / n, si = t % n;
    auto block_of = [&](int i) { return i < a.n_si ? 0 : (i < a.n_massive ? 1 : 2); };
    auto sources_of = [&](int block) { return block == 1 ? a.n_si : a.n_massive; };
    const bool has_pair = t < n * n, has_element = t < 6 * n, has_sum = t < 3 * n;
    const int block = block_of(pi);
    const bool pair = has_pair && pj < sources_of(block) && pj != pi && 0 < a.g.id[has_pair ? pi : 0] && 0 <= a.g.id[pj];
    const double Ri = has_pair ? a.g.radius[pi] : 0.0, mi = has_pair ? a.g.mass[pi] : 0.0;
    const double Rj = a.g.radius[pj], mj = a.g.mass[pj];
    const int n_terms = has_sum ? sources_of(block_of(si)) : 0;
    const Tile tile{pi, pi + 1, 0, sources_of(block), 0, 0, block, 0};
    GravArgs g = a.g;
    const bool record = g.record != 0, hill = g.hill != 0;
    if (t == 0) {
        M.max_bits = 0ull;
        M.n_eject = 0u;
        *g.ev.count = 0u;
        if (a.first) *g.hv.count = 0u;
    }
    if (has_element) {
        M.y[er][ei] = a.y[(size_t)er * a.stride + ei];
        if (!a.first) M.k[0][er][ei] = a.k0[(size_t)er * a.stride + ei];
    }
    __syncthreads();

    // accelerations of the positions p (velocities v) into the stage vector r
    auto gravity = [&](int r, const double (*p)[SMALL_MAX], const double (*v)[SMALL_MAX]) {
        g.px = p[0];
        g.py = p[1];
        g.pz = p[2];
        g.vx = v[0];
        g.vy = v[1];
        g.vz = v[2];
        g.rho = M.rho;
        g.record = record && r > 0;  // events of stage 0 are dropped (int_rungekutta8.cu:730-733)
        g.hill = hill && r == 0;
        g.seq = (r > 0 ? a.attempt << 8 : 0u) | (unsigned)r;
        if (has_pair) {
            PairOut o{0.0, 0.0, 0.0};
            if (pair) {
                const double hi = g.hill ? M.rho[pi] : 0.0, hj = g.hill ? M.rho[pj] : 0.0;
                // few warps: the FP64 pipe's shorter square root and division; many: the integer ones
                if (n <= 16)
                    pair_term<true, true>(g, tile, pi, pj, p[0][pi], p[1][pi], p[2][pi], Ri, mi, hi, p[0][pj], p[1][pj],
                                          p[2][pj], mj, Rj, hj, o);
                else
                    pair_term<true, false>(g, tile, pi, pj, p[0][pi], p[1][pi], p[2][pi], Ri, mi, hi, p[0][pj], p[1][pj],
                                           p[2][pj], mj, Rj, hj, o);
            }
            M.term[0][pj][pi] = o.tx;
            M.term[1][pj][pi] = o.ty;
            M.term[2][pj][pi] = o.tz;
        }
        __syncthreads();
        if (has_sum) {
            double acc = 0.0;
            for (int j = 0; j < n_terms; j++) acc = acc + M.term[sc][j][si];
            M.k[r][3 + sc][si] = acc;
        }
        __syncthreads();
    };

    if (a.first) {  // stage 0: (v, a(y))
        if (hill && t < n) {
            const double dx = M.y[0][t] - M.y[0][0], dy = M.y[1][t] - M.y[1][0], dz = M.y[2][t] - M.y[2][0];
            M.rho[t] = rn_sqrt(dx * dx + dy * dy + dz * dz);
        }
        if (has_sum) M.k[0][sc][si] = M.y[3 + sc][si];
        __syncthreads();
        gravity(0, &M.y[0], &M.y[3]);
        if (has_element) a.k0[(size_t)er * a.stride + ei] = M.k[0][er][ei];
    }
    for (int r = 1; r < 13; r++) {
        if (r == 11) {  // y_{n+1}, and without step-size control nothing more
            if (has_element) {
                auto k = [&](int q) { return M.k[q][er][ei]; };
                const double out = M.y[er][ei] + a.dt * (a.b[0] * k(0) + a.b[1] * k(5) + a.b[2] * (k(6) + k(7)) +
                                                         a.b[3] * (k(8) + k(9)) + a.b[4] * k(10));
                a.y_out[(size_t)er * a.stride + ei] = out;
                if (er < 3) M.pos[er][ei] = out;
            }
            __syncthreads();
            if (t < n && 0 < a.g.id[t] && a.type[t] != RG_BODY_STAR) {  // the ejection / hit-star screen (stages.cu)
                const double x = M.pos[0][t], y = M.pos[1][t], z = M.pos[2][t];
                const double r2 = x * x + y * y + z * z;
                if ((0.0 < a.thr_ej && a.thr_ej2 < r2) || (0.0 < a.thr_hit && a.thr_hit2 > r2)) atomicAdd(&M.n_eject, 1u);
            }
            __syncthreads();
            if (!a.adaptive) break;
        }
        if (has_element) {
            double sum = a.a[r][0] * M.k[a.stage[r][0]][er][ei];
            for (int q = 1; q < a.nterm[r]; q++) sum = sum + a.a[r][q] * M.k[a.stage[r][q]][er][ei];
            const double out = M.y[er][ei] + a.dt * sum;
            if (er < 3)
                M.pos[er][ei] = out;
            else
                M.k[r][er - 3][ei] = out;
        }
        __syncthreads();
        gravity(r, M.pos, &M.k[r][0]);
    }
    if (a.adaptive && has_element && ei < a.n_err) {
        const double v = M.k[0][er][ei] + M.k[10][er][ei] - M.k[11][er][ei] - M.k[12][er][ei];
        if (0.0 < v) atomicMax(&M.max_bits, (unsigned long long)__double_as_longlong(v));
    }
    __syncthreads();
    if (t == 0) {  // what the host needs, straight into its pinned memory
        a.out->max_bits = M.max_bits;
        a.out->n_event = atomicAdd(g.ev.count, 0u);
        a.out->n_hill = atomicAdd(g.hv.count, 0u);
        a.out->n_eject = M.n_eject;
    }
}

int launch_small_rkf78(const SmallStepArgs& a, cudaStream_t st)
{
    static std::atomic<bool> attr_set[64];  // a per-device attribute, set once per device
    int dev = 0;
    RG_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
        RG_CUDA_CHECK(cudaFuncSetAttribute(small_rkf78_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)sizeof(SmallSmem)));
        if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
    }
    const int threads = (std::max(a.n * a.n, 6 * a.n) + 31) / 32 * 32;
    small_rkf78_kernel<<<1, threads, sizeof(SmallSmem), st>>>(a);
    RG_CUDA_CHECK(cudaGetLastError());
    return 0;
}

}  // namespace redgb
