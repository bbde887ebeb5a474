// ens_stage.cu -- a stage of the ensemble's mixed-precision RKF7(8) attempt in one kernel: the stage
// sums of every body (ens_combine_df_kernel's arithmetic) and the symmetric heavy-light evaluation
// at them (grav_df_sym's), with the same bits as the two kernels.
//
// Bound: apart, the stage sums wait for HBM (they read y and up to nine stage vectors, 48 bytes a
// body each: 65 to 69 % of its rate) with the FP32 pipes idle, and the pairs use the pipes (61 %
// issue) with HBM idle.  Here warps in one phase run beside warps in the other, the stage positions
// stay in registers instead of going through memory (24 bytes written and read a body), and a stage
// has one launch, one prologue and one tail.  Measured: 128 attempts of 256 disks (1.1 million
// bodies) 238 -> 215 ms (267 -> 240 ms with the disks' states read), with the elements loaded when
// used 227 ms; attempts of eight disks of 512 bodies, all latency, 30 % more a second.  Now issue
// bounds it (65 % of cycles; six stage vectors and the pairs are 88 million warp instructions).
#include <atomic>
#include <string>

#include "../../include/redgb.h"
#include "common.cuh"
#include "kernels.h"
#include "pair_df.cuh"
#include "tma.cuh"

namespace redgb {

int set_error(int code, const std::string& msg);

namespace {

constexpr int HMAX = STAGE_SYM_HEAVY;  // heavy bodies of a disk

// df_mul with its product's rounding kept out of multiply-adds, as the stage sums' unit is built
__device__ __forceinline__ DF mul_nc(DF a, DF b)
{
    DF p;
    p.hi = __fmul_rn(a.hi, b.hi);
    p.lo = fmaf(a.hi, b.hi, -p.hi);
    p.lo = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, p.lo));
    return df_fast_sum(p.hi, p.lo);
}

// element e of the stage: y + sum_q w_q k_q
template <int NTERM>
__device__ __forceinline__ double stage_element(const StageSymArgs& a, const DF* w, long long e)
{
    const double y = __ldg(a.y + e);
    DF k[NTERM];
#pragma unroll
    for (int q = 0; q < NTERM; q++) {
        const float2 f = __ldg(reinterpret_cast<const float2*>(a.k[q]) + e);
        k[q] = DF{f.x, f.y};
    }
    DF sum = mul_nc(w[0], k[0]);
#pragma unroll
    for (int q = 1; q < NTERM; q++) sum = df_add(sum, mul_nc(w[q], k[q]));
    return __dadd_rn(y, __dadd_rn(f2d_bits(sum.hi), f2d_bits(sum.lo)));
}

// The light bodies' elements come through shared memory, each thread's own by cp.async AHEAD rows
// before they are used (across the pairs of the body before), so that no wait for them is seen:
// loaded when used, long-scoreboard stalls were two fifths of all and the kernel issued on 57 % of
// cycles.
constexpr int AHEAD = 3;  // rows in flight: a body's velocity or position rows
template <int NTERM>
struct Feed {
    double slot[AHEAD][NTERM + 1][256];  // y, then the stage vectors' pairs
};

template <int NTERM>
__device__ __forceinline__ void feed_row(const StageSymArgs& a, Feed<NTERM>& F, int slot, long long e)
{
#pragma unroll
    for (int q = 0; q <= NTERM; q++) {
        const double* const from = (q == 0 ? a.y : a.k[q - 1]) + e;
        const unsigned to = (unsigned)__cvta_generic_to_shared(&F.slot[slot][q][threadIdx.x]);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(from) : "memory");
    }
}
__device__ __forceinline__ void feed_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void feed_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD - 1) : "memory"); }

template <int NTERM>
__device__ __forceinline__ double fed_element(const Feed<NTERM>& F, int slot, const DF* w)
{
    const double y = F.slot[slot][0][threadIdx.x];
    DF sum{0.0f, 0.0f};
#pragma unroll
    for (int q = 0; q < NTERM; q++) {
        const float2 f = reinterpret_cast<const float2&>(F.slot[slot][q + 1][threadIdx.x]);
        const DF t = mul_nc(w[q], DF{f.x, f.y});
        sum = q == 0 ? t : df_add(sum, t);
    }
    return __dadd_rn(y, __dadd_rn(f2d_bits(sum.hi), f2d_bits(sum.lo)));
}

struct Body {
    double r[3], v[3];
};

// exact_event_tests (pair_df.cuh) of a pair whose states are at hand; no Hill tests after the step start
__device__ __noinline__ void stage_event(const GravArgs& g, const Tile& tile, int i, int j, const Body& bi, const Body& bj,
                                         const Body& b0)
{
    const double dx = __dadd_rn(bj.r[0], -bi.r[0]), dy = __dadd_rn(bj.r[1], -bi.r[1]), dz = __dadd_rn(bj.r[2], -bi.r[2]);
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    const double d = sqrt(r2);
    const int li = i - tile.base, lj = j - tile.base;
    if (!(g.record && li > 0 && li > lj && d < __dmul_rn(tile_f_rad(g, tile), __dadd_rn(g.radius[i], g.radius[j])))) return;
    const unsigned int slot = atomicAdd(g.ev.count, 1u);
    if (g.sys_events) atomicAdd(&g.sys_events[tile.sys], 1u);
    if (slot >= g.ev.cap) return;
    DevEvent* e = &g.ev.rec[slot];
    e->seq = record_seq(g, tile, 0);
    e->kind = 0;
    e->i = i;
    e->j = j;
    e->sys = tile.sys;
    e->pad = 0;
    e->d = d;
    e->t = g.sys_t ? g.sys_t[tile.sys] : 0.0;
    for (int c = 0; c < 3; c++) {
        e->ri[c] = bi.r[c];
        e->rj[c] = bj.r[c];
        e->vi[c] = bi.v[c];
        e->vj[c] = bj.v[c];
        e->r0[c] = b0.r[c];
        e->v0[c] = b0.v[c];
    }
}

}  // namespace

template <int NTERM>
__global__ void __launch_bounds__(256, DF_SYM_RESIDENT) ens_stage_sym(StageSymArgs a)
{
    const GravArgs& g = a.g;
    pdl_wait();  // first: every CTA waits for the kernel before it (the launch may overlap them)
    __shared__ SplitPos s_h[HMAX];
    __shared__ float s_R[HMAX], s_close2[HMAX];
    __shared__ Body s_b[HMAX];
    __shared__ int s_src[HMAX], s_sink[HMAX];
    __shared__ DF s_red[8][3 * HMAX];
    __shared__ DF s_hh[HMAX][HMAX][3];
    __shared__ DF s_w[NTERM];
    __shared__ int s_last;
    extern __shared__ __align__(16) unsigned char stage_smem[];
    Feed<NTERM>& F = *reinterpret_cast<Feed<NTERM>*>(stage_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int sg = a.cta_seg[blockIdx.x]; sg < a.cta_seg[blockIdx.x + 1]; sg++) {
        const Tile tile = g.tiles[sg];
        if (!g.sys_active[tile.sys]) continue;         // uniform over the CTA
        const int nh = tile.src_end - tile.src_begin;  // <= HMAX
        const float frad = tile_frad_f(g, tile);
        // rows 3 4 5 0 1 2 of this thread's bodies, one after the other
        auto feed = [&](int i, int row, int slot) {
            if (i < tile.sink_end) feed_row<NTERM>(a, F, slot, (long long)row * a.stride + i);
            feed_commit();
        };
#pragma unroll 1
        for (int j = 0; j < AHEAD; j++) feed(tile.sink_begin + (int)threadIdx.x, 3 + j, j);
        __syncthreads();  // the previous segment's shared data are consumed
        if ((int)threadIdx.x < NTERM) s_w[threadIdx.x] = split_df(__dmul_rn(a.dt[tile.sys], a.c[threadIdx.x]));
        __syncthreads();
        // the heavy bodies' stage state, in every CTA; part 1 writes their velocities
        if ((int)threadIdx.x < 6 * nh) {
            const int h = threadIdx.x / 6, row = threadIdx.x % 6;
            const double o = stage_element<NTERM>(a, s_w, (long long)row * a.stride + tile.src_begin + h);
            if (row < 3) {
                s_b[h].r[row] = o;
            } else {
                const float2 f = to_f2(o);
                s_b[h].v[row - 3] = f2_to_double(f);
                if (tile.part == 1)
                    reinterpret_cast<float2*>(a.vel)[(long long)(row - 3) * a.stride + tile.src_begin + h] = f;
            }
        }
        __syncthreads();
        if ((int)threadIdx.x < nh) {
            const int h = tile.src_begin + threadIdx.x;
            const float2 m = a.mass_f2[h];
            SplitPos ph;
            split_coord(s_b[threadIdx.x].r[0], ph.xy.x, ph.xy.y);
            split_coord(s_b[threadIdx.x].r[1], ph.xy.z, ph.xy.w);
            split_coord(s_b[threadIdx.x].r[2], ph.zm.x, ph.zm.y);
            ph.zm.z = m.x;
            ph.zm.w = m.y;
            const int id = g.id[h];
            s_h[threadIdx.x] = ph;
            s_src[threadIdx.x] = 0 <= id;  // a source term (pp_disk.cu:246-247)
            s_sink[threadIdx.x] = 0 < id;  // a sink's row (pp_disk.cu:235-236)
            s_R[threadIdx.x] = g.rf[h];
            s_close2[threadIdx.x] = close_r2(ph);
        }
        __syncthreads();
        const int row0 = a.tile_row0[sg];
        const float margin = 1.001f;  // of the event screens, as df_screen's
        if (tile.part == 1) {  // part 0: the heavy-heavy pairs, as grav_df_few forms them
            const int t = threadIdx.x;
            if (t < nh * nh) {
                const int hs = t / nh, hq = t % nh;  // sink, source
                DF tx{0.0f, 0.0f}, ty{0.0f, 0.0f}, tz{0.0f, 0.0f};
                if (hs != hq && s_sink[hs] && s_src[hq]) {
                    float r2f;
                    df_term(s_h[hs], s_h[hq], tx, ty, tz, r2f);
                    if (r2f < s_close2[hs])
                        df_term_fp64(s_b[hs].r[0], s_b[hs].r[1], s_b[hs].r[2], s_b[hq].r[0], s_b[hq].r[1], s_b[hq].r[2],
                                     s_h[hq].zm.z, s_h[hq].zm.w, tx, ty, tz, r2f);
                    const float lim = frad * (s_R[hs] + s_R[hq]) * margin;
                    if (g.record && hs > hq && r2f < lim * lim)
                        stage_event(g, tile, tile.src_begin + hs, tile.src_begin + hq, s_b[hs], s_b[hq], s_b[0]);
                }
                s_hh[hs][hq][0] = tx;
                s_hh[hs][hq][1] = ty;
                s_hh[hs][hq][2] = tz;
            }
            __syncthreads();
            if (t < 3 * nh) {
                const int hs = t / 3, c = t % 3;
                Acc2 v{0.0f, 0.0f};
                for (int q = 0; q < nh; q++) acc_df(v, s_hh[hs][q][c]);
                a.partial[((long long)c * a.rows + row0 + hs) * a.pitch] = f2d_bits(v.s) + f2d_bits(v.c);
            }
        }
        Acc2 racc[HMAX][3];
#pragma unroll
        for (int h = 0; h < HMAX; h++)
#pragma unroll
            for (int c = 0; c < 3; c++) racc[h][c] = Acc2{0.0f, 0.0f};
        for (int i = tile.sink_begin + (int)threadIdx.x; i < tile.sink_end; i += blockDim.x) {
            const int idi = g.id[i];
            const float Ri = g.rf[i];
            const float2 mi2 = a.mass_f2[i];
            // the next stage vector's velocity rows, then the position (half = 1), by the same code:
            // that of six rows does not stay in the instruction cache
            double r[3];
#pragma unroll 1
            for (int half = 0; half < 2; half++) {
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    feed_wait();
                    r[j] = fed_element<NTERM>(F, j, s_w);
                    // the row AHEAD on, into the slot just read: the body's position, or the next one's velocity
                    feed(half ? i + (int)blockDim.x : i, half ? 3 + j : j, j);
                    if (!half) reinterpret_cast<float2*>(a.vel)[(long long)j * a.stride + i] = to_f2(r[j]);
                }
            }
            const double xi = r[0], yi = r[1], zi = r[2];
            SplitPos pi;
            split_coord(xi, pi.xy.x, pi.xy.y);
            split_coord(yi, pi.xy.z, pi.xy.w);
            split_coord(zi, pi.zm.x, pi.zm.y);
            pi.zm.z = mi2.x;
            pi.zm.w = mi2.y;
            const bool sink_ok = 0 < idi, src_ok = 0 <= idi;
            Acc2 ox{0.0f, 0.0f}, oy{0.0f, 0.0f}, oz{0.0f, 0.0f};
            if (src_ok) {
                const float close_i = close_r2(pi);
                const DF mi{pi.zm.z, pi.zm.w};
#pragma unroll
                for (int h = 0; h < HMAX; h++) {
                    if (h >= nh) continue;
                    const bool own = sink_ok && s_src[h];
                    const bool rev = s_sink[h] != 0;
                    if (!(own || rev)) continue;
                    const SplitPos ph = s_h[h];
                    DF dx = df_diff(ph.xy.x, ph.xy.y, pi.xy.x, pi.xy.y);
                    DF dy = df_diff(ph.xy.z, ph.xy.w, pi.xy.z, pi.xy.w);
                    DF dz = df_diff(ph.zm.x, ph.zm.y, pi.zm.x, pi.zm.y);
                    DF r2 = df_add_same_sign(df_add_same_sign(df_mul(dx, dx), df_mul(dy, dy)), df_mul(dz, dz));
                    if (r2.hi < fmaxf(close_i, s_close2[h])) {  // the FP64 displacement (df_term_fp64)
                        dx = split_df(__dadd_rn(s_b[h].r[0], -xi));
                        dy = split_df(__dadd_rn(s_b[h].r[1], -yi));
                        dz = split_df(__dadd_rn(s_b[h].r[2], -zi));
                        r2 = df_add_same_sign(df_add_same_sign(df_mul(dx, dx), df_mul(dy, dy)), df_mul(dz, dz));
                    }
                    if (!(r2.hi < 1.0e30f)) r2 = DF{1.0e30f, 0.0f};  // a merged body parked at 1e20 AU
                    const float y0 = rsqrt_approx(r2.hi);
                    const DF p = df_mul(r2, df_two_prod(y0, y0));
                    const float hh = (1.0f - p.hi) - p.lo;
                    const DF y = df_fast_sum(y0, 0.5f * y0 * hh);
                    const DF y3 = df_mul(df_mul(y, y), y);
                    if (own) {
                        const DF w = df_mul(y3, DF{ph.zm.z, ph.zm.w});
                        acc_df(ox, df_mul(w, dx));
                        acc_df(oy, df_mul(w, dy));
                        acc_df(oz, df_mul(w, dz));
                        const float lim = frad * (Ri + s_R[h]) * margin;
                        if (g.record && r2.hi < lim * lim) {
                            Body b;
                            b.r[0] = xi;
                            b.r[1] = yi;
                            b.r[2] = zi;
                            for (int c = 0; c < 3; c++)  // (written above by this thread)
                                b.v[c] = f2_to_double(__ldcg(reinterpret_cast<const float2*>(a.vel) + (long long)c * a.stride + i));
                            stage_event(g, tile, i, tile.src_begin + h, b, s_b[h], s_b[0]);
                        }
                    }
                    if (rev) {
                        const DF w = df_mul(y3, mi);
                        const DF tx = df_mul(w, dx), ty = df_mul(w, dy), tz = df_mul(w, dz);
                        acc_df(racc[h][0], DF{-tx.hi, -tx.lo});
                        acc_df(racc[h][1], DF{-ty.hi, -ty.lo});
                        acc_df(racc[h][2], DF{-tz.hi, -tz.lo});
                    }
                }
            }
            const DF x = df_two_sum(ox.s, ox.c), y = df_two_sum(oy.s, oy.c), z = df_two_sum(oz.s, oz.c);
            reinterpret_cast<float2*>(g.ax)[i] = make_float2(x.hi, x.lo);
            reinterpret_cast<float2*>(g.ay)[i] = make_float2(y.hi, y.lo);
            reinterpret_cast<float2*>(g.az)[i] = make_float2(z.hi, z.lo);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
        for (int h = 0; h < HMAX; h++) {
            if (h < nh) {  // uniform over the CTA
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    Acc2 v = racc[h][c];
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) {
                        const Acc2 o{__shfl_xor_sync(0xffffffffu, v.s, off), __shfl_xor_sync(0xffffffffu, v.c, off)};
                        v = two_sum_merge(v, o);
                    }
                    if (lane == 0) s_red[warp][3 * h + c] = df_two_sum(v.s, v.c);
                }
            }
        }
        __syncthreads();
        if ((int)threadIdx.x < 3 * nh) {
            const int h = threadIdx.x / 3, c = threadIdx.x % 3;
            DF v = s_red[0][threadIdx.x];
            for (int w = 1; w < (int)(blockDim.x >> 5); w++) v = df_add(v, s_red[w][threadIdx.x]);
            a.partial[((long long)c * a.rows + row0 + h) * a.pitch + tile.part] = df_to_double(v);
        }
        // the system's last segment adds its heavy rows' parts in order (no waiting: the
        // others are done)
        const int np = a.row_nparts[row0];
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            s_last = atomicAdd(&a.ticket[tile.sys], 1u) == (unsigned int)(np - 2);  // np - 1 segments
        }
        __syncthreads();
        if (s_last) {
            __threadfence();
            if (threadIdx.x == 0) a.ticket[tile.sys] = 0u;
            if ((int)threadIdx.x < 3 * nh) {
                const int h = threadIdx.x / 3, c = threadIdx.x % 3;
                const double* P = a.partial + ((long long)c * a.rows + row0 + h) * a.pitch;
                double v = 0.0;
#pragma unroll 8
                for (int q = 0; q < np; q++) v += __ldcg(P + q);
                double* out = c == 0 ? g.ax : (c == 1 ? g.ay : g.az);
                store_acc(g, out, a.row_sink[row0 + h], v);
            }
        }
    }
}

int launch_ens_stage_sym(const StageSymArgs& a, int nterm, int n_cta, cudaStream_t st)
{
    if (n_cta <= 0) return 0;
    // the term counts of the RKF7(8) stages (rk_tables.h); any other would leave the stage unwritten
    if (nterm < 1 || nterm > 9 || nterm == 5) return set_error(RG_ERR_ARG, "a stage of so many terms has no kernel");
    cudaLaunchAttribute pdl[1];
    pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)n_cta);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cfg.attrs = pdl;
    cfg.numAttrs = 1;
    static std::atomic<bool> attr_set[64];  // a per-device attribute, set once per device
    int dev = 0;
    RG_CUDA_CHECK(cudaGetDevice(&dev));
    const bool set = dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire);
#define RG_STAGE(T)                                                                                                \
    do {                                                                                                           \
        if (set)                                                                                                   \
            RG_CUDA_CHECK(cudaFuncSetAttribute(ens_stage_sym<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,      \
                                               (int)sizeof(Feed<T>)));                                             \
        if (nterm == T) {                                                                                          \
            cfg.dynamicSmemBytes = sizeof(Feed<T>);                                                                \
            RG_CUDA_CHECK(cudaLaunchKernelEx(&cfg, ens_stage_sym<T>, a));                                          \
        }                                                                                                          \
    } while (0)
    RG_STAGE(1);
    RG_STAGE(2);
    RG_STAGE(3);
    RG_STAGE(4);
    RG_STAGE(6);
    RG_STAGE(7);
    RG_STAGE(8);
    RG_STAGE(9);
#undef RG_STAGE
    if (set && dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
    RG_CUDA_CHECK(cudaGetLastError());
    return 0;
}

}  // namespace redgb
