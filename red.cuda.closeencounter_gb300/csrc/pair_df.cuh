// pair_df.cuh -- a heavy pair's term in double-float arithmetic, its event screen and the FP64 event
// tests, shared by the mixed-precision gravity kernels.
#pragma once

#include "common.cuh"
#include "dfloat.cuh"

namespace redgb {

// |r_i - r_base| in FP32 from the split positions' leading parts (event screens)
__device__ __forceinline__ float star_dist_f(const SplitPos& pi, const SplitPos& p0)
{
    const float dx = pi.xy.x - p0.xy.x, dy = pi.xy.z - p0.xy.z, dz = pi.zm.x - p0.zm.x;
    return sqrtf(dx * dx + dy * dy + dz * dz);
}

__device__ __forceinline__ float rsqrt_approx(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ Acc2 two_sum_merge(Acc2 a, Acc2 b)
{
    two_sum_add(a, b.s);
    a.c += b.c;
    return a;
}

// an output row element and a velocity row element in the stage vectors' format (GravArgs::
// acc_f2, vel_f2: double-float pairs in the ensemble's mixed form, FP64 otherwise)
__device__ __forceinline__ void store_acc(const GravArgs& g, double* row, int i, double v)
{
    if (g.acc_f2)
        reinterpret_cast<float2*>(row)[i] = to_f2(v);
    else
        row[i] = v;
}

__device__ __forceinline__ double load_vel(const GravArgs& g, const double* row, int i)
{
    return g.vel_f2 ? f2_to_double(reinterpret_cast<const float2*>(row)[i]) : row[i];
}

__device__ __forceinline__ void exact_event_tests(const GravArgs& g, const Tile& tile, int i, int j, double xi,
                                                  double yi, double zi, double Ri, double mi, double rhoi)
{
    // __dadd_rn / __dmul_rn are never contracted into FMA: units of the mixed form are built
    // with FMA contraction on, and these decisions must round exactly as the FP64 kernel's do.
    const double xj = g.px[j], yj = g.py[j], zj = g.pz[j];
    const double dx = __dadd_rn(xj, -xi), dy = __dadd_rn(yj, -yi), dz = __dadd_rn(zj, -zi);
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    const double d = sqrt(r2);
    const int li = i - tile.base, lj = j - tile.base;
    const bool rad = g.record && li > 0 && li > lj && d < __dmul_rn(tile_f_rad(g, tile), __dadd_rn(Ri, g.radius[j]));
    bool hill = false;
    if (g.hill && tile.block != 2 && li > 0 && li > lj && lj > 0) {
        const double h = __dmul_rn(0.5, __dadd_rn(rhoi, g.rho[j]));
        const double lhs = __dmul_rn(__dmul_rn(d, d), d);
        const double rhs = __dmul_rn(__ddiv_rn(__dmul_rn(g.hill_f3, __dadd_rn(mi, g.mass[j])), __dmul_rn(3.0, g.mass[tile.base])),
                                     __dmul_rn(__dmul_rn(h, h), h));
        hill = lhs < rhs;
    }
    for (int kind = 0; kind < 2; kind++) {
        if (!(kind == 0 ? rad : hill)) continue;
        const EventBuf& eb = kind == 0 ? g.ev : g.hv;
        unsigned int slot = atomicAdd(eb.count, 1u);
        if (kind == 0 && g.sys_events) atomicAdd(&g.sys_events[tile.sys], 1u);
        if (slot < eb.cap) {
            DevEvent* e = &eb.rec[slot];
            e->seq = record_seq(g, tile, kind);
            e->kind = kind;
            e->i = i + g.i_shift;
            e->j = j;
            e->sys = tile.sys;
            e->pad = 0;
            e->d = d;
            e->t = g.sys_t ? g.sys_t[tile.sys] : 0.0;
            const int b0 = tile.base;
            e->ri[0] = xi; e->ri[1] = yi; e->ri[2] = zi;
            e->rj[0] = xj; e->rj[1] = yj; e->rj[2] = zj;
            e->vi[0] = load_vel(g, g.vx, i); e->vi[1] = load_vel(g, g.vy, i); e->vi[2] = load_vel(g, g.vz, i);
            e->vj[0] = load_vel(g, g.vx, j); e->vj[1] = load_vel(g, g.vy, j); e->vj[2] = load_vel(g, g.vz, j);
            e->r0[0] = g.px[b0]; e->r0[1] = g.py[b0]; e->r0[2] = g.pz[b0];
            e->v0[0] = load_vel(g, g.vx, b0); e->v0[1] = load_vel(g, g.vy, b0); e->v0[2] = load_vel(g, g.vz, b0);
        }
    }
}

// ---------------------------------------------------------------------------------------
// Heavy pairs in double-float arithmetic.
//
// The pairs whose terms need more than FP32 accuracy -- sinks against the star and giant
// planets, and the star and giants' own rows -- would cost GB300 its scarce FP64 issue
// (grav_fp64_rowseq and grav_fp64_rows spend about 35 FP64 operations per pair).
// Here they run on the FP32 pipes in unevaluated sums of two floats (hi + lo, about 44
// significant bits), built from the error-free transformations two-sum (Knuth) and
// two-product by FMA, with the double-double addition and multiplication of Hida, Li and
// Bailey (2001) carried out in float.  The inputs are the split positions and masses of
// split_positions_kernel (x = x_hi + x_lo to 2^-48 |x|), the displacement is formed from
// them exactly up to that split, 1/r^3 comes from the FP32 rsqrt refined by one Newton
// step evaluated in double-float (relative error about 2.5e-14), and the sums stay in
// double-float until one conversion to FP64 per sink and component.  Event decisions are
// screened in FP32 with the same 1e-3 margin as the mixed kernel and re-taken in FP64.


// the term m_j (r_j - r_i) / |r_j - r_i|^3 of one pair; r2f = |r_j - r_i|^2 in FP32
// the term from a double-float displacement r_j - r_i and the source's split mass
__device__ __forceinline__ void df_term_disp(DF dx, DF dy, DF dz, float mh, float ml, DF& tx, DF& ty, DF& tz,
                                             float& r2f)
{
    DF r2 = df_add_same_sign(df_add_same_sign(df_mul(dx, dx), df_mul(dy, dy)), df_mul(dz, dz));  // squares: no cancellation
    // a merged body parked at 1e20 AU (pp_disk.cu:1184) overflows r^2 in FP32; its mass is 0
    if (!(r2.hi < 1.0e30f)) r2 = DF{1.0e30f, 0.0f};
    const float y0 = rsqrt_approx(r2.hi);
    const DF p = df_mul(r2, df_two_prod(y0, y0));
    const float h = (1.0f - p.hi) - p.lo;  // 1 - r^2 y0^2, small: FP32 suffices
    const DF y = df_fast_sum(y0, 0.5f * y0 * h);
    const DF w = df_mul(df_mul(df_mul(y, y), y), DF{mh, ml});
    tx = df_mul(w, dx);
    ty = df_mul(w, dy);
    tz = df_mul(w, dz);
    r2f = r2.hi;
}

// the term from the split positions: the displacement (x_j^hi - x_i^hi) + (x_j^lo - x_i^lo)
// carries the positions to 2^-48 |x| (the split keeps 48 of FP64's 53 significant bits)
__device__ __forceinline__ void df_term(const SplitPos& si, const SplitPos& pj, DF& tx, DF& ty, DF& tz, float& r2f)
{
    df_term_disp(df_diff(pj.xy.x, pj.xy.y, si.xy.x, si.xy.y), df_diff(pj.xy.z, pj.xy.w, si.xy.z, si.xy.w),
                 df_diff(pj.zm.x, pj.zm.y, si.zm.x, si.zm.y), pj.zm.z, pj.zm.w, tx, ty, tz, r2f);
}

// r^2 below which a pair of this sink takes the FP64 displacement: beyond it the split
// positions' error, 2^-48 (|x_i| + |x_j|) per component, stays below ~1e-12 of |r_j - r_i|
__device__ __forceinline__ float close_r2(const SplitPos& p)
{
    const float m = fmaxf(fabsf(p.xy.x), fmaxf(fabsf(p.xy.z), fabsf(p.zm.x))) * (1.0f / 256.0f);
    return m * m;
}

// the term from the FP64 positions: the displacement is one FP64 subtraction per component
// (exact for neighbours, Sterbenz), kept to 2^-48 of itself -- for close pairs, where the
// split positions' 2^-48 |x| would be a large part of |r_j - r_i|
__device__ __forceinline__ void df_term_fp64(double xi, double yi, double zi, double xj, double yj, double zj,
                                             float mh, float ml, DF& tx, DF& ty, DF& tz, float& r2f)
{
    df_term_disp(split_df(__dadd_rn(xj, -xi)), split_df(__dadd_rn(yj, -yi)), split_df(__dadd_rn(zj, -zi)), mh, ml,
                 tx, ty, tz, r2f);
}

// FP32 screen of the event tests of pair_term (pp_disk.cu:262-280) with a 1e-3 margin;
// candidates are decided in FP64 by exact_event_tests
// frad: the tile's collision factor in FP32 (tile_frad_f, formed once per CTA: a per-pair load
// and conversion would run on GB300's FP64 pipe for every heavy pair)
__device__ __forceinline__ float tile_frad_f(const GravArgs& g, const Tile& tile)
{
    return g.sys_f_rad ? (float)g.sys_f_rad[tile.sys] : g.f_rad_f;
}

__device__ __forceinline__ void df_screen(const GravArgs& g, const Tile& tile, int i, int j, float r2f, float Ri,
                                          float Rj, float rhoi, float rhoj, float mi, float mj, float inv3M,
                                          float frad)
{
    const int li = i - tile.base, lj = j - tile.base;
    if (!(li > 0 && li > lj)) return;
    const float margin = 1.001f;
    bool cand = false;
    if (g.record) {
        const float lim = frad * (Ri + Rj) * margin;
        cand = r2f < lim * lim;
    }
    if (g.hill && tile.block != 2 && lj > 0) {
        const float h = 0.5f * (rhoi + rhoj);
        const float d3 = r2f * sqrtf(r2f);
        cand = cand || d3 < g.hill_f3_f * (mi + mj) * inv3M * (h * h * h) * (margin * margin * margin);
    }
    if (cand)
        exact_event_tests(g, tile, i, j, g.px[i], g.py[i], g.pz[i], g.radius[i], g.mass[i], g.hill ? g.rho[i] : 0.0);
}

}  // namespace redgb
