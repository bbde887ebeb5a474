// pair_fp64.cuh -- one (sink, source) pair in the reference's FP64 arithmetic: the term and the
// event tests, shared by the FP64 gravity kernels.  Include from units built with -fmad=false.
#pragma once

#include "common.cuh"
#include "exact_fp64.h"

namespace redgb {

struct PairOut {
    double tx, ty, tz;
    double r2;  // set by pair_term
};

// the event tests of a pair at distance d and their records
__device__ __forceinline__ void pair_events(const GravArgs& g, const Tile& tile, int i, int j, double xi, double yi,
                                            double zi, double Ri, double mi, double rhoi, double xj, double yj,
                                            double zj, double mj, double Rj, double rhoj, double d)
{
    const int li = i - tile.base, lj = j - tile.base;
    bool rad = g.record && li > 0 && li > lj && d < tile_f_rad(g, tile) * (Ri + Rj);
    bool hill = false;
    if (g.hill && tile.block != 2 && li > 0 && li > lj && lj > 0) {
        const double h = 0.5 * (rhoi + rhoj);
        const double lhs = d * d * d;
        const double rhs = ((g.hill_f3 * (mi + mj)) / (3.0 * g.mass[tile.base])) * (h * h * h);
        hill = lhs < rhs;
    }
    if (rad || hill) {
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
                e->vi[0] = g.vx[i]; e->vi[1] = g.vy[i]; e->vi[2] = g.vz[i];
                e->vj[0] = g.vx[j]; e->vj[1] = g.vy[j]; e->vj[2] = g.vz[j];
                e->r0[0] = g.px[b0]; e->r0[1] = g.py[b0]; e->r0[2] = g.pz[b0];
                e->v0[0] = g.vx[b0]; e->v0[1] = g.vy[b0]; e->v0[2] = g.vz[b0];
            }
        }
    }
}

// One (sink, source) pair: the term added to a_i and the event tests of pp_disk.cu:265
// (radius criterion) and of the mutual Hill sphere (cube form, no cube root).
// EVENTS = false: the term alone, for a pair whose event tests another evaluation has made.
// PIPE: the square root and the division on the FP64 pipe (the same bits), where the pipe has
// room and the integer pipes have not.
template <bool EVENTS = true, bool PIPE = false>
__device__ __forceinline__ void pair_term(const GravArgs& g, const Tile& tile, int i, int j, double xi, double yi,
                                          double zi, double Ri, double mi, double rhoi, double xj, double yj,
                                          double zj, double mj, double Rj, double rhoj, PairOut& o)
{
    const double dx = xj - xi;
    const double dy = yj - yi;
    const double dz = zj - zi;
    const double r2 = o.r2 = dx * dx + dy * dy + dz * dz;
    const double d = PIPE ? __dsqrt_rn(r2) : rn_sqrt(r2);  // rn_*: on the integer pipes (exact_fp64.h)
    const double w = PIPE ? __ddiv_rn(mj, d * r2) : rn_div(mj, d * r2);
    o.tx = w * dx;
    o.ty = w * dy;
    o.tz = w * dz;
    if (EVENTS) pair_events(g, tile, i, j, xi, yi, zi, Ri, mi, rhoi, xj, yj, zj, mj, Rj, rhoj, d);
}

}  // namespace redgb
