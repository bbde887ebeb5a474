// row_sum.h -- the bits of the serial FP64 sum acc + t_0 + t_1 + ... by a warp whose lanes each
// add one segment of the terms, all at once.
//
// A dependent FP64 addition costs 71 cycles on GB300, so a row of n terms added one after the
// other takes 71 n cycles whatever else the GPU does.  Here lane l adds its own segment from a
// guessed start: acc plus the sum of the segments before it, which is off from the true
// running sum by the roundings on the way -- a few units in the last place.  What the lane's
// chain would have given from the true start follows without another chain:
//
//  * Let the true start be d ulps above the guess.  An addition whose result stays in the
//    binade of its accumulator, Q = ulp, adds RN(t / Q) quanta, the same for every start, so the
//    offset stays d -- except when t / Q is a half-integer (a tie, to even): then the result
//    depends on the start's parity.
//  * Into the next binade up, the result is (x + d) / 2 rounded, x = a / Q + t / Q; d changes by a
//    rule of x's lowest bits.  Into a lower binade the offset is d 2^k of the finer ulps.
//
// So each lane records the few of its additions that change an offset (ties, binade changes)
// (row_mark, row_code) as it adds; then the lanes' offsets follow from one another: through
// lanes without codes by a prefix sum of the differences between a lane's end and the next
// lane's guess, through the others by applying their codes in order (row_apply), a few integer
// operations each.  The rules need every accumulator to stay in the binade it was in for any
// offset that occurs: a lane with a result within 2^32 ulps of a binade's end (or zero, not
// finite, far from the binade before) is "hard", and is added again from its true start.
//
#pragma once

#include <limits.h>

#include "exact_fp64.h"

namespace redgb {
namespace rs {

constexpr int64_t MAX_OFF = 1 << 18;   // largest offset the codes are used with

// within 2^32 ulps of a binade's end (the fraction's upper 20 bits all zeros or all ones)
XF_HD bool near_edge(uint64_t u) { return (((uint32_t)(u >> 32) + 1u) & 0xfffffu) < 2u; }

// x << s and x >> s, 0 for s outside [0, 63]
XF_HD uint64_t shl64(uint64_t x, int s)
{
#if defined(__CUDA_ARCH__)
    uint64_t r;
    asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
    return r;
#else
    return (unsigned)s < 64u ? x << s : 0ull;
#endif
}

XF_HD uint64_t shr64(uint64_t x, int s)
{
#if defined(__CUDA_ARCH__)
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
    return r;
#else
    return (unsigned)s < 64u ? x >> s : 0ull;
#endif
}

// Whether the addition s = RN(a + t), term k of its lane, changes an offset of a: a record of it
// for row_code, or 0.  A tie in the same binade: the lowest bit of t is half an ulp of a.
XF_HD uint32_t row_mark(uint64_t ua, uint64_t ut, uint64_t us, int k, bool* hard)
{
    const uint32_t ha = (uint32_t)(ua >> 32), hs = (uint32_t)(us >> 32), ht = (uint32_t)(ut >> 32), lt = (uint32_t)ut;
    const int ea = (int)(ha >> 20 & 0x7ffu), es = (int)(hs >> 20 & 0x7ffu), et = (int)(ht >> 20 & 0x7ffu);
    const uint32_t low = lt ? lt : ht | 0x100000u;  // (the leading bit; a zero term never ties: ea >= 64)
#if defined(__CUDA_ARCH__)
    const int z = __clz(__brev(low)) + (lt ? 0 : 32);
#else
    const int z = __builtin_ctz(low) + (lt ? 0 : 32);
#endif
    const int up = es - ea;
    if (up == 0 && et + z != ea - 1 && ((hs + 1u) & 0xfffffu) >= 2u && (unsigned)(es - 64) < 1983u) return 0u;
    *hard = *hard || near_edge(us) || (unsigned)(es - 64) >= 1983u || (unsigned)(ea - 64) >= 1983u || up > 6 || up < -12;
    return (uint32_t)ea << 20 | (uint32_t)(ha >> 31) << 19 | (uint32_t)k << 13 | ((uint32_t)(up + 12) & 31u) << 8 |
           ((uint32_t)ua & 0xffu);
}

// What that addition does to an offset d.  With Q = ulp(a), x = (a + t) / Q and N = floor(x): into a
// binade k up, d becomes G(N + d) - G(N), G the rounding to a multiple of 2^k (x's fraction only
// matters when N is half-way: `even`, no fraction, rounds such an N to even); a tie in the same
// binade is the same with x, d and Q halved (p = k = 1, N = 2 floor(x) + 1); into a binade p
// lower, d becomes d 2^p (whatever is rounded: the finer quantum divides the shift).
// Code: p | k << 5 | even << 8 | (N mod 2^(k + 1)) << 9 | G(N) << 17.
XF_HD uint32_t row_code(uint32_t rec, uint64_t ut)
{
    const int ea = (int)(rec >> 20), up = (int)(rec >> 8 & 31u) - 12, et = (int)((uint32_t)(ut >> 52) & 0x7ffu);
    const uint64_t mt = et ? ((ut & xf::M52) | xf::H52) : 0ull;
    const int sh = ea - et;  // |t| / Q = mt / 2^sh
    const bool rem = shl64(mt, 64 - sh) != 0 || (sh >= 64 && mt != 0);
    const uint32_t q = (uint32_t)(sh >= 0 ? shr64(mt, sh) : shl64(mt, -sh));
    const uint32_t A = rec >> 19 & 1u ? 0u - (rec & 0xffu) : rec & 0xffu;
    const uint32_t T = ut >> 63 ? 0u - q - (rem ? 1u : 0u) : q;
    const uint32_t N = A + T;
    const bool tie = up == 0;
    const int k = tie ? 1 : (up > 0 ? up : 0), p = tie ? 1 : (up < 0 ? -up : 0);
    const uint32_t even = tie || (up > 0 && !rem) ? 1u : 0u;
    const uint32_t n = k ? (tie ? 2u * N + 1u : N) & ((2u << k) - 1u) : 0u;
    const uint32_t g = (n + ((1u << k) >> 1) - even + (n >> k & even)) >> k;
    return (uint32_t)p | (uint32_t)k << 5 | even << 8 | n << 9 | g << 17;
}

// A code unpacked for a run through many of them, with `in` added to the offset before it: d becomes
// (v + half + (v >> k & even)) >> k with v = d 2^p + n.  Offsets of any size, as long as v keeps to
// 2^29 (`most` collects its bits, all of them where d 2^p does not fit 32 bits).
struct RowRule {
    int n, half, shifts, even;  // shifts: p | k << 16
};
XF_HD bool row_rule(uint32_t code, int in, RowRule* r)
{
    const int p = (int)(code & 31u), k = (int)(code >> 5 & 7u), even = (int)(code >> 8 & 1u);
    const int64_t n = (int64_t)(code >> 9 & 0xffu) + (int64_t)in * (1 << p);
    r->n = (int)n;
    r->half = ((1 << k) >> 1) - even - (int)(code >> 17) * (1 << k);
    r->shifts = p | k << 16;
    r->even = even;
    return n < (1 << 29) && n > -(1 << 29);
}
XF_HD int row_follow(const RowRule& r, int d, int* most)
{
    const int k = r.shifts >> 16, p = r.shifts & 31;
    const int v0 = (int)((uint32_t)d << p), v = v0 + r.n;
    *most |= (v0 ^ (v0 >> 31)) | ((v0 >> p) == d ? 0 : INT_MAX);
    return (v + r.half + (v >> k & r.even)) >> k;
}

// the offset after an addition with this code, |d| < MAX_OFF
XF_HD int row_apply(uint32_t code, int d)
{
    const int p = (int)(code & 31u), k = (int)(code >> 5 & 7u), even = (int)(code >> 8 & 1u);
    const int n = (int)(code >> 9 & 0xffu) + d * (1 << p);
    return ((n + ((1 << k) >> 1) - even + (n >> k & even)) >> k) - (int)(code >> 17);
}

// a value in units of 2^(top - 1073), truncated; 0 for one that is not finite
XF_HD int64_t row_units(uint64_t v, int top)
{
    const int e = (int)((uint32_t)(v >> 52) & 0x7ffu);
    const uint64_t m = e ? ((v & xf::M52) | xf::H52) : 0ull;
    const int64_t u = (int64_t)shr64(m, top - e + 2);
    return (v >> 63) ? -u : u;
}

XF_HD uint64_t row_from_units(int64_t u, int top)
{
    if (u == 0) return 0;
    const uint64_t m = u < 0 ? 0ull - (uint64_t)u : (uint64_t)u;
#if defined(__CUDA_ARCH__)
    const int z = __clzll((long long)m);
#else
    const int z = __builtin_clzll(m);
#endif
    const int e = top + 13 - z;  // the leading one at bit 63 - z, of units 2^(top - 1073)
    if (e < 1 || e > 2046) return 0;
    return (u < 0 ? 1ull << 63 : 0ull) | (uint64_t)e << 52 | ((m << z) >> 11 & xf::M52);
}

// the double d ulps above x in value (|d| small, x not near its binade's ends)
XF_HD uint64_t row_shift(uint64_t u, int d) { return (u >> 63) ? u - (uint64_t)(int64_t)d : u + (uint64_t)(int64_t)d; }

// x - y in ulps for x, y of one sign and binade with a difference below `limit`; false otherwise
XF_HD bool row_diff(uint64_t x, uint64_t y, int* d, int64_t limit = MAX_OFF)
{
    *d = 0;
    if (x == y) return true;
    if ((x >> 52) != (y >> 52) || ((x >> 52) & 0x7ff) == 0 || ((x >> 52) & 0x7ff) == 2047) return false;
    const int64_t v = (x >> 63) ? (int64_t)(y - x) : (int64_t)(x - y);
    if (v >= limit || v <= -limit) return false;
    *d = (int)v;
    return true;
}

}  // namespace rs

#if defined(__CUDACC__)

constexpr int ROW_SEG_MAX = 36;  // terms per lane and call
constexpr int ROW_CTA_WARPS = 16;  // most warps of cta_row_sum

// the plain chain: acc + T_0 + ... + T_{m-1}, by every lane alike
__device__ __forceinline__ double row_chain(double acc, const double* T, int seg, int pitch, int m)
{
    for (int l = 0; l * seg < m; l++) {
        const double* const t = T + l * pitch;
        const int n = min(seg, m - l * seg);
#pragma unroll 4
        for (int k = 0; k < n; k++) acc = __dadd_rn(acc, t[k]);
    }
    return acc;
}
// Whether it is shorter than adding `lanes` segments again: each costs its additions and some ten more.
// (Sums through zero at every other term, as of bodies in antipodal pairs: an RKF7(8) attempt of 1003 such
// bodies 1770 us with every lane added again, 700 so.)
__device__ __forceinline__ bool row_chain_pays(int lanes, int seg, int m) { return lanes * (seg + 10) > m; }

// acc + T_0 + ... + T_{m-1}, rounded after every addition in that order, m <= 32 seg,
// seg <= ROW_SEG_MAX: term e is at T[e / seg * pitch + e % seg].  Every lane of the warp calls
// this with the same arguments and returns the sum.  codes: 32 ROW_SEG_MAX entries of shared
// memory of this warp's own.  (GB300's FP64 pipe takes a warp's addition every 64 cycles per SM
// sub-partition, so each lane adds its terms once; the guesses are sums of integers.)
__device__ __forceinline__ double warp_row_sum(double acc, const double* T, int seg, int pitch, int m,
                                               uint32_t* codes)
{
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int n = max(0, min(seg, m - lane * seg));
    const double* t = T + lane * pitch;
    // the guesses: acc + the sums of the segments before, in units of 2^-51 of the largest value
    int top = (int)((uint32_t)(xf::dbits(acc) >> 52) & 0x7ffu);
    for (int k = 0; k < n; k++) top = max(top, (int)((uint32_t)(xf::dbits(t[k]) >> 52) & 0x7ffu));
    top = __reduce_max_sync(ALL, top);
    int64_t u = lane == 0 ? rs::row_units(xf::dbits(acc), top) : 0;
    for (int k = 0; k < n; k++) u += rs::row_units(xf::dbits(t[k]), top);
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const long long o = __shfl_up_sync(ALL, (long long)u, off);
        if (lane >= off) u += o;
    }
    const uint64_t g = rs::row_from_units(__shfl_up_sync(ALL, (long long)u, 1), top);
    double a = lane == 0 ? acc : __longlong_as_double((long long)g);
    // the lanes' chains, with the codes of the additions that change an offset; an addition is in
    // flight while the one before it is classified
    const uint64_t guess = xf::dbits(a);
    bool hard = rs::near_edge(guess);
    int nc = 0;
    uint32_t* const code = codes + lane * ROW_SEG_MAX;
    if (n > 0) {
        double tk = t[0], s = __dadd_rn(a, tk);
        for (int k = 0; k < n; k++) {
            const double tn = k + 1 < n ? t[k + 1] : 0.0;
            const double sn = __dadd_rn(s, tn);
            const uint32_t rec = rs::row_mark(xf::dbits(a), xf::dbits(tk), xf::dbits(s), k, &hard);
            if (rec) code[nc++] = rec;
            a = s;
            tk = tn;
            s = sn;
        }
    }
#pragma unroll 2
    for (int q = 0; q < nc; q++) code[q] = rs::row_code(code[q], xf::dbits(t[code[q] >> 13 & 63u]));
    __syncwarp();  // (the codes are read by other lanes)
    const uint64_t end = xf::dbits(a);
    const uint64_t before = __shfl_up_sync(ALL, (unsigned long long)end, 1);
    int d = 0;  // how far the end of the lane before is above the lane's guess; then the prefix of these
    bool loose = !rs::row_diff(before, guess, &d);
    if (lane == 0) {
        loose = false;
        d = 0;
    }
    // (a lane whose offset is 0 needs no rule: its chain is the true one)
    if (!__any_sync(ALL, loose || d != 0)) return __longlong_as_double((long long)__shfl_sync(ALL, (unsigned long long)end, 31));
    int P = d;  // the lanes' offsets if none had codes
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_up_sync(ALL, P, off);
        if (lane >= off) P += o;
    }
    constexpr int LIM = (int)(rs::MAX_OFF / 2);
    const bool slow = hard || loose || P >= LIM || P <= -LIM;
    unsigned todo = __ballot_sync(ALL, lane > 0 && (nc > 0 || slow));
    unsigned slows = __ballot_sync(ALL, slow);
    if (row_chain_pays(__popc(slows & ~1u), seg, m)) return row_chain(acc, T, seg, pitch, m);
    uint64_t tend = end;  // of a lane that has been through the loop below: its true end
    bool done = lane == 0;
    int off = 0;  // offset of a lane = P + off, for the lanes after the last one done
    if ((slows & ~1u) == 0) {
        // no slow lane (as a rule): every lane of the warp runs through the codes, with the next
        // lane's count and prefix and the next code on their way while one is applied.  A sum that
        // hovers (a coplanar system's z) has codes in most lanes: 168 of them took 28 k cycles by
        // the lanes' own passes, below, and take 13.8 k here.
        unsigned rest = todo;
        int most = 0;
        int L = __ffs(rest) - 1;
        int cnt = __shfl_sync(ALL, nc, L & 31), p = __shfl_sync(ALL, P, L & 31);
        uint32_t e = codes[(L & 31) * ROW_SEG_MAX];
        while (rest) {
            rest &= rest - 1;
            const int Ln = __ffs(rest) - 1;
            const int cntn = __shfl_sync(ALL, nc, Ln & 31), pn = __shfl_sync(ALL, P, Ln & 31);
            const uint32_t first = codes[(Ln & 31) * ROW_SEG_MAX];
            const uint32_t* const cl = codes + (L & 31) * ROW_SEG_MAX;
            int dl = p + off;
#pragma unroll 1
            for (int q = 1; q <= cnt; q++) {
                const uint32_t en = cl[min(q, ROW_SEG_MAX - 1)];
                dl = rs::row_apply(e, dl);
                most |= dl ^ (dl >> 31);
                e = en;
            }
            off = dl - p;
            most |= off ^ (off >> 31);
            L = Ln;
            cnt = cntn;
            p = pn;
            e = first;
        }
        if (most < LIM) {
            const uint64_t last = rs::row_shift(end, P + off);
            return __longlong_as_double((long long)__shfl_sync(ALL, (unsigned long long)last, 31));
        }
        off = 0;
    }
    while (todo) {
        const int L = __ffs(todo) - 1;
        todo &= todo - 1;
        const bool is_slow = slows >> L & 1;
        // a slow lane: its true start, the true end of the lane before it
        uint64_t start = 0;
        if (is_slow) {
            const uint64_t mine = done ? tend : rs::row_shift(end, P + off);
            start = __shfl_sync(ALL, (unsigned long long)mine, L - 1);
        }
        int next = 0;
        if (lane == L) {
            int dl = P + off;
            bool serial = false, force = false;
            if (is_slow) serial = !rs::row_diff(start, guess, &dl) || (hard && dl != 0);
            if (!serial && dl != 0 && nc > 0) {
                uint32_t next_code = code[0];
                int most = 0;
                for (int q = 0; q < nc; q++) {
                    const uint32_t e = next_code;
                    next_code = code[q + 1 < nc ? q + 1 : q];
                    dl = rs::row_apply(e, dl);
                    most |= dl ^ (dl >> 31);
                    if (most >= (int)rs::MAX_OFF) break;
                }
                serial = most >= (int)rs::MAX_OFF;
            }
            if (serial) {
                if (!is_slow) start = rs::row_shift(guess, P + off);
                double b = __longlong_as_double((long long)start);
                for (int q = 0; q < n; q++) b = __dadd_rn(b, t[q]);
                tend = xf::dbits(b);
                force = !rs::row_diff(tend, end, &dl);
            } else {
                tend = rs::row_shift(end, dl);
            }
            done = true;
            next = dl - P;
            // offsets after it the codes are not used with: the next lane is a slow one
            if (force || next >= LIM || next <= -LIM) next = INT_MIN;
        }
        off = __shfl_sync(ALL, next, L);
        if (off == INT_MIN) {
            if (L < 31) {
                todo |= 1u << (L + 1);
                slows |= 1u << (L + 1);
            }
            off = 0;
        }
    }
    const uint64_t mine = done ? tend : rs::row_shift(end, P + off);
    return __longlong_as_double((long long)__shfl_sync(ALL, (unsigned long long)mine, 31));
}

// The same sum by a group of W warps (a CTA, or warps with a named barrier of their own), each lane one
// of 32 W segments: the lanes' passes get as many times shorter, the codes are still applied in
// order, by the first warp, one after the other from one list.  A slow lane is added again from its
// true start when its turn comes; a row with too many of them or of codes, or with offsets out of
// range, is summed by the first warp alone.
// Measured: a hovering row of 1027 terms (some 250 codes) 15.5 k cycles of eight warps,
// warp_row_sum 28 k.
constexpr int ROW_HARD = 8;  // most lanes of a row that are added again
struct RowGroup {
    int id, threads, me;  // named barrier, its threads, this one of them
    __device__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
    __device__ bool any(bool p) const
    {
        int r;
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.or.pred q, %2, %3, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                     : "=r"(r)
                     : "r"((int)p), "r"(id), "r"(threads)
                     : "memory");
        return r != 0;
    }
};
template <int RULES, int WARPS>  // RULES: most codes of a row that are applied
struct GroupRowSmem {
    rs::RowRule rule[RULES];
    struct {
        int lane, rule, in;  // the lane, its place among the rules, the offset's change since the lane with codes before
        unsigned long long before, end;
    } hard[ROW_HARD];
    int P[32 * WARPS];  // of the lanes with codes
    int top[WARPS];
    long long units[WARPS];
    unsigned long long end[WARPS], last;
    int diff[WARPS], count[WARPS], coded[WARPS];
    int last_in;
    double sum;
};

// acc + T_0 + ... + T_{m-1}: term e is at T[e / seg * pitch + e % seg], seg <= ROW_SEG_MAX, m <= 32 W
// seg; every thread of the group calls this and gets the sum.  codes: max(m, 32 ROW_SEG_MAX)
// entries of shared memory at least.
template <int RULES, int WARPS>
__device__ __forceinline__ double group_row_sum(const RowGroup& grp, double acc, const double* T, int seg, int pitch,
                                                int m, uint32_t* codes, GroupRowSmem<RULES, WARPS>& S)
{
    constexpr unsigned ALL = 0xffffffffu;
    const int me = grp.me, W = grp.threads >> 5, warp = me >> 5, lane = me & 31;
    const int n = max(0, min(seg, m - me * seg));
    const double* const t = T + me * pitch;
    int top = (int)((uint32_t)(xf::dbits(acc) >> 52) & 0x7ffu);
    for (int k = 0; k < n; k++) top = max(top, (int)((uint32_t)(xf::dbits(t[k]) >> 52) & 0x7ffu));
    top = __reduce_max_sync(ALL, top);
    if (lane == 0) S.top[warp] = top;
    grp.sync();
    for (int w = 0; w < W; w++) top = max(top, S.top[w]);
    long long u = me == 0 ? rs::row_units(xf::dbits(acc), top) : 0;
    for (int k = 0; k < n; k++) u += rs::row_units(xf::dbits(t[k]), top);
    const long long own = u;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const long long o = __shfl_up_sync(ALL, u, off);
        if (lane >= off) u += o;
    }
    if (lane == 31) S.units[warp] = u;
    grp.sync();
    long long base = u - own;
    for (int w = 0; w < warp; w++) base += S.units[w];
    double a = me == 0 ? acc : __longlong_as_double((long long)rs::row_from_units(base, top));
    const uint64_t guess = xf::dbits(a);
    bool hard = rs::near_edge(guess);
    int nc = 0;
    uint32_t* const code = codes + me * seg;
    for (int k = 0; k < n; k++) {
        const double tk = t[k], s = __dadd_rn(a, tk);
        const uint32_t rec = rs::row_mark(xf::dbits(a), xf::dbits(tk), xf::dbits(s), k, &hard);
        if (rec) code[nc++] = rec;
        a = s;
    }
    for (int q = 0; q < nc; q++) code[q] = rs::row_code(code[q], xf::dbits(t[code[q] >> 13 & 63u]));
    const uint64_t end = xf::dbits(a);
    if (lane == 31) S.end[warp] = end;
    if (me == grp.threads - 1) S.last = end;
    grp.sync();
    uint64_t before = __shfl_up_sync(ALL, (unsigned long long)end, 1);
    if (lane == 0 && warp > 0) before = S.end[warp - 1];
    int d = 0;
    bool loose = !rs::row_diff(before, guess, &d, 1 << 20);
    if (me == 0) {
        loose = false;
        d = 0;
    }
    if (!grp.any(loose || d != 0)) return __longlong_as_double((long long)S.last);
    // the lanes' offsets if none had codes, and where a lane's codes stand among all (the first
    // lane's change nothing: its offset is 0)
    const bool again = me > 0 && (hard || loose), has = me > 0 && (again || nc > 0);
    const int mine = again ? 1 : (me > 0 ? nc : 0);
    int P = d, at = mine | (again ? 1 << 20 : 0), order = has;  // at: above bit 20 the slow lanes
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_up_sync(ALL, P, off), oc = __shfl_up_sync(ALL, at, off), oo = __shfl_up_sync(ALL, order, off);
        if (lane >= off) {
            P += o;
            at += oc;
            order += oo;
        }
    }
    if (lane == 31) {
        S.diff[warp] = P;
        S.count[warp] = at;
        S.coded[warp] = order;
    }
    grp.sync();
    int total = 0;
    for (int w = 0; w < W; w++) {
        if (w < warp) {
            P += S.diff[w];
            at += S.count[w];
            order += S.coded[w];
        }
        total += S.count[w];
    }
    const int n_hard = total >> 20, n_rule = total & 0xfffff;
    if (has) S.P[order - 1] = P;
    bool slow = grp.any(n_rule > RULES || n_hard > ROW_HARD);
    const int since = P - (order - (int)has > 0 ? S.P[order - (int)has - 1] : 0);
    if (me == grp.threads - 1) S.last_in = has ? 0 : since;
    bool fit = true;
    if (!slow && has) {
        const int first = (at & 0xfffff) - mine;
        if (again) {
            auto& h = S.hard[(at >> 20) - 1];
            h.lane = me;
            h.rule = first;
            h.in = since - d;
            h.before = before;
            h.end = end;
        } else {
            for (int q = 0; q < nc; q++) fit = rs::row_rule(code[q], q == 0 ? since : 0, &S.rule[first + q]) && fit;
        }
    }
    constexpr int LIM = 1 << 29;
    slow = grp.any(slow || !fit);
    if (warp == 0) {
        int off = 0, most = slow ? LIM : 0;
        uint64_t tend = 0;  // the true end of the last lane added again
        int q = 0;
        for (int k = 0; k <= n_hard && !slow; k++) {
            const int to = k < n_hard ? S.hard[k].rule : n_rule;
#pragma unroll 4
            for (; q < to; q++) off = rs::row_follow(S.rule[q], off, &most);
            if (k == n_hard || most >= LIM) break;
            const auto& h = S.hard[k];
            const bool follows = k > 0 && S.hard[k - 1].lane == h.lane - 1;
            double b = __longlong_as_double((long long)(follows ? tend : rs::row_shift(h.before, off + h.in)));
            for (int e = 0; e < min(seg, m - h.lane * seg); e++) b = __dadd_rn(b, T[h.lane * pitch + e]);
            tend = xf::dbits(b);
            if (!rs::row_diff(tend, h.end, &off, LIM)) most = LIM;
            q = to + 1;
        }
        double sum = acc;
        if (most < LIM)
            sum = __longlong_as_double((long long)rs::row_shift(S.last, off + S.last_in));
        else if (row_chain_pays(n_hard, seg, m))
            sum = row_chain(sum, T, seg, pitch, m);
        else  // (the codes' space is free: they are not used)
            for (int w = 0; w < W && w * 32 * seg < m; w++)
                sum = warp_row_sum(sum, T + w * 32 * pitch, seg, pitch, min(m - w * 32 * seg, 32 * seg), codes);
        if (lane == 0) S.sum = sum;
    }
    grp.sync();
    return S.sum;
}

// by a whole CTA of at most ROW_CTA_WARPS warps, from zero, the terms one after the other
using CtaRowSmem = GroupRowSmem<1024, ROW_CTA_WARPS>;
__device__ __forceinline__ double cta_row_sum(const double* T, int m, uint32_t* codes, CtaRowSmem& S)
{
    const int seg = (m + (int)blockDim.x - 1) / (int)blockDim.x;
    return group_row_sum(RowGroup{0, (int)blockDim.x, (int)threadIdx.x}, 0.0, T, seg, seg, m, codes, S);
}
#endif

}  // namespace redgb
