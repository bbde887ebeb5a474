// gravity_cert.cu -- FP64 direct-summation gravity, bit-identical to the reference's serial
// sums, with most pair terms never computed in FP64.
//
// The reference adds a sink's terms t_j one after the other: acc = RN(acc + t_j)
// (pp_disk.cu:404-572).  While acc stays in one binade its values are the multiples of the
// quantum Q = ulp(acc), and then RN(acc + t_j) = acc + Q r_j with r_j = t_j / Q rounded to the
// nearest integer: all the sum ever sees of a term is that integer.  The star's pull comes
// first and dominates, so a typical term is 2^25 quanta, and its integer is known from an
// approximation good to 2^-40 -- which double-float arithmetic gives on the FP32 pipes, 64 times
// as wide as GB300's FP64 pipe -- unless t_j / Q lies within the approximation's error of a
// half-integer.  So for each pair the kernel forms t_j / Q in double-float with a bound E on its
// error (below), takes the nearest integer and checks that its distance from t_j / Q plus E is
// below one half; a pair that fails (1 to 2 % of them, or one too large for the integer form)
// is computed by the reference's own FP64 operations (pair_term) and rounded exactly.  Integers
// are added in any order with the same result, so the sources are shared out over a warp's
// lanes and the sum stays the serial sum, as long as no running sum left the binade: an epoch
// of sources is accepted when |acc| is further from both ends of its binade than the sum of
// its integers' magnitudes, and otherwise redone slice by slice, with exact terms added in order
// (warp_serial_sum) where the sum does leave.  Sums that are small beside their terms (the z
// component of a sink close to the disk's plane) are left to the row kernel (gravity_fp64.cu).
//
// Measured (one evaluation of 16 385 self-gravitating bodies, 2.07 GHz): 2.45 ms, 2.0 of them
// here, 0.4 in the row kernel; the FP64 form it replaces took 9.0 ms with the FP64 pipe 76 % busy
// (18 FP64 operations per pair at 16 cycles per warp and SM).  Bound: the FP32 pipe.  A packed instruction (f32x2.cuh) takes
// 2 cycles, 3 when its three operands are all new; 127 of them serve two pairs, beside 60
// instructions on the other pipes.  The warps are independent (a CTA-wide form with a barrier
// per source tile took 3.4 to 7 ms), four per scheduler; five or six with fewer registers
// measured the same.
//
// Error bound.  Coordinates are x = hi + lo + err with hi a multiple of a system-wide grid g (so
// hi differences are exact) and lo in FP32; alpha = g 2^-24.  |lo| reaches 0.75 g (a coordinate
// half-way between two grid points, and the split's own remainder): its rounding is 0.625 alpha at
// most, the difference of two, up to 1.5 g, rounds by one alpha.  Not all three at once: a rounding
// of 0.5 alpha or more is a tie, which leaves lo an even multiple of alpha, and the difference of two
// such ones is exact; so a displacement is good to (0.625 + 0.5 + 1) alpha (DISP_ERR; reached).
// r^2 is summed with two-sums and the products' FMA errors, 1/r from rsqrt.approx (2^-22.9)
// with its residual h = 1 - r^2 y0^2 formed by FMAs (3 2^-46), y^3 = y0^3 (1 + 1.5 h + 1.875 h^2);
// every product keeps its FMA error term.  Relative error of w = m y^3: in units of 2^-44, 1.1
// (h) + 0.6 (corr) + 1.0 (the error terms' and the term's last roundings) + 0.5 (their product
// with the displacement's low part) + 0.5 (r^2's error terms) + 0.8 (the fast two-sum of the
// remainder where its operands are in the other order) < 4.8, taken as 1.2 2^-42 with the
// reference's own FP64 roundings (2^-49); plus 3 sqrt(3) 2.125 alpha / r = 11.05 alpha / r, taken as
// 11.2.  A component's error is then at most w (|dx| (1.2 2^-42 + 11.2 alpha / r) + 3 alpha_c); |dx| is
// bounded by dx^2 / (2 eta) + eta / 2, which needs no absolute value in the packed form.
#include <atomic>
#include <string>

#include "../../include/redgb.h"
#include "common.cuh"
#include "dfloat.cuh"
#include "exact_fp64.h"
#include "f32x2.cuh"
#include "kernels.h"
#include "pair_fp64.cuh"

namespace redgb {

int set_error(int code, const std::string& msg);

namespace {

constexpr int HEAD = 16;              // leading sources (star, planets) taken exactly; a multiple of 4
constexpr float MAGIC = 12582912.0f;  // 1.5 2^23: adding it rounds to an integer, |v| <= 2^22
constexpr unsigned MAGIC_BITS = 0x4B400000u;
constexpr float RADIX = 65536.0f;     // a term is H 2^16 + L quanta
constexpr int RADIX_BITS = 16;
constexpr float BIG = 4.1e6f;         // |t / Q| / 2^16 below this (MAGIC's range is 4.19e6)
// accepted when f^2 + E < 1/4 - 2^-13: then |f| + E + 2^-13 < 1/2 (the rounding of f itself: 2^-23)
constexpr float CERTAIN = 0.24987f;
constexpr int64_t UNCERTAIN = 1ll << 36;  // terms this large are rarely certain (E > 2^-5)
constexpr float DISP_ERR = 2.125f;    // of a displacement's component, in alpha
constexpr float DISP_W = 11.2f;       // of w, in alpha / r
static_assert(DISP_W > 1.01f * 5.19616f * DISP_ERR, "3 sqrt(3) times a component's");
constexpr float MIN_R2 = 8.3e-25f;    // 2^-80: closer pairs (and the sink itself) are taken exactly
constexpr float MIN_MASS = 5.3e-23f;  // 2^-74: lighter masses have no exact split
constexpr float FAR = 1.0e15f;        // beyond the splits' range
constexpr int CERT_WARPS = 1;         // independent warps per CTA (2: 1.9 % slower at 16 385 and 131 074 bodies)

// per warp: SW sinks, 32 / SW lanes on each.  Four where the sinks fill the chip with warps (2, 4 and
// 8 sinks per warp: 3.0, 2.5 and 2.8 ms per evaluation of 16 385 bodies when this was first
// measured, 2.47 against 2.38 ms now; 916 against 871 us for 9001), two below ten such warps an SM,
// where twice the warps hide more latency (2001 / 2999 / 4501 bodies: 153 / 212 / 343 us, with four
// 180 / 236 / 369 us; 6001 bodies: the same).
constexpr int CERT_FULL = 10;  // warps an SM

template <int SW>
struct alignas(16) CertSmem {  // rows are read and copied to 16 bytes at a time
    static constexpr int NQ = 32 / SW;       // slices
    static constexpr int SLICE = 32;         // sources of a lane per epoch: one flag bit each
    static constexpr int PART = 8;           // of them staged at a time (cp.async), two parts in flight
    static constexpr int PITCH = PART + 4;   // slices 4 floats apart: lanes on different slices read different banks
    float src[2][8][NQ * PITCH];             // xh xl yh yl zh zl mh ml
    union {
        double term[3][32];      // exact terms of a round
        struct {
            long long r[32][3];  // a round of flagged pairs: quanta
            int bad[32];         // bits: components that have none
        } f;
    };
    double sink[6][SW];                      // x, y, z, R, m, rho
    double acc[3][SW];
    long long part[NQ][3][SW];               // a lane's sum of quanta
    float bnd[NQ][3][SW];                    // and of their magnitudes (infinite: it has no quanta)
    float sig[3][SW];                        // 2^-16 / Q; 0 for acc = 0 and for a sum left to the row kernel
    unsigned short fitem[32];
};

__device__ __forceinline__ float pow2f(int e)  // e in [-126, 127]
{
    return __uint_as_float((unsigned)(e + 127) << 23);
}

__device__ __forceinline__ int expo(float v) { return (int)((__float_as_uint(v) >> 23) & 0xffu) - 127; }

// 2^-16 / Q of a running sum: 0 for zero, NaN outside [2^-40, 2^120] and for one that is not finite
__device__ __forceinline__ float sigma_of(double acc)
{
    const int ea = (int)((xf::dbits(acc) >> 52) & 0x7ff);
    if (acc == 0.0) return 0.0f;
    if (ea < 983 || ea > 1143) return __uint_as_float(0x7fc00000u);
    return pow2f(1075 - RADIX_BITS - ea);
}

// a coordinate |h| <= c = 2^23 g on the tile's grid: hi a multiple of g, lo the rest (|h| + c lies
// in [c, 2 c], where FP32's spacing is g)
__device__ __forceinline__ void regrid(float h, float l, float c, float& hi, float& lo)
{
    c = copysignf(c, h);
    hi = __fadd_rn(__fadd_rn(h, c), -c);
    lo = __fadd_rn(__fadd_rn(h, -hi), l);
}

// constants of the pair loop, each twice (packed)
struct CertConst {
    f2 neg, one, two, c15, c1875, M, R;  // -1, 1, 2, 1.5, 1.875, MAGIC, RADIX
    f2 Yk, Ya;                           // 2^16 1.2 2^-42, 2^16 11.2 alpha (the larger one)
    f2 i2_xy, h_xy, a_xy;                // 1 / (2 eta), eta / 2, 2^16 3 alpha
    f2 i2_z, h_z, a_z;
};

// a packed constant that stays in registers (rebuilt from immediates it costs two moves per use)
__device__ __forceinline__ f2 pinned(float v)
{
    f2 r = f2_dup(v);
    asm volatile("" : "+l"(r));
    return r;
}

__device__ __forceinline__ f2 two_sum2(f2 a, f2 b, f2& e)
{
    const f2 s = f2_add(a, b);
    const f2 bb = f2_sub(s, a);
    e = f2_add(f2_sub(a, f2_sub(s, bb)), f2_sub(b, bb));
    return s;
}

__device__ __forceinline__ float rsqrt_seed(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// acc + total quanta when no running sum of them can have left acc's binade; bound: the sum of
// their magnitudes
__device__ __forceinline__ bool accept(double& acc, long long total, float bound)
{
    const int ea = (int)((xf::dbits(acc) >> 52) & 0x7ff);
    if (ea == 0 || ea == 2047) return false;
    const int64_t A = xf::quanta_of(acc);
    const int64_t mag = A < 0 ? -A : A;
    const int64_t room = min(mag - (int64_t)xf::H52, 2 * (int64_t)xf::H52 - mag);
    if (!(bound * 1.01f < __ll2float_rd(room))) return false;
    acc = xf::from_quanta(A + total, ea);
    return true;
}

struct CertSink {
    f2 xh, xl, yh, yl, zh, zl;
    f2 sx, sy, sz;
};

struct CertSum {
    unsigned hx, hy, hz, lx, ly, lz;
    float big;  // sum over the pairs of the largest component's |t / Q| 2^-16
};

// one component: integers of t / Q (high part, low part, both with MAGIC's bits), |t / Q| 2^-16
// and f^2 + E
__device__ __forceinline__ void cert_comp(const CertConst& k, f2 w, f2 ew, f2 sig, f2 d, f2 nd, f2 l, f2 px, f2 Y, f2 i2,
                                          f2 hh, f2 al, f2& hb, f2& lb, f2& th, f2& chk)
{
    const f2 W = f2_mul(w, sig), V = f2_mul(ew, sig);
    th = f2_mul(W, d);
    const f2 nth = f2_mul(W, nd);
    f2 te = f2_fma(W, d, nth);
    te = f2_fma(W, l, te);
    const f2 tl = f2_fma(V, d, te);
    hb = f2_add(th, k.M);
    const f2 hr = f2_sub(th, f2_sub(hb, k.M));
    const f2 r = f2_add(hr, tl), re = f2_add(f2_sub(hr, r), tl);  // r + re = hr + tl
    lb = f2_fma(r, k.R, k.M);
    const f2 f = f2_fma(re, k.R, f2_fma(r, k.R, f2_sub(k.M, lb)));
    const f2 D = f2_fma(px, i2, hh);
    const f2 G = f2_fma(D, Y, al);
    chk = f2_fma(f, f, f2_mul(W, G));
}

// one of the two pairs: its integers added when it is certain, else its flag bit set (compares
// that a NaN fails)
__device__ __forceinline__ void cert_take(float cx, float cy, float cz, float tx, float ty, float tz, float r2, float cut,
                                          unsigned hx, unsigned hy, unsigned hz, unsigned lx, unsigned ly, unsigned lz,
                                          unsigned bit, CertSum& s, unsigned& flags)
{
    const float big = fmaxf(fmaxf(fabsf(tx), fabsf(ty)), fabsf(tz));
    asm("{\n\t.reg .pred p;\n\t"
        "setp.lt.f32 p, %8, %15;\n\t"
        "setp.lt.and.f32 p, %9, %15, p;\n\t"
        "setp.lt.and.f32 p, %10, %15, p;\n\t"
        "setp.lt.and.f32 p, %11, %16, p;\n\t"
        "setp.ge.and.f32 p, %12, %13, p;\n\t"
        "@p add.u32 %0, %0, %17;\n\t"
        "@p add.u32 %1, %1, %18;\n\t"
        "@p add.u32 %2, %2, %19;\n\t"
        "@p add.u32 %3, %3, %20;\n\t"
        "@p add.u32 %4, %4, %21;\n\t"
        "@p add.u32 %5, %5, %22;\n\t"
        "@p add.f32 %6, %6, %11;\n\t"
        "@!p or.b32 %7, %7, %14;\n\t}"
        : "+r"(s.hx), "+r"(s.hy), "+r"(s.hz), "+r"(s.lx), "+r"(s.ly), "+r"(s.lz), "+f"(s.big), "+r"(flags)
        : "f"(cx), "f"(cy), "f"(cz), "f"(big), "f"(r2), "f"(cut), "r"(bit), "f"(CERTAIN), "f"(BIG), "r"(hx), "r"(hy),
          "r"(hz), "r"(lx), "r"(ly), "r"(lz));
}

// (ah + al) - (bh + bl) on one grid: the hi difference is exact
__device__ __forceinline__ void cert_diff(f2 ah, f2 al, f2 bh, f2 bl, f2& d, f2& l)
{
    const f2 h = f2_sub(ah, bh), r = f2_sub(al, bl);
    d = f2_add(h, r);
    l = f2_add(f2_sub(h, d), r);
}

// two sources against one sink; bit0: the flag bit of the first
__device__ __forceinline__ void cert_pair2(const CertSink& k, const CertConst& q, f2 xh, f2 xl, f2 yh, f2 yl, f2 zh,
                                           f2 zl, f2 mh, f2 ml, float cut, unsigned bit0, CertSum& s, unsigned& flags)
{
    // displacements dx + lx, |lx| <= 2^-24 |dx|
    f2 dx, dy, dz, lx, ly, lz;
    cert_diff(xh, xl, k.xh, k.xl, dx, lx);
    cert_diff(yh, yl, k.yh, k.yl, dy, ly);
    cert_diff(zh, zl, k.zh, k.zl, dz, lz);
    const f2 ndx = f2_mul(dx, q.neg), ndy = f2_mul(dy, q.neg), ndz = f2_mul(dz, q.neg);
    // r^2 = s0 + sl
    const f2 px = f2_mul(dx, dx), py = f2_mul(dy, dy), pz = f2_mul(dz, dz);
    const f2 ne = f2_add(f2_add(f2_fma(ndx, dx, px), f2_fma(ndy, dy, py)), f2_fma(ndz, dz, pz));
    f2 e1, e2;
    const f2 s2 = two_sum2(two_sum2(px, py, e1), pz, e2);
    const f2 c = f2_fma(dx, lx, f2_fma(dy, ly, f2_mul(dz, lz)));
    f2 sl = f2_fma(c, q.two, f2_sub(f2_add(e1, e2), ne));
    const f2 s0 = f2_add(s2, sl);
    sl = f2_add(f2_sub(s2, s0), sl);
    float ra, rb;
    f2_unpack(s0, ra, rb);
    const f2 y0 = f2_pack(rsqrt_seed(ra), rsqrt_seed(rb));
    const f2 n0 = f2_mul(y0, q.neg);
    const f2 b = f2_mul(y0, y0), nb = f2_mul(y0, n0);
    const f2 neb = f2_fma(y0, n0, b);
    f2 h = f2_fma(s0, nb, q.one);
    h = f2_fma(s0, neb, h);
    h = f2_fma(sl, nb, h);
    const f2 corr = f2_mul(h, f2_fma(h, q.c1875, q.c15));
    const f2 c3 = f2_mul(b, y0), nc3 = f2_mul(b, n0);
    const f2 ec = f2_fma(neb, n0, f2_fma(b, y0, nc3));
    const f2 w = f2_mul(c3, mh);
    f2 ew = f2_fma(c3, mh, f2_mul(nc3, mh));
    ew = f2_fma(ec, mh, ew);
    ew = f2_fma(c3, ml, ew);
    ew = f2_fma(w, corr, ew);
    const f2 Y = f2_fma(y0, q.Ya, q.Yk);
    f2 hbx, hby, hbz, lbx, lby, lbz, tx, ty, tz, gx, gy, gz;
    cert_comp(q, w, ew, k.sx, dx, ndx, lx, px, Y, q.i2_xy, q.h_xy, q.a_xy, hbx, lbx, tx, gx);
    cert_comp(q, w, ew, k.sy, dy, ndy, ly, py, Y, q.i2_xy, q.h_xy, q.a_xy, hby, lby, ty, gy);
    cert_comp(q, w, ew, k.sz, dz, ndz, lz, pz, Y, q.i2_z, q.h_z, q.a_z, hbz, lbz, tz, gz);
    float x0, x1, y0f, y1f, z0, z1, u0, u1, v0, v1, w0, w1;
    f2_unpack(gx, x0, x1);
    f2_unpack(gy, y0f, y1f);
    f2_unpack(gz, z0, z1);
    f2_unpack(tx, u0, u1);
    f2_unpack(ty, v0, v1);
    f2_unpack(tz, w0, w1);
    cert_take(x0, y0f, z0, u0, v0, w0, ra, cut, (unsigned)hbx, (unsigned)hby, (unsigned)hbz, (unsigned)lbx, (unsigned)lby,
              (unsigned)lbz, bit0, s, flags);
    cert_take(x1, y1f, z1, u1, v1, w1, rb, cut, (unsigned)(hbx >> 32), (unsigned)(hby >> 32), (unsigned)(hbz >> 32),
              (unsigned)(lbx >> 32), (unsigned)(lby >> 32), (unsigned)(lbz >> 32), bit0 << 1, s, flags);
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

}  // namespace

// The rows of one evaluation: every body's coordinates on its system's grid and its mass, as 8
// FP32 rows (hi, lo), and the system's scale.  Body j of the system with first body `base` is
// at cert_row(base, sys) + j - base, so every system starts on a 16-byte boundary.
__host__ __device__ __forceinline__ long long cert_row(int base, int sys) { return ((base + 3) & ~3) + 4LL * sys; }

struct CertPrepArgs {
    const double *x, *y, *z, *mass, *radius, *rho;  // rho: Hill screens only
    const int* id;
    const int* sys_base;    // first body of each system, or nullptr: one system of n bodies
    const int* sys_n;       // and its bodies
    const int* sys_active;
    int n_sys;
    int n;
    int blocks;             // CTAs per system
    int screen;
    float* rows;
    long long stride;
    unsigned int* n_list;   // counts of rows left to grav_fp64_rows: none yet
    float* scale;           // 8 per system: max |x|, |y|; max |z|; the screens' maxima of R, m, rho;
                            // bits: components in which every displacement is zero
};

constexpr int PREP_NT = 1024;

// |v| from the high word (no FP64-pipe conversion), at most 2e-6 above it; 0 below FP32's normal
// range, 2e38 above it and for infinities and NaNs
__device__ __forceinline__ float magnitude(const double* v, long long k)
{
    const unsigned h = reinterpret_cast<const unsigned*>(v)[2 * k + 1] & 0x7fffffffu;
    const unsigned e = h >> 20;
    if (e < 897u) return 0.0f;
    if (e > 1149u) return 2.0e38f;
    return __uint_as_float((h - (896u << 20)) << 3) * 1.000002f;
}

// One CTA per PREP_NT bodies of a system, the systems one after the other over the whole grid (an
// ensemble has more of them than a grid has rows); each CTA first takes the maxima over its system
// (a few reads per thread from L2: less than a second launch costs).  The grid must not be
// coarsened by a few bodies far out (ejected ones), so its range ends at 16 times the mean
// |coordinate|; bodies beyond it are marked (NaN) and taken exactly.
__global__ void __launch_bounds__(PREP_NT) cert_prep_kernel(CertPrepArgs a)
{
    const long long cta = blockIdx.x + (long long)gridDim.x * blockIdx.y;
    const long long sys_of = cta / a.blocks;
    if (sys_of >= a.n_sys) return;
    const int sys = (int)sys_of, block = (int)(cta - sys_of * a.blocks);
    if (cta == 0 && threadIdx.x < CERT_COUNTERS) a.n_list[threadIdx.x] = 0u;
    const int b0 = a.sys_base ? a.sys_base[sys] : 0, b1 = b0 + (a.sys_base ? a.sys_n[sys] : a.n);
    const int j = b0 + block * PREP_NT + threadIdx.x;
    if (b0 + block * PREP_NT >= b1 || (a.sys_active && !a.sys_active[sys])) return;
    __shared__ float red[PREP_NT / 32][8];
    __shared__ float all[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float cap_xy = FAR, cap_z = FAR;
    float m_xy = 0.0f, m_z = 0.0f;
    bool flat[3] = {true, true, true};  // every body has the first one's coordinate
    for (int pass = 0; pass < 4; pass++) {
        // [0..1] maxima, [2..3] sums, [4] count, [5..7] screen maxima
        float v[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        for (int k = b0 + threadIdx.x; k < b1; k += PREP_NT) {
            const float xy = fmaxf(magnitude(a.x, k), magnitude(a.y, k)), z = magnitude(a.z, k);
            if (pass == 0) {
                flat[0] = flat[0] && xf::dbits(a.x[k]) == xf::dbits(a.x[b0]);
                flat[1] = flat[1] && xf::dbits(a.y[k]) == xf::dbits(a.y[b0]);
                flat[2] = flat[2] && xf::dbits(a.z[k]) == xf::dbits(a.z[b0]);
            }
            if (xy < cap_xy && z < cap_z) {
                v[0] = fmaxf(v[0], xy);
                v[1] = fmaxf(v[1], z);
                v[2] += xy;
                v[3] += z;
                v[4] += 1.0f;
            }
            // (a merged body waits at 1e20 AU with id < 0: one of them would open the Hill screen to every
            // pair; a step of 8003 bodies 3.3 -> 14.8 ms.  The loads side by side: 31 -> 24 us at 16 385)
            if (a.screen && pass == 0 && k >= b0 + HEAD) {
                const int id = a.id[k];
                const float R = magnitude(a.radius, k), m = magnitude(a.mass, k), rho = a.rho ? magnitude(a.rho, k) : 0.0f;
                v[5] = fmaxf(v[5], 0 <= id ? R : 0.0f);
                v[6] = fmaxf(v[6], 0 <= id ? m : 0.0f);
                v[7] = fmaxf(v[7], 0 <= id ? rho : 0.0f);
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const float o = __shfl_xor_sync(0xffffffffu, v[q], off);
                v[q] = q >= 2 && q <= 4 ? v[q] + o : fmaxf(v[q], o);
            }
        if (lane == 0)
            for (int q = 0; q < 8; q++) red[warp][q] = v[q];
        __syncthreads();
        if (warp == 0) {
            for (int q = 0; q < 8; q++) v[q] = red[lane][q];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const float o = __shfl_xor_sync(0xffffffffu, v[q], off);
                    v[q] = q >= 2 && q <= 4 ? v[q] + o : fmaxf(v[q], o);
                }
            if (lane == 0)
                for (int q = 0; q < 8; q++)
                    if (pass == 0 || q < 5) all[q] = v[q];
        }
        __syncthreads();
        m_xy = all[0];
        m_z = all[1];
        const float n = fmaxf(all[4], 1.0f);
        const float c_xy = 16.0f * all[2] / n, c_z = 16.0f * all[3] / n;
        __syncthreads();
        if (m_xy <= c_xy && m_z <= c_z) break;  // uniform
        cap_xy = fminf(cap_xy, c_xy * 1.0001f);
        cap_z = fminf(cap_z, c_z * 1.0001f);
    }
    int flat_bits = 0;
    for (int q = 0; q < 3; q++) flat_bits |= __syncthreads_and(flat[q]) ? 1 << q : 0;
    if (block == 0 && threadIdx.x < 6)
        a.scale[8 * sys + threadIdx.x] = threadIdx.x < 2 ? all[threadIdx.x]
                                                         : (threadIdx.x < 5 ? all[threadIdx.x + 3] : __int_as_float(flat_bits));
    if (j >= b1) return;
    const float c_xy = pow2f(max(-50, expo(m_xy)) + 1), c_z = pow2f(max(-50, expo(m_z)) + 1);  // 2^23 g
    float h, l, r[8];
    bool in = true;
    split_bits(a.x[j], h, l);
    in = in && fabsf(h) <= c_xy;
    regrid(h, l, c_xy, r[0], r[1]);
    split_bits(a.y[j], h, l);
    in = in && fabsf(h) <= c_xy;
    regrid(h, l, c_xy, r[2], r[3]);
    split_bits(a.z[j], h, l);
    in = in && fabsf(h) <= c_z;
    regrid(h, l, c_z, r[4], r[5]);
    // an inactive or massless source adds nothing; a mass too small for its split, or not
    // finite, is taken exactly
    const double m = a.mass[j];
    const bool source = 0 <= a.id[j] && m != 0.0;
    r[6] = r[7] = 0.0f;
    if (source) split_bits(m, r[6], r[7]);
    if (source && !(r[6] >= MIN_MASS && r[6] < 1.0e30f)) in = false;
    if (!in) {  // as a sink such a body is out of the grid; as a source NaN, or no mass
        r[0] = source ? __uint_as_float(0x7fc00000u) : 4.0f * c_xy;
        r[1] = r[2] = r[3] = r[4] = r[5] = 0.0f;
    }
    float* out = a.rows + cert_row(b0, sys) + (j - b0);
#pragma unroll
    for (int q = 0; q < 8; q++) out[q * a.stride] = r[q];
}

// One warp per SW sinks of a tile; lane l has sink l % SW and the slice l / SW of every epoch of
// 32 NQ sources.  The warps are independent: the latencies of a warp's exact pairs and sums
// hide behind the others' packed arithmetic.
//
// A component whose sum is small beside its terms (a sink close to the disk's plane: its z sum)
// has few certain terms.  Once more than an eighth of an epoch's pairs are uncertain in it, or it
// has left its binade in four epochs (in one where the rows are short), the sink goes to a list of rows, the component is dropped
// here, and grav_fp64_rows adds it from exact terms.  A sink outside the grid goes there whole, with
// its event tests: its exact pairs in one warp would be the last thing running (one body at 100 AU
// in a disk of 8003 bodies with collisions on: an RKF7(8) attempt 21.7 ms, 8.9 without it).  So does
// a sink whose flagged pairs no failing component explains (sources outside the grid, wide screens) and
// are more than an eighth: an exact pair here costs eleven of the row kernel's.  And so do all, once
// three quarters of the sinks begun have rows in the list (a row costs what three or four
// sinks do here); and a sink whose sums are all left to the row kernel is done here.  An RK4 step of 8003
// bodies with collisions on, of them 10 / 30 % out to thousands of AU 22.2 / 30.3 -> 9.8 / 10.7 ms, 10 %
// above an otherwise flat disk 29.8 -> 10.2 ms (every pair on the FP64 pipe: 9.7 ms).
template <int SW, bool SCREEN>
__global__ void __launch_bounds__(32 * CERT_WARPS, 16 / CERT_WARPS)
    grav_fp64_cert(GravArgs g, CertRows cr)
{
    using Sm = CertSmem<SW>;
    static_assert(sizeof(Sm) % 16 == 0 && Sm::PITCH % 4 == 0 && HEAD % 4 == 0, "16-byte copies");
    constexpr int NQ = Sm::NQ, PITCH = Sm::PITCH, SLICE = Sm::SLICE, PART = Sm::PART, EPOCH = SLICE * NQ;
    constexpr unsigned ALL = 0xffffffffu, SINKS = (1u << SW) - 1u;
    __shared__ __align__(16) Sm smem[CERT_WARPS];
    Sm& M = smem[threadIdx.x >> 5];

    Tile tile = g.tiles[blockIdx.x];
    if (g.sys_active && !g.sys_active[tile.sys]) return;
    tile.sink_begin += SW * (blockIdx.y * CERT_WARPS + (threadIdx.x >> 5));  // this warp's sinks
    if (tile.sink_begin >= tile.sink_end) return;
    const int lane = threadIdx.x & 31;
    const int s = lane % SW, q = lane / SW;
    const int c = q;  // component owned by a lane < 3 SW
    const bool owner = lane < 3 * SW;
    const int i = tile.sink_begin + s;
    const bool active = i < tile.sink_end && 0 < g.id[i];
    const unsigned act = __ballot_sync(ALL, active);  // bit s: sink s feels forces
    if (lane < SW) {
        M.sink[0][s] = active ? g.px[i] : 0.0;
        M.sink[1][s] = active ? g.py[i] : 0.0;
        M.sink[2][s] = active ? g.pz[i] : 0.0;
        M.sink[3][s] = active ? g.radius[i] : 0.0;
        M.sink[4][s] = active ? g.mass[i] : 0.0;
        M.sink[5][s] = active && g.hill ? g.rho[i] : 0.0;
    }
    const long long stride = cr.stride;
    const float* const base = cr.rows + cert_row(tile.base, tile.sys) - tile.base;  // [j]: body j
    CertSink k;
    bool outside;  // the grid: left to the row kernel whole, event tests and all
    const bool counted = tile.src_end - tile.src_begin > 4 * EPOCH;  // rows long enough to learn from the others' fate
    if (counted && lane == 0) atomicAdd(cr.n_list + 1, (unsigned)__popc(act & SINKS));
    {
        const float* p = base + (active ? i : tile.base);
        const float lim = pow2f(max(-50, expo(cr.scale[8 * tile.sys])) + 1);
        outside = active && !(fabsf(p[0]) <= lim);
        k.xh = f2_dup(p[0]);
        k.xl = f2_dup(p[stride]);
        k.yh = f2_dup(p[2 * stride]);
        k.yl = f2_dup(p[3 * stride]);
        k.zh = f2_dup(p[4 * stride]);
        k.zl = f2_dup(p[5 * stride]);
    }
    const float* sc = cr.scale + 8 * tile.sys;
    const int flat = __float_as_int(sc[5]);
    CertConst tc;
    {
        const float m_xy = sc[0], m_z = sc[1];
        const int e_xy = max(-50, expo(m_xy)), e_z = max(-50, expo(m_z));
        const float al_xy = pow2f(e_xy - 46), al_z = pow2f(e_z - 46);  // g 2^-24, g = 2^(e - 22)
        tc.neg = pinned(-1.0f);
        tc.one = pinned(1.0f);
        tc.two = pinned(2.0f);
        tc.c15 = pinned(1.5f);
        tc.c1875 = pinned(1.875f);
        tc.M = pinned(MAGIC);
        tc.R = pinned(RADIX);
        tc.Yk = pinned(1.2f * pow2f(RADIX_BITS - 42));
        tc.Ya = pinned(DISP_W * RADIX * fmaxf(al_xy, al_z));
        tc.h_xy = pinned(0.25f * m_xy);  // eta = max / 2
        tc.i2_xy = pinned(m_xy > 0.0f ? 1.0f / m_xy : 0.0f);
        tc.h_z = pinned(0.125f * m_z);  // eta = max / 4: few bodies are near the largest height
        tc.i2_z = pinned(m_z > 0.0f ? 2.0f / m_z : 0.0f);
        tc.a_xy = pinned(3.0f * RADIX * al_xy);
        tc.a_z = pinned(3.0f * RADIX * al_z);
    }
    // r^2 below which an event test of this sink may pass (the limits grow with the sources'
    // radius, mass and distance): such pairs are taken exactly, with their tests
    float event_cut = MIN_R2;
    if (SCREEN && active) {
        const float Ri = __double2float_ru(g.radius[i]), mi = __double2float_ru(g.mass[i]);
        if (g.record) {
            const float lim = (float)tile_f_rad(g, tile) * (Ri + sc[2]) * 1.001f;
            event_cut = fmaxf(event_cut, lim * lim);
        }
        if (g.hill) {
            const float inv3M = (float)(1.0 / (3.0 * g.mass[tile.base]));
            const float k3 = cbrtf(g.hill_f3_f * (mi + sc[3]) * inv3M), rho = __double2float_ru(g.rho[i]);
            float lim = k3 * 0.5f * (rho + sc[4]);
            // (a source at the distance d is at most d further from the star: one body far out does not
            // open the screens of the others)
            if (k3 < 1.0f) lim = fminf(lim, k3 * rho / (1.0f - 0.5f * k3));
            lim *= 1.001f;
            event_cut = fmaxf(event_cut, lim * lim);
        }
    }
    double acc = 0.0;
    bool deferred = false;  // an owner's sum is left to grav_fp64_rows
    __syncwarp();

    // the term of one exact pair of the sink s2
    auto exact_pair = [&](int s2, int j, bool events, PairOut& o) {
        o = PairOut{0.0, 0.0, 0.0};
        const int i2 = tile.sink_begin + s2;
        // (all loads first: their latency is paid once)
        const double xj = g.px[j], yj = g.py[j], zj = g.pz[j], mj = g.mass[j];
        const double Rj = SCREEN ? g.radius[j] : 0.0, rhoj = SCREEN && g.hill ? g.rho[j] : 0.0;
        if (j == i2 || 0 > g.id[j]) return;
        if (SCREEN && events)
            pair_term<true, true>(g, tile, i2, j, M.sink[0][s2], M.sink[1][s2], M.sink[2][s2], M.sink[3][s2], M.sink[4][s2],
                            M.sink[5][s2], xj, yj, zj, mj, Rj, rhoj, o);
        else
            pair_term<false, true>(g, tile, i2, j, M.sink[0][s2], M.sink[1][s2], M.sink[2][s2], 0.0, 0.0, 0.0, xj, yj,
                             zj, mj, 0.0, 0.0, o);
    };
    // sources [jb, jb + nj), nj <= 32, against the sink s2: the exact terms added in order to its
    // sums `comps` in M.acc
    auto exact_round = [&](int s2, int comps, int jb, int nj, bool events) {
        PairOut o{0.0, 0.0, 0.0};
        if (lane < nj) exact_pair(s2, jb + lane, events, o);
        __syncwarp();
        M.term[0][lane] = o.tx;
        M.term[1][lane] = o.ty;
        M.term[2][lane] = o.tz;
        __syncwarp();
        for (int cc = 0; cc < 3; cc++) {
            if (!(comps >> cc & 1)) continue;
            SerialSumState st{0, 0};
            const double v = warp_serial_sum(M.acc[cc][s2], M.term[cc], nj, st);
            __syncwarp();
            if (lane == 0) M.acc[cc][s2] = v;
            __syncwarp();
        }
    };
    auto publish = [&]() {
        __syncwarp();
        if (owner) {
            M.acc[c][s] = acc;
            float sigma = (act >> s & 1) && !deferred ? sigma_of(acc) : 0.0f;
            if (sigma != sigma) {  // out of range (all but zero, as a coplanar body's z): every pair would be exact
                deferred = true;
                sigma = 0.0f;
            }
            M.sig[c][s] = sigma;
        }
        __syncwarp();
    };

    int j0 = tile.src_begin;
    const int head = min(HEAD, tile.src_end - j0);
    for (int h0 = 0; h0 < head; h0 += 32 / SW) {  // 32 / SW sources against the SW sinks, a pair per lane
        const int nh = min(32 / SW, head - h0);
        PairOut o{0.0, 0.0, 0.0};
        if (q < nh && active) exact_pair(s, j0 + h0 + q, true, o);
        M.term[0][lane] = o.tx;
        M.term[1][lane] = o.ty;
        M.term[2][lane] = o.tz;
        __syncwarp();
        if (owner)
            for (int f = 0; f < nh; f++) acc = acc + M.term[c][f * SW + s];
        __syncwarp();
    }
    deferred = outside && owner;
    publish();
    j0 += head;
    const int j_head = j0;

    // the rows of part h of an epoch: slice u's sources jt + u sl + [PART h, PART h + PART)
    auto fetch = [&](int jt, int h) {
        const int nj = min(EPOCH, tile.src_end - jt);
        const int sl = nj == EPOCH ? SLICE : ((nj + NQ * 4 - 1) / (NQ * 4)) * 4;
        if (nj > 0)
            for (int e = lane; e < 8 * NQ * (PART / 4); e += 32) {
                const int r = e / (NQ * (PART / 4)), u = e / (PART / 4) % NQ, o = e % (PART / 4) * 4, k = PART * h + o;
                if (k < sl && u * sl + k < nj) cp_async16(&M.src[h & 1][r][u * PITCH + o], base + r * stride + jt + u * sl + k);
            }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(j0, 0);
    fetch(j0, 1);
    int again = 0;                // times the epoch has been taken again for flagged sinks
    int n_redo = 0, n_exact = 0;  // n_exact: this lane's flagged pairs that no failing component explains
    // epochs a sum may leave its binade in: taken again, one costs up to its pairs exactly, a row an eighth of its own
    const int redo_most = min(4, 1 + (tile.src_end - tile.src_begin) / (8 * EPOCH));
    int tests = outside ? j_head : tile.src_end;  // the first source whose event tests are the row kernel's
    unsigned live = act & ~__ballot_sync(ALL, outside) & SINKS;  // sinks with sums left here (or events to find)
    unsigned listed = act & SINKS & ~live;                       // sinks with a row in the list
    for (; j0 < tile.src_end; j0 += EPOCH) {
        const int nj = min(EPOCH, tile.src_end - j0);
        const int sl = nj == EPOCH ? SLICE : ((nj + NQ * 4 - 1) / (NQ * 4)) * 4;
        const int cnt = max(0, min(sl, nj - q * sl));
        const int passed = j0 - j_head;
        const bool look = passed < 8 * EPOCH || passed % (16 * EPOCH) == 0;  // whether the sinks had better go whole
        unsigned begun = 0u, rows = 0u;
        if (counted && look && lane == 0) begun = __ldcg(cr.n_list + 1), rows = __ldcg(cr.n_list + 2);
        CertSum sum{0u, 0u, 0u, 0u, 0u, 0u, 0.0f};
        unsigned flags = 0u;
        const float sx = M.sig[0][s], sy = M.sig[1][s], sz = M.sig[2][s];
        k.sx = f2_dup(sx);
        k.sy = f2_dup(sy);
        k.sz = f2_dup(sz);
        const float cut = SCREEN && j0 < i ? event_cut : MIN_R2;
        int n_done = 0;
#pragma unroll 1
        for (int h = 0; h < SLICE / PART; h++) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");  // all but the next part
            __syncwarp();
            const int n = (live >> s & 1) ? min(PART, cnt - PART * h) : 0;
            const float* b = &M.src[h & 1][0][q * PITCH];
            constexpr int P = NQ * PITCH;
            unsigned bit = 1u << (PART * h);
#pragma unroll 2
            for (int e = 0; e < n; e += 2, b += 2, bit <<= 2) {
                const auto row = [&](int r) { return *reinterpret_cast<const f2*>(b + r * P); };
                f2 mh = row(6), ml = row(7);
                if (e + 2 > n) {  // the body past the last source adds nothing
                    mh &= 0xffffffffull;
                    ml &= 0xffffffffull;
                }
                cert_pair2(k, tc, row(0), row(1), row(2), row(3), row(4), row(5), mh, ml, cut, bit, sum, flags);
                n_done += 2;
            }
            __syncwarp();  // every lane has read the part: its buffer is free
            fetch(h + 2 < SLICE / PART ? j0 : j0 + EPOCH, (h + 2) & 3);
        }
        n_done -= __popc(flags);
        if (cnt < 32) flags &= (1u << cnt) - 1u;
        if (!SCREEN) {  // a sink with most of its pairs flagged: nothing of it is left here
            int n = __popc(flags);
            for (int off = SW; off < 32; off <<= 1) n += __shfl_xor_sync(ALL, n, off);
            const bool most = 2 * n > nj;
            deferred = deferred || (most && owner);
            if (most) flags = 0u;
        }
        // with event tests: a sink with most of its pairs flagged loses its smallest sum, which is the one they
        // are uncertain in as a rule, or, if that does not help, goes to the row kernel whole; and the warp
        // takes the epoch again.  (Their exact pairs cost eleven times the row's: an RKF7(8) attempt of 30 disks
        // of 303 bodies, a tenth of them above an otherwise flat disk, 9.1 ms, 4.1 so; of ordinary ones
        // 1.60 and 1.33 ms.)
        if (SCREEN && __any_sync(ALL, 2 * __popc(flags) > cnt)) {  // (one lane of such a sink has most of its own)
            int n = __popc(flags);
            for (int off = SW; off < 32; off <<= 1) n += __shfl_xor_sync(ALL, n, off);
            const bool most = n > 32 && 2 * n > nj && (live >> s & 1u);
            const int size = owner && !deferred && acc != 0.0 ? (int)((xf::dbits(acc) >> 52) & 0x7ff) : 4096;
            const int s0 = __shfl_sync(ALL, size, s), s1 = __shfl_sync(ALL, size, SW + s), s2 = __shfl_sync(ALL, size, 2 * SW + s);
            const int least = s2 <= min(s0, s1) ? 2 : (s1 <= s0 ? 1 : 0);  // z first: a disk's plane
            if (__any_sync(ALL, most)) {
                const bool whole = most && again > 0;
                if (owner && most && (whole || c == least)) deferred = true;
                if (whole) tests = j0;
                live &= ~__ballot_sync(ALL, whole);
                again++;
                publish();
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                __syncwarp();
                fetch(j0, 0);
                fetch(j0, 1);
                j0 -= EPOCH;
                continue;
            }
        }
        again = 0;
        // each high and low integer carries MAGIC's bits
        const unsigned nb = (unsigned)n_done * MAGIC_BITS;
        long long px = (long long)(int)(sum.hx - nb) * 65536 + (int)(sum.lx - nb);
        long long py = (long long)(int)(sum.hy - nb) * 65536 + (int)(sum.ly - nb);
        long long pz = (long long)(int)(sum.hz - nb) * 65536 + (int)(sum.lz - nb);
        float bx = sum.big * RADIX + 2.0f * (float)n_done, by = bx, bz = bx;
        // the flagged pairs, shared out over the warp: each round the lanes list up to 32 of their
        // pairs, each lane computes one of them exactly, and the owners add the quanta
        int left = __popc(flags);
        unsigned fail = 0u;  // of the flagged pairs, too large for the integers: per component, 10 bits each
        while (__any_sync(ALL, left > 0)) {
            int incl = left;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int v = __shfl_up_sync(ALL, incl, d);
                if (lane >= d) incl += v;
            }
            const int off = incl - left;
            const int n_items = min(32, __shfl_sync(ALL, incl, 31));
            int take = max(0, min(left, 32 - off));
            const int taken = take;
            left -= take;
            for (int f = off; take > 0; take--, f++) {
                const int bit = __ffs(flags) - 1;
                flags &= flags - 1;
                M.fitem[f] = (unsigned short)((lane << 5) | bit);
            }
            __syncwarp();
            if (lane < n_items) {
                const unsigned it = M.fitem[lane];
                const int ol = (int)(it >> 5), s2 = ol % SW;
                PairOut o;
                exact_pair(s2, j0 + ol / SW * sl + (int)(it & 31u), true, o);
                int bad = 0;
                const double v[3] = {o.tx, o.ty, o.tz};
#pragma unroll
                for (int f = 0; f < 3; f++) {
                    const int ea = (int)((xf::dbits(M.acc[f][s2]) >> 52) & 0x7ff);
                    int64_t r = 0;
                    const bool ok = v[f] == 0.0 || (ea > 0 && ea < 2047 && xf::quantize(v[f], ea, &r));
                    M.f.r[lane][f] = ok ? (long long)r : 0ll;
                    bad |= ok ? 0 : 1 << f;
                    bad |= !ok || (r < 0 ? -r : r) > UNCERTAIN ? 8 << f : 0;
                }
                M.f.bad[lane] = bad;
            }
            __syncwarp();
            for (int f = off; f < off + taken; f++) {
                const unsigned bad = (unsigned)M.f.bad[f];
                const long long rx = M.f.r[f][0], ry = M.f.r[f][1], rz = M.f.r[f][2];
                const float inf = __uint_as_float(0x7f800000u);
                px += rx;
                py += ry;
                pz += rz;
                bx += bad & 1 ? inf : __ll2float_ru(rx < 0 ? -rx : rx);
                by += bad & 2 ? inf : __ll2float_ru(ry < 0 ? -ry : ry);
                bz += bad & 4 ? inf : __ll2float_ru(rz < 0 ? -rz : rz);
                fail += (bad >> 3 & 1u) | (bad >> 4 & 1u) << 10 | (bad >> 5 & 1u) << 20;
                n_exact += bad >> 3 == 0u;
            }
            __syncwarp();  // the round's lists are read before the next round writes them
        }
        M.part[q][0][s] = px;
        M.part[q][1][s] = py;
        M.part[q][2][s] = pz;
        M.bnd[q][0][s] = bx;
        M.bnd[q][1][s] = by;
        M.bnd[q][2][s] = bz;
        __syncwarp();
        // the owners accept the epoch's quanta when no running sum can have left the binade
        bool ok = true;
        if (owner && (act >> s & 1) && !deferred) {
            long long total = 0;
            float bound = 0.0f;
            for (int u = 0; u < NQ; u++) {
                total += M.part[u][c][s];
                bound += M.bnd[u][c][s];
            }
            // (a zero sum of zero displacements stays zero)
            ok = accept(acc, total, bound) || (acc == 0.0 && (flat >> c & 1) && bound < 1.0e30f);
        }
        for (int off = SW; off < 32; off <<= 1) fail += __shfl_xor_sync(ALL, fail, off);
        bool whole = false;
        if (look) {
            int n = n_exact;
            for (int off = SW; off < 32; off <<= 1) n += __shfl_xor_sync(ALL, n, off);
            const bool many = __any_sync(ALL, begun >= 512u && 4ull * rows > 3ull * begun);  // (by every lane)
            // as many to come as up to here, against a row's cost: that of an eighth of its pairs, or of 50
            const long long left = tile.src_end - (j0 + nj), all = max(400, tile.src_end - tile.src_begin);
            whole = many || (n > 32 && 8 * n * left > (passed + nj) * all);
        }
        if (owner && !deferred && (act >> s & 1)) {
            n_redo += ok ? 0 : (acc == 0.0 ? 4 : 1);  // (a sum that is zero so far will hover)
            deferred = deferred || whole || (int)(fail >> (10 * c) & 1023u) * 8 > nj || n_redo >= redo_most;
            ok = ok || deferred;
        }
        // sums (bit c SW + s) whose epoch is taken slice by slice
        const unsigned redo = __ballot_sync(ALL, !ok);
        const unsigned gone = __ballot_sync(ALL, deferred);
        const unsigned done = gone & gone >> SW & gone >> 2 * SW & live, some = (gone | gone >> SW | gone >> 2 * SW) & live;
        if (done >> s & 1u) tests = min(j0 + EPOCH, tile.src_end);
        live &= ~done;
        if (counted && lane == 0 && (some & ~listed)) atomicAdd(cr.n_list + 2, (unsigned)__popc(some & ~listed));
        listed |= some;
        // the others slice by slice: its quanta while the sum stays in the epoch's binade, else
        // its exact terms added in order
        for (unsigned left_sums = redo; left_sums; left_sums &= left_sums - 1) {
            const int w = __ffs(left_sums) - 1, s2 = w % SW, c2 = w / SW;
            double a = M.acc[c2][s2];
            const int ea = (int)((xf::dbits(a) >> 52) & 0x7ff);
            for (int u = 0; u * sl < nj; u++) {
                if ((int)((xf::dbits(a) >> 52) & 0x7ff) == ea && accept(a, M.part[u][c2][s2], M.bnd[u][c2][s2])) continue;
                if (lane == 0) M.acc[c2][s2] = a;
                __syncwarp();
                exact_round(s2, 1 << c2, j0 + u * sl, min(sl, nj - u * sl), false);
                a = M.acc[c2][s2];
            }
            if (lane == w) acc = a;
        }
        if (!live) break;  // (uniform)
        publish();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (owner && i < tile.sink_end && !deferred) {
        double* out = c == 0 ? g.ax : (c == 1 ? g.ay : g.az);
        out[i] = acc;
    }
    const unsigned gone = __ballot_sync(ALL, deferred);
    if (lane < SW) {
        const int mask = (int)(gone >> s & 1u) | (int)(gone >> (SW + s) & 1u) << 1 | (int)(gone >> (2 * SW + s) & 1u) << 2;
        if (mask) {
            Tile row = tile;
            row.sink_begin = i;
            row.sink_end = tests;
            row.part = mask | (int)((__float_as_uint(event_cut) + 8u) & ~7u);
            cr.list[atomicAdd(cr.n_list, 1u)] = row;
        }
    }
}

long long cert_stride(int n, int n_sys) { return cert_row(n, n_sys) + 4; }

int launch_cert_prep(const GravArgs& g, const int* sys_base, const int* sys_n, int n_sys, int max_n, const CertRows& cr,
                     cudaStream_t st)
{
    if (max_n <= 0 || n_sys <= 0) return 0;
    const int blocks = (max_n - 1) / PREP_NT + 1;
    CertPrepArgs a{g.px, g.py, g.pz, g.mass, g.radius, g.hill ? g.rho : nullptr, g.id, sys_base, sys_n, g.sys_active, n_sys,
                   max_n, blocks, g.record || g.hill, cr.rows, cr.stride, cr.n_list, cr.scale};
    const long long ctas = (long long)blocks * n_sys, row = 1ll << 30;  // (a grid has 2^31 - 1 columns, 65 535 rows)
    const dim3 grid((unsigned)(ctas < row ? ctas : row), (unsigned)((ctas + row - 1) / row));
    cert_prep_kernel<<<grid, PREP_NT, 0, st>>>(a);
    RG_CUDA_CHECK(cudaGetLastError());
    return 0;
}

int launch_grav_fp64_cert(const GravArgs& g, const CertRows& cr, int S, cudaStream_t st)
{
    if (g.n_tiles <= 0) return 0;
    // the CTAs of an SM need more than the default shared-memory carve-out: a per-device attribute of each
    // kernel, set once per device (setting it again from another thread is harmless)
    static std::atomic<bool> attr_set[64];
    int dev = 0;
    RG_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
        for (auto kernel : {grav_fp64_cert<2, true>, grav_fp64_cert<2, false>, grav_fp64_cert<4, true>, grav_fp64_cert<4, false>})
            RG_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                               cudaSharedmemCarveoutMaxShared));
        if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
    }
    const bool few = (long long)g.n_tiles * S <= 4LL * CERT_FULL * NUM_SMS_HINT;
    const int per_cta = (few ? 2 : 4) * CERT_WARPS;
    const dim3 grid(g.n_tiles, (S + per_cta - 1) / per_cta);
    auto kernel = few ? (g.record || g.hill ? grav_fp64_cert<2, true> : grav_fp64_cert<2, false>)
                      : (g.record || g.hill ? grav_fp64_cert<4, true> : grav_fp64_cert<4, false>);
    kernel<<<grid, 32 * CERT_WARPS, 0, st>>>(g, cr);
    RG_CUDA_CHECK(cudaGetLastError());
    return 0;
}

}  // namespace redgb
