// The displacements of the certified FP64 form (gravity_cert.cu: split, grid, difference) against exact
// ones, in alpha = g 2^-24: random coordinates, and ones chosen so that every rounding is at its
// worst (half-way between two grid points, on both sides).
//
//   cert_disp_gpu  ->  "pairs N worst W bound B"
#include <cstdio>
#include <string>

#include "../../red.cuda.closeencounter_gb300/csrc/gravity_cert.cu"

namespace redgb {
int set_error(int code, const std::string&) { return code; }
int cuda_fail(cudaError_t, const char*, const char*, int) { return 1; }

__device__ unsigned long long mix(unsigned long long x)
{
    x ^= x >> 31, x *= 0x9E3779B97F4A7C15ull;
    x ^= x >> 29, x *= 0xBF58476D1CE4E5B9ull;
    return x ^ x >> 32;
}

__global__ void displacements(unsigned long long n, unsigned long long* worst)
{
    const float c = 4.0f;                      // 2^23 g
    const double g = (double)c / 8388608.0, alpha = g / 16777216.0;
    double most = 0.0;
    for (unsigned long long t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (unsigned long long)gridDim.x * blockDim.x) {
        double v[2];
        for (int q = 0; q < 2; q++) {
            const unsigned long long r = mix(4 * t + q + 1);
            const double u = (double)(r >> 12 & 0xfffffffull) / 268435456.0;
            // worst cases: in the binade c 2^-(e + 1), half-way between grid points and u of the split's remainder on
            const int e = (int)(r & 7u);
            const unsigned long long k = (1ull << (22 - e)) + (r >> 40 & ((1ull << (22 - e)) - 1ull));
            v[q] = t & 1 ? ((double)k + 0.5 + ldexp(0.25 * u, -e)) * g : ldexp((double)(r >> 12), -52) * c;
            if (q == 1 || t & 2) v[q] = -v[q];
        }
        float h, l, ah, al, bh, bl;
        split_bits(v[0], h, l);
        regrid(h, l, c, ah, al);
        split_bits(v[1], h, l);
        regrid(h, l, c, bh, bl);
        f2 d2, l2;
        cert_diff(f2_dup(ah), f2_dup(al), f2_dup(bh), f2_dup(bl), d2, l2);
        float d, e, unused;
        f2_unpack(d2, d, unused);
        f2_unpack(l2, e, unused);
        const double s = __dadd_rn(v[0], -v[1]), bb = __dadd_rn(s, -v[0]);
        const double low = __dadd_rn(__dadd_rn(v[0], -__dadd_rn(s, -bb)), __dadd_rn(-v[1], -bb));  // exact: s + low
        const double err = fabs(((s - (double)d) - (double)e) + low) / alpha;
        most = fmax(most, err);
    }
    atomicMax(worst, (unsigned long long)__double_as_longlong(most));
}
}  // namespace redgb

int main()
{
    unsigned long long* w = nullptr;
    const unsigned long long n = 1ull << 30;
    if (cudaMalloc((void**)&w, 8) != cudaSuccess || cudaMemset(w, 0, 8) != cudaSuccess) return 2;
    redgb::displacements<<<152 * 8, 256>>>(n, w);
    double worst = 0.0;
    if (cudaMemcpy(&worst, w, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    printf("pairs %llu worst %.4f bound %.4f\n", n, worst, (double)redgb::DISP_ERR);
    return worst <= (double)redgb::DISP_ERR && worst > 2.0 ? 0 : 1;
}
