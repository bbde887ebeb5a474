// GPU check of cta_row_sum (row_sum.h): one CTA of 8 or 16 warps per row of serial_sum_cases.h,
// against a plain serial loop of __dadd_rn, counted on the device.
//
//   cta_row_sum_gpu ROWS  ->  one line per family and size: "family F warps W rows R bad B"
#include <cstdio>
#include <cstdlib>

#include "../../red.cuda.closeencounter_gb300/csrc/row_sum.h"
#include "serial_sum_cases.h"

struct Smem {
    double term[SC_MAX_LEN + 1];
    uint32_t codes[SC_MAX_LEN + 64];
    redgb::CtaRowSmem sum;
    int n;
};

__global__ void __launch_bounds__(512) check(uint64_t seed, int fam, long long rows, unsigned long long* bad)
{
    __shared__ Smem S;
    for (long long r = blockIdx.x; r < rows; r += gridDim.x) {
        __syncthreads();
        if (threadIdx.x == 0) {
            double acc0 = 0.0;
            S.n = 1 + sc_row(seed, fam, (uint64_t)r, &acc0, S.term + 1);
            S.term[0] = acc0;
        }
        __syncthreads();
        const int n = S.n;
        const double acc = redgb::cta_row_sum(S.term, n, S.codes, S.sum);
        if (threadIdx.x == blockDim.x - 1) {
            double ref = 0.0;
            for (int k = 0; k < n; k++) ref = __dadd_rn(ref, S.term[k]);
            if (!(acc != acc && ref != ref) && __double_as_longlong(acc) != __double_as_longlong(ref)) atomicAdd(bad, 1ull);
        }
    }
}

int main(int argc, char** argv)
{
    const long long rows = argc > 1 ? atoll(argv[1]) : 20000;
    unsigned long long* bad = nullptr;
    if (cudaMalloc(&bad, 10 * sizeof(unsigned long long)) != cudaSuccess) return 2;
    cudaMemset(bad, 0, 10 * sizeof(unsigned long long));
    for (int q = 0; q < 10; q++) check<<<152 * 2, q < 5 ? 256 : 512>>>(815, q % 5, rows, bad + q);
    unsigned long long h[10];
    if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) {
        printf("cuda error %s\n", cudaGetErrorString(cudaGetLastError()));
        return 3;
    }
    int rc = 0;
    for (int q = 0; q < 10; q++) {
        printf("family %d warps %d rows %lld bad %llu\n", q % 5, q < 5 ? 8 : 16, rows, h[q]);
        rc |= h[q] != 0;
    }
    cudaFree(bad);
    return rc;
}
