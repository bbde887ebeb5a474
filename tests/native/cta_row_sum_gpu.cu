// GPU check of cta_row_sum (row_sum.h): one CTA of 8 or 16 warps per row of serial_sum_cases.h,
// against a plain serial loop of __dadd_rn, counted on the device.
//
// Then group_row_sum: two groups of two warps in a CTA, rows in chunks of 1152 terms.
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

constexpr int CHUNK = 1152, LANES = 64;
struct GroupSmem {
    double term[2][LANES * (CHUNK / LANES | 1)];
    uint32_t codes[2][CHUNK];
    redgb::GroupRowSmem<640, 2> sum[2];
    double acc0[2];
    int n[2];
};

__global__ void __launch_bounds__(128) check_groups(uint64_t seed, int fam, long long rows, double* buf,
                                                    unsigned long long* bad)
{
    extern __shared__ __align__(16) unsigned char raw[];
    GroupSmem& S = *reinterpret_cast<GroupSmem*>(raw);
    const int q = threadIdx.x / LANES;
    const redgb::RowGroup grp{1 + q, LANES, (int)threadIdx.x % LANES};
    double* const t = buf + (2 * blockIdx.x + q) * (long long)SC_MAX_LEN;
    for (long long r = 2 * blockIdx.x + q; r < rows; r += 2 * gridDim.x) {
        if (grp.me == 0) S.n[q] = sc_row(seed, fam, (uint64_t)r, &S.acc0[q], t);
        __threadfence_block();
        grp.sync();
        const int n = S.n[q];
        double acc = S.acc0[q];
        for (int b = 0; b < n; b += CHUNK) {
            const int m = min(CHUNK, n - b), seg = (m + LANES - 1) / LANES, pitch = seg | 1;
            grp.sync();
            for (int e = grp.me; e < m; e += LANES) S.term[q][e / seg * pitch + e % seg] = t[b + e];
            grp.sync();
            acc = redgb::group_row_sum(grp, acc, S.term[q], seg, pitch, m, S.codes[q], S.sum[q]);
        }
        if (grp.me == LANES - 1) {
            double ref = S.acc0[q];
            for (int k = 0; k < n; k++) ref = __dadd_rn(ref, t[k]);
            if (!(acc != acc && ref != ref) && __double_as_longlong(acc) != __double_as_longlong(ref)) atomicAdd(bad, 1ull);
        }
        grp.sync();
    }
}

int main(int argc, char** argv)
{
    const long long rows = argc > 1 ? atoll(argv[1]) : 20000;
    unsigned long long* bad = nullptr;
    if (cudaMalloc(&bad, 15 * sizeof(unsigned long long)) != cudaSuccess) return 2;
    cudaMemset(bad, 0, 15 * sizeof(unsigned long long));
    for (int q = 0; q < 10; q++) check<<<152 * 2, q < 5 ? 256 : 512>>>(815, q % 5, rows, bad + q);
    double* buf = nullptr;
    const int grid = 152 * 2;
    if (cudaMalloc(&buf, (size_t)2 * grid * SC_MAX_LEN * sizeof(double)) != cudaSuccess) return 2;
    if (cudaFuncSetAttribute(check_groups, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GroupSmem)) != cudaSuccess)
        return 2;
    for (int q = 0; q < 5; q++) check_groups<<<grid, 128, sizeof(GroupSmem)>>>(77, q, rows, buf, bad + 10 + q);
    unsigned long long h[15];
    if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) {
        printf("cuda error %s\n", cudaGetErrorString(cudaGetLastError()));
        return 3;
    }
    int rc = 0;
    for (int q = 0; q < 15; q++) {
        printf("family %d warps %d rows %lld bad %llu\n", q % 5, q < 5 ? 8 : (q < 10 ? 16 : 2), rows, h[q]);
        rc |= h[q] != 0;
    }
    cudaFree(bad);
    cudaFree(buf);
    return rc;
}
