// GPU check of warp_row_sum (row_sum.h) as the gravity kernels compile it: one warp per row of
// serial_sum_cases.h, in calls of up to 32 x 36 terms, against lane 0's plain serial loop of
// __dadd_rn, counted on the device; then the cycles per term of both on a row whose sum keeps
// changing binade.
//
//   row_sum_gpu ROWS  ->  one line per family: "family F rows R bad B", and "cycles ..."
#include <cstdio>
#include <cstdlib>

#include "../../red.cuda.closeencounter_gb300/csrc/row_sum.h"
#include "serial_sum_cases.h"

constexpr int WARPS = 2;
constexpr int CHUNK = 32 * redgb::ROW_SEG_MAX;

struct Smem {
    double term[WARPS][32 * (redgb::ROW_SEG_MAX | 1)];
    uint32_t codes[WARPS][CHUNK];
};

__device__ double row(double acc, const double* t, int n, Smem& S, int warp)
{
    const int lane = threadIdx.x & 31;
    for (int b = 0; b < n; b += CHUNK) {
        const int m = min(CHUNK, n - b), seg = (m + 31) / 32, pitch = seg | 1;
        __syncwarp();
        for (int e = lane; e < m; e += 32) S.term[warp][e / seg * pitch + e % seg] = t[b + e];
        __syncwarp();
        acc = redgb::warp_row_sum(acc, S.term[warp], seg, pitch, m, S.codes[warp]);
    }
    return acc;
}

__global__ void __launch_bounds__(32 * WARPS) check(uint64_t seed, int fam, long long rows, double* buf,
                                                    unsigned long long* bad)
{
    __shared__ Smem S;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long gw = (long long)blockIdx.x * WARPS + warp;
    double* t = buf + gw * SC_MAX_LEN;
    for (long long r = gw; r < rows; r += (long long)gridDim.x * WARPS) {
        double acc0 = 0.0;
        int n = 0;
        if (lane == 0) n = sc_row(seed, fam, (uint64_t)r, &acc0, t);
        n = __shfl_sync(0xffffffffu, n, 0);
        acc0 = __shfl_sync(0xffffffffu, acc0, 0);
        __syncwarp();
        double ref = acc0;
        if (lane == 0)
            for (int k = 0; k < n; k++) ref = __dadd_rn(ref, t[k]);
        ref = __shfl_sync(0xffffffffu, ref, 0);
        const double acc = row(acc0, t, n, S, warp);
        const bool ok = (acc != acc && ref != ref) || __double_as_longlong(acc) == __double_as_longlong(ref);
        if (lane == 0 && !ok) atomicAdd(bad, 1ull);
        __syncwarp();
    }
}

__global__ void __launch_bounds__(32) latency(double* t, int n, long long* out)
{
    __shared__ Smem S;
    const int lane = threadIdx.x;
    if (lane == 0) {  // random signs: the sum hovers about zero
        ScRng g{31};
        for (int k = 0; k < n; k++) t[k] = (g.below(2) ? -1.0 : 1.0) * sc_random_mag(g, -4, 0);
    }
    __syncwarp();
    double a = 0.0, b = 0.0;
    for (int rep = 0; rep < 2; rep++) {
        const long long t0 = clock64();
        b = row(0.0, t, n, S, 0);
        const long long t1 = clock64();
        a = 0.0;
        for (int k = 0; k < n; k++) a = __dadd_rn(a, S.term[0][k / 32 * 33 + k % 32]);  // latency only
        const long long t2 = clock64();
        out[0] = t1 - t0;
        out[1] = t2 - t1;
    }
    double ref = 0.0;
    for (int k = 0; k < n; k++) ref = __dadd_rn(ref, t[k]);
    out[2] = __double_as_longlong(ref) == __double_as_longlong(b);
    if (a == 12345.0) out[2] = 2;
}

int main(int argc, char** argv)
{
    const long long rows = argc > 1 ? atoll(argv[1]) : 20000;
    const int grid = 152 * 2;
    double* buf = nullptr;
    unsigned long long* bad = nullptr;
    long long* out = nullptr;
    if (cudaMalloc(&buf, (size_t)grid * WARPS * SC_MAX_LEN * sizeof(double)) != cudaSuccess) return 2;
    if (cudaMalloc(&bad, 5 * sizeof(unsigned long long)) != cudaSuccess) return 2;
    if (cudaMalloc(&out, 3 * sizeof(long long)) != cudaSuccess) return 2;
    cudaMemset(bad, 0, 5 * sizeof(unsigned long long));
    for (int fam = 0; fam < 5; fam++) check<<<grid, 32 * WARPS>>>(4711, fam, rows, buf, bad + fam);
    unsigned long long h[5];
    if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) {
        printf("cuda error %s\n", cudaGetErrorString(cudaGetLastError()));
        return 3;
    }
    int rc = 0;
    for (int fam = 0; fam < 5; fam++) {
        printf("family %d rows %lld bad %llu\n", fam, rows, h[fam]);
        rc |= h[fam] != 0;
    }
    const int n = 1024;
    latency<<<1, 32>>>(buf, n, out);
    long long c[3];
    if (cudaMemcpy(c, out, sizeof(c), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    printf("cycles per term: serial %.1f warp_row_sum %.1f same %lld\n", (double)c[1] / n, (double)c[0] / n, c[2]);
    rc |= c[2] != 1;
    cudaFree(buf);
    cudaFree(bad);
    cudaFree(out);
    return rc;
}
