// The event-screen maxima that launch_cert_prep (gravity_cert.cu) leaves per system: over the bodies
// that can be in an event, so not over inactive ones (id < 0), wherever a merger has parked them.
//
//   cert_screen_gpu  ->  "systems N bad B"
#include <cstdio>
#include <string>
#include <vector>

#include "../../red.cuda.closeencounter_gb300/csrc/gravity_cert.cu"

namespace redgb {
int set_error(int code, const std::string& msg)
{
    fprintf(stderr, "%s\n", msg.c_str());
    return code;
}
int cuda_fail(cudaError_t e, const char* what, const char*, int) { return set_error(1, std::string(what) + cudaGetErrorString(e)); }
}  // namespace redgb

using namespace redgb;

template <class T>
T* up(const std::vector<T>& v)
{
    T* p = nullptr;
    if (cudaMalloc((void**)&p, v.size() * sizeof(T)) != cudaSuccess ||
        cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess)
        exit(2);
    return p;
}

int main()
{
    const int sizes[] = {17, 40, 300, 1100, 2500};
    const int n_sys = 5;
    std::vector<int> base, count, id;
    std::vector<double> x, y, z, m, R, rho, want(3 * n_sys, 0.0);
    for (int s = 0; s < n_sys; s++) {
        base.push_back((int)id.size());
        count.push_back(sizes[s]);
        for (int k = 0; k < sizes[s]; k++) {
            const bool gone = k == sizes[s] - 1 || k == sizes[s] / 2;  // a parked merger; an ejected body
            const double v[3] = {gone ? 0.5 : 1e-5 * (1 + k % 7), gone ? 0.25 : 1e-9 * (1 + k % 11), gone ? 1e20 : 1.0 + k % 13};
            id.push_back(gone ? -k - 1 : (k == 20 ? 0 : k + 1));
            x.push_back(gone ? 1e20 : 1.0 + k % 13);
            y.push_back(0.0);
            z.push_back(0.001 * k);
            R.push_back(v[0]);
            m.push_back(v[1]);
            rho.push_back(v[2]);
            for (int q = 0; q < 3; q++)
                if (k >= 16 && !gone && v[q] > want[3 * s + q]) want[3 * s + q] = v[q];
        }
    }
    const int n = (int)id.size();
    GravArgs g{};
    g.px = up(x);
    g.py = up(y);
    g.pz = up(z);
    g.mass = up(m);
    g.radius = up(R);
    g.rho = up(rho);
    g.id = up(id);
    g.record = g.hill = 1;
    CertRows cr{};
    cr.stride = cert_stride(n, n_sys);
    cr.rows = up(std::vector<float>(8 * cr.stride));
    cr.scale = up(std::vector<float>(8 * n_sys));
    cr.n_list = up(std::vector<unsigned int>(CERT_COUNTERS, 7u));
    if (launch_cert_prep(g, up(base), up(count), n_sys, 2500, cr, nullptr)) return 2;
    std::vector<float> scale(8 * n_sys);
    unsigned int n_list = 1;
    if (cudaMemcpy(scale.data(), cr.scale, scale.size() * sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(&n_list, cr.n_list, sizeof(n_list), cudaMemcpyDeviceToHost) != cudaSuccess)
        return 2;
    int bad = n_list != 0;
    for (int s = 0; s < n_sys; s++)
        for (int q = 0; q < 3; q++) {  // magnitude(): at most 2e-6 above the value, never below it
            const double got = scale[8 * s + 2 + q], w = want[3 * s + q];
            const bool ok = got >= w && got <= w * (1.0 + 4e-6);
            if (!ok) printf("system %d maximum %d: %g, not %g\n", s, q, got, w);
            bad += !ok;
        }
    printf("systems %d bad %d\n", n_sys, bad);
    return bad ? 1 : 0;
}
