// The double-FP32 far field on two points, with a log table that covers their distance and with one that does not: the
// second launch ends, and says so in its error word.
#include <cmath>
#include <cstdio>
#include <vector>

#include "../h2weak_gb300/csrc/kernels.cuh"

using namespace h2w;
template <class T> T *up(const std::vector<T> &v) {
    T *p = nullptr;
    cudaMalloc(&p, v.size() * sizeof(T));
    cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
    return p;
}
int run(double d, int e0, int ne, int *flag) {  // distance d, table from 2^e0 over ne exponents
    const std::vector<double> pts{0.0, 0.0, 0.0, d, 0.0, 0.0};
    double *dp = up(pts);
    float *df = up(std::vector<float>(16, 0.f));
    launch_ptsdf(dp, 3, 2, df, 0);
    FlyItem it{};
    it.nrows = it.ncols = 1;
    std::vector<float> tab((size_t)512 * ne);
    fly_df_table(e0, ne, tab.data());
    KParams kp{};
    kp.dim = 3;
    kp.choice = 1;
    kp.loga = std::log(1e-4);
    FlyK32 k{};
    k.sep = 1;
    k.tab_e0 = e0;
    k.ntab = 128 * ne;
    double *ws = up(std::vector<double>{0.0, 1.0});  // row 0 gets the entry times row 1
    int32_t *err = up(std::vector<int32_t>{0});
    const cudaError_t e = launch_fly_df64(up(std::vector<FlyItem>{it}), 1, up(std::vector<unsigned long long>{0}),
                                          up(std::vector<int32_t>{0}), up(std::vector<int32_t>{1}), up(std::vector<int32_t>{1}),
                                          df, up(tab), ws, kp, k, err, 0);
    double out = 0;
    cudaMemcpy(&out, ws, 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(flag, err, 4, cudaMemcpyDeviceToHost);
    const double want = std::log(d) / std::log(1e-4);
    printf("d %g table 2^%d..: error word %d, entry off by %.1e (%s)\n", d, e0, *flag, std::fabs(out - want), cudaGetErrorString(e));
    return e == cudaSuccess && std::fabs(out - want) <= 1e-12 * std::fabs(want) + 1e-13;
}
int main() {
    int bad = 0, flag = 0;
    bad += !run(0.7, -4, 5, &flag) || flag != 0;    // R^2 = 0.49
    bad += !run(0.26, -4, 5, &flag) || flag != 0;   // 0.0676, just above 2^-4
    run(0.2, -4, 5, &flag);                         // 0.04: below
    bad += flag != 5;
    run(1.5, -4, 5, &flag);                         // 2.25: above 2^1
    bad += flag != 5;
    return bad;
}
