// Operators that share a device's memory: the runtime's allocations run against a budget here, and
// operators that fit without their copies fit with them, for the copies are given back.
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <cmath>
#include <cstdio>
#include <map>
#include <vector>

#include "h2w.h"

namespace {
size_t budget = (size_t)1 << 60, used = 0, peak = 0;
std::map<void *, size_t> size_of;
template <class F> F next(const char *name) { return (F)dlsym(RTLD_NEXT, name); }
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    static const auto real = next<cudaError_t (*)(void **, size_t)>("cudaMalloc");
    *p = nullptr;
    if (used + n > budget) return cudaErrorMemoryAllocation;
    const cudaError_t e = real(p, n);
    if (e == cudaSuccess) {
        size_of[*p] = n;
        used += n;
        if (used > peak) peak = used;
    }
    return e;
}
cudaError_t cudaFree(void *p) {
    static const auto real = next<cudaError_t (*)(void *)>("cudaFree");
    const auto it = size_of.find(p);
    if (it != size_of.end()) {
        used -= it->second;
        size_of.erase(it);
    }
    return real(p);
}
cudaError_t cudaMemGetInfo(size_t *fr, size_t *tot) {
    static const auto real = next<cudaError_t (*)(size_t *, size_t *)>("cudaMemGetInfo");
    const cudaError_t e = real(fr, tot);
    const size_t left = budget > used ? budget - used : 0;
    if (*fr > left) *fr = left;
    return e;
}
}

namespace {
int bad = 0;
void check(bool ok, const char *what) {
    if (!ok) {
        ++bad;
        printf("failed: %s (%.1f of %.1f MB)\n", what, used / 1e6, budget / 1e6);
    }
}
h2w_handle *make(int side, int levels, bool copies) {
    h2w_config c{};
    c.dim = 2;
    c.form = H2W_FORM_NESTED;
    c.choice = H2W_KERNEL_RBF;
    c.tol_pow = 8;
    c.nlevels = levels;
    h2w_handle *h = nullptr;
    if (h2w_create(&c, &h) != H2W_OK) return nullptr;
    if (!copies) h2w_set_option(h, H2W_OPT_COPIES, 0);
    if (h2w_gen_grid(h, side) != H2W_OK || h2w_build_tree(h) != H2W_OK || h2w_assemble(h, H2W_ASSEMBLE_NCA) != H2W_OK) {
        printf("%s\n", h2w_last_error(h));
        h2w_destroy(h);
        return nullptr;
    }
    return h;
}
int64_t made(h2w_handle *h) {
    int64_t v = -1;
    h2w_get_option(h, H2W_OPT_COPIES_MADE, &v);
    return v;
}
double off(const std::vector<double> &a, const std::vector<double> &b) {
    double e = 0, n = 0;
    for (size_t i = 0; i < a.size(); ++i) e += (a[i] - b[i]) * (a[i] - b[i]), n += b[i] * b[i];
    return std::sqrt(e / n);
}
}  // namespace

int main() {
    const int side = 100, levels = 4;
    const size_t N = (size_t)side * side;
    std::vector<double> x(8 * N), want(8 * N), y(8 * N);
    for (size_t i = 0; i < x.size(); ++i) x[i] = std::sin(0.37 * (double)i);
    h2w_handle *h = make(side, levels, false);
    check(h && made(h) == 0, "an operator without copies");
    if (!h) return 1;
    const size_t one = used, more = peak - used;
    check(h2w_matvec(h, x.data(), want.data(), 8, H2W_PREC_FP64, H2W_HOST, nullptr) == H2W_OK, "a product without copies");
    h2w_destroy(h);

    // five operators where five fit without copies
    const size_t base = used;
    budget = base + 5 * one + more + one / 2;
    std::vector<h2w_handle *> ops;
    for (int i = 0; i < 5; ++i) {
        h = make(side, levels, true);
        check(h, "an operator among five");
        if (!h) break;
        if (i == 0) check(made(h) & 1, "the first operator's copy");
        ops.push_back(h);
    }
    if (ops.size() == 5) check(made(ops[0]) == 0, "the first operator's copy was given back");
    for (h2w_handle *o : ops) {
        check(h2w_matvec(o, x.data(), y.data(), 1, H2W_PREC_FP64, H2W_HOST, nullptr) == H2W_OK, "a product among five");
        check(off({y.begin(), y.begin() + (long)N}, {want.begin(), want.begin() + (long)N}) < 1e-13, "its result");
    }
    for (h2w_handle *o : ops) h2w_destroy(o);

    // one operator with both copies, then a solve whose Krylov vectors need their room
    budget = used + 8 * one;
    h = make(side, levels, true);
    check(h, "an operator with room");
    if (!h) return 1;
    check(h2w_matvec(h, x.data(), y.data(), 8, H2W_PREC_FP64, H2W_HOST, nullptr) == H2W_OK, "a product of several vectors");
    check(off(y, want) < 1e-13, "its results");
    check(made(h) == 3, "both copies");
    budget = used + one / 2;
    const int m = (int)(3 * one / 4 / (8 * N));
    std::vector<double> b(want.begin(), want.begin() + (long)N), s(N, 1.0);
    int it = 0;
    double res = 0;
    const int rc = h2w_gmres(h, b.data(), s.data(), m, 10, H2W_HOST, &it, &res);
    check(rc == H2W_OK, h2w_last_error(h));
    check(off(s, {x.begin(), x.begin() + (long)N}) < 1e-6, "the solution");
    check(made(h) != 3, "a copy was given back");
    check(h2w_matvec(h, x.data(), y.data(), 8, H2W_PREC_FP64, H2W_HOST, nullptr) == H2W_OK && off(y, want) < 1e-13,
          "a product of several vectors after that");
    h2w_destroy(h);
    check(used == base, "everything freed");
    printf("%d steps of room, %d failures\n", m, bad);
    return bad != 0;
}
