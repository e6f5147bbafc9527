// Launchers of kernels with more than 48 KB of dynamic shared memory against a runtime that only keeps books: two
// devices in one process, and each launch on a device needs the attribute to have been set on that device.
#include <cstdio>
#include <map>
#include <set>
#include <utility>

#include "../h2weak_gb300/csrc/kernels.cuh"

namespace {
int device = 0, launches = 0, bad = 0;
std::map<std::pair<int, const void *>, int> attr;  // (device, kernel) -> bytes allowed
void launched(const void *f, size_t smem) {
    ++launches;
    const auto it = attr.find({device, f});
    if (smem > 48 * 1024 && (it == attr.end() || (size_t)it->second < smem)) {
        ++bad;
        printf("device %d: %zu bytes of shared memory without the attribute\n", device, smem);
    }
}
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int *d) {
    *d = device;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) {
    *v = a == cudaDevAttrMultiProcessorCount ? 100 + d : 228 * 1024;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) attr[{device, f}] = v;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes *a, const void *) {
    *a = cudaFuncAttributes{};
    a->numRegs = 64;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3, dim3, void **, size_t smem, cudaStream_t) {
    launched(f, smem);
    return cudaSuccess;
}
// a <<<>>> launch: the kernel of an entry, then its launch
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **, size_t smem, cudaStream_t) {
    launched((const void *)k, smem);
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
}

int main() {
    using namespace h2w;
    int failed = 0;
    for (int round = 0; round < 2; ++round)
        for (device = 0; device < 3; ++device) {
            const int before = launches;
            GmresDev g{};
            g.N = 200000;
            g.m = 500;
            g.nblk = gmres_blocks(g.N);
            failed += gmres_step(g, nullptr, 0) != cudaSuccess;
            MoArgs a{};
            a.ld = 16;
            a.ncg = 1;
            a.l1[0] = a.l1[1] = a.l1[2] = 100;
            failed += launch_mo(a, 0) != cudaSuccess;
            const MrPhases *coop = nullptr;
            failed += launch_mr_f64_flow(64, false, 0, 0, 10, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0) != cudaSuccess;
            failed += launch_mr_f64_flow(64, true, 0, 0, 10, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0) != cudaSuccess;
            failed += launch_mr_f64(64, 0, 0, 0, 1, coop, 0, 0, 0, 0, 0, 0, 0, 0) != cudaSuccess;
            failed += launch_mw_f32_flow(64, 0, 0, 10, 0, 0, 0, 0, 0, 0, 0, (double *)nullptr, 0, 0) != cudaSuccess;
            failed += launch_mrt_f32(64, 0, 0, 0, 1, coop, 0, 0, 0, 0, (double *)nullptr, 0, 0, 0) != cudaSuccess;
            failed += launch_mlp_forward(nullptr, nullptr, 100, nullptr, 0) != cudaSuccess;
            if (launches - before < 8) ++failed;
        }
    printf("%d launches, %d without the attribute, %d refused\n", launches, bad, failed);
    return bad || failed;
}
