// The NCA pivot search, one thread-block cluster per block (I, J) (sm_103a).
//
// Pivoting and stopping follow ACA_only_nodes (1D/codes/aca.hpp:296-446): first row with a
// non-negligible entry, column pivot = first largest |.| among unused columns of the
// residual row, row pivot = first largest |.| among unused rows of the residual column,
// stop when ||u|| ||v|| <= tol normS or the rank reaches min(n1, n2) (a block whose rank
// reaches its scratch capacity rcap first reports -rank). Residual rows and columns are
// formed entry by entry in pivot order with separate multiply and subtract, so for
// identical entries they are bitwise those of the reference; norms and dot products are
// tree reductions (they only enter the stopping test).
//
// What bounds it: the FP64 pipe (two operations a clock and SM: an entry takes a square
// root and a division, a residual two operations a kept term) where there are as many
// blocks as SMs, and the chain of steps of a pivot where there are fewer. So the CTAs of a
// cluster split a block's rows and columns, as many as the SMs allow; their candidates,
// norms and dot products are read by every member from distributed shared memory in
// the same order (the same decisions everywhere), two cluster barriers a pivot; largest
// magnitudes are compared as integers, the dot products of eight kept terms are
// reduced together (9 shuffled additions for 8 sums), and square roots and the
// stopping test are one warp's.
// Searches of an operator (2D, 9973 points, 1/r): 75 ms with one CTA a block, and groups
// of 76 CTAs of a cooperative launch for the four widest; 19 here. 3D, 20011 points, 1/r: 480
// and 100.
#include <climits>

#include "entry.cuh"

namespace h2w {
namespace {

constexpr int NC_T = 256, NC_W = NC_T / 32, NC_U = 8;

struct NcBest {
    unsigned long long key;  // |value| as an integer, plus one (0: no candidate)
    int32_t i;
};
struct NcPart {
    NcBest b;
    double s;
};

__device__ __forceinline__ void nc_offer(NcBest &b, double v, int i) {
    const unsigned long long k = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    if (k <= 0x7ff0000000000000ull && (k + 1 > b.key || (k + 1 == b.key && i < b.i))) b = {k + 1, i};  // a NaN is no candidate
}
// the warp's largest, lowest index among equals, in every lane
__device__ __forceinline__ NcBest nc_warp_best(NcBest b) {
    const unsigned hi = (unsigned)(b.key >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = hi == mh ? (unsigned)b.key : 0u, ml = __reduce_max_sync(0xffffffffu, lo);
    const int mi = __reduce_min_sync(0xffffffffu, hi == mh && (unsigned)b.key == ml ? b.i : INT_MAX);
    return {(unsigned long long)mh << 32 | ml, mi};
}
__device__ __forceinline__ double nc_warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// the sums over the lanes of d[0 .. 7]: lanes with (lane & 3) == 0 get that of d[lane >> 2]
__device__ __forceinline__ double nc_reduce8(const double (&d)[8], int lane) {
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    double e[4], f[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) e[i] = (b4 ? d[i + 4] : d[i]) + __shfl_xor_sync(0xffffffffu, b4 ? d[i] : d[i + 4], 16);
#pragma unroll
    for (int i = 0; i < 2; ++i) f[i] = (b3 ? e[i + 2] : e[i]) + __shfl_xor_sync(0xffffffffu, b3 ? e[i] : e[i + 2], 8);
    double g = (b2 ? f[1] : f[0]) + __shfl_xor_sync(0xffffffffu, b2 ? f[0] : f[1], 4);
    g += __shfl_xor_sync(0xffffffffu, g, 2);
    return g + __shfl_xor_sync(0xffffffffu, g, 1);
}
__device__ __forceinline__ void nc_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// p's address in the shared memory of cluster member r
template <class T> __device__ __forceinline__ const T *nc_member(const T *p, int r) {
    uint64_t a;
    asm("mapa.u64 %0, %1, %2;" : "=l"(a) : "l"((uint64_t)p), "r"(r));
    return reinterpret_cast<const T *>(a);
}
__device__ __forceinline__ bool nc_bit(const uint32_t *m, int i) { return (m[i >> 5] >> (i & 31)) & 1u; }

// v - sum of c[l] x[l ld], term by term; the loads of NC_U terms before their subtractions
__device__ __forceinline__ double nc_residual(double v, const double *c, const double *x, size_t ld, int rank) {
    int l = 0;
#pragma unroll 1
    for (; l + NC_U <= rank; l += NC_U) {
        double t[NC_U];
#pragma unroll
        for (int k = 0; k < NC_U; ++k) t[k] = x[(size_t)(l + k) * ld];
#pragma unroll
        for (int k = 0; k < NC_U; ++k) v = __dsub_rn(v, __dmul_rn(c[l + k], t[k]));
    }
#pragma unroll 1
    for (; l < rank; ++l) v = __dsub_rn(v, __dmul_rn(c[l], x[(size_t)l * ld]));
    return v;
}

// Dynamic shared memory: coefficients (rmax, even), the CTA's dot products (2 (rmax + 4)), pivot
// masks of the rows and columns.
__global__ void __launch_bounds__(NC_T, 2) nca_kernel(const NcaProb *__restrict__ probs, const int32_t *__restrict__ idx,
                                                   KParams kp, double tol, double *scr, int32_t *__restrict__ rank_out,
                                                   int32_t *__restrict__ prow, int32_t *__restrict__ pcol, int32_t *status,
                                                   int mask1_words, int mask2_words, int rmax, int C) {
    extern __shared__ __align__(16) unsigned char nc_smem[];
    double *coef = reinterpret_cast<double *>(nc_smem);
    double *dots = coef + (rmax + 1) / 2 * 2;  // du and dv of term l at 2 l, 2 l + 1
    uint32_t *rmask = reinterpret_cast<uint32_t *>(dots + 2 * (rmax + 4)), *cmask = rmask + mask1_words;
    // the warps' candidates; this CTA's for the residual row (pivots alternate: one that is ahead
    // writes the next row's while another still reads) and for the residual column
    __shared__ NcPart wpart[NC_W], rpart[2], cpart;
    __shared__ double wsum[NC_W], normS;
    __shared__ int go;

    const int blk = blockIdx.x / C, me = blockIdx.x % C;
    const NcaProb pb = probs[blk];
    const int n1 = pb.n1, n2 = pb.n2, rcap = pb.rcap, mn = n1 < n2 ? n1 : n2;
    const int32_t *I = idx + pb.ri, *J = idx + pb.ci;
    double *U = scr + pb.u, *V = scr + pb.v;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int a0 = (int)((int64_t)n1 * me / C), a1 = (int)((int64_t)n1 * (me + 1) / C);  // this CTA's rows
    const int b0 = (int)((int64_t)n2 * me / C), b1 = (int)((int64_t)n2 * (me + 1) / C);  // and columns
    const double tiny = 1e-36;

    // this CTA's candidate and sum of squares, for the others from the next cluster barrier on
    auto publish = [&](NcBest b, double s, NcPart *out) {
        b = nc_warp_best(b);
        s = nc_warp_sum(s);
        if (lane == 0) wpart[warp] = {b, s};
        __syncthreads();
        if (warp == 0) {
            const NcPart p = lane < NC_W ? wpart[lane] : NcPart{{0, INT_MAX}, 0.0};
            b = nc_warp_best(p.b);
            s = p.s;
#pragma unroll
            for (int o = NC_W / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) *out = {b, s};
        }
    };
    // the cluster's candidate, in every thread; its norm in warp 0
    auto best_of = [&](const NcPart *p) {
        return nc_warp_best(lane < C ? nc_member(p, lane)->b : NcBest{0, INT_MAX});
    };
    auto norm_of = [&](const NcPart *p) { return sqrt(nc_warp_sum(lane < C ? nc_member(p, lane)->s : 0.0)); };

    for (int q = tid; q < mask1_words; q += NC_T) rmask[q] = 0u;
    for (int q = tid; q < mask2_words; q += NC_T) cmask[q] = 0u;
    if (tid == 0 && me == 0) rank_out[blk] = 0;
    if (mn == 0 || rcap == 0) return;  // all members: nobody reads another's shared memory

    // first pivot row: the first whose largest |entry| exceeds 1e-36
    int ri = -1, ci = -1;
    double vsq = 0.0;
#pragma unroll 1
    for (int l = 0; l < n1 && ri < 0; ++l) {
        NcBest b{0, INT_MAX};
        vsq = 0.0;
        const int gi = I[l];
        for (int s = b0 + tid; s < b1; s += NC_T) {
            const double v = kentry(kp, gi, J[s]);
            V[s] = v;
            vsq += v * v;
            nc_offer(b, v, s);
        }
        publish(b, vsq, rpart);
        nc_barrier();
        b = best_of(rpart);
        if (b.key > 0 && __longlong_as_double((long long)(b.key - 1)) > tiny) {
            ri = l;
            ci = b.i;
        } else {
            nc_barrier();  // read by all before the next row's
        }
    }
    int rank = 0, nri = INT_MAX;
    bool over = false;
    if (ri >= 0) {
#pragma unroll 1
        for (;;) {
            // here: the residual row's slices in V_rank, its pivot column ci known, its partial in rpart[rank & 1]
            double *Vr = V + (size_t)rank * n2, *Ur = U + (size_t)rank * n1;
            // residual column ci
            const double piv = __ldcg(Vr + ci);  // another member's store: from the L2
            for (int l = tid; l < rank; l += NC_T) coef[l] = __ldcg(V + (size_t)l * n2 + ci);
            __syncthreads();
            NcBest b{0, INT_MAX};
            double usq = 0.0;
            {
                const int gj = J[ci];
#pragma unroll 1
                for (int t = a0 + tid; t < a1; t += NC_T) {
                    const double c = nc_residual(kentry(kp, I[t], gj), coef, U + t, (size_t)n1, rank);
                    const double u = __ddiv_rn(c, piv);
                    Ur[t] = u;
                    usq += u * u;
                    if (t != ri && !nc_bit(rmask, t)) nc_offer(b, c, t);
                }
            }
            publish(b, usq, &cpart);
            // dots of this CTA's slices of every kept u and v with the newest ones (not of the
            // first: its normS stays zero); four terms a warp at a time, u's and v's sums reduced together
            if (rank > 0) {
                __syncthreads();  // Ur and Vr are whole
#pragma unroll 1
                for (int l0 = 4 * warp; l0 <= rank; l0 += 4 * NC_W) {
                    double d[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
                    size_t o[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) o[k] = (size_t)min(l0 + k, rank);
#pragma unroll 2
                    for (int t = a0 + lane; t < a1; t += 32) {
                        const double u = Ur[t];
#pragma unroll
                        for (int k = 0; k < 4; ++k) d[2 * k] = fma(U[o[k] * n1 + t], u, d[2 * k]);
                    }
#pragma unroll 2
                    for (int s = b0 + lane; s < b1; s += 32) {
                        const double v = Vr[s];
#pragma unroll
                        for (int k = 0; k < 4; ++k) d[2 * k + 1] = fma(V[o[k] * n2 + s], v, d[2 * k + 1]);
                    }
                    const double g = nc_reduce8(d, lane);
                    if ((lane & 3) == 0) dots[2 * l0 + (lane >> 2)] = g;  // room for four terms past the last
                }
            }
            nc_barrier();
            nri = best_of(&cpart).i;
            // normS: every member adds the members' dots in their order
            double ns = 0.0;
            if (rank > 0) {
                for (int l = tid; l <= rank; l += NC_T) {
                    double du = 0.0, dv = 0.0;
                    for (int r = 0; r < C; ++r) {
                        const double2 p = *reinterpret_cast<const double2 *>(nc_member(dots + 2 * l, r));
                        du += p.x;
                        dv += p.y;
                    }
                    ns += 2.0 * fabs(du * dv);
                }
                if (warp * 32 <= rank) {
                    ns = nc_warp_sum(ns);
                    if (lane == 0) wsum[warp] = ns;
                }
                __syncthreads();
            }
            if (warp == 0) {
                const double nu = norm_of(&cpart), nv = norm_of(rpart + (rank & 1));
                ns = lane < NC_W && lane * 32 <= rank && rank > 0 ? wsum[lane] : 0.0;
#pragma unroll
                for (int o = NC_W / 2; o > 0; o >>= 1) ns += __shfl_xor_sync(0xffffffffu, ns, o);
                if (lane == 0) {
                    if (rank == 0) {
                        normS = 0.0;
                    } else if (!(nu < 1e-36 || nv < 1e-36)) {
                        const double uv = nu * nv;
                        normS = sqrt(normS * normS + uv * uv + ns);
                    }
                    // 0: this pivot is dropped, 1: the last, 2: another
                    go = rank > 0 && (nu < 1e-36 || nv < 1e-36) ? 0 : nu * nv > tol * normS ? 2 : 1;
                    if (go > 0) {
                        if (me == 0) {
                            prow[pb.piv + rank] = ri;
                            pcol[pb.piv + rank] = ci;
                        }
                        rmask[ri >> 5] |= 1u << (ri & 31);
                        cmask[ci >> 5] |= 1u << (ci & 31);
                    }
                }
            }
            __syncthreads();
            const int g = go;
            if (g == 0) break;
            ++rank;
            ri = nri;
            if (g == 1 || rank >= mn) break;
            if (rank >= rcap) {
                over = true;
                break;
            }
            if (ri < 0 || ri >= n1) {  // no finite candidate row
                if (tid == 0) atomicOr(status, 2);
                break;
            }
            // residual row ri
            for (int l = tid; l < rank; l += NC_T) coef[l] = __ldcg(U + (size_t)l * n1 + ri);
            __syncthreads();
            Vr += n2;
            b = {0, INT_MAX};
            vsq = 0.0;
            {
                const int gi = I[ri];
#pragma unroll 1
                for (int s = b0 + tid; s < b1; s += NC_T) {
                    const double v = nc_residual(kentry(kp, gi, J[s]), coef, V + s, (size_t)n2, rank);
                    Vr[s] = v;
                    vsq += v * v;
                    if (!nc_bit(cmask, s)) nc_offer(b, v, s);
                }
            }
            publish(b, vsq, rpart + (rank & 1));
            nc_barrier();
            ci = best_of(rpart + (rank & 1)).i;
            if (ci < 0 || ci >= n2) {  // no finite candidate column (non-finite entries)
                if (tid == 0) atomicOr(status, 2);
                break;
            }
        }
    }
    // an overflowing block reports -rank: the host runs it again with more scratch
    if (tid == 0 && me == 0) rank_out[blk] = over ? -rank : rank;
    nc_barrier();  // nobody leaves while its shared memory may be read
}

}  // namespace

cudaError_t launch_nca(const NcaProb *probs, int nprob, const int32_t *idx, const KParams &kp, double tol,
                       double *scratch, int32_t *rank, int32_t *prow, int32_t *pcol, int32_t *status, int max_n1,
                       int max_n2, int max_rcap, cudaStream_t st) {
    if (nprob == 0) return cudaSuccess;
    const int m1 = (max_n1 + 31) / 32, m2 = (max_n2 + 31) / 32;
    const size_t smem = (size_t)((max_rcap + 1) / 2 * 2 + 2 * (max_rcap + 4)) * 8 + (size_t)(m1 + m2) * 4;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(nca_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(nca_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    // CTAs a block: as many as keep two an SM at most, and a thread an entry. Against one an SM:
    // 64 blocks of 9000 rows and columns 19 instead of 27 ms, 16 of 1500 the same; four an SM: 3D
    // 15 instead of 19, 2D 4 instead of 3.
    int C = 1;
    while (C < 16 && (int64_t)nprob * C <= sms && (int64_t)C * NC_T < (int64_t)max_n1 + max_n2) C *= 2;
    for (;; C /= 2) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at{};
        cfg.gridDim = dim3((unsigned)(nprob * C));
        cfg.blockDim = dim3(NC_T);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = (unsigned)C;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        if (C > 1) {
            int n = 0;
            e = cudaOccupancyMaxActiveClusters(&n, nca_kernel, &cfg);
            if (e != cudaSuccess || n < 1) {
                cudaGetLastError();
                continue;
            }
        }
        e = cudaLaunchKernelEx(&cfg, nca_kernel, probs, idx, kp, tol, scratch, rank, prow, pcol, status, m1, m2, max_rcap, C);
        count_launch();
        return e != cudaSuccess ? e : cudaGetLastError();
    }
}

}  // namespace h2w
