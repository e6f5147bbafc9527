// sm_103a kernels of the GB300 H2* / (H2+H)* library.
//
//  * kentry            kernel-matrix entries, operation order and rounding of
//                      the reference's getMatrixEntry (no FMA contraction)
//  * factor_kernel     LU of K(I,J) in pivot order = the ACA's L and R
//  * xfer_kernel       rows K(p,J) R^-1 L^-1 (transfer matrices), columns
//                      R^-1 L^-1 K(I,p), and the 1D U / V^T factors
//  * fill_kernel       dense blocks K(I,J) straight into the packed operator
//  * brg_kernel        the matvec: block-row GEMV over a work list of targets,
//                      each the sum of row-major panels times gathered sources
//  * GMRES kernels     CGS2 Arnoldi step, normalisation, Givens rotations
#include <atomic>
#include <cfloat>

#include "kernels.cuh"
#include "sync.cuh"
#include "entry.cuh"

namespace h2w {

static std::atomic<int64_t> g_launches{0};
int64_t launch_count() { return g_launches.load(); }
void count_launch(int64_t n) { g_launches.fetch_add(n); }

// ---------------------------------------------------------- reductions ---
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// Block-wide sum; every thread gets the total. sh: >= 32 doubles.
__device__ double block_sum(double v, double *sh) {
    v = warp_sum(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    double t = 0.0;
    for (int q = 0; q < nw; ++q) t += sh[q];
    return t;
}
constexpr int GM_THREADS = 256;

// ------------------------------------------------------------- factors ---
// F (r x r, row-major) <- K(I,J) factorised in pivot order: R on and above
// the diagonal, unit-lower L below it, with the ACA's operation order
// (R(l,j) = A(l,j) - sum_m L(l,m) R(m,j); L(t,l) = (A(t,l) - sum_m R(m,l) L(t,m)) / R(l,l)).
__global__ void factor_kernel(const FactorJob *__restrict__ jobs, const int32_t *__restrict__ idx, KParams kp,
                              double *__restrict__ F) {
    const FactorJob jb = jobs[blockIdx.x];
    const int r = jb.r;
    double *A = F + jb.f;
    const int32_t *I = idx + jb.ii, *J = idx + jb.jj;
    for (int e = threadIdx.x; e < r * r; e += blockDim.x) {
        int i = e / r, j = e % r;
        A[e] = kentry(kp, I[i], J[j]);
    }
    __syncthreads();
    for (int l = 0; l < r; ++l) {
        for (int j = l + threadIdx.x; j < r; j += blockDim.x) {
            double v = A[l * r + j];
            for (int m = 0; m < l; ++m) v = __dsub_rn(v, __dmul_rn(A[l * r + m], A[m * r + j]));
            A[l * r + j] = v;
        }
        __syncthreads();
        const double piv = A[l * r + l];
        for (int t = l + 1 + threadIdx.x; t < r; t += blockDim.x) {
            double v = A[t * r + l];
            for (int m = 0; m < l; ++m) v = __dsub_rn(v, __dmul_rn(A[m * r + l], A[t * r + m]));
            A[t * r + l] = __ddiv_rn(v, piv);
        }
        __syncthreads();
    }
}

cudaError_t launch_factor(const FactorJob *jobs, int njobs, const int32_t *idx, const KParams &kp, double *F,
                          cudaStream_t st) {
    if (njobs == 0) return cudaSuccess;
    factor_kernel<<<njobs, 128, 0, st>>>(jobs, idx, kp, F);
    count_launch(); return cudaGetLastError();
}

// ----------------------------------------------------------- transfers ---
// One thread per point p of a job.
//  X_ROW_RL: y = K(p,J) R^-1 L^-1  (far L2P rows; vertex / 1D M2M^T rows)
//  X_ROW_R : y = K(p,J) R^-1       (1D U rows)
//  X_COL_LR: y = R^-1 L^-1 K(I,p)  (semi-nested R^-1 L^-1 Ar columns)
//  X_COL_L : y = L^-1 K(I,p)       (1D V^T columns)
// The substitutions follow Eigen's triangularView::solve order as restated
// in the oracle, so transfer rows are bitwise the reference's for equal entries.
__global__ void xfer_kernel(const XferJob *__restrict__ jobs, const int32_t *__restrict__ idx, KParams kp,
                            const double *__restrict__ F, double *__restrict__ op) {
    const XferJob jb = jobs[blockIdx.y];
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= jb.n) return;
    const int r = jb.r;
    const double *A = F + jb.f;  // row-major r x r: R upper, L strictly lower
    const int32_t *J = idx + jb.jj;
    const int gp = idx[jb.pi + p];
    const bool row = jb.mode == X_ROW_RL || jb.mode == X_ROW_R;
    // Column-major outputs. ROW modes: element (p, j) of the n x r result at
    // a1 + j*ld1 + p; COL modes: element (i, p) of the r x n result at
    // a1 + p*ld1 + i. The output location is the working vector.
    double *y = row ? op + jb.a1 + p : op + jb.a1 + (int64_t)p * jb.ld1;
    const int64_t ys = row ? jb.ld1 : 1;
    for (int j = 0; j < r; ++j) y[j * ys] = kentry(kp, gp, J[j]);  // K(p,J) == K(J,p) bitwise
    if (row) {
        // z R = b (forward), then y L = z (backward, unit diagonal)
        for (int j = 0; j < r; ++j) {
            double s = y[j * ys];
            for (int q = 0; q < j; ++q) s = __dsub_rn(s, __dmul_rn(y[q * ys], A[q * r + j]));
            y[j * ys] = __ddiv_rn(s, A[j * r + j]);
        }
        if (jb.mode == X_ROW_RL)
            for (int j = r - 1; j >= 0; --j) {
                double s = y[j * ys];
                for (int q = j + 1; q < r; ++q) s = __dsub_rn(s, __dmul_rn(y[q * ys], A[q * r + j]));
                y[j * ys] = s;
            }
        // transposed copy: element (j, p) of the r x n result at a2 + p*ld2 + j
        if (jb.a2 >= 0)
            for (int j = 0; j < r; ++j) op[jb.a2 + (int64_t)p * jb.ld2 + j] = y[j * ys];
    } else {
        // L x = b (forward, unit diagonal), then R x = x (backward)
        for (int i = 0; i < r; ++i) {
            double s = y[i];
            for (int q = 0; q < i; ++q) s = __dsub_rn(s, __dmul_rn(A[i * r + q], y[q]));
            y[i] = s;
        }
        if (jb.mode == X_COL_LR)
            for (int i = r - 1; i >= 0; --i) {
                double s = y[i];
                for (int q = i + 1; q < r; ++q) s = __dsub_rn(s, __dmul_rn(A[i * r + q], y[q]));
                y[i] = __ddiv_rn(s, A[i * r + i]);
            }
    }
}

cudaError_t launch_xfer(const XferJob *jobs, int njobs, int max_n, const int32_t *idx, const KParams &kp,
                        const double *F, double *op, cudaStream_t st) {
    if (njobs == 0 || max_n == 0) return cudaSuccess;
    const int bs = 64;
    for (int j0 = 0; j0 < njobs; j0 += 65535) {
        int nj = njobs - j0 < 65535 ? njobs - j0 : 65535;
        dim3 grid((unsigned)((max_n + bs - 1) / bs), (unsigned)nj);
        xfer_kernel<<<grid, bs, 0, st>>>(jobs + j0, idx, kp, F, op);
        count_launch();
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// --------------------------------------------------------------- fills ---
__global__ void fill_kernel(const FillJob *__restrict__ jobs, const int32_t *__restrict__ idx, KParams kp,
                            double *__restrict__ op) {
    const FillJob jb = jobs[blockIdx.y];
    const int64_t total = (int64_t)jb.nr * jb.nc;
    const int32_t *R = idx + jb.ri, *C = idx + jb.ci;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        int c = (int)(e / jb.nr), i = (int)(e % jb.nr);
        op[jb.a + (int64_t)c * jb.lda + i] = kentry(kp, R[i], C[c]);
    }
}

cudaError_t launch_fill(const FillJob *jobs, int njobs, const int32_t *idx, const KParams &kp, double *op,
                        cudaStream_t st) {
    if (njobs == 0) return cudaSuccess;
    for (int j0 = 0; j0 < njobs; j0 += 65535) {
        int nj = njobs - j0 < 65535 ? njobs - j0 : 65535;
        dim3 grid(8, (unsigned)nj);
        fill_kernel<<<grid, 256, 0, st>>>(jobs + j0, idx, kp, op);
        count_launch();
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

__global__ void convert_f32_kernel(const double *__restrict__ s, float *__restrict__ d, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        d[i] = (float)s[i];
}
cudaError_t launch_convert_f32(const double *src, float *dst, int64_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    convert_f32_kernel<<<1216, 256, 0, st>>>(src, dst, n);
    count_launch(); return cudaGetLastError();
}

// ------------------------------------------------------- block-row GEMV ---
// Persistent block-row GEMV over column-major panels. A CTA takes targets
// t0 + blockIdx.x, + gridDim.x, ... (heaviest first, the host sorts them),
// copies the target's packed record into shared memory, gathers its sources
// (x through perm, or the workspace) into shared memory, then lets
// lane l of a warp own row l of a 32-row group while the warps of the CTA
// split the columns: every load is a coalesced 32-row column segment and
// each lane keeps several independent loads in flight. Partial sums of the
// column slices meet in shared memory.
constexpr int BRG_THREADS = 256;
constexpr int BRG_WARPS = BRG_THREADS / 32;

// Target record (int64 words), built by the host plan:
//   [0] dst   [1] nrows | flags << 32   [2] np | ns << 32
//   np panels x 3 words: a, lda | w << 32, xoff
//   ns segments x 2 words: src, len | (xoff << 1 | gather) << 32  (xoff: offset in the target's gathered x)
template <class T> struct Vec16;
template <> struct Vec16<double> { using type = double2; static constexpr int n = 2; };
template <> struct Vec16<float> { using type = float4; static constexpr int n = 4; };
__device__ __forceinline__ void vfma(double *acc, const double2 v, const double x) {
    acc[0] += v.x * x;
    acc[1] += v.y * x;
}
__device__ __forceinline__ void vfma(float *acc, const float4 v, const float x) {
    acc[0] += v.x * x;
    acc[1] += v.y * x;
    acc[2] += v.z * x;
    acc[3] += v.w * x;
}

template <class T> struct BrgShared {
    T xs[BRG_XS_ELEMS];
    T red[BRG_WARPS * 32 * Vec16<T>::n];
    int64_t rec[BRG_REC_WORDS];
};

// One target: rows [dst, dst+nrows) from its packed record (see above).
template <class T>
__device__ __forceinline__ void brg_target(BrgShared<T> &sh, int64_t t, const int64_t *__restrict__ roff,
                                           const int64_t *__restrict__ blob, const T *__restrict__ A, T *ws,
                                           const double *__restrict__ xin, double *yout,
                                           const int32_t *__restrict__ perm) {
    T *xs = sh.xs;
    T *red = sh.red;
    int64_t *rec = sh.rec;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t o = roff[t];
    const int nw = (int)(roff[t + 1] - o);
    for (int q = tid; q < nw; q += BRG_THREADS) rec[q] = blob[o + q];
    __syncthreads();
    const int64_t dst = rec[0];
    const int nrows = (int)(rec[1] & 0xffffffff), flags = (int)(rec[1] >> 32);
    const int np = (int)(rec[2] & 0xffffffff), ns = (int)(rec[2] >> 32);
    const int64_t *pan = rec + 3;
    const int64_t *seg = pan + 3 * np;
    // gather: every thread walks the segments for its elements
    {
        int sidx = 0;
        int64_t s_src = 0;
        int s_lo = 0, s_hi = -1, s_g = 0;
        auto seek = [&](int e) {
            while (e >= s_hi && sidx < ns) {
                const int64_t w1 = seg[2 * sidx + 1];
                s_src = seg[2 * sidx];
                const int len = (int)(w1 & 0xffffffff);
                const int code = (int)(w1 >> 32);
                s_lo = code >> 1;
                s_hi = s_lo + len;
                s_g = code & 1;
                ++sidx;
            }
        };
        // elements of the concatenated sources, in segment order
        int total = 0;
        if (ns > 0) {
            const int64_t wl = seg[2 * (ns - 1) + 1];
            total = (int)(wl >> 33) + (int)(wl & 0xffffffff);
        }
        for (int e0 = tid; e0 < total; e0 += 4 * BRG_THREADS) {
            int64_t idx4[4];
            int xo4[4], g4[4];
            int cnt = 0;
            for (int u = 0; u < 4; ++u) {
                const int e = e0 + u * BRG_THREADS;
                if (e >= total) break;
                seek(e);
                if (e < s_lo) {  // padding gap between panels
                    idx4[u] = -1;
                } else {
                    idx4[u] = s_src + (e - s_lo);
                }
                xo4[u] = e;
                g4[u] = s_g;
                ++cnt;
            }
            T v4[4];
            for (int u = 0; u < cnt; ++u) {
                const int64_t ix = idx4[u];
                if (ix < 0) v4[u] = T(0);
                else if (g4[u]) v4[u] = (T)xin[perm ? (int64_t)perm[ix] : ix];
                else v4[u] = ws[ix];
            }
            for (int u = 0; u < cnt; ++u) xs[xo4[u]] = v4[u];
        }
    }
    __syncthreads();
    // Rows in blocks of RB = 32*VN. Within a block, a warp's lane l owns the
    // VN-row slice rq = l % RQ (16-byte vector loads down a column) and
    // column phase cs = l / RQ, so one load instruction covers 32/RQ columns.
    // The warps of the CTA split the columns of each block.
    using V16 = typename Vec16<T>::type;
    constexpr int VN = Vec16<T>::n;
    constexpr int RB = 32 * VN;
    const int nblk = (nrows + RB - 1) / RB;
    for (int bb = 0; bb < nblk; bb += BRG_WARPS) {
        const int nb_here = nblk - bb < BRG_WARPS ? nblk - bb : BRG_WARPS;
        const int S = BRG_WARPS / nb_here;        // warps (column slices) per row block
        const int myb = warp % nb_here, sl = warp / nb_here;
        const int rb = (bb + myb) * RB;
        const int rows = nrows - rb < RB ? nrows - rb : RB;
        int RQ = 1;
        while (RQ * VN < rows) RQ <<= 1;          // row slices of this block (power of two <= 32)
        const int CS = 32 / RQ;                   // column phases per load
        const int rq = lane % RQ, cs = lane / RQ;
        const int r_lo = rb + rq * VN;            // first row of the lane's slice
        T acc[VN];
#pragma unroll
        for (int v = 0; v < VN; ++v) acc[v] = T(0);
        if (sl < S && r_lo < nrows) {
            for (int q = 0; q < np; ++q) {
                const int64_t pa = pan[3 * q];
                const int lda = (int)(pan[3 * q + 1] & 0xffffffff), w = (int)(pan[3 * q + 1] >> 32);
                const int xoff = (int)pan[3 * q + 2];
                const int c0 = (int)(((int64_t)w * sl) / S), c1 = (int)(((int64_t)w * (sl + 1)) / S);
                const T *xp = xs + xoff;
                const int64_t ld = lda;
                const T *base = A + pa + r_lo;
                if (((pa & 3) == 0) && ((lda & 3) == 0)) {
                    int c = c0 + cs;
                    for (; c + 3 * CS < c1; c += 4 * CS) {
                        const V16 v0 = *reinterpret_cast<const V16 *>(base + (int64_t)c * ld);
                        const V16 v1 = *reinterpret_cast<const V16 *>(base + (int64_t)(c + CS) * ld);
                        const V16 v2 = *reinterpret_cast<const V16 *>(base + (int64_t)(c + 2 * CS) * ld);
                        const V16 v3 = *reinterpret_cast<const V16 *>(base + (int64_t)(c + 3 * CS) * ld);
                        const T x0 = xp[c], x1 = xp[c + CS], x2 = xp[c + 2 * CS], x3 = xp[c + 3 * CS];
                        vfma(acc, v0, x0);
                        vfma(acc, v1, x1);
                        vfma(acc, v2, x2);
                        vfma(acc, v3, x3);
                    }
                    for (; c < c1; c += CS) vfma(acc, *reinterpret_cast<const V16 *>(base + (int64_t)c * ld), xp[c]);
                } else {
                    const int nv = nrows - r_lo < VN ? nrows - r_lo : VN;
                    for (int c = c0 + cs; c < c1; c += CS) {
                        const T xc = xp[c];
                        const T *col = base + (int64_t)c * ld;
#pragma unroll
                        for (int v = 0; v < VN; ++v)
                            if (v < nv) acc[v] += col[v] * xc;
                    }
                }
            }
        }
        // reduce over the column phases of the warp
#pragma unroll
        for (int v = 0; v < VN; ++v)
            for (int o = RQ; o < 32; o <<= 1) acc[v] += __shfl_xor_sync(0xffffffffu, acc[v], o);
        if (cs == 0 && sl < S)
#pragma unroll
            for (int v = 0; v < VN; ++v) red[warp * RB + rq * VN + v] = acc[v];
        __syncthreads();
        // combine the column slices of each block and write
        for (int e = tid; e < nb_here * RB; e += BRG_THREADS) {
            const int mb = e / RB, r = e % RB;
            const int i = (bb + mb) * RB + r;
            if (i >= nrows) continue;
            T v = T(0);
            for (int q = 0; q < S; ++q) v += red[(mb + q * nb_here) * RB + r];
            const int64_t d = dst + i;
            if (flags & T_SCATTER) {
                const T ov = (flags & T_ACCUM) ? ws[d] + v : v;
                yout[perm ? (int64_t)perm[d] : d] = (double)ov;
            } else if (flags & T_ATOMIC) {
                atomicAdd(ws + d, v);
            } else if (flags & T_ACCUM) {
                ws[d] += v;
            } else {
                ws[d] = v;
            }
        }
        __syncthreads();
    }
}

template <class T>
__global__ void __launch_bounds__(BRG_THREADS, 4)
    brg_kernel(const int64_t *__restrict__ roff, const int64_t *__restrict__ blob, int64_t t0, int64_t t1,
               const T *__restrict__ A, T *ws, const double *__restrict__ xin, double *yout,
               const int32_t *__restrict__ perm) {
    __shared__ BrgShared<T> sh;
    for (int64_t t = t0 + blockIdx.x; t < t1; t += gridDim.x) brg_target<T>(sh, t, roff, blob, A, ws, xin, yout, perm);
}

// The whole matvec in one cooperative launch: phases separated by grid
// barriers; targets of a phase striped over the CTAs.
template <class T>
__global__ void __launch_bounds__(BRG_THREADS, 4)
    brg_coop_kernel(const int64_t *__restrict__ roff, const int64_t *__restrict__ blob,
                    const int64_t *__restrict__ pstart, int nphase, const T *__restrict__ A, T *ws,
                    const double *__restrict__ xin, double *yout, const int32_t *__restrict__ perm, unsigned *bar,
                    int32_t *err, long long spin) {
    __shared__ BrgShared<T> sh;
    for (int p = 0; p < nphase; ++p) {
        const int64_t t1 = pstart[p + 1];
        for (int64_t t = pstart[p] + blockIdx.x; t < t1; t += gridDim.x)
            brg_target<T>(sh, t, roff, blob, A, ws, xin, yout, perm);
        if (p + 1 < nphase) grid_barrier(bar, gridDim.x, err, spin);
    }
}

// Dataflow form of brg_coop_kernel (no grid barriers), for FP64 products of operators without room for
// the copy that sv.cu streams: targets claimed in stored (topological) order from a
// global counter; each waits until its producer count rem[t] is zero (bounded spin: on timeout
// *err = 3 and the CTA proceeds), runs, fences its writes and decrements the counts of its
// consumers cidx[coff[t] .. coff[t+1]). Cooperative launch: every CTA is resident, so the
// producers of a waiting target are all claimed and running. 2D integral equation, 65536 points: 218 us,
// 320 with grid barriers (154 on the copy); 3D semi-nested RBF, 20011 points: 667, 752 (428).
__global__ void __launch_bounds__(BRG_THREADS, 4)
    brg_flow_kernel(const int64_t *__restrict__ roff, const int64_t *__restrict__ blob, int64_t nt, int32_t *ctr,
                    int32_t *rem, const int64_t *__restrict__ coff, const int32_t *__restrict__ cidx,
                    const double *__restrict__ A, double *ws, const double *__restrict__ xin, double *yout,
                    const int32_t *__restrict__ perm, int32_t *err) {
    __shared__ BrgShared<double> sh;
    __shared__ int64_t s_next;
    int64_t t = blockIdx.x;
    while (t < nt) {
        if (threadIdx.x == 0) {
            long long it = 0;
            while (*((volatile int32_t *)(rem + t)) > 0) {
                if (++it > (1LL << 20)) {  // about 0.1 s
                    atomicExch(err, 3);
                    break;
                }
                __nanosleep(32);
            }
            __threadfence();
        }
        __syncthreads();
        brg_target<double>(sh, t, roff, blob, A, ws, xin, yout, perm);
        __syncthreads();
        if (threadIdx.x < 32) {
            __threadfence();  // this CTA's results are visible before its consumers are released
            for (int64_t e = coff[t] + threadIdx.x; e < coff[t + 1]; e += 32) atomicSub(rem + cidx[e], 1);
            if (threadIdx.x == 0) s_next = gridDim.x + atomicAdd(ctr, 1);
        }
        __syncthreads();
        t = s_next;
    }
}

// Many independent problems in one cooperative launch: the problem index of
// a target sits in bits 8.. of its record's flag word, and the target runs
// on that problem's operator, workspace, point permutation and vector
// segment (xoff into the concatenated input and output vectors). active
// (may be NULL): a problem whose entry is not -1 (a converged system of the
// lockstep solver) is skipped.
template <class T>
__global__ void __launch_bounds__(BRG_THREADS, 4)
    brgb_coop_kernel(const int64_t *__restrict__ roff, const int64_t *__restrict__ blob,
                     const int64_t *__restrict__ pstart, int nphase, const BatchProb *__restrict__ probs,
                     const int32_t *__restrict__ active, const double *__restrict__ xin, double *yout,
                     unsigned *bar, int32_t *err) {
    __shared__ BrgShared<T> sh;
    for (int p = 0; p < nphase; ++p) {
        const int64_t t1 = pstart[p + 1];
        for (int64_t t = pstart[p] + blockIdx.x; t < t1; t += gridDim.x) {
            const int pid = (int)(blob[roff[t] + 1] >> 40);
            if (active && active[pid] != -1) continue;
            const BatchProb pr = probs[pid];
            brg_target<T>(sh, t, roff, blob, reinterpret_cast<const T *>(pr.A), reinterpret_cast<T *>(pr.ws),
                          xin + pr.xoff, yout + pr.xoff, pr.perm);
        }
        if (p + 1 < nphase) grid_barrier(bar, gridDim.x, err);
    }
}

template <class T>
static cudaError_t launch_brg_t(const int64_t *roff, const int64_t *blob, int64_t t0, int64_t t1, const T *A, T *ws,
                                const double *xin, double *yout, const int32_t *perm, cudaStream_t st) {
    if (t1 <= t0) return cudaSuccess;
    static PerDevice<int> per_sm_of;
    int &per_sm = per_sm_of.here();
    if (per_sm == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, brg_kernel<T>, BRG_THREADS, 0);
        if (per_sm <= 0) per_sm = 1;
    }
    const int64_t nt = t1 - t0;
    const int64_t cap = (int64_t)device_sms() * per_sm;
    const int grid = (int)(nt < cap ? nt : cap);
    brg_kernel<T><<<grid, BRG_THREADS, 0, st>>>(roff, blob, t0, t1, A, ws, xin, yout, perm);
    count_launch();
    return cudaGetLastError();
}

template <class T>
static cudaError_t launch_coop_t(const int64_t *roff, const int64_t *blob, const int64_t *pstart, int nphase,
                                 const T *A, T *ws, const double *xin, double *yout, const int32_t *perm,
                                 unsigned *bar, int32_t *err, long long spin, cudaStream_t st) {
    if (nphase <= 0) return cudaSuccess;
    if (spin <= 0) spin = GRID_SPIN_LIMIT;
    static PerDevice<int> per_sm_of;
    int &per_sm = per_sm_of.here();
    if (per_sm == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, brg_coop_kernel<T>, BRG_THREADS, 0);
        if (per_sm <= 0) return cudaErrorCooperativeLaunchTooLarge;
    }
    const int grid = device_sms() * per_sm;
    void *args[] = {(void *)&roff, (void *)&blob, (void *)&pstart, (void *)&nphase, (void *)&A, (void *)&ws,
                    (void *)&xin, (void *)&yout, (void *)&perm, (void *)&bar, (void *)&err, (void *)&spin};
    cudaError_t e = cudaLaunchCooperativeKernel((const void *)brg_coop_kernel<T>, dim3(grid), dim3(BRG_THREADS), args,
                                                0, st);
    count_launch();
    return e;
}

cudaError_t launch_brg_flow_f64(const int64_t *roff, const int64_t *blob, int64_t nt, int32_t *ctr, int32_t *rem,
                                const int64_t *coff, const int32_t *cidx, const double *A, double *ws,
                                const double *xin, double *yout, const int32_t *perm, int32_t *err, cudaStream_t st) {
    if (nt <= 0) return cudaSuccess;
    static PerDevice<int> per_sm_of;
    int &per_sm = per_sm_of.here();
    if (per_sm == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, brg_flow_kernel, BRG_THREADS, 0);
        if (per_sm <= 0) return cudaErrorCooperativeLaunchTooLarge;
    }
    const int grid = device_sms() * per_sm;
    void *args[] = {(void *)&roff, (void *)&blob, (void *)&nt, (void *)&ctr, (void *)&rem,  (void *)&coff, (void *)&cidx,
                    (void *)&A,    (void *)&ws,   (void *)&xin, (void *)&yout, (void *)&perm, (void *)&err};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void *)brg_flow_kernel, dim3(grid), dim3(BRG_THREADS), args, 0, st);
    count_launch();
    return e;
}

cudaError_t launch_coop_f64(const int64_t *roff, const int64_t *blob, const int64_t *pstart, int nphase,
                            const double *A, double *ws, const double *xin, double *yout, const int32_t *perm,
                            unsigned *bar, int32_t *err, cudaStream_t st, long long spin) {
    return launch_coop_t<double>(roff, blob, pstart, nphase, A, ws, xin, yout, perm, bar, err, spin, st);
}
cudaError_t launch_coop_f32(const int64_t *roff, const int64_t *blob, const int64_t *pstart, int nphase,
                            const float *A, float *ws, const double *xin, double *yout, const int32_t *perm,
                            unsigned *bar, int32_t *err, cudaStream_t st, long long spin) {
    return launch_coop_t<float>(roff, blob, pstart, nphase, A, ws, xin, yout, perm, bar, err, spin, st);
}

template <class T>
static cudaError_t launch_brgb_t(const int64_t *roff, const int64_t *blob, const int64_t *pstart, int nphase,
                                 const BatchProb *probs, const int32_t *active, const double *xin, double *yout,
                                 unsigned *bar, int32_t *err, cudaStream_t st) {
    if (nphase <= 0) return cudaSuccess;
    static PerDevice<int> per_sm_of;
    int &per_sm = per_sm_of.here();
    if (per_sm == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, brgb_coop_kernel<T>, BRG_THREADS, 0);
        if (per_sm <= 0) return cudaErrorCooperativeLaunchTooLarge;
    }
    const int grid = device_sms() * per_sm;
    void *args[] = {(void *)&roff, (void *)&blob, (void *)&pstart, (void *)&nphase, (void *)&probs,
                    (void *)&active, (void *)&xin, (void *)&yout,  (void *)&bar,    (void *)&err};
    cudaError_t e = cudaLaunchCooperativeKernel((const void *)brgb_coop_kernel<T>, dim3(grid), dim3(BRG_THREADS), args,
                                                0, st);
    count_launch();
    return e;
}
cudaError_t launch_brgb_f64(const int64_t *roff, const int64_t *blob, const int64_t *pstart, int nphase,
                            const BatchProb *probs, const int32_t *active, const double *xin, double *yout,
                            unsigned *bar, int32_t *err, cudaStream_t st) {
    return launch_brgb_t<double>(roff, blob, pstart, nphase, probs, active, xin, yout, bar, err, st);
}
cudaError_t launch_brg_f64(const int64_t *roff, const int64_t *blob, int64_t t0, int64_t t1, const double *A,
                           double *ws, const double *xin, double *yout, const int32_t *perm, cudaStream_t st) {
    return launch_brg_t<double>(roff, blob, t0, t1, A, ws, xin, yout, perm, st);
}
cudaError_t launch_brg_f32(const int64_t *roff, const int64_t *blob, int64_t t0, int64_t t1, const float *A,
                           float *ws, const double *xin, double *yout, const int32_t *perm, cudaStream_t st) {
    return launch_brg_t<float>(roff, blob, t0, t1, A, ws, xin, yout, perm, st);
}

template <class T>
__global__ void scatter_kernel2(const T *__restrict__ yp, double *__restrict__ y, const int32_t *__restrict__ perm,
                                int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[perm[i]] = (double)yp[i];
}
cudaError_t launch_scatter_f64(const double *yp, double *y, const int32_t *perm, int64_t n, cudaStream_t st) {
    scatter_kernel2<double><<<608, 256, 0, st>>>(yp, y, perm, n);
    count_launch(); return cudaGetLastError();
}
__global__ void gather_kernel(const double *__restrict__ x, double *__restrict__ xp, const int32_t *__restrict__ perm,
                              int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        xp[i] = x[perm[i]];
}
cudaError_t launch_gather_f64(const double *x, double *xp, const int32_t *perm, int64_t n, cudaStream_t st) {
    gather_kernel<<<608, 256, 0, st>>>(x, xp, perm, n);
    count_launch(); return cudaGetLastError();
}
cudaError_t launch_scatter_f32(const float *yp, double *y, const int32_t *perm, int64_t n, cudaStream_t st) {
    scatter_kernel2<float><<<608, 256, 0, st>>>(yp, y, perm, n);
    count_launch(); return cudaGetLastError();
}

// -------------------------------------------------------- dense oracle ---
__global__ void dense_kernel(KParams kp, int64_t N, const double *__restrict__ x, double *__restrict__ y,
                             int64_t row0) {
    __shared__ double sh[32];
    const int64_t r = row0 + blockIdx.x;
    double acc = 0.0;
    for (int64_t j = threadIdx.x; j < N; j += blockDim.x) acc += kentry(kp, (int)r, (int)j) * x[j];
    acc = block_sum(acc, sh);
    if (threadIdx.x == 0) y[blockIdx.x] = acc;
}
// Dense FP64 rows y[i] = sum_j K(rows[i], j) x[j] for a list of rows.
__global__ void dense_rows_kernel(KParams kp, int64_t N, const double *__restrict__ x,
                                  const int64_t *__restrict__ rows, double *__restrict__ y) {
    __shared__ double sh[32];
    const int64_t r = rows[blockIdx.x];
    double acc = 0.0;
    for (int64_t j = threadIdx.x; j < N; j += blockDim.x) acc += kentry(kp, (int)r, (int)j) * x[j];
    acc = block_sum(acc, sh);
    if (threadIdx.x == 0) y[blockIdx.x] = acc;
}
cudaError_t launch_dense_rows(const KParams &kp, int64_t N, const double *x, const int64_t *rows, int64_t nrows,
                              double *y, cudaStream_t st) {
    for (int64_t b = 0; b < nrows; b += 2147483647LL) {
        int64_t nb = nrows - b < 2147483647LL ? nrows - b : 2147483647LL;
        dense_rows_kernel<<<(unsigned)nb, 256, 0, st>>>(kp, N, x, rows + b, y + b);
        count_launch();
    }
    return cudaGetLastError();
}
cudaError_t launch_dense_matvec(const KParams &kp, int64_t N, const double *x, double *y, int64_t row0, int64_t nrows,
                                cudaStream_t st) {
    for (int64_t b = 0; b < nrows; b += 2147483647LL) {
        int64_t nb = nrows - b < 2147483647LL ? nrows - b : 2147483647LL;
        dense_kernel<<<(unsigned)nb, 256, 0, st>>>(kp, N, x, y + b, row0 + b);
        count_launch();
    }
    return cudaGetLastError();
}

// --------------------------------------------------------------- GMRES ---
// Classical Gram-Schmidt with one reorthogonalisation (CGS2), FP64, on a
// device-resident Krylov basis. CTA b owns rows [b*chunk, (b+1)*chunk).
__device__ __forceinline__ void gm_rows(int64_t N, int nblk, int64_t &r0, int64_t &r1) {
    int64_t chunk = (N + nblk - 1) / nblk;
    r0 = (int64_t)blockIdx.x * chunk < N ? (int64_t)blockIdx.x * chunk : N;
    r1 = r0 + chunk < N ? r0 + chunk : N;
}

__device__ void gm_apply(double &dx, double &dy, double cs, double sn) {
    double temp = __dadd_rn(__dmul_rn(cs, dx), __dmul_rn(sn, dy));
    dy = __dadd_rn(__dmul_rn(-sn, dx), __dmul_rn(cs, dy));
    dx = temp;
}

// One Arnoldi step after the product w = A v_i: two Gram-Schmidt passes, the norm, the
// next basis vector, the Givens rotations of column i, the convergence test and (cond)
// the loop condition of the captured step, as one cooperative launch with three grid
// barriers. A CTA keeps its rows of w in shared memory (ws_rows > 0; else in g.w), and
// those of the first vcap basis vectors, which the first pass reads from memory
// and the other three sweeps from there. Dots: a warp per basis vector (and row share,
// while there are fewer vectors than warps), whose lanes stride the rows: with few rows a
// CTA the shuffles of a warp sum cost the FP64 pipe as much as the multiply-adds, so
// there is one sum a vector, not one a vector and warp. Every CTA then sums the
// partials of all CTAs itself, a warp a vector. What bounds it: latency, the barriers and
// the chains of reads between them; past 1e5 rows, the FP64 pipe. A 7-step solve of 32768
// rows: 29 us a step (cold caches), where five launches, whose CTAs each summed the
// partials in one thread, took 54.
constexpr int GMS_THREADS = 512, GMS_WARPS = GMS_THREADS / 32;

// A CTA's rows of basis vector k
struct GmCols {
    const double *V;  // this CTA's rows of vector 0
    int64_t N;
    double *vsh;      // copies of the first vcap
    int rows, vcap;
    __device__ __forceinline__ const double *col(int k) const { return k < vcap ? vsh + (size_t)k * rows : V + (size_t)k * N; }
};

// out[k] = sum over this CTA's rows of V[., k] w, k <= i, then over all CTAs in h[k];
// first: the copies are made
__device__ void gm_dots_all(const GmresDev &g, const GmCols &C, int i, bool first, const double *w, double *red,
                            double *part, double *h) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nk = i + 1, S = nk < GMS_WARPS ? GMS_WARPS / nk : 1, rows = C.rows;
    __syncthreads();  // w is written
    for (int e = warp; e < nk * S; e += GMS_WARPS) {
        const int k = e % nk, sl = e / nk;
        const double *v = first ? C.V + (size_t)k * C.N : C.col(k);
        double *to = first && k < C.vcap ? C.vsh + (size_t)k * rows : nullptr;
        double acc = 0.0;
#pragma unroll 4
        for (int t = sl * 32 + lane; t < rows; t += 32 * S) {
            const double x = v[t];
            if (to) to[t] = x;
            acc = fma(x, w[t], acc);
        }
        acc = warp_sum(acc);
        if (lane == 0) red[e] = acc;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nk; k += GMS_THREADS) {
        double s = 0.0;
        for (int sl = 0; sl < S; ++sl) s += red[sl * nk + k];
        part[(size_t)k * g.nblk + blockIdx.x] = s;
    }
    grid_barrier(g.bar, gridDim.x, g.err);
    for (int k = warp; k < nk; k += GMS_WARPS) {
        double s = 0.0;
        for (int b = lane; b < g.nblk; b += 32) s += __ldcg(part + (size_t)k * g.nblk + b);
        s = warp_sum(s);
        if (lane == 0) h[k] = s;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(GMS_THREADS)
    gm_step(GmresDev g, int ws_rows, int vcap, cudaGraphConditionalHandle hnd, int cond) {
    extern __shared__ double gsh[];
    __shared__ double s_hn, s_ih, sh[32];
    double *h1 = gsh, *h2 = h1 + g.m + 1, *red = h2 + g.m + 1, *wsh = red + g.m + 1 + GMS_WARPS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int i = *g.iter;
    const bool done = g.scal[2] != 0.0;  // CTA 0 changes these two only after the last barrier
    if (done) {
        if (cond && blockIdx.x == 0 && tid == 0) cudaGraphSetConditional(hnd, 0u);
        return;
    }
    int64_t r0, r1;
    gm_rows(g.N, g.nblk, r0, r1);
    const int rows = (int)(r1 - r0);
    double *w = ws_rows > 0 ? wsh : g.w + r0;
    const GmCols C{g.V + r0, g.N, wsh + ws_rows, rows, vcap};
    if (ws_rows > 0)
        for (int t = tid; t < rows; t += GMS_THREADS) w[t] = g.w[r0 + t];
    const size_t ps = (size_t)g.nblk * (g.m + 1);
    double nrm = 0.0;
    for (int pass = 0; pass < 2; ++pass) {
        double *h = pass == 0 ? h1 : h2;
        gm_dots_all(g, C, i, pass == 0, w, red, g.part + pass * ps, h);
        nrm = 0.0;
        for (int t = tid; t < rows; t += GMS_THREADS) {
            double x = w[t];
#pragma unroll 4
            for (int k = 0; k <= i; ++k) x -= C.col(k)[t] * h[k];
            w[t] = x;
            nrm = fma(x, x, nrm);
        }
    }
    nrm = block_sum(nrm, sh);
    if (tid == 0) g.part[2 * ps + blockIdx.x] = nrm;
    grid_barrier(g.bar, gridDim.x, g.err);
    if (warp == 0) {
        double s = 0.0;
        for (int b = lane; b < g.nblk; b += 32) s += __ldcg(g.part + 2 * ps + b);
        s = warp_sum(s);
        if (lane == 0) {
            s_hn = sqrt(s);
            s_ih = 1.0 / s_hn;
        }
    }
    __syncthreads();
    const double hn = s_hn;
    // the first warp of CTA 0 does the rotations meanwhile
    const bool rot = blockIdx.x == 0 && warp == 0;
    if (!rot) {
        const double ih = s_ih;
        const int first = blockIdx.x == 0 ? 32 : 0;
        double *Vn = g.V + (size_t)(i + 1) * g.N + r0;
        for (int t = tid - first; t < rows; t += GMS_THREADS - first) {
            const double v = ih * w[t];
            Vn[t] = v;
            g.vcur[r0 + t] = v;
        }
        return;
    }
    // Givens rotations on column i (*/codes/gmres.hpp:30-75,156-162); resid = |s(i+1)| / ||b||.
    // h1: the column; red and h2: the earlier rotations
    for (int k = lane; k <= i; k += 32) {
        h1[k] += h2[k];
        if (k < i) {
            red[k] = g.cs[k];
            h2[k] = g.sn[k];
        }
    }
    __syncwarp();
    if (lane == 0) {
        double next = hn;
        for (int k = 0; k < i; ++k) gm_apply(h1[k], h1[k + 1], red[k], h2[k]);
        double dx = h1[i], dy = next, cs, sn;
        if (dy == 0.0) { cs = 1.0; sn = 0.0; }
        else if (fabs(dy) > fabs(dx)) {
            double temp = dx / dy;
            sn = 1.0 / sqrt(1.0 + temp * temp);
            cs = temp * sn;
        } else {
            double temp = dy / dx;
            cs = 1.0 / sqrt(1.0 + temp * temp);
            sn = temp * cs;
        }
        g.cs[i] = cs;
        g.sn[i] = sn;
        gm_apply(h1[i], next, cs, sn);
        g.H[(size_t)i * (g.m + 1) + i + 1] = next;
        gm_apply(g.s[i], g.s[i + 1], cs, sn);
        const double resid = fabs(g.s[i + 1]) / g.scal[0];
        g.scal[1] = resid;
        if (resid < g.scal[6]) g.scal[2] = 1.0;
        else if (i + 1 < g.m) *g.iter = i + 1;
        const int c = ++g.iter[1];
        if (cond) cudaGraphSetConditional(hnd, (!(resid < g.scal[6]) && c < g.m) ? 1u : 0u);
    }
    __syncwarp();
    for (int k = lane; k <= i; k += 32) g.H[(size_t)i * (g.m + 1) + k] = h1[k];
}

__global__ void gm_backsub(GmresDev g, double *__restrict__ y);

int gmres_blocks(int64_t N) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // one CTA an SM at most, and at least a row a thread: more CTAs only add partials to sum
    const int64_t want = (N + GMS_THREADS - 1) / GMS_THREADS;
    return (int)(want < 1 ? 1 : want < sms ? want : sms > 0 ? sms : 1);
}

// One-time function attributes of the Arnoldi kernels (done before any
// stream capture of an Arnoldi step).
void gmres_prepare() {
    static PerDevice<bool> cfg_of;
    bool &cfg = cfg_of.here();
    if (!cfg) {
        cudaFuncSetAttribute(gm_step, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(gm_backsub, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cfg = true;
    }
}

cudaError_t gmres_step(const GmresDev &g, const cudaGraphConditionalHandle *hnd, cudaStream_t st) {
    gmres_prepare();
    const int64_t chunk = (g.N + g.nblk - 1) / g.nblk;
    const size_t head = ((size_t)3 * (g.m + 1) + GMS_WARPS) * sizeof(double), most = 200 * 1024;
    if (head > most) return cudaErrorInvalidValue;
    int ws_rows = head + (size_t)chunk * 8 <= most ? (int)chunk : 0;
    const size_t left = ws_rows > 0 ? (most - head) / 8 - (size_t)chunk : 0;
    int vcap = (int)(left / (size_t)chunk < (size_t)g.m + 1 ? left / (size_t)chunk : (size_t)g.m + 1);
    const size_t smem = head + ((size_t)ws_rows + (size_t)vcap * chunk) * 8;
    GmresDev ga = g;
    cudaGraphConditionalHandle h = hnd ? *hnd : cudaGraphConditionalHandle{};
    int cond = hnd ? 1 : 0;
    void *args[] = {(void *)&ga, (void *)&ws_rows, (void *)&vcap, (void *)&h, (void *)&cond};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void *)gm_step, dim3(g.nblk), dim3(GMS_THREADS), args, smem, st);
    count_launch();
    return e;
}

// r = b - Ax (Ax NULL: r = b); beta = ||r||; V[:,0] = vcur = r / beta; s = beta e1; iter = 0;
// normb = ||b|| (1 if b = 0); converged (scal[2] = 2) if beta / normb <= tol
__global__ void gm_resid_part(GmresDev g, const double *__restrict__ b, const double *__restrict__ Ax) {
    __shared__ double sh[32];
    int64_t r0, r1;
    gm_rows(g.N, g.nblk, r0, r1);
    double acc = 0.0, bb = 0.0;
    for (int64_t t = r0 + threadIdx.x; t < r1; t += blockDim.x) {
        const double v = b[t], r = Ax ? v - Ax[t] : v;  // Ax == NULL: x0 = 0
        g.w[t] = r;
        acc += r * r;
        bb += v * v;
    }
    acc = block_sum(acc, sh);
    bb = block_sum(bb, sh);
    if (threadIdx.x == 0) {
        g.part[blockIdx.x] = acc;
        g.part[g.nblk + blockIdx.x] = bb;
    }
}
__global__ void gm_start_fin(GmresDev g) {
    __shared__ double sh[32];
    double r2 = 0.0, b2 = 0.0;
    for (int b = threadIdx.x; b < g.nblk; b += blockDim.x) {
        r2 += g.part[b];
        b2 += g.part[g.nblk + b];
    }
    r2 = block_sum(r2, sh);
    b2 = block_sum(b2, sh);
    __shared__ double s_v[3];
    if (threadIdx.x == 0) {  // one root and quotient a CTA: the FP64 pipe is slow at them
        s_v[0] = sqrt(r2);
        s_v[1] = 1.0 / s_v[0];
        s_v[2] = b2 == 0.0 ? 1.0 : sqrt(b2);
    }
    __syncthreads();
    const double beta = s_v[0], ib = s_v[1], normb = s_v[2];
    if (blockIdx.x == 0) {
        for (int k = threadIdx.x; k <= g.m; k += blockDim.x) {
            g.s[k] = k == 0 ? beta : 0.0;
            g.cs[k] = 0.0;
            g.sn[k] = 0.0;
        }
        if (threadIdx.x == 0) {
            g.scal[0] = normb;
            g.scal[1] = beta / normb;
            g.scal[2] = beta / normb <= g.scal[6] ? 2.0 : 0.0;
            g.scal[3] = beta;
            g.iter[0] = 0;
            g.iter[1] = 0;  // Arnoldi steps taken
        }
    }
    int64_t r0, r1;
    gm_rows(g.N, g.nblk, r0, r1);
    for (int64_t t = r0 + threadIdx.x; t < r1; t += blockDim.x) {
        double v = g.w[t] * ib;
        g.V[t] = v;
        g.vcur[t] = v;
    }
}
cudaError_t gmres_start(const GmresDev &g, const double *b, const double *Ax, cudaStream_t st) {
    gm_resid_part<<<g.nblk, GM_THREADS, 0, st>>>(g, b, Ax);
    gm_start_fin<<<g.nblk, GM_THREADS, 0, st>>>(g);
    count_launch(2); return cudaGetLastError();
}

// The triangular least-squares system H(0:k,0:k) y = s(0:k), k the last column
// (*/codes/gmres.hpp:77-90), into y; nothing if converged at the start. One CTA: a
// column's updates in parallel, the columns in turn, each entry's operations in
// the order of the plain double loop.
__global__ void gm_backsub(GmresDev g, double *__restrict__ y) {
    extern __shared__ double ysh[];
    if (g.scal[2] == 2.0) return;
    const int k = g.iter[0];
    for (int j = threadIdx.x; j <= k; j += blockDim.x) ysh[j] = g.s[j];
    for (int i = k; i >= 0; --i) {
        const double *Hc = g.H + (size_t)i * (g.m + 1);
        __syncthreads();
        const double yi = ysh[i] / Hc[i];  // (every thread: they wait for it anyway)
        __syncthreads();
        for (int j = threadIdx.x; j < i; j += blockDim.x) ysh[j] = __dsub_rn(ysh[j], __dmul_rn(Hc[j], yi));
        if (threadIdx.x == 0) ysh[i] = yi;
    }
    __syncthreads();
    for (int j = threadIdx.x; j <= k; j += blockDim.x) y[j] = ysh[j];
}
// x += sum_{j<=k} V[:,j] y[j]
__global__ void gm_xupdate(GmresDev g, double *__restrict__ x, const double *__restrict__ y) {
    if (g.scal[2] == 2.0) return;
    const int k = g.iter[0];
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < g.N; t += (int64_t)gridDim.x * blockDim.x) {
        double v = x[t];
#pragma unroll 4
        for (int j = 0; j <= k; ++j) v += g.V[(size_t)j * g.N + t] * y[j];
        x[t] = v;
    }
}
cudaError_t gmres_update(const GmresDev &g, double *x, double *y, cudaStream_t st) {
    gm_backsub<<<1, 128, (size_t)(g.m + 1) * sizeof(double), st>>>(g, y);
    const int64_t nb = (g.N + GM_THREADS - 1) / GM_THREADS;
    gm_xupdate<<<(unsigned)(nb < 1216 ? nb : 1216), GM_THREADS, 0, st>>>(g, x, y);
    count_launch(2); return cudaGetLastError();
}

__global__ void norm_part(const double *__restrict__ x, int64_t n, double *part) {
    __shared__ double sh[32];
    double acc = 0.0;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        acc += x[t] * x[t];
    acc = block_sum(acc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = acc;
}
__global__ void norm_fin(const double *part, int nblk, double *out) {
    __shared__ double sh[32];
    double s = 0.0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) s += part[b];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) *out = sqrt(s);
}
cudaError_t vec_norm(const double *x, int64_t n, double *part, int nblk, double *out, cudaStream_t st) {
    norm_part<<<nblk, GM_THREADS, 0, st>>>(x, n, part);
    norm_fin<<<1, GM_THREADS, 0, st>>>(part, nblk, out);
    count_launch(2); return cudaGetLastError();
}

__global__ void axpby_kernel(double a, const double *x, double b, const double *y, double *z, int64_t n) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        z[t] = a * x[t] + b * y[t];
}
cudaError_t vec_axpby(double a, const double *x, double b, const double *y, double *z, int64_t n, cudaStream_t st) {
    axpby_kernel<<<608, 256, 0, st>>>(a, x, b, y, z, n);
    count_launch(); return cudaGetLastError();
}
__global__ void d2f_kernel(const double *x, float *y, int64_t n) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        y[t] = (float)x[t];
}
__global__ void f2d_kernel(const float *x, double *y, int64_t n) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        y[t] = (double)x[t];
}
cudaError_t vec_f64_to_f32(const double *x, float *y, int64_t n, cudaStream_t st) {
    d2f_kernel<<<608, 256, 0, st>>>(x, y, n);
    count_launch(); return cudaGetLastError();
}
cudaError_t vec_f32_to_f64(const float *x, double *y, int64_t n, cudaStream_t st) {
    f2d_kernel<<<608, 256, 0, st>>>(x, y, n);
    count_launch(); return cudaGetLastError();
}

}  // namespace h2w
