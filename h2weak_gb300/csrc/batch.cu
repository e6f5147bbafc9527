// Segmented GMRES for many independent problems (sm_103a).
//
// P systems of different sizes run the reference's unrestarted GMRES
// (*/codes/gmres.hpp:92-200) in lockstep over one concatenated vector:
// problem p owns a contiguous row range, every CTA works on rows of one
// problem only, so a CTA's partial sums belong to one problem and a
// per-problem reduction over that problem's CTAs gives its dot products.
// CGS2 orthogonalisation, Givens rotations, stopping test and back
// substitution are per problem; one problem's numbers never mix with
// another's. A converged problem keeps its state.
#include "kernels.cuh"

namespace h2w {

constexpr int GMS_THREADS = 256;
constexpr int GMS_WARPS = GMS_THREADS / 32;

__device__ __forceinline__ double gms_warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ size_t gms_h(const GmresSeg &g, int p, int row, int col) {
    return ((size_t)p * g.m + col) * (g.m + 1) + row;
}

// out[blk*(m+1) + k] = sum over the block's rows of a_k[t] * b[t], k < kn,
// a_k = a + k*Ntot: a warp a vector (and row share, while there are fewer vectors than
// warps), so that the FP64 pipe sees one warp sum a vector. red: 4 * GMS_WARPS doubles.
__device__ void gms_block_dots(const GmresSeg &g, const double *a, const double *b, int kn, double *red,
                               double *out) {
    const int64_t r0 = g.brow[blockIdx.x];
    const int rows = (int)(g.brow[blockIdx.x + 1] - r0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = kn < GMS_WARPS ? GMS_WARPS / kn : 1;
    out += (size_t)blockIdx.x * (g.m + 1);
    for (int e = warp; e < kn * S; e += GMS_WARPS) {
        const int k = e % kn, sl = e / kn;
        const double *v = a + (size_t)k * g.Ntot + r0;
        double acc = 0.0;
#pragma unroll 4
        for (int t = sl * 32 + lane; t < rows; t += 32 * S) acc = fma(v[t], b[r0 + t], acc);
        acc = gms_warp_sum(acc);
        if (lane == 0) {
            if (S == 1) out[k] = acc;
            else red[e] = acc;
        }
    }
    if (S == 1) return;
    __syncthreads();
    for (int k = threadIdx.x; k < kn; k += GMS_THREADS) {
        double s = 0.0;
        for (int sl = 0; sl < S; ++sl) s += red[sl * kn + k];
        out[k] = s;
    }
}

// Blocks of problems that are no longer running (converged) skip the
// Arnoldi step's vector work: their state is frozen.
__global__ void gms_dots(GmresSeg g) {
    __shared__ double red[4 * GMS_WARPS];
    if (g.conv[g.bprob[blockIdx.x]] != -1) return;
    gms_block_dots(g, g.V, g.w, *g.iter + 1, red, g.part);
}

// hsum[p*(m+1) + k] = sum over problem p's blocks of part[b*(m+1) + k], k <= i
// (all = 1) or k = 0 (all = 0); block p
__global__ void gms_reduce(GmresSeg g, int all) {
    const int p = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kn = all ? *g.iter + 1 : 1;
    const int b0 = g.pblk[p], b1 = g.pblk[p + 1];
    for (int k = warp; k < kn; k += blockDim.x >> 5) {  // a warp a sum
        double s = 0.0;
        for (int b = b0 + lane; b < b1; b += 32) s += g.part[(size_t)b * (g.m + 1) + k];
        s = gms_warp_sum(s);
        if (lane == 0) g.hsum[(size_t)p * (g.m + 1) + k] = s;
    }
}

// h = hsum of the block's problem; H(:, i) (=|+=) h (the problem's first
// block); w -= V h; then new dots (pass 0) or ||w||^2 partials (pass 1)
__global__ void gms_update(GmresSeg g, int pass) {
    extern __shared__ double gms_sm[];
    double *h = gms_sm;
    double *red = gms_sm + (g.m + 1);
    const int i = *g.iter, p = g.bprob[blockIdx.x];
    if (g.conv[p] != -1) return;
    for (int k = threadIdx.x; k <= i; k += blockDim.x) h[k] = g.hsum[(size_t)p * (g.m + 1) + k];
    __syncthreads();
    if (blockIdx.x == g.pblk[p])
        for (int k = threadIdx.x; k <= i; k += blockDim.x) {
            double *Hk = g.H + gms_h(g, p, k, i);
            *Hk = pass == 0 ? h[k] : *Hk + h[k];
        }
    const int64_t r0 = g.brow[blockIdx.x], r1 = g.brow[blockIdx.x + 1];
    for (int64_t t = r0 + threadIdx.x; t < r1; t += GMS_THREADS) {
        double v = g.w[t];
        for (int k = 0; k <= i; ++k) v -= g.V[(size_t)k * g.Ntot + t] * h[k];
        g.w[t] = v;
    }
    __syncthreads();
    if (pass == 0) gms_block_dots(g, g.V, g.w, i + 1, red, g.part);
    else gms_block_dots(g, g.w, g.w, 1, red, g.part);
}

// H(i+1, i) = ||w||; V[:, i+1] = vcur = w / ||w|| (a zero segment stays zero)
__global__ void gms_normalise(GmresSeg g) {
    const int i = *g.iter, p = g.bprob[blockIdx.x];
    if (g.conv[p] != -1) return;
    __shared__ double s_ih;
    if (threadIdx.x == 0) {  // one root and quotient a CTA: the FP64 pipe is slow at them
        const double hn = sqrt(g.hsum[(size_t)p * (g.m + 1)]);
        if (blockIdx.x == g.pblk[p]) g.H[gms_h(g, p, i + 1, i)] = hn;
        s_ih = hn > 0.0 ? 1.0 / hn : 0.0;
    }
    __syncthreads();
    const double ih = s_ih;
    double *Vn = g.V + (size_t)(i + 1) * g.Ntot;
    const int64_t r0 = g.brow[blockIdx.x], r1 = g.brow[blockIdx.x + 1];
    for (int64_t t = r0 + threadIdx.x; t < r1; t += GMS_THREADS) {
        const double v = ih * g.w[t];
        Vn[t] = v;
        g.vcur[t] = v;
    }
}

__device__ __forceinline__ void gms_apply(double &dx, double &dy, double cs, double sn) {
    const double temp = __dadd_rn(__dmul_rn(cs, dx), __dmul_rn(sn, dy));
    dy = __dadd_rn(__dmul_rn(-sn, dx), __dmul_rn(cs, dy));
    dx = temp;
}

// Givens rotations of column i of every running problem (*/codes/gmres.hpp:30-75,156-162),
// a warp a problem, its column and earlier rotations in shared memory: the chain
// over them otherwise waits for memory at each rotation.
__global__ void gms_givens(GmresSeg g) {
    extern __shared__ double gms_sm[];
    const int p = blockIdx.x, lane = threadIdx.x, i = *g.iter;
    if (g.conv[p] != -1) return;
    double *cs = g.cs + (size_t)p * (g.m + 1), *sn = g.sn + (size_t)p * (g.m + 1), *s = g.s + (size_t)p * (g.m + 1);
    double *Hc = g.H + gms_h(g, p, 0, i);
    double *h = gms_sm, *c = h + g.m + 1, *d = c + g.m + 1;
    for (int k = lane; k <= i + 1; k += 32) h[k] = Hc[k];
    for (int k = lane; k < i; k += 32) {
        c[k] = cs[k];
        d[k] = sn[k];
    }
    __syncwarp();
    if (lane == 0) {
        for (int k = 0; k < i; ++k) gms_apply(h[k], h[k + 1], c[k], d[k]);
        double dx = h[i], dy = h[i + 1], c_, s_;
        if (dy == 0.0) { c_ = 1.0; s_ = 0.0; }
        else if (fabs(dy) > fabs(dx)) {
            const double temp = dx / dy;
            s_ = 1.0 / sqrt(1.0 + temp * temp);
            c_ = temp * s_;
        } else {
            const double temp = dy / dx;
            c_ = 1.0 / sqrt(1.0 + temp * temp);
            s_ = temp * c_;
        }
        cs[i] = c_;
        sn[i] = s_;
        gms_apply(h[i], h[i + 1], c_, s_);
        gms_apply(s[i], s[i + 1], c_, s_);
        const double resid = fabs(s[i + 1]) / g.normb[p];
        g.resid[p] = resid;
        if (resid < *g.tolp) g.conv[p] = i;
    }
    __syncwarp();
    for (int k = lane; k <= i + 1; k += 32) Hc[k] = h[k];
}
// The next column, and (cond) the loop condition: while a problem is running
__global__ void gms_next(GmresSeg g, cudaGraphConditionalHandle hnd, int cond) {
    int running = 0;
    for (int p = threadIdx.x; p < g.P; p += blockDim.x) running |= g.conv[p] == -1;
    running = __syncthreads_or(running);
    if (threadIdx.x == 0) {
        const int c = ++g.iter[1], i = g.iter[0];
        if (i + 1 < g.m) g.iter[0] = i + 1;
        if (cond) cudaGraphSetConditional(hnd, (running && c < g.m) ? 1u : 0u);
    }
}

// w = b - Ax (Ax == NULL: w = b) and per-block partials of ||w||^2
__global__ void gms_resid(GmresSeg g, const double *__restrict__ b, const double *__restrict__ Ax) {
    __shared__ double red[4 * GMS_WARPS];
    const int64_t r0 = g.brow[blockIdx.x], r1 = g.brow[blockIdx.x + 1];
    for (int64_t t = r0 + threadIdx.x; t < r1; t += GMS_THREADS) g.w[t] = Ax ? b[t] - Ax[t] : b[t];
    __syncthreads();
    gms_block_dots(g, g.w, g.w, 1, red, g.part);
}
__global__ void gms_colnorm_part(GmresSeg g, const double *__restrict__ v) {
    __shared__ double red[4 * GMS_WARPS];
    gms_block_dots(g, v, v, 1, red, g.part);
}
// out[p] = sqrt(sum of problem p's partials); zero_to_one: a zero norm becomes 1
__global__ void gms_colnorm_fin(GmresSeg g, double *out, int zero_to_one) {
    const int p = blockIdx.x;
    double s = 0.0;
    for (int b = g.pblk[p] + threadIdx.x; b < g.pblk[p + 1]; b += 32) s += g.part[(size_t)b * (g.m + 1)];
    s = gms_warp_sum(s);
    if (threadIdx.x == 0) {
        s = sqrt(s);
        out[p] = (zero_to_one && s == 0.0) ? 1.0 : s;
    }
}
// beta = ||w|| (hsum); V[:, 0] = vcur = w / beta; s = beta e1; per-problem state
__global__ void gms_start_fin(GmresSeg g, double tol) {
    const int p = g.bprob[blockIdx.x];
    __shared__ double s_beta, s_ib;
    if (threadIdx.x == 0) {
        s_beta = sqrt(g.hsum[(size_t)p * (g.m + 1)]);
        s_ib = s_beta > 0.0 ? 1.0 / s_beta : 0.0;
    }
    __syncthreads();
    const double beta = s_beta, ib = s_ib;
    if (blockIdx.x == g.pblk[p] && threadIdx.x == 0) {
        double *cs = g.cs + (size_t)p * (g.m + 1), *sn = g.sn + (size_t)p * (g.m + 1), *s = g.s + (size_t)p * (g.m + 1);
        for (int k = 0; k <= g.m; ++k) { s[k] = 0.0; cs[k] = 0.0; sn[k] = 0.0; }
        s[0] = beta;
        const double r = beta / g.normb[p];
        g.resid[p] = r;
        g.conv[p] = r <= tol ? -2 : -1;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        g.iter[0] = 0;
        g.iter[1] = 0;
    }
    const int64_t r0 = g.brow[blockIdx.x], r1 = g.brow[blockIdx.x + 1];
    for (int64_t t = r0 + threadIdx.x; t < r1; t += GMS_THREADS) {
        const double v = g.w[t] * ib;
        g.V[t] = v;
        g.vcur[t] = v;
    }
}
// y_p = H_p(0:k, 0:k) \ s_p(0:k), k = the problem's last Arnoldi column
// (converged: conv; running: last; converged at the start: none), each entry's
// operations in the reference's order (*/codes/gmres.hpp:77-90); a CTA a problem, a
// column's updates in parallel in shared memory
__global__ void gms_backsolve(GmresSeg g, int last) {
    extern __shared__ double gms_sm[];
    const int p = blockIdx.x, cv = g.conv[p];
    const int k = cv >= 0 ? cv : (cv == -1 ? last : -1);
    double *y = g.y + (size_t)p * (g.m + 1);
    for (int j = threadIdx.x; j <= k; j += blockDim.x) gms_sm[j] = g.s[(size_t)p * (g.m + 1) + j];
    for (int i = k; i >= 0; --i) {
        const double *Hc = g.H + gms_h(g, p, 0, i);
        __syncthreads();
        const double yi = gms_sm[i] / Hc[i];
        __syncthreads();
        for (int j = threadIdx.x; j < i; j += blockDim.x) gms_sm[j] -= Hc[j] * yi;
        if (threadIdx.x == 0) gms_sm[i] = yi;
    }
    __syncthreads();
    for (int j = threadIdx.x; j <= g.m; j += blockDim.x) y[j] = j <= k ? gms_sm[j] : 0.0;
}
// x += V y over the Arnoldi columns of each row's problem (0..k_p: its
// converged column, `last` while running, none when converged at the start;
// later columns of a converged problem are never written and never read)
__global__ void gms_xupdate(GmresSeg g, double *__restrict__ x, int last) {
    const int p = g.bprob[blockIdx.x];
    const int cv = g.conv[p];
    const int kp = cv >= 0 ? cv : (cv == -1 ? last : -1);
    const double *y = g.y + (size_t)p * (g.m + 1);
    const int64_t r0 = g.brow[blockIdx.x], r1 = g.brow[blockIdx.x + 1];
    for (int64_t t = r0 + threadIdx.x; t < r1; t += GMS_THREADS) {
        double v = x[t];
        for (int j = 0; j <= kp; ++j) v += g.V[(size_t)j * g.Ntot + t] * y[j];
        x[t] = v;
    }
}
__global__ void gather64_kernel(const double *__restrict__ x, double *__restrict__ y, const int64_t *__restrict__ idx,
                                int64_t n) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        y[t] = x[idx[t]];
}
__global__ void scatter64_kernel(const double *__restrict__ x, double *__restrict__ y, const int64_t *__restrict__ idx,
                                 int64_t n) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        y[idx[t]] = x[t];
}
cudaError_t launch_gather64(const double *x, double *y, const int64_t *idx, int64_t n, cudaStream_t st) {
    gather64_kernel<<<1216, 256, 0, st>>>(x, y, idx, n);
    count_launch();
    return cudaGetLastError();
}
cudaError_t launch_scatter64(const double *x, double *y, const int64_t *idx, int64_t n, cudaStream_t st) {
    scatter64_kernel<<<1216, 256, 0, st>>>(x, y, idx, n);
    count_launch();
    return cudaGetLastError();
}

cudaError_t gms_norms(const GmresSeg &g, const double *v, double *out, int zero_to_one, cudaStream_t st) {
    gms_colnorm_part<<<g.nblk, GMS_THREADS, 0, st>>>(g, v);
    gms_colnorm_fin<<<g.P, 32, 0, st>>>(g, out, zero_to_one);
    count_launch(2);
    return cudaGetLastError();
}
cudaError_t gms_start(const GmresSeg &g, const double *b, const double *Ax, double tol, cudaStream_t st) {
    gms_resid<<<g.nblk, GMS_THREADS, 0, st>>>(g, b, Ax);
    gms_reduce<<<g.P, 32, 0, st>>>(g, 0);
    gms_start_fin<<<g.nblk, GMS_THREADS, 0, st>>>(g, tol);
    count_launch(3);
    return cudaGetLastError();
}
cudaError_t gms_arnoldi(const GmresSeg &g, const cudaGraphConditionalHandle *hnd, cudaStream_t st) {
    const size_t smu = ((size_t)(g.m + 1) + 4 * GMS_WARPS) * 8;
    gms_dots<<<g.nblk, GMS_THREADS, 0, st>>>(g);
    gms_reduce<<<g.P, 256, 0, st>>>(g, 1);
    gms_update<<<g.nblk, GMS_THREADS, smu, st>>>(g, 0);
    gms_reduce<<<g.P, 256, 0, st>>>(g, 1);
    gms_update<<<g.nblk, GMS_THREADS, smu, st>>>(g, 1);
    gms_reduce<<<g.P, 32, 0, st>>>(g, 0);
    gms_normalise<<<g.nblk, GMS_THREADS, 0, st>>>(g);
    gms_givens<<<g.P, 32, (size_t)3 * (g.m + 1) * 8, st>>>(g);
    gms_next<<<1, 256, 0, st>>>(g, hnd ? *hnd : cudaGraphConditionalHandle{}, hnd ? 1 : 0);
    count_launch(9);
    return cudaGetLastError();
}
cudaError_t gms_finish(const GmresSeg &g, double *x, int last, int kmax, cudaStream_t st) {
    gms_backsolve<<<g.P, 128, (size_t)(g.m + 1) * 8, st>>>(g, last);
    count_launch();
    if (kmax >= 0) {
        gms_xupdate<<<g.nblk, GMS_THREADS, 0, st>>>(g, x, last);
        count_launch();
    }
    return cudaGetLastError();
}

}  // namespace h2w
