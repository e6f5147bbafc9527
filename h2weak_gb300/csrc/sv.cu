// Single-vector product on the dataflow launch, warp-specialised (sm_103a).
//
// One cooperative launch performs a whole product (or a range of its target
// stream) of one operator, or of every operator of a batch. A target is a
// block row of the compressed operator: rows [dst, dst + nrows) of the
// workspace get the nrows x W matrix of all its panels (stored contiguously,
// column-major at leading dimension pad4(nrows)) times its W gathered
// sources. The work of a CTA is split by role:
//
//  * P (operator): takes targets (the first two by block index, then from the
//    claim counters), and streams each target's matrix in column chunks into a
//    ring of stages by bulk copies. The operator depends on
//    nothing, so P runs ahead of every wait on the data: the ring holds the
//    matrices of the next targets while the current one waits for its sources.
//  * G (sources, two warps in turn): waits for the target's producer count, then copies its
//    sources (and the rows it adds to, and the output positions of its rows)
//    into the target's slot by asynchronous 4- or 8-byte copies that complete
//    on the slot's mbarrier; up to `nslots` targets are in preparation.
//  * CW consumer warps multiply the stages as they land, reduce the partial
//    sums of each row through shared memory and write the rows;
//  * R (release): fences the written rows and decrements the producer counts
//    of the groups that wait for them, whose list it read in advance.
//
// Which columns a thread adds up decides how much is lost to rounding. In FP64 a thread has neighbouring
// ones, for terms that cancel are mostly neighbours (the matrix is stored so that the threads read neighbouring
// vectors of it all the same, sv_slice_kernel); only the rows of a leaf's own points, whose diagonal outweighs the
// rest and stands among the last columns, take every CG-th column, so that little is added after it. Against
// every CG-th column everywhere, error of a product, quadratic mean over 64 vectors: 1D integral equation, 32768
// points, 7.0e-14 and 3.5e-14 of the result (3.5e-14 in the launch by phases), 2D RBF 9973 3.5e-16 and 1.9e-16 (2.5e-16);
// neighbouring columns everywhere: 2D integral equation 65536 2.7e-16, 1.6e-16 so. In FP32 every CG-th
// column with SvSum does best.
//
// Two kinds of CTA share an SM: some take the chain of dependent passes first and
// mostly wait, so that each pass starts at once when its producers are done; the
// others stream the work that depends on the input alone meanwhile (SvArgs).
//
// Deadlock-free by order: within a list, and from lists 0 and 1 to list 2,
// dependencies point from earlier to later targets, and none between lists 0 and 1.
// Every CTA is resident and finishes its targets in the order it took them, and it
// leaves a list only when that is claimed to the end, so targets of list 1 are taken
// by CTAs that started with list 0, or targets of list 0 by CTAs that started with
// list 1, but not both. One of the two lists is then wholly in CTAs that started with
// it, where its earliest unfinished target always runs; then the other's; then list 2's.
// Every wait is bounded all the same: one that runs out sets *err (1 grid barrier,
// 3 dependency, 4 mbarrier) and the CTA stops, after its copies in flight have landed.
//
// The launch prepares itself: the workspace is zeroed, the producer counts
// are reset, and the input goes (converted) to leaf order behind the
// workspace, while P already streams; one grid barrier before the first
// source is read. Sources then all come from one array of the kernel's type.
//
// What bounds it: HBM for FP32 operators that exceed the L2, the FP64 pipe (two
// multiply-adds a clock and SM, 5.0 TB/s of operator) for FP64 ones, and the
// chain of dependent passes (2 L + 1, about 3 us each) for small problems.
// Measured against one kernel whose CTAs gathered, multiplied and released a target
// at a time: 2D integral equation, 65536 points (62e6 entries): FP64 207 -> 152 us,
// FP32 138 -> 80; 3D semi-nested RBF, 20011 points (2e8): FP64 665 -> 428, FP32 330 -> 168
// (4.8 TB/s); the FP64 pipe is 79 % busy in the 2D product; 1D RBF, 4096 points, waited for: 92 -> 75, calls on
// several streams 69 -> 18 each.
#include <algorithm>

#include "kernels.cuh"

namespace h2w {
namespace {

// CW consumer warps: 4, or 8 where few CTAs fit an SM (wide targets)
template <int CW> struct SvDim {
    static constexpr int CT = 32 * CW;                         // consumer threads
    static constexpr int NT = CT + 128;                        // + P, two G, R
    static constexpr int STAGE = CW == 4 ? 8192 : 16384;       // bytes of one operator stage
    static constexpr int PER_SM = CW == 4 ? 5 : 3;
};
constexpr int SV_GW = 2;                      // G warps, taking targets in turn
constexpr int SV_MAX_SLOTS = 4, SV_MAX_STAGES = 24;
constexpr int SV_SM_BYTES = 226 * 1024;       // shared memory of an SM's CTAs
constexpr int SV_WAIT = 1 << 20;              // polls of one mbarrier wait
constexpr int SV_POLL = 1 << 20;              // polls of a producer count or the grid barrier (about a second)

template <class T> struct SvVec;
template <> struct SvVec<double> { using type = double2; static constexpr int n = 2; };
template <> struct SvVec<float> { using type = float4; static constexpr int n = 4; };
__device__ __forceinline__ void sv_fma(double *a, const double2 v, double x) {
    a[0] = fma(v.x, x, a[0]);
    a[1] = fma(v.y, x, a[1]);
}
__device__ __forceinline__ void sv_fma(float *a, const float4 v, float x) {
    a[0] = fmaf(v.x, x, a[0]);
    a[1] = fmaf(v.y, x, a[1]);
    a[2] = fmaf(v.z, x, a[2]);
    a[3] = fmaf(v.w, x, a[3]);
}

// A row's sum of its threads' partial sums. In FP32 the roundings are kept (Knuth's TwoSum) and added at
// the end: with up to 128 partial sums a row they made most of a product's error. Of the result's norm,
// quadratic mean over 40 vectors, added plainly and so: 1D integral equation, 32768 points, 3.4e-5 and 1.7e-5; 2D
// 65536 9.5e-8 and 8.6e-8; 3D RBF 9001 1.28e-7 and 1.06e-7. It costs 1 to 5 % of a product.
template <class T> struct SvSum {
    T s = T(0), c = T(0);
    __device__ __forceinline__ void add(T x) {
        if constexpr (sizeof(T) == 4) {
            const T t = __fadd_rn(s, x), b = __fsub_rn(t, s);
            c = __fadd_rn(c, __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(x, b)));
            s = t;
        } else {
            s += x;
        }
    }
    __device__ __forceinline__ void join(int o) {  // with the thread o away
        const T cx = sizeof(T) == 4 ? __shfl_xor_sync(0xffffffffu, c, o) : T(0);
        add(__shfl_xor_sync(0xffffffffu, s, o));
        if (sizeof(T) == 4) c += cx;
    }
    // (an infinite or undefined sum has no rounding to add)
    __device__ __forceinline__ T value() const { return sizeof(T) == 4 && fabs(s) <= T(3.402823466e38) ? s + c : s; }
};

struct SvSlot {  // one target in preparation
    int32_t t;   // < 0: the stream's end
    uint32_t dst, idx0, grp;
    int32_t nrows, W, flags, skip;
    int32_t RQ, CG, cpc;  // row vectors, column groups of the consumer threads, columns a stage
    int32_t per, rem, xs;  // group cg's sources: from cg per + min(cg, rem), xs apart
    uint32_t inv;         // thread / RQ = thread * inv >> 16
    int64_t vpos;         // its rows' position in the output vector (scatter targets)
};

// Shared memory: barriers and slots, partial sums (two buffers), the slots'
// sources, the stages (16-byte aligned).
template <class T, int CW> struct SvLayout {
    static constexpr size_t bars = 8 * (size_t)(2 * SV_MAX_STAGES + 4 * SV_MAX_SLOTS + 1);
    static constexpr size_t slots = sizeof(SvSlot) * SV_MAX_SLOTS;
    static constexpr size_t red = sizeof(T) * 2 * SvDim<CW>::CT * SvVec<T>::n;
    static constexpr size_t off_slots = (bars + 15) / 16 * 16;
    static constexpr size_t off_misc = off_slots + slots;  // fail flag, barrier generation
    static constexpr size_t off_red = (off_misc + 16 + 15) / 16 * 16;
    static constexpr size_t off_src = off_red + red;
    // a slot's sources: W values, then the rows it adds to, then output positions
    static size_t slot_bytes(int max_w) { return sizeof(T) * (size_t)(max_w + SV_MAX_ROWS) + 4 * SV_MAX_ROWS; }
    static size_t smem(int max_w, int nslots, int nst) {
        return off_src + (size_t)nslots * slot_bytes(max_w) + (size_t)nst * SvDim<CW>::STAGE;
    }
};

__device__ __forceinline__ uint32_t sv_sa(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void sv_init(uint64_t *b, uint32_t n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sv_sa(b)), "r"(n));
}
__device__ __forceinline__ void sv_arrive(uint64_t *b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sv_sa(b)) : "memory");
}
__device__ __forceinline__ void sv_arrive_tx(uint64_t *b, uint32_t tx) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sv_sa(b)), "r"(tx) : "memory");
}
// this thread's cp.async copies so far complete -> one arrival (counted in the barrier's total)
__device__ __forceinline__ void sv_arrive_copies(uint64_t *b) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(sv_sa(b)) : "memory");
}
__device__ __forceinline__ bool sv_try(uint64_t *b, uint32_t par) {
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done)
                 : "r"(sv_sa(b)), "r"(par)
                 : "memory");
    return done != 0;
}
// Bounded wait for phase `par`; false once any wait of the CTA has run out. The
// polling is out of line: the roles run different code side by side, a target's
// epilogue once per target, and the instruction caches hold little of it (unrolling
// these loops cost 15 % of a product).
__device__ __noinline__ bool sv_wait_more(uint64_t *b, uint32_t par, volatile int32_t *fail, int32_t *err) {
    for (int it = 0; it < SV_WAIT; ++it) {
        if (sv_try(b, par)) return true;
        if (*fail) return false;
    }
    *fail = 1;
    atomicExch(err, 4);
    return false;
}
__device__ __forceinline__ bool sv_wait(uint64_t *b, uint32_t par, volatile int32_t *fail, int32_t *err) {
    return sv_try(b, par) || sv_wait_more(b, par, fail, err);
}
// The same for a whole warp, with one answer for all lanes.
__device__ __forceinline__ bool sv_wait_warp(uint64_t *b, uint32_t par, volatile int32_t *fail, int32_t *err) {
    return __all_sync(0xffffffffu, sv_wait(b, par, fail, err));
}
// Position in a ring of n: index and the parity of its current round
struct SvRing {
    int i = 0;
    uint32_t par = 0;
    __device__ __forceinline__ void next(int n) {
        if (++i == n) {
            i = 0;
            par ^= 1u;
        }
    }
};
__device__ __forceinline__ void sv_bulk(void *dst, const void *src, uint32_t bytes, uint64_t *b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     sv_sa(dst)),
                 "l"(src), "r"(bytes), "r"(sv_sa(b))
                 : "memory");
}
__device__ __forceinline__ void sv_cp(uint32_t dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void sv_cp(uint32_t dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void sv_cp(uint32_t dst, const int32_t *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
// An acquiring load, where a fence would also wait for this thread's earlier copies
// (with one per target the product of a 65536-point 2D operator took 218 instead of 168 us).
__device__ __forceinline__ uint32_t sv_acquire(const void *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// the group's producers are done: bounded, out of line as the waits above
__device__ __noinline__ bool sv_until(const int32_t *rem, volatile int32_t *fail, int32_t *err) {
    for (int it = 0; it <= SV_POLL; ++it) {
        if ((int32_t)sv_acquire(rem) <= 0) return true;
        if (*fail) return false;
    }
    *fail = 1;
    atomicExch(err, 3);
    return false;
}

template <class T, int CW>
__global__ void __launch_bounds__(SvDim<CW>::NT, SvDim<CW>::PER_SM)
    sv_flow_kernel(const SvArgs<T> a, int max_w, int nslots, int nst) {
    using Lay = SvLayout<T, CW>;
    constexpr int CT = SvDim<CW>::CT, STAGE = SvDim<CW>::STAGE;
    using V = typename SvVec<T>::type;
    constexpr int VN = SvVec<T>::n;
    extern __shared__ __align__(128) char sv_smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(sv_smem), *empty = full + SV_MAX_STAGES;
    uint64_t *s_known = empty + SV_MAX_STAGES;  // slot's target named (P)
    uint64_t *s_src = s_known + SV_MAX_SLOTS;   // its sources landed (G's 32 lanes)
    uint64_t *s_done = s_src + SV_MAX_SLOTS;    // its rows written (consumer warps)
    uint64_t *s_free = s_done + SV_MAX_SLOTS;   // released (R)
    uint64_t *redbar = s_free + SV_MAX_SLOTS;   // consumer warps meet
    SvSlot *slots = reinterpret_cast<SvSlot *>(sv_smem + Lay::off_slots);
    volatile int32_t *fail = reinterpret_cast<volatile int32_t *>(sv_smem + Lay::off_misc);
    unsigned *gen0 = reinterpret_cast<unsigned *>(sv_smem + Lay::off_misc + 4);
    T *red = reinterpret_cast<T *>(sv_smem + Lay::off_red);
    const int slot_b = (int)sizeof(T) * (max_w + SV_MAX_ROWS) + 4 * SV_MAX_ROWS;
    char *src0 = sv_smem + Lay::off_src;
    char *stages = src0 + nslots * slot_b;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < SV_MAX_STAGES) {
        sv_init(full + tid, 1);
        sv_init(empty + tid, CW);
        if (tid < SV_MAX_SLOTS) {
            sv_init(s_known + tid, 1);
            sv_init(s_src + tid, 32);
            sv_init(s_done + tid, CW);
            sv_init(s_free + tid, 1);
        }
        if (tid == 0) {
            sv_init(redbar, CW);
            *fail = 0;
            // before this CTA arrives at the grid barrier, so the barrier cannot complete yet
            *gen0 = *reinterpret_cast<volatile unsigned *>(a.bar + 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == CW) {  // --------------------------------------------------- P
        if (lane != 0) return;
        // Targets in order: two by block index, then claims, after the grid barrier that
        // resets the counters. One target ahead of the one being streamed.
        const bool first = (int)blockIdx.x < a.na;
        const int cls = first ? a.na : (int)gridDim.x - a.na, me = first ? blockIdx.x : blockIdx.x - a.na;
        int li = 0, taken = 0;
        bool ready = !a.prep, ok = true;
        SvHdr h{}, hn{};
        int t = -2, tn = -2;  // -2: not yet, -1: no more
        SvRing sr, fr;        // slots, stages
        bool slot_used = false, stage_used = false;  // the rings have gone round once
        uint32_t sent = 0;
        for (int ends = 0; ok && ends < SV_GW;) {
            if (t != -2) {
                if (slot_used && !sv_wait(s_free + sr.i, sr.par ^ 1u, fail, a.err)) break;
                SvSlot &sl = slots[sr.i];
                sl.t = t;
                const int RQ = (h.nrows + 3) / 4 * 4 / VN;
                const bool skip = t >= 0 && a.active && a.active[h.pid] != -1;
                // whole rounds of the column groups a stage, while it holds one
                const int CG = RQ > 0 ? CT / RQ : 1, fit = RQ > 0 ? STAGE / (16 * RQ) : 1;
                const int cpc = fit > CG ? fit / CG * CG : fit;
                if (t >= 0) {
                    sl.dst = h.dst;
                    sl.idx0 = h.idx0;
                    sl.grp = h.grp;
                    sl.nrows = h.nrows;
                    sl.W = h.W;
                    sl.flags = h.flags;
                    sl.skip = skip;
                    sl.RQ = RQ;
                    sl.CG = CG;
                    sl.cpc = cpc;
                    const bool near = sizeof(T) == 8 && (h.flags & SV_NEIGHBOURS);
                    sl.per = near ? h.W / CG : 1;
                    sl.rem = near ? h.W - sl.per * CG : 0;
                    sl.xs = near ? 1 : CG;
                    sl.inv = (65536u + (uint32_t)RQ - 1) / (uint32_t)RQ;  // exact for thread numbers below 512
                    sl.vpos = (int64_t)h.dst - (a.vshift ? a.vshift[h.pid] : 0);
                } else {
                    ++ends;  // one for each G warp's turn
                }
                sv_arrive(s_known + sr.i);
                sr.next(nslots);
                if (sr.i == 0) slot_used = true;
                if (t >= 0 && !skip) {
                    const T *A = (a.Ap ? a.Ap[h.pid] : a.A) + h.a;
#pragma unroll 1
                    for (int c = 0; c < h.W; c += cpc) {
                        if (stage_used && !sv_wait(empty + fr.i, fr.par ^ 1u, fail, a.err)) {
                            ok = false;
                            break;
                        }
                        const uint32_t bytes = (uint32_t)min(cpc, h.W - c) * (uint32_t)RQ * 16u;
                        sv_arrive_tx(full + fr.i, bytes);
                        sv_bulk(stages + fr.i * STAGE, A + (int64_t)c * (RQ * VN), bytes, full + fr.i);
                        ++sent;
                        fr.next(nst);
                        if (fr.i == 0) stage_used = true;
                    }
                }
            }
            t = tn;
            h = hn;
            tn = -1;
#pragma unroll 1
            while (t != -1 && li < 3) {
                const int l = li == 2 ? 2 : (first ? li : 1 - li);
                const int n = a.l1[l] - a.l0[l];
                int i;
                if (li == 0 && taken < 2) {
                    i = me + cls * taken++;
                } else {
                    if (!ready) {
                        int it = 0;
                        while (ok && sv_acquire(a.bar + 1) == *gen0) {
                            if (++it > SV_POLL || *fail) {
                                atomicExch(a.err, 1);
                                *fail = 1;
                                ok = false;
                            }
                        }
                        if (!ok) break;
                        ready = true;
                    }
                    // the targets that a list's own CTAs took by block index come first
                    i = (l == 2 ? 0 : 2 * (li == 0 ? cls : (int)gridDim.x - cls)) + atomicAdd(a.ctr + l, 1);
                    if (i >= n) ++li;
                }
                if (i < n) {
                    tn = a.l0[l] + i;
                    hn = a.hdr[tn];
                    break;
                }
            }
        }
        // the copies in flight land before the CTA may end (the consumers may have stopped)
        for (int q = 0; q < nst && (uint32_t)q < sent; ++q) {
            fr.i = fr.i > 0 ? fr.i - 1 : (fr.par ^= 1u, nst - 1);
            for (int it = 0; it < SV_WAIT && !sv_try(full + fr.i, fr.par); ++it) {
            }
        }
        return;
    }
    if (warp > CW && warp <= CW + SV_GW) {  // ------------------------------- G
        bool ready = !a.prep;
        SvRing sr;
        for (int k = 0;; ++k, sr.next(nslots)) {
            if (k % SV_GW != warp - CW - 1) continue;
            if (!sv_wait_warp(s_known + sr.i, sr.par, fail, a.err)) break;
            const SvSlot &sl = slots[sr.i];
            if (sl.t < 0) {
                sv_arrive(s_src + sr.i);
                break;
            }
            // 256 columns a round, each round's rows read a round ahead, the first before the wait
            constexpr int U = 8;
            const uint32_t *ix = a.idx + sl.idx0 + lane;
            const uint32_t xd = sv_sa(src0 + sr.i * slot_b);
            const int W = sl.W, skip = sl.skip;
            bool good = true;
            uint32_t row[U], ahead[U];
#pragma unroll
            for (int u = 0; u < U; ++u) row[u] = 0;
#pragma unroll 1
            for (int c = -32 * U; c < W; c += 32 * U) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = c + 32 * U + u * 32;
                    ahead[u] = i + lane < W ? ix[i] : 0;
                }
                if (c < 0) {
                    if (lane == 0) {
                        int it = 0;
                        if (!ready)  // the launch's preparation, by every CTA
                            while (good && sv_acquire(a.bar + 1) == *gen0)
                                if (++it > SV_POLL || *fail) {
                                    good = false;
                                    atomicExch(a.err, 1);
                                }
                        it = 0;
                        while (good && !skip && !(sl.flags & SV_LATE) && (int32_t)sv_acquire(a.rem + sl.grp) > 0)
                            if (++it > SV_POLL || *fail) {
                                good = false;
                                atomicExch(a.err, 3);
                            }
                        if (!good) *fail = 1;
                    }
                    ready = true;
                    good = __shfl_sync(0xffffffffu, (int)good, 0);
                    __syncwarp();
                    if (!good || skip) break;
                } else {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int i = c + u * 32 + lane;
                        if (i < W) sv_cp(xd + (uint32_t)(i * (int)sizeof(T)), (const T *)a.ws + row[u]);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) row[u] = ahead[u];
            }
            if (!good) break;
            const int nrows = skip ? 0 : sl.nrows, flags = sl.flags;
            const uint32_t pd = xd + (uint32_t)(max_w * (int)sizeof(T));
#pragma unroll 1
            for (int i = lane; i < nrows; i += 32) {
                if ((flags & T_ACCUM) && !(flags & SV_LATE)) sv_cp(pd + (uint32_t)(i * (int)sizeof(T)), (const T *)a.ws + sl.dst + i);
                if ((flags & T_SCATTER) && a.perm)
                    sv_cp(pd + (uint32_t)(SV_MAX_ROWS * (int)sizeof(T) + 4 * i), a.perm + sl.vpos + i);
            }
            sv_arrive_copies(s_src + sr.i);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }
    if (warp == CW + SV_GW + 1) {  // ---------------------------------------- R
        for (SvRing sr;; sr.next(nslots)) {
            if (!sv_wait_warp(s_known + sr.i, sr.par, fail, a.err)) break;
            if (slots[sr.i].t < 0) break;
            const uint2 gi = a.grp[slots[sr.i].grp];
            const uint32_t mine = lane < gi.y ? a.cons[gi.x + lane] : 0;
            if (!sv_wait_warp(s_done + sr.i, sr.par, fail, a.err)) break;
            if (lane == 0) sv_arrive(s_free + sr.i);
            if (gi.y > 0) {
                // the rows before the counts
                asm volatile("fence.acq_rel.gpu;" ::: "memory");
                if (lane < gi.y) atomicSub(a.rem + mine, 1);
#pragma unroll 1
                for (uint32_t e = 32 + lane; e < gi.y; e += 32) atomicSub(a.rem + a.cons[gi.x + e], 1);
            }
        }
        return;
    }
    // -------------------------------------------------------------- consumers
    uint32_t met = 0;  // meetings of the consumer warps so far
    auto meet = [&]() -> bool {
        __syncwarp();
        if (lane == 0) sv_arrive(redbar);
        const bool r = sv_wait_warp(redbar, met & 1u, fail, a.err);
        ++met;
        return r;
    };
    if (a.prep) {
        const int64_t me = (int64_t)blockIdx.x * CT + tid, all = (int64_t)gridDim.x * CT;
        int4 *w4 = reinterpret_cast<int4 *>(a.ws);
        const int64_t nz = a.nzero * (int64_t)sizeof(T) / 16;
#pragma unroll 1
        for (int64_t i = me; i < nz; i += all) w4[i] = make_int4(0, 0, 0, 0);
        T *xl = a.ws + a.xoff;
#pragma unroll 1
        for (int64_t i = me; i < a.nx; i += all) xl[i] = (T)a.xin[a.perm ? (int64_t)a.perm[i] : i];
#pragma unroll 1
        for (int64_t i = me; i < a.ngrp; i += all) a.rem[i] = a.cnt[i];
        if (me < SV_CTRS) a.ctr[me] = 0;
        if (!meet()) return;
        if (tid == 0) {
            __threadfence();
            if (atomicAdd(a.bar, 1u) == gridDim.x - 1) {
                atomicExch(a.bar, 0u);
                __threadfence();
                atomicAdd(a.bar + 1, 1u);
            }
        }
    }
    SvRing fr;
    for (SvRing sr;; sr.next(nslots)) {
        if (!sv_wait_warp(s_src + sr.i, sr.par, fail, a.err)) return;
        const SvSlot &sl = slots[sr.i];
        if (sl.t < 0) return;
        if (!sl.skip) {
            const int nrows = sl.nrows, W = sl.W, RQ = sl.RQ, CG = sl.CG, cpc = sl.cpc;
            const T *xs = reinterpret_cast<const T *>(src0 + sr.i * slot_b);
            const int xstep = sizeof(T) == 8 ? sl.xs : CG;
            // thread = row slice q (VN rows, one 16-byte vector a column) x column group cg
            const int cg = (int)((uint32_t)tid * sl.inv >> 16), q = tid - cg * RQ;
            // FP32: four stages' terms (16 at most) summed apart before they go to the total. One sum of a
            // target's W / CG terms (256 of 4096 columns) lost more to rounding (3D semi-nested, 20011 points:
            // 1.09e-7 of the result, 9.8e-8 so; 7.7e-8 with SvSum)
            T acc[VN], tot[VN];
#pragma unroll
            for (int v = 0; v < VN; ++v) acc[v] = tot[v] = T(0);
            int done = 0;
            const T *x0 = xs + (sizeof(T) == 8 ? cg * sl.per + min(cg, sl.rem) : cg);  // the group's sources
#pragma unroll 1
            for (int c = 0; c < W; c += cpc) {
                if (!sv_wait_warp(full + fr.i, fr.par, fail, a.err)) return;
                const int nc = min(cpc, W - c);
                if (cg < CG) {
                    const V *As = reinterpret_cast<const V *>(stages + fr.i * STAGE) + cg * RQ + q;
                    const int step = CG * RQ;
                    const T *xc = sizeof(T) == 8 ? x0 : x0 + c;
                    int j = cg;
#pragma unroll 1
                    for (; j + 3 * CG < nc; j += 4 * CG, As += 4 * step, xc += 4 * xstep) {
                        const V v0 = As[0], v1 = As[step], v2 = As[2 * step], v3 = As[3 * step];
                        const T y0 = xc[0], y1 = xc[xstep], y2 = xc[2 * xstep], y3 = xc[3 * xstep];
                        sv_fma(acc, v0, y0);
                        sv_fma(acc, v1, y1);
                        sv_fma(acc, v2, y2);
                        sv_fma(acc, v3, y3);
                    }
#pragma unroll 1
                    for (; j < nc; j += CG, As += step, xc += xstep) sv_fma(acc, As[0], xc[0]);
                    if (sizeof(T) == 8) x0 = xc;
                }
                __syncwarp();
                if (lane == 0) sv_arrive(empty + fr.i);
                fr.next(nst);
                if (sizeof(T) == 4 && (++done & 3) == 0) {
#pragma unroll
                    for (int v = 0; v < VN; ++v) {
                        tot[v] += acc[v];
                        acc[v] = T(0);
                    }
                }
            }
            if (sizeof(T) == 4)
#pragma unroll
                for (int v = 0; v < VN; ++v) acc[v] += tot[v];
            // Rows: 2^l neighbouring threads share a row's CG partial sums (few, for each
            // step of a shuffle costs the FP64 pipe a whole warp). Two buffers in turn:
            // once the warps have met, all of them have read the sums of the meeting before.
            T *rb = red + (met & 1u) * (CT * VN);
#pragma unroll
            for (int v = 0; v < VN; ++v) rb[v * CT + tid] = acc[v];
            if (!meet()) return;
            int l = 0;
            while (l < 3 && (nrows << (l + 1)) <= CT) ++l;
            const int part = tid & ((1 << l) - 1), flags = sl.flags;
            // the rows added to: only now does a target of input columns wait for the part before it
            if (flags & SV_LATE) {
                if (!__all_sync(0xffffffffu, lane != 0 || sv_until(a.rem + sl.grp, fail, a.err))) return;
                __syncwarp();  // lane 0's acquire, for the rows that the other lanes read
            }
#pragma unroll 1
            for (int r0 = 0; r0 < nrows; r0 += CT >> l) {
                if (r0 + (warp * 32 >> l) >= nrows) break;  // the same for the whole warp
                const int r = r0 + (tid >> l);
                SvSum<T> sum;
                constexpr bool near = sizeof(T) == 8;  // neighbouring groups together
                const T *p = rb + (r % VN) * CT + r / VN;
                if (r < nrows)
#pragma unroll 1
                    for (int e = near ? part * CG >> l : part; e < (near ? (part + 1) * CG >> l : CG); e += near ? 1 : 1 << l)
                        sum.add(p[e * RQ]);
#pragma unroll 1
                for (int o = 1; o < (1 << l); o <<= 1) sum.join(o);
                if (part != 0 || r >= nrows) continue;
                T *w = a.ws + sl.dst + r;
                if (flags & T_ACCUM) sum.add(flags & SV_LATE ? __ldcg(w) : xs[max_w + r]);
                if (flags & T_SCATTER) {
                    const int32_t *pp = reinterpret_cast<const int32_t *>(xs + max_w + SV_MAX_ROWS);
                    a.yout[a.perm ? (int64_t)pp[r] : sl.vpos + r] = (double)sum.value();
                } else {
                    *w = sum.value();
                }
            }
        }
        __syncwarp();
        if (lane == 0) sv_arrive(s_done + sr.i);
    }
}

// CTAs per SM, target slots and stages for targets of at most max_w gathered
// columns. Four slots when they are small, two when one holds thousands of
// sources; as many CTAs as fit with at least three stages each (five at most: 40
// warps), the remaining shared memory to the stages. With fewer than four CTAs an
// SM each has 8 consumer warps instead of 4, so that the FP64 pipe and the shared memory
// always see 16 or more of them. SV_MAX_W columns leave room for two CTAs: one alone, with 16 warps, had
// nothing to do while they met at the end of a target (2D semi-nested FP64, 13908 points: 165 us with
// targets of 3535 columns, 93 with two CTAs; 3D, 13824 points: 225 and 195).
template <class T, int CW> cudaError_t sv_configure_cw(int per, int sms, SvConf &s) {
    using Lay = SvLayout<T, CW>;
    const size_t each = (size_t)(SV_SM_BYTES / per - 1024), base = Lay::smem(s.max_w, s.nslots, 0);
    s.ctas = 0;
    s.sms = sms;
    if (each < base + 3 * SvDim<CW>::STAGE) return cudaSuccess;
    s.cw = CW;
    s.nst = (int)std::min<size_t>((each - base) / SvDim<CW>::STAGE, SV_MAX_STAGES);
    s.smem = Lay::smem(s.max_w, s.nslots, s.nst);
    int fit = 0;
    cudaError_t e = cudaFuncSetAttribute(sv_flow_kernel<T, CW>, cudaFuncAttributeMaxDynamicSharedMemorySize, SV_SM_BYTES);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, sv_flow_kernel<T, CW>, SvDim<CW>::NT, s.smem);
    if (e == cudaSuccess) s.ctas = std::min(fit, per) * sms;
    return e;
}
template <class T> cudaError_t sv_configure_t(int max_w, SvConf &s) {
    s = SvConf{};
    s.max_w = (max_w + 3) & ~3;  // keeps the slots and stages 16-byte aligned
    if (max_w < 1 || max_w > SV_MAX_W) return cudaErrorInvalidValue;
    const size_t sb = SvLayout<T, 4>::slot_bytes(s.max_w);
    s.nslots = sb <= 8192 ? 4 : sb <= 16384 ? 3 : 2;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    for (int per = 5; e == cudaSuccess && per >= 2 && s.ctas == 0; --per)
        e = per >= 4 ? sv_configure_cw<T, 4>(per, sms, s) : sv_configure_cw<T, 8>(per, sms, s);
    if (e == cudaSuccess && s.ctas == 0) e = cudaErrorCooperativeLaunchTooLarge;
    return e;
}

template <class T> cudaError_t sv_launch(const SvArgs<T> &args, const SvConf &c, cudaStream_t st) {
    int64_t n[3];
    for (int l = 0; l < 3; ++l) n[l] = args.l1[l] - args.l0[l];
    const int64_t want = n[0] + n[1] + n[2];
    if (want <= 0 && !args.prep) return cudaSuccess;
    // at least four targets a CTA, or one CTA an SM: with fewer CTAs a small product's
    // preparation and barrier are shorter (1D, 4096 points: 55 -> 50 us)
    const int64_t ctas = std::max<int64_t>(std::min<int64_t>(want, c.sms), want / 4);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(ctas, c.ctas));
    SvArgs<T> a = args;
    // CTAs that start with list 0: its share of the work, given in thousandths, but at
    // least a fifth and at most four fifths of them while both lists have targets
    int na = (int)((int64_t)grid * args.na / 1000);
    na = n[0] == 0 ? 0 : n[1] == 0 ? grid : std::max(grid / 5, std::min(na, grid - grid / 5));
    a.na = na;
    int max_w = c.max_w, nslots = c.nslots, nst = c.nst;
    void *pv[] = {(void *)&a, (void *)&max_w, (void *)&nslots, (void *)&nst};
    const void *f = c.cw == 4 ? (const void *)sv_flow_kernel<T, 4> : (const void *)sv_flow_kernel<T, 8>;
    const int nt = c.cw == 4 ? SvDim<4>::NT : SvDim<8>::NT;
    const cudaError_t e = cudaLaunchCooperativeKernel(f, dim3(grid), dim3(nt), pv, c.smem, st);
    count_launch();
    return e;
}

// One CTA per slice, a panel of a target's matrix: source offset, leading dimension, rows, columns, the matrix's
// offset and leading dimension, the panel's first column in it, its columns in all (negative: columns stay in
// order). In FP64 column j of the matrix goes where its consumer group reads it: groups take W / CG neighbouring
// columns each, and position k CG + cg holds the k-th of group cg.
template <class D> __global__ void sv_slice_kernel(const double *__restrict__ src, const int64_t *__restrict__ sl, D *dst, int ct) {
    const int64_t *d = sl + 8 * (int64_t)blockIdx.x;
    const int64_t a = d[0], lda = d[1], o = d[4];
    const int rows = (int)d[2], w = (int)d[3], ld = (int)d[5], c0 = (int)d[6], W = abs((int)d[7]);
    const bool near = sizeof(D) == 8 && d[7] > 0;
    const int CG = ct / (ld / SvVec<D>::n), per = W / CG, rem = W - per * CG, more = rem * (per + 1);
    for (int e = threadIdx.x; e < ld * w; e += blockDim.x) {
        const int c = e / ld, r = e - c * ld, j = c0 + c;
        int to = j;
        if (near) {
            const int cg = j < more ? j / (per + 1) : rem + (j - more) / per;
            to = (j - cg * per - min(cg, rem)) * CG + cg;
        }
        dst[o + (int64_t)to * ld + r] = r < rows ? (D)src[a + (int64_t)c * lda + r] : D(0);
    }
}
template <class D>
cudaError_t sv_slices(const double *src, const int64_t *slices, int64_t n, const SvConf &conf, D *dst, cudaStream_t st) {
    for (int64_t b = 0; b < n; b += 1 << 30) {
        const int64_t m = n - b < (1 << 30) ? n - b : 1 << 30;
        sv_slice_kernel<D><<<(unsigned)m, 256, 0, st>>>(src, slices + 8 * b, dst, 32 * conf.cw);
        count_launch();
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t sv_configure(int max_w, SvConf &f64, SvConf &f32) {
    const cudaError_t e = sv_configure_t<double>(max_w, f64);
    return e != cudaSuccess ? e : sv_configure_t<float>(max_w, f32);
}
cudaError_t launch_sv(const SvArgs<double> &a, const SvConf &c, cudaStream_t st) { return sv_launch<double>(a, c, st); }
cudaError_t launch_sv(const SvArgs<float> &a, const SvConf &c, cudaStream_t st) { return sv_launch<float>(a, c, st); }
cudaError_t launch_sv_slices(const double *src, const int64_t *slices, int64_t n, const SvConf &c, double *dst, cudaStream_t st) {
    return sv_slices(src, slices, n, c, dst, st);
}
cudaError_t launch_sv_slices(const double *src, const int64_t *slices, int64_t n, const SvConf &c, float *dst, cudaStream_t st) {
    return sv_slices(src, slices, n, c, dst, st);
}

}  // namespace h2w
