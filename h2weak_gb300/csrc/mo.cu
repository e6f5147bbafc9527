// FP64 products of many vectors on the tensor cores (sm_103a, tcgen05 kind::f16).
//
// The tensor cores multiply FP16 and add in FP32, which is exact for integers of up to
// eight bits while the sums stay below 2^24. So both operands are written in base 256:
// 256 columns (a part) of a row of a target's matrix as fixed-point numbers of their largest
// entry's scale, ten signed digits each, the part's sources of each vector likewise, and the
// products of digits of the same weight are summed exactly in an accumulator of their own (the
// error-free splitting of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 2012, with digits
// of fixed width). Digits i of A and j of X have weight 256^-(i+j); the products with
// i + j <= 11 and half of those with i + j = 12 are formed. What is left out of a product
// (four digit products of weight 12 and the smaller ones, 2^-74) and the rounding to 80 bits are
// below 2^-73.8 of the row's largest entry in the part times the vector's largest source in it.
// (The two sums of lowest weight add five digit products a column and could in principle pass 2^24: then they
// round by less than a third of that.) Multiply-adds round at 2^-53 of the terms themselves. So
// a part's result that is below 2^-20 of the largest entry times the largest source, where the digits'
// bound no longer lies below theirs, is formed again by multiply-adds (mo_again), and so is every
// result of a vector with an infinity or a NaN in the part: each row has FP64's precision
// in its own terms, also of sparse or widely spread vectors (double-FP32 products, of
// 2^-44 a term: 2^-28). Against long double (stored entries of 900 to 2197 points) results are off by
// 7e-17 .. 1.5e-16 of their norm, those of multiply-adds in the order of the launch by phases by
// 4e-16 .. 1.1e-15; row by row, of the sum of a row's terms' magnitudes, 1e-16 .. 6e-15 and 2e-16 .. 6e-15.
// GB300's FP64 pipe does two multiply-adds a clock and SM; this form multiplies 64 rows x
// 32 columns x 16 vectors in 480 tensor clocks, 68 a clock. Times of a product, on the FP64 pipe
// and here, 64 vectors: 2D 65536 points 6.9 ms and 1.45 ms, 3D 13824 10.4 and 1.37; 19 vectors 3.6
// and 0.76, 5.5 and 0.72; as float-float 64 vectors 2.3 and 2.8. With eight digits, one scale a
// target and no guard it took 0.81 and 0.67 ms, but a term of 2^-k of the largest kept 62 - k bits: 1e-12 of a
// near-field entry for a unit vector. The guard costs 3 to 9 % on vectors without structure; unit
// vectors take up to twice as long as those.
// What bounds it is latency: digits, MMAs and read-out (160 accumulator columns a part, added up as
// integers) follow one another through the rings of one CTA an SM; issue slots are 36 % busy, the
// tensor pipe 21 %, the FP64 pipe 19 % (2D, 64 vectors).
//
// Accumulators: digits 2p+1 and 2p+2 of eight rows each alternate in the 128 rows of an
// MMA (A_p, p = 0 .. 4), so A_p times digit j adds weight 2p+1+j in one half of the
// lanes and the next in the other; the digits of X lie side by side along N, so A_p meets
// all of them in one MMA. Ten accumulators of 16 columns take 160 of the 512 columns of tensor
// memory, and as many are read out meanwhile: 64 vectors are four groups of 16, one after the other on the
// same CTA (A's digits come from the L2 again). After a part a sum is read out, added up in 64-bit
// integers, rounded to FP64 once and added to the row.
//
// Roles of a CTA (one an SM), on a dataflow stream as in sv.cu:
//  * P names targets (and column groups) and streams A's digits, stored in the operand
//    layout, by one bulk copy a chunk of 32 columns;
//  * G waits for the target's producers and copies the FP64 source rows into a ring;
//  * E finds the scale of each source column: every written block of rows has the largest
//    magnitude of each column beside it (mx), so no pass over the sources is needed;
//  * eight warps, in teams that take chunks in turn, turn source rows into digits;
//  * one thread issues the MMAs; eight warps read the accumulators out, write the rows
//    and their columns' largest magnitudes; R releases the consumers.
// The workspace is a plane of 16 columns per group (rows of a group contiguous), with the
// input behind its rows: the launch copies it there as it finds its magnitudes.
// All waits are bounded as in sv.cu (*err 1 grid barrier, 3 dependency, 4 mbarrier).
#include <algorithm>

#include "kernels.cuh"

namespace h2w {
namespace {

constexpr int MO_KC = 32, MO_ND = 10, MO_PART = 8;  // columns a chunk, digits, chunks between read-outs (a part)
constexpr int MO_GC = 16;                           // columns of a group
constexpr int MO_SLOTS = 6;
constexpr int MO_EPI = MO_GC / 2, MO_CONV = 8;     // read-out warps (0 ..), digit warps behind them
constexpr int MO_P = MO_EPI + MO_CONV, MO_G = MO_P + 1, MO_E = MO_P + 2, MO_M = MO_P + 3, MO_R = MO_P + 4;
constexpr int MO_NT = (MO_R + 1) * 32;
constexpr int MO_WAIT = 1 << 20, MO_POLL = 1 << 20;
constexpr int MO_BAD = INT32_MAX;                  // scale of a column with a non-finite source
constexpr int MO_A = 64 * MO_KC * 2 * MO_ND;       // bytes of A's digits of a chunk at 64 rows
constexpr int MO_PARTS = MO_MAX_W / (MO_PART * MO_KC);

struct MoSlot {
    int32_t t;
    uint32_t dst, idx0, grp, ob0, p0;  // p0: its first part
    int32_t nrows, W, flags, nob, rg, cg, last;  // last: the target's last column group
};
struct MoLay {
    static constexpr int GC = MO_GC;
    // rings: digits of A and X (a chunk a stage), source rows
    static constexpr int NS = 4, NR = 4;
    static constexpr int TEAM = 4 * GC / 32, TEAMS = MO_CONV / TEAM;  // digit warps a chunk, chunks at a time
    static constexpr int X = GC * MO_KC * 2 * MO_ND;                  // X's digits of a chunk
    static constexpr int raw = MO_KC * GC * 8;
    static constexpr int off_x = NS * MO_A, off_raw = off_x + NS * X;
    static constexpr int off_bar = off_raw + NR * raw;
    static constexpr int nbar = 2 * NS + 2 * NR + 5 * MO_SLOTS + 6;
    static constexpr int off_slot = (off_bar + 8 * nbar + 15) / 16 * 16;
    static constexpr int off_sx = (off_slot + (int)sizeof(MoSlot) * MO_SLOTS + 15) / 16 * 16;  
    static constexpr int sx = (MO_PARTS + 1) * GC;  // a slot's column scales in each part, then its largest results
    static constexpr int off_misc = off_sx + 4 * sx * MO_SLOTS;
    static constexpr int smem = off_misc + 32;
    static constexpr uint32_t acc_cols = MO_ND * GC, tmem_cols = 512;  // a power of two
    static_assert(off_x % 128 == 0 && off_raw % 128 == 0 && off_bar % 8 == 0 && off_sx % 16 == 0, "vector accesses");
    static_assert(2 * acc_cols <= tmem_cols && smem <= 227 * 1024, "one CTA an SM");
    // A parity wait tells two neighbouring rounds of a slot apart, no more: each waiter has
    // to see every round. So a slot of the rings always falls to the same team.
    static_assert(NS % TEAMS == 0 && NR % TEAMS == 0, "a ring's slots alternate between teams");
};

__device__ __forceinline__ uint32_t mo_sa(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mo_init(uint64_t *b, uint32_t n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mo_sa(b)), "r"(n));
}
__device__ __forceinline__ void mo_arrive(uint64_t *b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mo_sa(b)) : "memory");
}
__device__ __forceinline__ void mo_arrive_tx(uint64_t *b, uint32_t tx) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mo_sa(b)), "r"(tx) : "memory");
}
__device__ __forceinline__ bool mo_try(uint64_t *b, uint32_t par) {
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done)
                 : "r"(mo_sa(b)), "r"(par)
                 : "memory");
    return done != 0;
}
__device__ __noinline__ bool mo_wait_more(uint64_t *b, uint32_t par, volatile int32_t *fail, int32_t *err) {
    for (int it = 0; it < MO_WAIT; ++it) {
        if (mo_try(b, par)) return true;
        if (*fail) return false;
    }
    *fail = 1;
    atomicExch(err, 4);
    return false;
}
__device__ __forceinline__ bool mo_wait(uint64_t *b, uint32_t par, volatile int32_t *fail, int32_t *err) {
    return mo_try(b, par) || mo_wait_more(b, par, fail, err);
}
__device__ __forceinline__ bool mo_wait_warp(uint64_t *b, uint32_t par, volatile int32_t *fail, int32_t *err) {
    return __all_sync(0xffffffffu, mo_wait(b, par, fail, err));
}
struct MoRing {
    int i = 0;
    uint32_t par = 0;
    __device__ __forceinline__ void next(int n) {
        if (++i == n) {
            i = 0;
            par ^= 1u;
        }
    }
};
__device__ __forceinline__ void mo_bulk(void *dst, const void *src, uint32_t bytes, uint64_t *b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     mo_sa(dst)),
                 "l"(src), "r"(bytes), "r"(mo_sa(b))
                 : "memory");
}
__device__ __forceinline__ uint32_t mo_acquire(const void *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// shared-memory matrix descriptor: K-major, no swizzle, 8-row x 16-byte core matrices lbo
// bytes apart along K and 128 along the rows
__device__ __forceinline__ uint64_t mo_desc(uint32_t addr, uint32_t lbo) {
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void mo_mma(uint32_t tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem),
                 "l"(da), "l"(db), "r"(idesc), "r"(acc));
}
// instruction descriptor: D F32, A and B F16 (0), both K-major, M = 128
__host__ __device__ constexpr uint32_t mo_idesc(int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ void mo_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mo_sa(bar))
                 : "memory");
}
__device__ __forceinline__ void mo_tld4(uint32_t *v, uint32_t a) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(a));
}
__device__ __forceinline__ void mo_twait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// NB accumulators (blk columns apart) of four columns as base-256 numbers;
// the lanes of the upper weights (half) finish columns 2 and 3, the others 0 and 1:
// out[i] = lower weights' number x 256 + upper weights'
template <int NB> __device__ __forceinline__ void mo_sum(uint32_t addr, uint32_t blk, int half, int64_t *out) {
    uint32_t v[NB][4];
#pragma unroll
    for (int b = 0; b < NB; ++b) mo_tld4(v[b], addr + (uint32_t)b * blk);
    mo_twait();
    int64_t h[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        auto f = [&](int b) { return (int64_t)(int)__uint_as_float(v[b][c]); };
        h[c] = f(NB - 3) * 65536 + (f(NB - 2) * 256 + f(NB - 1));
        if (NB == 4) h[c] += f(0) * 16777216;
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int64_t keep = half ? h[c + 2] : h[c], send = half ? h[c] : h[c + 2];
        const int64_t got = __shfl_xor_sync(0xffffffffu, send, 8);
        out[c] = ((half ? got : keep) << 8) + (half ? keep : got);
    }
}

// x as a fixed-point number of 80 bits, |x| <= 2^78, at the scale of a largest biased
// exponent ex >= 1 (x 2^-(ex - 1020) 2^80), its bytes offset by 128: digit i of weight
// 256^-i is byte 10 - i minus 128. Exact to 2^-25 of the largest, rounded below. 2^78 is the
// largest power of two that ten signed digits hold.
struct MoFix {
    uint64_t lo;
    uint32_t hi;  // 16 bits
};
__device__ __forceinline__ MoFix mo_fixed(uint64_t b, int ex) {
    const uint32_t hw = (uint32_t)(b >> 32);
    const int e = (int)(hw >> 20) & 0x7ff;
    const uint32_t mh = (hw & 0xfffffu) | (e > 0 ? 0x100000u : 0u);
    const uint64_t m = (uint64_t)mh << 32 | (uint32_t)b;
    const int sh = 25 - min(max(ex - max(e, 1), 0), 80), up = max(sh, 0), down = max(-sh, 0);
    uint64_t lo = (m + ((1ull << down) >> 1)) >> down << up;
    uint32_t hi = (uint32_t)(m >> 32 >> (32 - up));
    if ((int32_t)hw < 0) {
        lo = 0ull - lo;
        hi = ~hi + (lo == 0 ? 1u : 0u);
    }
    const uint64_t o = lo + 0x8080808080808080ull;
    return {o, hi + 0x8080u + (o < lo ? 1u : 0u)};
}
// byte k of two offset numbers as F16 integers in [-128, 127], first in the low half:
// 0x64uu is 1024 + u
__device__ __forceinline__ uint32_t mo_digit2(const MoFix &a, const MoFix &b, int k) {
    const uint32_t wa = k < 4 ? (uint32_t)a.lo : k < 8 ? (uint32_t)(a.lo >> 32) : a.hi;
    const uint32_t wb = k < 4 ? (uint32_t)b.lo : k < 8 ? (uint32_t)(b.lo >> 32) : b.hi;
    const uint32_t t = (__byte_perm(wa, wb, (uint32_t)(k & 3) | (uint32_t)(4 + (k & 3)) << 8) & 0x00ff00ffu) | 0x64006400u;
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(t), "r"(0xe480e480u));  // - 1152
    return r;
}
// the digits of eight neighbouring columns (or rows), `step` bytes a digit
template <class F> __device__ __forceinline__ void mo_digits(const MoFix (&q)[8], F &&at) {
#pragma unroll
    for (int d = 0; d < MO_ND; ++d) {
        uint4 w;
        w.x = mo_digit2(q[0], q[1], MO_ND - 1 - d);
        w.y = mo_digit2(q[2], q[3], MO_ND - 1 - d);
        w.z = mo_digit2(q[4], q[5], MO_ND - 1 - d);
        w.w = mo_digit2(q[6], q[7], MO_ND - 1 - d);
        *reinterpret_cast<uint4 *>(at(d)) = w;
    }
}
// (H 2^48 + L) 2^e in FP64, |H| < 2^55, 0 <= L < 2^48: two exact conversions (an integer beside a
// power of two) of the bits from 52 up and below, one rounding; the power of two goes into the exponent
__device__ __forceinline__ double mo_value(int64_t H, int64_t L, int e) {
    const double hi = __longlong_as_double(0x4338000000000000ll + (H >> 4)) - 6755399441055744.0;
    const double lo = __longlong_as_double(0x4330000000000000ll | (H & 15) << 48 | L) - 4503599627370496.0;
    const double v = fma(hi, 4503599627370496.0, lo);
    const int hw = __double2hiint(v), be = (hw >> 20) & 0x7ff;
    if (be > 0 && be + e > 0 && be + e < 2047) return __hiloint2double(hw + (e << 20), __double2loint(v));
    return v == 0.0 ? v : scalbn(v, e);
}

// A part's product of one row with four columns on the FP64 pipe, for results that the digits may
// leave with fewer bits than multiply-adds: the whole warp, eight of the part's n columns a lane. col: their
// addresses (op: the row's), ix: their sources, x: vectors 0, 1, 4 and 5 in the workspace. Lane
// 16 a + 8 b gets the result of vector 4 a + b. Sparse vectors and rows come here most; their zeros take no FP64
// operation.
__device__ __forceinline__ double mo_again(const double *op, const int64_t *col, const uint32_t *ix, const double *x, int n) {
    constexpr int U = 4;
    const int lane = threadIdx.x & 31;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    bool some = false;
#pragma unroll 1
    for (int j = lane; j - lane < n; j += 32 * U) {
        uint32_t r[U];
        double m[U];
#pragma unroll
        for (int u = 0; u < U; ++u) r[u] = j + u * 32 < n ? ix[j + u * 32] : 0;
#pragma unroll
        for (int u = 0; u < U; ++u) m[u] = j + u * 32 < n ? op[col[j + u * 32]] : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            double2 v = make_double2(0.0, 0.0), w = v;
            if (j + u * 32 < n) {
                const double2 *xr = reinterpret_cast<const double2 *>(x + (int64_t)r[u] * MO_GC);
                v = __ldcg(xr);
                w = __ldcg(xr + 2);
            }
            const int h0 = __double2hiint(v.x) & 0x7fffffff, h1 = __double2hiint(v.y) & 0x7fffffff;
            const int h2 = __double2hiint(w.x) & 0x7fffffff, h3 = __double2hiint(w.y) & 0x7fffffff;
            const bool x0 = (h0 | h1 | h2 | h3 | __double2loint(v.x) | __double2loint(v.y) | __double2loint(w.x) |
                             __double2loint(w.y)) == 0;
            const bool m0 = ((__double2hiint(m[u]) & 0x7fffffff) | __double2loint(m[u])) == 0;
            const bool fin = max(max(h0, h1), max(h2, h3)) < 0x7ff00000;
            if (!__any_sync(0xffffffffu, !x0 && !(m0 && fin))) continue;
            some = true;
            s0 = fma(m[u], v.x, s0);
            s1 = fma(m[u], v.y, s1);
            s2 = fma(m[u], w.x, s2);
            s3 = fma(m[u], w.y, s3);
        }
    }
    if (!some) return 0.0;
    const bool hi = lane & 16, mid = lane & 8;
    const double a0 = (hi ? s2 : s0) + __shfl_xor_sync(0xffffffffu, hi ? s0 : s2, 16);
    const double a1 = (hi ? s3 : s1) + __shfl_xor_sync(0xffffffffu, hi ? s1 : s3, 16);
    s0 = (mid ? a1 : a0) + __shfl_xor_sync(0xffffffffu, mid ? a0 : a1, 8);
#pragma unroll
    for (int q = 4; q > 0; q >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, q);
    return s0;
}

// After a wait ran out the barriers of the copies in flight may lack arrivals of other roles
// for ever: 2 ms, a thousand times a copy's time, let them land before the CTA ends.
__device__ __noinline__ void mo_land() {
    for (int i = 0; i < 200; ++i) __nanosleep(10000);
}

__global__ void __launch_bounds__(MO_NT, 1) mo_kernel(const MoArgs a) {
    using L = MoLay;
    constexpr int GC = MO_GC;
    extern __shared__ __align__(1024) char mo_smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(mo_smem + L::off_bar), *empty = full + L::NS;
    uint64_t *rfull = empty + L::NS, *rempty = rfull + L::NR;
    uint64_t *s_known = rempty + L::NR, *s_dep = s_known + MO_SLOTS, *s_scale = s_dep + MO_SLOTS,
             *s_done = s_scale + MO_SLOTS, *s_free = s_done + MO_SLOTS;
    uint64_t *acc_full = s_free + MO_SLOTS, *acc_empty = acc_full + 2, *quit = acc_full + 4;
    MoSlot *slots = reinterpret_cast<MoSlot *>(mo_smem + L::off_slot);
    int32_t *sxs = reinterpret_cast<int32_t *>(mo_smem + L::off_sx);
    volatile int32_t *fail = reinterpret_cast<volatile int32_t *>(mo_smem + L::off_misc);
    unsigned *gen0 = reinterpret_cast<unsigned *>(mo_smem + L::off_misc + 4);
    uint32_t *tm = reinterpret_cast<uint32_t *>(mo_smem + L::off_misc + 8);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int LD = a.ld;
    if (tid == 0) {
        for (int i = 0; i < L::NS; ++i) {
            mo_init(full + i, 1 + L::TEAM);
            mo_init(empty + i, 1);
        }
        for (int i = 0; i < L::NR; ++i) {
            mo_init(rfull + i, 1);
            mo_init(rempty + i, L::TEAM);
        }
        for (int i = 0; i < MO_SLOTS; ++i) {
            mo_init(s_known + i, 1);
            mo_init(s_dep + i, 1);
            mo_init(s_scale + i, 1);
            mo_init(s_done + i, MO_EPI);
            mo_init(s_free + i, 1 + MO_CONV);  // R, and every digit warp: one with no chunk in it may be behind
        }
        for (int i = 0; i < 2; ++i) {
            mo_init(acc_full + i, 1);
            mo_init(acc_empty + i, MO_EPI);
        }
        mo_init(quit, MO_EPI);
        mo_init(quit + 1, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *fail = 0;
        *gen0 = *reinterpret_cast<volatile unsigned *>(a.bar + 1);  // before this CTA arrives there
    }
    for (int i = tid; i < L::sx * MO_SLOTS; i += MO_NT) sxs[i] = 0;
    if (warp == MO_M) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(mo_sa(tm)),
                     "r"(L::tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    // ---- the launch's preparation: counts, claim counters, rows nobody writes, the
    // workspace blocks' largest magnitudes; the input and its blocks' magnitudes
    {
        const int64_t me = (int64_t)blockIdx.x * MO_NT + tid, all = (int64_t)gridDim.x * MO_NT;
        for (int64_t i = me; i < a.ngrp; i += all) a.rem[i] = a.cnt[i];
        if (me < SV_CTRS) a.ctr[me] = 0;
        for (int64_t i = me; i < (int64_t)a.nzrow * LD; i += all) {
            const int c = (int)(i % LD);
            a.ws[((int64_t)(c / GC) * a.rows + a.zrow[i / LD]) * GC + c % GC] = 0.0;
        }
        for (int64_t i = me; i < (int64_t)a.nwb * LD; i += all) a.mx[i] = 0;
        const int pad = LD - a.ncg * GC;  // result columns that belong to no group
        for (int64_t i = me; i < (a.rows - a.xoff) * pad; i += all) a.yout[i / pad * LD + a.ncg * GC + i % pad] = 0.0;
        int32_t *sm = reinterpret_cast<int32_t *>(mo_smem);  // the rings are not in use yet
        const int per = MO_NT / LD;                          // threads of one column
        const int c = tid % LD, sub = tid / LD;
        double *plane = a.ws + ((int64_t)(c / GC) * a.rows + a.xoff) * GC + c % GC;
        for (int b = blockIdx.x; b < a.nxb; b += gridDim.x) {
            const int64_t r0 = a.xb[b], r1 = a.xb[b + 1];
            uint32_t m = 0;
            if (sub < per)
                for (int64_t r = r0 + sub; r < r1; r += per) {
                    const double x = a.xin[r * LD + c];
                    plane[r * GC] = x;
                    m = max(m, (uint32_t)__double2hiint(x) & 0x7fffffffu);
                }
            if (tid < LD) sm[tid] = 0;
            __syncthreads();
            if (sub < per) atomicMax(sm + c, (int32_t)m);
            __syncthreads();
            if (tid < LD) a.mx[(int64_t)(a.nwb + b) * LD + tid] = sm[tid];
            __syncthreads();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the copies overwrite what was used above
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tm;
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(a.bar, 1u) == gridDim.x - 1) {
            atomicExch(a.bar, 0u);
            __threadfence();
            atomicAdd(a.bar + 1, 1u);
        }
    }

    if (warp == MO_P) {  // -------------------------------------------------- P
        if (lane != 0) return;
        const bool first = (int)blockIdx.x < a.na;
        const int cls = first ? a.na : (int)gridDim.x - a.na, me = first ? blockIdx.x : blockIdx.x - a.na;
        const int ncg = a.ncg;
        int li = 0, taken = 0;
        bool ready = false, ok = true;
        MoHdr h{}, hn{};
        int t = -2, tn = -2;
        MoRing sr, fr;
        bool slot_used = false, stage_used = false;
        while (ok) {
#pragma unroll 1
            for (int cg = 0; ok && t != -2 && cg < ncg; ++cg) {
                if (slot_used && !mo_wait(s_free + sr.i, sr.par ^ 1u, fail, a.err)) {
                    ok = false;
                    break;
                }
                MoSlot &sl = slots[sr.i];
                sl.t = t;
                const int rg = 2 * ((h.nrows + 7) / 8);
                if (t >= 0) {
                    sl.dst = h.dst;
                    sl.idx0 = h.idx0;
                    sl.grp = h.grp;
                    sl.ob0 = h.ob0;
                    sl.nrows = h.nrows;
                    sl.W = h.W;
                    sl.flags = h.flags;
                    sl.nob = h.nob;
                    sl.p0 = h.p0;
                    sl.rg = rg;
                    sl.cg = cg;
                    sl.last = cg == ncg - 1;
                }
                mo_arrive(s_known + sr.i);
                sr.next(MO_SLOTS);
                if (sr.i == 0) slot_used = true;
                if (t < 0) {
                    ok = false;
                    break;
                }
                const char *A = a.img + h.img;
                const uint32_t bytes = (uint32_t)(256 * MO_ND * rg);
#pragma unroll 1
                for (int c = 0; c < h.W; c += MO_KC) {
                    if (stage_used && !mo_wait(empty + fr.i, fr.par ^ 1u, fail, a.err)) {
                        ok = false;
                        break;
                    }
                    mo_arrive_tx(full + fr.i, bytes);
                    mo_bulk(mo_smem + fr.i * MO_A, A, bytes, full + fr.i);
                    A += bytes;
                    fr.next(L::NS);
                    if (fr.i == 0) stage_used = true;
                }
            }
            if (!ok) break;
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
                        while (ok && mo_acquire(a.bar + 1) == *gen0)
                            if (++it > MO_POLL || *fail) {
                                atomicExch(a.err, 1);
                                *fail = 1;
                                ok = false;
                            }
                        if (!ok) break;
                        ready = true;
                    }
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
        if (*fail) mo_land();
        return;
    }
    if (warp == MO_G) {  // -------------------------------------------------- G
        MoRing sr, rr;
        bool used = false, ready = false;
        for (;; sr.next(MO_SLOTS)) {
            if (!mo_wait_warp(s_known + sr.i, sr.par, fail, a.err)) break;
            const MoSlot &sl = slots[sr.i];
            if (sl.t < 0) break;
            const uint32_t *ix = a.idx + sl.idx0;
            const double *plane = a.ws + (int64_t)sl.cg * a.rows * GC;
            const int W = sl.W;
            uint32_t row = lane < W ? ix[lane] : 0;
            bool good = true;
            if (lane == 0) {
                int it = 0;
                if (!ready)
                    while (good && mo_acquire(a.bar + 1) == *gen0)
                        if (++it > MO_POLL || *fail) {
                            good = false;
                            atomicExch(a.err, 1);
                        }
                it = 0;
                while (good && (int32_t)mo_acquire(a.rem + sl.grp) > 0)
                    if (++it > MO_POLL || *fail) {
                        good = false;
                        atomicExch(a.err, 3);
                    }
                if (!good) *fail = 1;
            }
            ready = true;
            if (!__shfl_sync(0xffffffffu, (int)good, 0)) break;
            __syncwarp();
            asm volatile("fence.proxy.async.global;" ::: "memory");  // the copies read what other CTAs stored
            if (lane == 0) mo_arrive(s_dep + sr.i);
            bool lost = false;
#pragma unroll 1
            for (int c = 0; c < W; c += MO_KC) {
                const uint32_t ahead = c + MO_KC + lane < W ? ix[c + MO_KC + lane] : 0;
                if (used && !mo_wait_warp(rempty + rr.i, rr.par ^ 1u, fail, a.err)) {
                    lost = true;
                    break;
                }
                const int kw = min(MO_KC, W - c);
                // runs of consecutive rows as one copy each
                const uint32_t prev = __shfl_up_sync(0xffffffffu, row, 1);
                const bool in = lane < kw;
                const bool start = in && (lane == 0 || row != prev + 1);
                const unsigned brk = __ballot_sync(0xffffffffu, start || !in);
                double *R = reinterpret_cast<double *>(mo_smem + L::off_raw + rr.i * L::raw);
                if (lane == 0) mo_arrive_tx(rfull + rr.i, (uint32_t)kw * GC * 8u);
                __syncwarp();
                if (start) {
                    const unsigned after = brk & ~((2u << lane) - 1u);
                    const int end = after ? __ffs(after) - 1 : 32;
                    mo_bulk(R + lane * GC, plane + (int64_t)row * GC, (uint32_t)(end - lane) * GC * 8u, rfull + rr.i);
                }
                rr.next(L::NR);
                if (rr.i == 0) used = true;
                row = ahead;
            }
            if (lost) break;
        }
        if (*fail) mo_land();
        return;
    }
    if (warp == MO_E) {  // -------------------------------------------------- E
        constexpr int PER = 32 * 4 / GC;  // blocks a warp reads at once (a lane reads four columns)
        const int c4 = (lane * 4) % GC, sub = lane * 4 / GC;
        bool ready = false;
        for (MoRing sr;; sr.next(MO_SLOTS)) {
            if (!mo_wait_warp(s_known + sr.i, sr.par, fail, a.err)) break;
            const MoSlot &sl = slots[sr.i];
            if (sl.t < 0) break;
            const int parts = (sl.W + MO_PART * MO_KC - 1) / (MO_PART * MO_KC), col = sl.cg * GC + c4;
            // the producers' magnitudes: a wait of its own, for G is behind with its copies
            bool good = true;
            if (lane == 0) {
                int it = 0;
                while (good && !ready && mo_acquire(a.bar + 1) == *gen0)
                    if (++it > MO_POLL || *fail) {
                        good = false;
                        atomicExch(a.err, 1);
                    }
                it = 0;
                while (good && (int32_t)mo_acquire(a.rem + sl.grp) > 0)
                    if (++it > MO_POLL || *fail) {
                        good = false;
                        atomicExch(a.err, 3);
                    }
                if (!good) *fail = 1;
            }
            ready = true;
            if (!__shfl_sync(0xffffffffu, (int)good, 0)) break;
            __syncwarp();
#pragma unroll 1
            for (int p = 0; p < parts; ++p) {
                const uint2 list = a.plist[sl.p0 + p];
                const uint32_t *bl = a.blist + list.x;
                int4 m = make_int4(0, 0, 0, 0);
#pragma unroll 4
                for (int b = sub; b < (int)list.y; b += PER) {
                    const int4 v = __ldcg(reinterpret_cast<const int4 *>(a.mx + (int64_t)bl[b] * LD + col));
                    m.x = max(m.x, v.x);
                    m.y = max(m.y, v.y);
                    m.z = max(m.z, v.z);
                    m.w = max(m.w, v.w);
                }
#pragma unroll
                for (int o = GC / 4; o < 32; o <<= 1) {
                    m.x = max(m.x, __shfl_xor_sync(0xffffffffu, m.x, o));
                    m.y = max(m.y, __shfl_xor_sync(0xffffffffu, m.y, o));
                    m.z = max(m.z, __shfl_xor_sync(0xffffffffu, m.z, o));
                    m.w = max(m.w, __shfl_xor_sync(0xffffffffu, m.w, o));
                }
                if (lane * 4 < GC) {
                    auto sc = [](int v) { return v >= 0x7ff00000 ? MO_BAD : v >> 20; };  // 0: zeros or subnormal numbers
                    *reinterpret_cast<int4 *>(sxs + sr.i * L::sx + p * GC + c4) = make_int4(sc(m.x), sc(m.y), sc(m.z), sc(m.w));
                }
            }
            __syncwarp();
            if (lane == 0) mo_arrive(s_scale + sr.i);
        }
        return;
    }
    if (warp == MO_M) {  // -------------------------------------------------- MMA
        MoRing sr, fr, ar;
        bool acc_used = false;
        // descriptors: fixed fields, then addresses in 16-byte units
        const uint64_t db0 = mo_desc(mo_sa(mo_smem + L::off_x), GC * 16u * MO_ND);
        for (;; sr.next(MO_SLOTS)) {
            if (!mo_wait_warp(s_known + sr.i, sr.par, fail, a.err)) break;
            if (slots[sr.i].t < 0) break;
            const int W = slots[sr.i].W, nch = (W + MO_KC - 1) / MO_KC;
            const uint32_t alb = (uint32_t)slots[sr.i].rg * 128u;
            const uint64_t da0 = mo_desc(mo_sa(mo_smem), alb);
            bool lost = false;
#pragma unroll 1
            for (int q = 0; q < nch; ++q) {
                const bool head = q % MO_PART == 0, tail = q % MO_PART == MO_PART - 1 || q == nch - 1;
                if (head && acc_used && !mo_wait_warp(acc_empty + ar.i, ar.par ^ 1u, fail, a.err)) lost = true;
                if (!lost && !mo_wait_warp(full + fr.i, fr.par, fail, a.err)) lost = true;
                if (lost) break;
                if (lane == 0) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t da = da0 + (uint64_t)(fr.i * (MO_A / 16)), db = db0 + (uint64_t)(fr.i * (L::X / 16));
                    const uint32_t acc = tmem + (uint32_t)ar.i * L::acc_cols;
                    // A_p against its ND - 2p digits of X at once (GC (ND - 2p) <= 256 columns)
#pragma unroll
                    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
                        for (int p = 0; p < MO_ND / 2; ++p)
                            mo_mma(acc + (uint32_t)(2 * p * GC), da + (uint64_t)((4 * p + 2 * ks) * (alb >> 4)),
                                   db + (uint64_t)(ks * 2 * MO_ND * GC), mo_idesc((MO_ND - 2 * p) * GC),
                                   p == 0 && ks == 0 ? (head ? 0u : 1u) : 1u);
                    mo_commit(empty + fr.i);
                    if (tail) mo_commit(acc_full + ar.i);
                }
                __syncwarp();
                fr.next(L::NS);
                if (tail) {
                    ar.next(2);
                    if (ar.i == 0) acc_used = true;
                }
            }
            if (lost) break;
        }
        // the read-out warps are done with the tensor memory, and so are the MMAs
        if (*fail && lane == 0) mo_commit(quit + 1);
        for (int it = 0; it < MO_WAIT && !mo_try(quit, 0); ++it) {
        }
        if (*fail)
            for (int it = 0; it < MO_WAIT && !mo_try(quit + 1, 0); ++it) {
            }
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::tmem_cols));
        return;
    }
    if (warp == MO_R) {  // -------------------------------------------------- R
        for (MoRing sr;; sr.next(MO_SLOTS)) {
            if (!mo_wait_warp(s_known + sr.i, sr.par, fail, a.err)) break;
            const MoSlot &sl = slots[sr.i];
            if (sl.t < 0) break;
            const uint2 gi = sl.last ? a.grp[sl.grp] : make_uint2(0, 0);
            const uint32_t mine = lane < gi.y ? a.cons[gi.x + lane] : 0;
            const int nob = sl.nob, cg = sl.cg;
            const uint32_t ob0 = sl.ob0;
            if (!mo_wait_warp(s_done + sr.i, sr.par, fail, a.err)) break;
            int32_t *big = sxs + sr.i * L::sx + MO_PARTS * GC;
            if (lane < GC) {
                const int32_t v = big[lane];
                big[lane] = 0;
                for (int b = 0; b < nob; ++b) atomicMax(a.mx + (int64_t)(ob0 + b) * LD + cg * GC + lane, v);
            }
            __syncwarp();
            if (lane == 0) mo_arrive(s_free + sr.i);
            if (gi.y > 0) {
                asm volatile("fence.acq_rel.gpu;" ::: "memory");  // rows and magnitudes before the counts
                __syncwarp();
                if (lane < gi.y) atomicSub(a.rem + mine, 1);
#pragma unroll 1
                for (uint32_t e = 32 + lane; e < gi.y; e += 32) atomicSub(a.rem + a.cons[gi.x + e], 1);
            }
        }
        return;
    }
    if (warp >= MO_EPI) {  // ------------------------------------------- digits
        // unit = source column n x eight rows of the chunk: 16 bytes of each digit
        const int team = (warp - MO_EPI) / L::TEAM, u = (warp - MO_EPI) % L::TEAM * 32 + lane, n = u % GC, kg = u / GC;
        MoRing sr, rr, fr;
        bool used = false;
        int turn = 0;
        for (;; sr.next(MO_SLOTS)) {
            if (!mo_wait_warp(s_known + sr.i, sr.par, fail, a.err)) return;
            if (slots[sr.i].t < 0) return;
            const int W = slots[sr.i].W;
            if (!mo_wait_warp(s_scale + sr.i, sr.par, fail, a.err)) return;
#pragma unroll 1
            for (int c = 0; c < W; c += MO_KC) {
                if (turn == team) {
                    if (!mo_wait_warp(rfull + rr.i, rr.par, fail, a.err)) return;
                    if (used && !mo_wait_warp(empty + fr.i, fr.par ^ 1u, fail, a.err)) return;
                    const uint64_t *R = reinterpret_cast<const uint64_t *>(mo_smem + L::off_raw + rr.i * L::raw) + kg * 8 * GC + n;
                    const int ex = max(sxs[sr.i * L::sx + c / (MO_PART * MO_KC) * GC + n], 1);
                    MoFix q[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) q[i] = mo_fixed(R[i * GC], ex);
                    char *X = mo_smem + L::off_x + fr.i * L::X + (kg * MO_ND * GC + n) * 16;  // [8 rows][digit][column]
                    mo_digits(q, [&](int d) { return X + d * GC * 16; });
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        mo_arrive(rempty + rr.i);
                        mo_arrive(full + fr.i);
                    }
                }
                turn = turn + 1 == L::TEAMS ? 0 : turn + 1;
                rr.next(L::NR);
                fr.next(L::NS);
                if (fr.i == 0) used = true;
            }
            if (lane == 0) mo_arrive(s_free + sr.i);
        }
    }
    // ------------------------------------------------------------------ read-out
    // warps w and w + 4 read lanes 32 (w % 4) .., eight columns each, in two rounds of four. Lanes l
    // and l + 8 hold the same rows' accumulators of neighbouring weights; the lower lane
    // finishes two of the columns (c, c + 1; then c + 4, c + 5), the upper the others.
    const int quad = warp & 3, c0 = 8 * (warp >> 2), half = (lane >> 3) & 1;
    const int row = 16 * quad + 8 * (lane >> 4) + (lane & 7), c = c0 + 2 * half;
    MoRing sr, ar;
    for (;; sr.next(MO_SLOTS)) {
        if (!mo_wait_warp(s_known + sr.i, sr.par, fail, a.err)) break;
        const MoSlot &sl = slots[sr.i];
        if (sl.t < 0) break;
        const int nrows = sl.nrows, flags = sl.flags, nch = (sl.W + MO_KC - 1) / MO_KC;
        const bool on = 16 * quad < nrows && c0 < GC, mine = on && row < nrows;
        double *w = a.ws + ((int64_t)sl.cg * a.rows + sl.dst + row) * GC + c;
        bool lost = false;
#pragma unroll 1
        for (int q0 = 0; q0 < nch; q0 += MO_PART) {
            const bool last = q0 + MO_PART >= nch, add = q0 > 0 || (flags & T_ACCUM);
            const int ea = a.sa[((int64_t)sl.p0 + q0 / MO_PART) * 64 + row];  // the row's scale in this part
            double prev[4] = {0.0, 0.0, 0.0, 0.0};
            if (add) {  // the rows that are added to, on their way while the MMAs run
                if (q0 == 0 && !mo_wait_warp(s_dep + sr.i, sr.par, fail, a.err)) {
                    lost = true;
                    break;
                }
                if (mine) {
                    const double2 p0 = reinterpret_cast<const double2 *>(w)[0], p1 = reinterpret_cast<const double2 *>(w)[2];
                    prev[0] = p0.x;
                    prev[1] = p0.y;
                    prev[2] = p1.x;
                    prev[3] = p1.y;
                }
            }
            if (!mo_wait_warp(acc_full + ar.i, ar.par, fail, a.err)) {
                lost = true;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (on) {
                const uint32_t acc = tmem + (uint32_t)ar.i * L::acc_cols + ((uint32_t)(32 * quad) << 16) + (uint32_t)c0;
                double r[4];
                unsigned small = 0;  // columns whose result is below the guard
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    int64_t H[2], Mi[2], Lo[2];
                    mo_sum<4>(acc + 4 * g, GC, half, H);
                    mo_sum<3>(acc + 4 * g + 4 * GC, GC, half, Mi);
                    mo_sum<3>(acc + 4 * g + 7 * GC, GC, half, Lo);
                    const int32_t *sx = sxs + sr.i * L::sx + q0 / MO_PART * GC + c + 4 * g;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int s = sx[i], k = 2 * g + i;
                        Mi[i] += Lo[i] >> 24;  // 24 bits of each below the first
                        r[k] = mo_value(H[i] + (Mi[i] >> 24), (Mi[i] & 0xffffff) << 24 | (Lo[i] & 0xffffff),
                                        max(ea, 1) + min(max(s, 1), 0x7ff) - 2040 - 96);
                        const int have = max((__double2hiint(r[k]) >> 20) & 0x7ff, (__double2hiint(prev[k]) >> 20) & 0x7ff);
                        if (s == MO_BAD || (ea > 0 && s > 0 && have < ea + s - 1021 - a.guard)) small |= 1u << k;
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mo_arrive(acc_empty + ar.i);
                if (!mine) small = 0;
                if (__any_sync(0xffffffffu, small != 0)) {
                    // the sources' rows are there (the digits came from them); G's arrival orders these reads too
                    if (!mo_wait_warp(s_dep + sr.i, sr.par, fail, a.err)) {
                        lost = true;
                        break;
                    }
#pragma unroll 1
                    for (unsigned todo = __ballot_sync(0xffffffffu, small != 0); todo; todo &= todo - 1) {
                        const int src = __ffs(todo) - 1;
                        const double z = mo_again(a.op + 16 * quad + 8 * (src >> 4) + (src & 7),
                                                  a.col + ((int64_t)sl.p0 + q0 / MO_PART) * (MO_PART * MO_KC),
                                                  a.idx + sl.idx0 + q0 * MO_KC,
                                                  a.ws + (int64_t)sl.cg * a.rows * GC + c0 + 2 * ((src >> 3) & 1),
                                                  min(MO_PART * MO_KC, sl.W - q0 * MO_KC));
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const double zk = __shfl_sync(0xffffffffu, z, 8 * k);
                            if (lane == src && (small >> k & 1u)) r[k] = zk;
                        }
                    }
                }
                if (add)
#pragma unroll
                    for (int k = 0; k < 4; ++k) r[k] += prev[k];
                if (mine) {
                    double *o = last && (flags & T_SCATTER) ? a.yout + (int64_t)(sl.dst + row) * LD + sl.cg * GC + c : w;
                    reinterpret_cast<double2 *>(o)[0] = make_double2(r[0], r[1]);
                    reinterpret_cast<double2 *>(o)[2] = make_double2(r[2], r[3]);
                }
                if (last && !(flags & T_SCATTER)) {
                    int32_t *big = sxs + sr.i * L::sx + MO_PARTS * GC + c;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        uint32_t m = mine ? (uint32_t)__double2hiint(r[k]) & 0x7fffffffu : 0u;
                        m = half ? __reduce_max_sync(0xff00ff00u, m) : __reduce_max_sync(0x00ff00ffu, m);
                        if ((lane & 0x17) == 0) atomicMax(big + k + (k & 2), (int32_t)m);
                    }
                }
            } else if (lane == 0) {
                mo_arrive(acc_empty + ar.i);
            }
            ar.next(2);
        }
        if (lost) break;
        __syncwarp();
        if (lane == 0) mo_arrive(s_done + sr.i);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (lane == 0) mo_arrive(quit);
}

// y (n x ld, interleaved) from the workspace planes' rows r0 ..
__global__ void mo_unplane_kernel(const double *__restrict__ ws, int64_t rows, int64_t r0, int ncg, int ld, int64_t n,
                                  double *__restrict__ y) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n * ld; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = e / ld;
        const int c = (int)(e - r * ld);
        y[e] = c < ncg * MO_GC ? ws[((int64_t)(c / MO_GC) * rows + r0 + r) * MO_GC + c % MO_GC] : 0.0;
    }
}

// The digits of target t's matrix in the operand layout, and its rows' scales in each part (biased
// exponents, 0: no normal number), and the addresses of its columns: one CTA a target; slices sl[s0[t] ..]: (address, leading
// dimension, rows, columns, -, -)
__global__ void mo_image_kernel(const MoHdr *__restrict__ hdr, const int64_t *__restrict__ s0, const int64_t *__restrict__ sl,
                                const double *__restrict__ op, char *__restrict__ img, int32_t *__restrict__ sa,
                                int64_t *__restrict__ adr, int32_t *bad) {
    __shared__ int64_t col[MO_MAX_W];
    __shared__ int32_t mx[MO_PARTS][64];
    const int t = blockIdx.x, tid = threadIdx.x;
    const MoHdr h = hdr[t];
    const int W = h.W, parts = (W + MO_PART * MO_KC - 1) / (MO_PART * MO_KC);
    if (W > MO_MAX_W || h.nrows > 64) {
        if (tid == 0) atomicExch(bad, 1);
        return;
    }
    int at = 0;
    for (int64_t q = s0[t]; q < s0[t + 1]; ++q) {
        const int64_t ad = sl[6 * q], ld = sl[6 * q + 1];
        const int w = (int)sl[6 * q + 3];
        for (int c = tid; c < w && at + c < W; c += blockDim.x) col[at + c] = ad + c * ld;
        at += w;
    }
    for (int i = tid; i < parts * 64; i += blockDim.x) mx[i / 64][i % 64] = 0;
    __syncthreads();
    for (int e = tid; e < h.nrows * W; e += blockDim.x) {
        const int c = e / h.nrows, r = e - c * h.nrows;
        atomicMax(&mx[c / (MO_PART * MO_KC)][r], (int32_t)((uint32_t)__double2hiint(op[col[c] + r]) & 0x7fffffffu));
    }
    __syncthreads();
    for (int i = tid; i < parts * 64; i += blockDim.x) {
        int32_t &m = mx[i / 64][i % 64];
        if (m >= 0x7ff00000) atomicExch(bad, 1);
        m >>= 20;
        sa[(int64_t)h.p0 * 64 + i] = m;
    }
    for (int c = tid; c < W; c += blockDim.x) adr[(int64_t)h.p0 * (MO_PART * MO_KC) + c] = col[c];
    __syncthreads();
    const int rg = 2 * ((h.nrows + 7) / 8), rows = rg * 4, nch = (W + MO_KC - 1) / MO_KC;
    for (int u = tid; u < nch * 4 * rows; u += blockDim.x) {
        const int r = u % rows, kg = u / rows % 4, ch = u / (4 * rows);
        MoFix q[8];
        for (int i = 0; i < 8; ++i) {
            const int c = ch * MO_KC + kg * 8 + i;
            const double v = r < h.nrows && c < W ? op[col[c] + r] : 0.0;
            q[i] = mo_fixed((uint64_t)__double_as_longlong(v), max(mx[ch / MO_PART][r], 1));
        }
        char *o = img + h.img + (int64_t)ch * (256 * MO_ND * rg) + kg * rg * 128 + (2 * (r / 8)) * 128 + (r % 8) * 16;
        mo_digits(q, [&](int d) { return o + (d / 2) * 4 * rg * 128 + (d & 1) * 128; });
    }
}

cudaError_t mo_launch(const MoArgs &args, cudaStream_t st) {
    using L = MoLay;
    static PerDevice<bool> attr_of;
    bool &attr = attr_of.here();
    cudaError_t e = attr ? cudaSuccess : cudaFuncSetAttribute(mo_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::smem);
    if (e != cudaSuccess) return e;
    attr = true;
    const int sms = device_sms();
    int64_t n[3];
    for (int l = 0; l < 3; ++l) n[l] = args.l1[l] - args.l0[l];
    const int64_t want = std::max<int64_t>(n[0] + n[1] + n[2], 1);
    const int grid = (int)std::min<int64_t>(want, sms);
    MoArgs a = args;
    const int na = (int)((int64_t)grid * args.na / 1000);
    a.na = n[0] == 0 ? 0 : n[1] == 0 ? grid : std::max(grid / 5, std::min(na, grid - grid / 5));
    void *pv[] = {(void *)&a};
    e = cudaLaunchCooperativeKernel((const void *)mo_kernel, dim3(grid), dim3(MO_NT), pv, L::smem, st);
    count_launch();
    return e;
}

}  // namespace

int64_t mo_image_bytes(int nrows, int W) { return (int64_t)((W + MO_KC - 1) / MO_KC) * (256 * MO_ND) * 2 * ((nrows + 7) / 8); }
int mo_part_columns() { return MO_PART * MO_KC; }
cudaError_t launch_mo_image(const MoHdr *hdr, int64_t nt, const int64_t *s0, const int64_t *slices, const double *op,
                            char *img, int32_t *sa, int64_t *adr, int32_t *bad, cudaStream_t st) {
    if (nt <= 0) return cudaSuccess;
    mo_image_kernel<<<(unsigned)nt, 256, 0, st>>>(hdr, s0, slices, op, img, sa, adr, bad);
    count_launch();
    return cudaGetLastError();
}
cudaError_t launch_mo(const MoArgs &a, cudaStream_t st) {
    const bool ok = (a.ld == 16 || a.ld == 32 || a.ld == 64) && a.ncg >= 1 && a.ncg * MO_GC <= a.ld;
    return ok ? mo_launch(a, st) : cudaErrorInvalidValue;
}
cudaError_t launch_mo_unplane(const MoArgs &a, int64_t r0, int64_t n, double *y, cudaStream_t st) {
    mo_unplane_kernel<<<1216, 256, 0, st>>>(a.ws, a.rows, r0, a.ncg, a.ld, n, y);
    count_launch();
    return cudaGetLastError();
}

}  // namespace h2w
