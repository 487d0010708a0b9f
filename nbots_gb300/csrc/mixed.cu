// Mixed-precision Jacobi-PCG with reliable updates, one cooperative launch.
//
// GB300 runs FP32 at many times its FP64 rate, and the stiffness matrices
// here have condition numbers near 1e8, where plain FP32 CG needs several
// times more iterations than FP64.  Measured on the lognormal cantilever
// (1M dof), the inflation comes from three places: the precision of the
// matrix values (even 32 significant bits cost 1.33x the iterations: the
// inner operator must match the FP64 one behind the residual), FP32 search
// directions p and FP32 products A p, and an FP32 correction x.  The
// iteration count alone is not the whole story: with about 40-bit matrix
// values and an FP32 residual the counts match FP64, yet the solution
// keeps an error of 1e-8 to 1e-7 (varying with rounding details) in the
// smooth modes, whose share of the residual is too small for the stopping
// test to see.  A CPU emulation of this solver on the cantilever traced it
// to the FP32 residual (its rounding each iteration feeds those modes) and
// to the matrix precision; with both raised the error matches FP64's.  So
// the inner iteration runs on the FP32 pipes with:
//   matrix      FP32 hi + a 23-bit remainder in units of 2^-46 hi
//               (about 47 significant bits in 7 B/value instead of 8),
//   p, A p      FP32 hi + FP32 lo per dof (float-float),
//   x, r        float-float,
// products and sums by error-free transformations (TwoProduct with FMA,
// TwoSum), dot products with compensated FP32 sums per thread and
// float-float sums across threads and blocks.  A reliable update (Sleijpen
// & van der Vorst 1996) adds x to the FP64 solution and recomputes
// r = b - A u in FP64 with the FP64 values whenever |r| has fallen by
// `delta` since the last one; p is kept, so the Krylov progress survives.
// Convergence is judged on the FP64 residual only (row_residual).  Three grid barriers per
// iteration in the global-gather form (L1 | L2 | L3 of
// cg_precond_jacobi.c:50-74), two sums over the grid in the ghost-node form
// below and in the slice form (mixed_slice.cuh): folding L3
// into the next SpMV (each block rebuilding z + beta p for the columns it
// reads) measured slower, 77 vs 66 us per iteration at 1M dof, because the
// float-float rebuild per column costs more issue slots and gather bytes
// than the barrier it saves.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <type_traits>
#include <vector>

#include "allreduce.cuh"
#include "ghost_plan.cuh"
#include "perm.cuh"
#include "persist.cuh"

using namespace nbg;

// Keep each block's own-row vectors in shared memory when they fit
// (overridable at build time for tuning).
#ifndef NBG_MIXED_RESIDENT
#define NBG_MIXED_RESIDENT 1
#endif
// The vectors p, A p, x and r are float-float, stored as float4 {hi of both
// dofs, lo of both} per node row: one 16-byte load or store per row and
// vector, one gather per block entry.  (With bfloat16 low parts for p and
// A p the 4M-dof unstructured T3 case needed 26,067 iterations against
// FP64's 22,323; with FP32 ones 22,563.)
#ifndef NBG_MIXED_UNROLL
#define NBG_MIXED_UNROLL 4  // entries in flight per lane in the SpMV
#endif
// One 1024-thread block per SM: with two 512-thread blocks the SM serves one
// block's warps first and the other block's SpMV ends several microseconds
// later, which the next barrier then waits for.
#ifndef NBG_MIXED_THREADS
#define NBG_MIXED_THREADS 1024
#endif
#ifndef NBG_MIXED_MIN_BLOCKS
#define NBG_MIXED_MIN_BLOCKS 1
#endif
constexpr int kMixThreads = NBG_MIXED_THREADS;
constexpr int kMixMinBlocks = NBG_MIXED_MIN_BLOCKS;
// Batched launches give every system at least one block, so they use
// smaller blocks (more of them per SM) than the single-system launch.
#ifndef NBG_BATCH_THREADS
#define NBG_BATCH_THREADS 256
#endif
#ifndef NBG_BATCH_MIN_BLOCKS
#define NBG_BATCH_MIN_BLOCKS 4
#endif
constexpr int kBatThreads = NBG_BATCH_THREADS;
constexpr int kBatMinBlocks = NBG_BATCH_MIN_BLOCKS;
constexpr int kUnroll = NBG_MIXED_UNROLL;
// The ghost-node form's grid barriers by counting (grid_barrier_count),
// whose arrival is a reduction with no return value: 0.2422 against 0.2443
// s per 1M-dof solve with the arrival that returns the old word
// (grid_barrier).
#ifndef NBG_BARRIER_COUNT
#define NBG_BARRIER_COUNT 1
#endif
namespace {

struct MixArgs {
    nbg_bsr_t A;
    const double* b;
    double* u;
    float4* p;             // search direction, global (gathered by neighbours)
    float4 *x4, *r4, *w4;  // x, r, A p of the rows: own rows when they do not fit in
                           // shared memory (the ghost form keeps x and r there)
    const float *ph, *pl;  // the standalone operator's input, hi and lo apart
    uint32_t max_iter;
    double tol, delta;
    unsigned flags;
    uint32_t keep;     // share of each block's matrix stream kept in L2, of 2^32 (all ones: all)
};

// Whether the matrix of slice `at` of a block's n stays in L2 between
// iterations: a share `keep` of the slices.  With the first ones kept, DRAM had
// nothing to do while every warp worked on them (1M-dof ghost form: 33.8
// against 34.2 us per iteration); spread with a period, some pairs of warps,
// which take every (kThreads / 64)th slice, had theirs all in L2 and others all
// from DRAM (482,000 dof, half kept: 18.7 against 16.9).  So the fractional
// parts of multiples of the golden ratio, along each pair's slices.  Batched
// launches keep all or nothing (the test costs them 4 %).
__device__ __forceinline__ bool kept_at(uint32_t j, uint32_t keep) {
    return j * 0x9E3779B9u < keep || keep == 0xFFFFFFFFu;
}
template <int kThreads>
__device__ __forceinline__ bool kept(const MixArgs& a, uint32_t at, uint32_t n) {
    if (kThreads != kMixThreads) return a.keep != 0;
    constexpr uint32_t kPairs = kThreads / 64;
    return kept_at(at % kPairs * ((n + kPairs - 1) / kPairs) + at / kPairs, a.keep);
}

// One system of a launch: its slices, its blocks and its synchronisation.
struct Group {
    double* part;  // L1 [0,K), L2 [K,3K), init/update [3K,6K), K = pstride
    unsigned* bar;
    int* status;
    double* res;              // niter, updates, status, rr64, bb, b.u
    unsigned char* sums;      // words of the two fixed-point sums, 2 kExactBytes
    uint32_t s_begin, s_end;  // slices
    uint32_t g_base, g_size;  // blocks [g_base, g_base + g_size) of the launch
    uint32_t pstride;
};



// Scalar state of one solve, kept by thread 0 of every block of the group
// (each block derives the same values from the same partial sums).  Per
// iteration it runs on the FP32 pipes: p.w, r.z and |r|^2 arrive as
// float-float sums, the step lengths are float-float quotients (ff_div) and
// the update test compares FP32 leading parts.  GB300 issues FP64 at a small
// fraction of its FP32 rate: one FP64 division on thread 0 held its block
// for about half a microsecond, twice per iteration.  FP64 stays where the
// result is judged, on the true residual at the start and at each reliable
// update.
struct MixScalars {
    FF rz;                          // r.z of the current residual
    double rr64, bb, target2;       // true |r|^2, |b|^2, stopping threshold
    float rmax2, target2f, delta2;  // update test
    float last;                     // recursive |r|^2 at the last update
    uint32_t k, nupd;
    int converged;

    __device__ __forceinline__ void clear() {
        rz = FF{0.f, 0.f};
        rr64 = bb = target2 = 0.0;
        rmax2 = target2f = delta2 = last = 0.f;
        k = nupd = 0;
        converged = 0;
    }
    // The start's sums {|r|^2, |b|^2, r.z} (FP64): 2 stop, 0 iterate.
    __device__ __forceinline__ int start(const double (&t)[3], const MixArgs& a) {
        rr64 = t[0];
        bb = t[1];
        rz = ff_from_double(t[2]);
        target2 = (a.flags & NBG_CG_RELATIVE) ? a.tol * a.tol * bb : a.tol * a.tol;
        target2f = (float)target2;
        delta2 = (float)(a.delta * a.delta);
        rmax2 = (float)rr64;
        converged = rr64 <= target2;  // not where it is NaN
        return (!(rr64 > target2) || a.max_iter == 0) ? 2 : 0;
    }
    __device__ __forceinline__ FF alpha(FF pw) const { return ff_div(rz, pw); }
    // The recursive residual's {r.z, |r|^2}: 1 when a reliable update is
    // due, else 0 with beta.
    __device__ __forceinline__ int step(FF rz_new, FF rr, uint32_t max_iter, FF& beta) {
        if (rr.hi > rmax2) rmax2 = rr.hi;
        k++;
        const int upd = rr.hi <= delta2 * rmax2 || rr.hi <= target2f || k >= max_iter;
        if (!upd) {
            beta = ff_div(rz_new, rz);
            rz = rz_new;
        } else {
            last = rr.hi;
        }
        return upd;
    }
    // Whether the solve may end with the update that step() asked for; from every
    // thread of the block.
    __device__ __forceinline__ bool may_end(uint32_t max_iter) const {
        return last <= 4.f * target2f || k >= max_iter;
    }
    // A reliable update's {|r|^2, r.z, r.p} (FP64), r the recomputed residual
    // and p the last direction: 2 stop, else 0 with beta.  checked: |r|^2 is the
    // one that the solve is judged on (row_residual).  The recursive
    // residual was orthogonal to p, the recomputed one is only up to the
    // rounding of b - A u.  Near the FP64 floor of a system r.(z + beta p)
    // then differs from r.z, and with r.z as the next step's numerator the
    // error stayed in every later step until the iteration diverged (the
    // 20,000-point T3 L-shape at relres 8e-12: 36 after 40,000 iterations).
    // From a relative difference of kOffLeast on the step takes r.(z + beta p);
    // smaller ones do not show (13 models, Q4 and T3, from 1e-6 to 1e-11: the same
    // iterations, to 1 %, with 0 and 1e-7, and closer to the floor either one ahead).
    static constexpr float kOffLeast = 1e-7f;
    __device__ __forceinline__ int replaced(const double (&t)[3], bool checked, uint32_t max_iter,
                                            FF& beta) {
        rr64 = t[0];
        rmax2 = (float)rr64;
        nupd++;
        converged = checked && rr64 <= target2;
        const int stop = converged || rr64 != rr64 || k >= max_iter;
        if (!stop) {
            const FF rzn = ff_from_double(t[1]);
            beta = ff_div(rzn, rz);
            rz = rzn;
            const FF off = ff_mul(beta, ff_from_double(t[2]));
            if (!(fabsf(off.hi) <= kOffLeast * rzn.hi)) {
                const FF rp = ff_add(rzn, off);
                if (rp.hi > 0.1f * rzn.hi) rz = rp;
                else beta = FF{0.f, 0.f};  // p points uphill: start again from z
            }
        }
        return stop ? 2 : 0;
    }
};

// Half of w = A p for node row (s, r): lanes l and l + 16 share row
// r = 16 h + (l & 15) of slice s, taking alternate entries, so a warp works on
// half a slice at a time (the block's 2 (s1 - s0) half slices spread evenly
// over its warps) and each load still covers two 16-entry runs.  The two
// partial float-float sums are combined with one exchange; TwoSum is
// symmetric, so both lanes hold the same bits.  Every lane of the warp must
// call it (the exchange is warp-wide).
// kSplit: p from the separate hi and lo arrays (the standalone operator),
// else from the solver's interleaved copy.
template <bool kSplit = false>
__device__ __forceinline__ void spmv_half_split(const MixArgs& a, uint32_t s, uint32_t r,
                                                uint32_t par, bool live, uint64_t pol, FF& y0,
                                                FF& y1) {
    const float4* __restrict__ bh = reinterpret_cast<const float4*>(a.A.b32);
    const uint2* __restrict__ bl = reinterpret_cast<const uint2*>(a.A.blo);
    const uint32_t* __restrict__ bx = reinterpret_cast<const uint32_t*>(a.A.bxt);
    const float2* __restrict__ ph = reinterpret_cast<const float2*>(a.ph);
    const float2* __restrict__ pl = reinterpret_cast<const float2*>(a.pl);
    const float4* __restrict__ p4 = a.p;
    // scalar accumulators: with p gathered from global memory the packed
    // FP32x2 form of spmv_half_local measured 5 % slower here (4M-dof T3:
    // 192 against 183 us per iteration); the roundings are the same
    FFAcc c0{0.f, 0.f}, c1{0.f, 0.f};
    // rows past Nn in the last slice hold no entries: such lanes only
    // take part in the exchange
    const uint32_t k0 = a.A.slice_off[s] + par, k1 = live ? a.A.slice_off[s + 1] : 0;
#pragma unroll(kUnroll)
    for (uint32_t k = k0; k < k1; k += 2) {
        const size_t e = (size_t)k * 32 + r;
        const uint32_t c = ld_hint(a.A.bcol + e, pol);
        const float4 m = ld_hint(bh + e, pol);  // a00 a10 a01 a11
        const float4 sc = rem23_scale4(ld_hint(bl + e, pol), ld_hint(bx + e, pol));
        float4 pv;
        if (kSplit) {
            const float2 h = ph[c], l = pl[c];
            pv = make_float4(h.x, h.y, l.x, l.y);
        } else {
            pv = p4[c];
        }
        c0.fma2s(m.x, sc.x, pv.x, pv.z);
        c0.fma2s(m.z, sc.z, pv.y, pv.w);
        c1.fma2s(m.y, sc.y, pv.x, pv.z);
        c1.fma2s(m.w, sc.w, pv.y, pv.w);
    }
    FF t[2] = {c0.result(), c1.result()};
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const float h = __shfl_xor_sync(0xffffffffu, t[j].hi, 16);
        const float l = __shfl_xor_sync(0xffffffffu, t[j].lo, 16);
        t[j] = ff_add(t[j], FF{h, l});
    }
    y0 = t[0];
    y1 = t[1];
}

// Own-row vectors of this block, indexed by local node row (i - 32 * s0):
// those that fit in shared memory, the others in the global workspace.  kOwn:
// 3 all four, 2 A p and r, 1 A p, 0 none.  Past level 3 the systems are larger
// than L2 and the iteration is bound by DRAM, to which a vector in global
// memory adds its reads and writes, 32 B per node row and iteration each for
// A p and r: 1.28e6 T3 nodes, 500 iterations, 50.4 -> 47.5 ms at level 1
// instead of 0; 24 batched systems, 252 MB, 281 -> 277.5 ms at level 2.
struct Own {
    float4 *p, *x, *r, *w;  // {hi, hi, lo, lo}
    const float2* dv;
};
// Up to 192 KB per SM for them: the L1 cache left beside more holds too few of
// the SpMV's gathers (us per iteration with nothing, A p, and A p and r in shared
// memory: T3 of 1.28M nodes 99.0, 92.8 at 135 KB; 1.8M 146.9, 135.3 at 190 KB; 2.0M
// 163.2, 191.3 at 211 KB; Q4 of 1.02M 78.1, 75.3, 89.1 at 215 KB).
constexpr size_t kOwnSmem = 192 * 1024;
constexpr size_t own_node_bytes(int own) { return own == 3 ? 64 : 16 * (size_t)own; }

template <int kOwn>
__device__ __forceinline__ Own own_vectors(const MixArgs& a, unsigned char* smem, uint32_t s0,
                                           uint32_t nrows) {
    Own o;
    const size_t base = (size_t)s0 * 32;
    float4* const sh = reinterpret_cast<float4*>(smem);
    o.p = kOwn == 3 ? sh + 2 * nrows : a.p + base;
    o.x = kOwn == 3 ? sh + 3 * nrows : a.x4 + base;
    o.r = kOwn >= 2 ? sh + nrows : a.r4 + base;
    o.w = kOwn >= 1 ? sh : a.w4 + base;
    o.dv = reinterpret_cast<const float2*>(a.A.dinv32) + base;
    return o;
}

// rp + r.p of one node row, p float-float
__device__ __forceinline__ double dot_with(double r0, double r1, float4 p, double rp) {
    return fma(r0, (double)p.x + (double)p.z, fma(r1, (double)p.y + (double)p.w, rp));
}

// r = b - A u in FP64 of node row i (s, lane), A u by FMAs: the iteration goes on
// with it.  Accumulates |r|^2 and optionally |b|^2.  check: |r|^2 is of A u in
// nbots' own arithmetic, the residual that nb_sparse_multiply_vector gives for
// u, on which every form of the solver is judged.  Near the FP64 floor of a system
// the two differ by a third of the tolerance, and the error of the rounded one is
// the larger by a fifth (64 x 32 lognormal: 2.2e-13 and 1.8e-13 of |b|).  Its
// FP64 operations, two for each FMA, are spent where the solve may end only.
__device__ __forceinline__ double2 row_residual(const MixArgs& a, uint32_t s, uint32_t lane,
                                                bool check, double& rr, double* bb) {
    const uint32_t i = s * 32 + lane;
    const double2* __restrict__ u = reinterpret_cast<const double2*>(a.u);
    const double2 bi = reinterpret_cast<const double2*>(a.b)[i];
    double2 an;
    const double2 au = check ? spmv_row_f64<true>(a.A, s, lane, u, &an)
                             : spmv_row_f64(a.A, s, lane, u);
    if (!check) an = au;
    const double j0 = bi.x - an.x, j1 = bi.y - an.y;
    rr = fma(j0, j0, fma(j1, j1, rr));
    if (bb) *bb = fma(bi.x, bi.x, fma(bi.y, bi.y, *bb));
    return make_double2(bi.x - au.x, bi.y - au.y);
}

// r = b - A u for the own rows (row_residual), stored as float-float; z = r / Aii
// (float-float); accumulates |r|^2 (FP64), r.z and optionally |b|^2 and r.p;
// with set_p, p = z (own copy and the global one).
template <int kThreads>
__device__ __forceinline__ void true_residual(const MixArgs& a, const Own& o, uint32_t s0,
                                              uint32_t s1, bool check, double& rr, FFAcc& rz,
                                              double* bb, double* rp, bool set_p) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nw = kThreads / 32;
    for (uint32_t s = s0 + warp; s < s1; s += nw) {
        const uint32_t i = s * 32 + lane, li = i - s0 * 32;
        if (i >= a.A.Nn) continue;
        const double2 ri = row_residual(a, s, lane, check, rr, bb);
        if (rp) *rp = dot_with(ri.x, ri.y, o.p[li], *rp);
        const FF f0 = ff_from_double(ri.x), f1 = ff_from_double(ri.y);
        o.r[li] = make_float4(f0.hi, f1.hi, f0.lo, f1.lo);
        const float2 di = o.dv[li];
        const FF z0 = ff_mulf(f0, di.x), z1 = ff_mulf(f1, di.y);
        rz.fma2(f0.hi, f0.lo, z0.hi, z0.lo);
        rz.fma2(f1.hi, f1.lo, z1.hi, z1.lo);
        if (set_p) {
            const float4 p = make_float4(z0.hi, z1.hi, z0.lo, z1.lo);
            o.p[li] = p;
            a.p[i] = p;  // the same slot when the own rows are in global memory
        }
    }
}

// The two sums of an iteration, in fixed point (allreduce.cuh; 1M-dof ghost
// form 31.6 us per iteration against 32.9 with block sums, a counting barrier
// and the partials' loads behind it), with kFence
// also as a barrier for the vectors in global memory; where a window does not
// serve, by partials and a barrier (`sync`).  finish(sums ...) runs in thread 0.
// Nonzero return: stop.  Both forms of the single-system solver use it, with
// the same values per thread, so they get the same bits.
struct MixSums {
    int sh[kSumShared];
    ExactSum pw, rz;
    float scale[3];  // windows of p.w, r.z, |r|^2
    int again;

    __device__ __forceinline__ void init(unsigned char* words) {  // by one thread
        pw.init(words);
        rz.init(words + kExactBytes);
        scale[0] = scale[1] = scale[2] = 0.f;
    }
};

struct NoMixSums {};

template <int NV, bool kFence, class Sync, class Finish, class Meanwhile>
__device__ __forceinline__ int mixed_sum(MixSums& m, ExactSum& site, int first, FF (&v)[NV],
                                         const Group& g, uint32_t rank, float2* ffred,
                                         float2* part, Sync sync, Finish finish,
                                         Meanwhile meanwhile) {
    float scale[NV];
    int window[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) {
        scale[k] = m.scale[first + k];
        window[k] = window_exponent(scale[k]);
    }
    exact_begin<NV>(v, scale, m.sh);
    __syncthreads();
    if (threadIdx.x < 32) {
        long long x;
        int e;
        const int st = site.sum<NV, kFence>(m.sh, blockDim.x >> 5, g.g_size, g.status, window,
                                            kLeastFF, x, e,
                                            [] { if (kFence) bar_arrive(1); });
        FF t[NV];
        const FF mine = exact_ff(x, e);
#pragma unroll
        for (int k = 0; k < NV; k++)
            t[k] = {__shfl_sync(0xffffffffu, mine.hi, k), __shfl_sync(0xffffffffu, mine.lo, k)};
        if (threadIdx.x == 0) {
            m.again = st;
            if (!st) {
#pragma unroll
                for (int k = 0; k < NV; k++) m.scale[first + k] = window_scale(t[k].hi);
                finish(t);
            }
        }
    } else {
        // memory traffic waits until the fence is over, which would wait for it
        if (kFence) bar_sync(1);
        meanwhile();
    }
    __syncthreads();
    if (m.again) {
        if (m.again == 2) return 1;
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] = fast_two_sum(v[k].hi, v[k].lo);
        group_publish_ff<NV>(v, ffred, part, rank);
        if (sync()) return 1;
        FF t[NV];
        group_reduce0_ff<NV>(part, g.g_size, t);
        if (threadIdx.x == 0) {
#pragma unroll
            for (int k = 0; k < NV; k++) m.scale[first + k] = window_scale(t[k].hi);
            finish(t);
        }
        __syncthreads();
    }
    return 0;
}

// The solver of one system on the blocks [g_base, g_base + g_size) of the
// launch: its own slices, group barrier, partial sums and result.  The
// scalar recurrences (step lengths, residual norms, stopping and update
// decisions) run in thread 0 (MixScalars) and reach the block through
// shared memory as FP32 pairs and flags.
// kExact: sums in fixed point, else by partials.
template <int kOwn, int kThreads, bool kExact>
__device__ __forceinline__ void mixed_solve(const MixArgs& a, const Group& g, unsigned char* smem) {
    constexpr bool kRes = kOwn == 3;
    constexpr int kRB = kThreads == kMixThreads ? kReduceBatch : 1;
    __shared__ std::conditional_t<kExact, MixSums, NoMixSums> ms;
    __shared__ double red[3 * 32];
    float2* const ffred = reinterpret_cast<float2*>(red);
    __shared__ float s_alpha[2], s_beta[2];
    __shared__ int s_flag;  // 0 iterate, 1 reliable update, 2 stop
    __shared__ MixScalars sc;  // thread 0 only, but for may_end()
    const unsigned G = g.g_size;
    const uint32_t rank = blockIdx.x - g.g_base;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nw = kThreads / 32;
    uint32_t s0, s1;
    group_slice_range(g.s_begin, g.s_end, rank, G, s0, s1);
    const uint32_t Nn = a.A.Nn;
    const Own o = own_vectors<kOwn>(a, smem, s0, (s1 - s0) * 32);
    float4* const gp = a.p;
    double* const part0 = g.part;
    double* const part1 = g.part + g.pstride;
    double* const part2 = g.part + 3 * g.pstride;
    // the arrival that returns the old word: with the counting barrier the
    // global-gather and batched launches ran slower (4M-dof T3: 4.19 against
    // 4.07 s; the 96-system batch: 1.43 against 1.36 s)
    auto sync = [&]() { return grid_barrier(g.bar, G, rank, g.status); };

    if (threadIdx.x == 0) {
        sc.clear();
        if constexpr (kExact) ms.init(g.sums);
    }
    {   // init: x = 0, r = b - A u (FP64), p = z
        for (uint32_t s = s0 + warp; s < s1; s += nw) {
            const uint32_t i = s * 32 + lane, li = i - s0 * 32;
            if (i < Nn) o.x[li] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncwarp();
        double rrl = 0.0, bbl = 0.0;
        FFAcc rzk{0.f, 0.f};
        true_residual<kThreads>(a, o, s0, s1, true, rrl, rzk, &bbl, nullptr, true);
        const FF t = rzk.result();
        double v[3] = {rrl, bbl, (double)t.hi + (double)t.lo};
        group_publish<3>(v, red, part2, rank);
    }
    if (sync()) goto done;
    {
        double t[3];
        group_reduce0<3>(part2, G, t);
        if (threadIdx.x == 0) {
            s_flag = sc.start(t, a);
            if constexpr (kExact) {
                ms.scale[1] = window_scale(sc.rz.hi);
                ms.scale[2] = window_scale((float)sc.rr64);
            }
        }
        __syncthreads();
    }
    while (s_flag != 2) {
        {   // L1: w = A p, p.w (two lanes per node row)
            FFAcc pw{0.f, 0.f};
            const uint32_t par = lane >> 4, nh = 2 * (s1 - s0);
            // warp w takes half slices w, w + nw, ...
            for (uint32_t h = warp; h < nh; h += nw) {
                const uint32_t s = s0 + (h >> 1), r = ((h & 1) << 4) | (lane & 15);
                const uint32_t i = s * 32 + r, li = i - s0 * 32;
                // a slice's rows past Nn are padding: skip them whole (both lanes)
                if (s * 32 + ((h & 1) << 4) >= Nn) continue;
                FF y0, y1;
                const uint64_t pol = l2_policy(kept<kThreads>(a, s - s0, s1 - s0));
                spmv_half_split(a, s, r, par, i < Nn, pol, y0, y1);
                if (par || i >= Nn) continue;
                o.w[li] = make_float4(y0.hi, y1.hi, y0.lo, y1.lo);
                const float4 p = o.p[li];
                pw.fma2(p.x, p.z, y0.hi, y0.lo);
                pw.fma2(p.y, p.w, y1.hi, y1.lo);
            }
            auto finish = [&](const FF (&pws)[1]) {
                const FF al = sc.alpha(pws[0]);
                s_alpha[0] = al.hi;
                s_alpha[1] = al.lo;
            };
            if constexpr (kExact) {
                FF v[1] = {{pw.s, pw.c}};
                if (mixed_sum<1, true>(ms, ms.pw, 0, v, g, rank, ffred, reinterpret_cast<float2*>(part0),
                                 sync, finish, [] {}))
                    goto done;
            } else {
                FF v[1] = {pw.result()};
                group_publish_ff<1>(v, ffred, reinterpret_cast<float2*>(part0), rank);
                if (sync()) goto done;
                FF t[1];
                group_reduce0_ff<1, kRB>(reinterpret_cast<const float2*>(part0), G, t);
                if (threadIdx.x == 0) finish(t);
                __syncthreads();
            }
        }
        {   // L2: x += alpha p, r -= alpha w, z = r / Aii (own rows only)
            const FF alpha = {s_alpha[0], s_alpha[1]};
            FFAcc rzk{0.f, 0.f}, rrk{0.f, 0.f};
            for (uint32_t s = s0 + warp; s < s1; s += nw) {
                const uint32_t i = s * 32 + lane, li = i - s0 * 32;
                if (i >= Nn) continue;
                const float4 p = o.p[li], w = o.w[li], xo = o.x[li], ri = o.r[li];
                const float2 di = o.dv[li];
                const FF x0 = ff_add({xo.x, xo.z}, ff_mul(alpha, {p.x, p.z}));
                const FF x1 = ff_add({xo.y, xo.w}, ff_mul(alpha, {p.y, p.w}));
                o.x[li] = make_float4(x0.hi, x1.hi, x0.lo, x1.lo);
                const FF aw0 = ff_mul(alpha, {w.x, w.z}), aw1 = ff_mul(alpha, {w.y, w.w});
                const FF r0 = ff_add({ri.x, ri.z}, {-aw0.hi, -aw0.lo});
                const FF r1 = ff_add({ri.y, ri.w}, {-aw1.hi, -aw1.lo});
                o.r[li] = make_float4(r0.hi, r1.hi, r0.lo, r1.lo);
                const FF z0 = ff_mulf(r0, di.x), z1 = ff_mulf(r1, di.y);
                rzk.fma2(r0.hi, r0.lo, z0.hi, z0.lo);
                rzk.fma2(r1.hi, r1.lo, z1.hi, z1.lo);
                rrk.fma2(r0.hi, r0.lo, r0.hi, r0.lo);
                rrk.fma2(r1.hi, r1.lo, r1.hi, r1.lo);
            }
            auto finish = [&](const FF (&t2)[2]) {
                FF be;
                s_flag = sc.step(t2[0], t2[1], a.max_iter, be);
                if (!s_flag) {
                    s_beta[0] = be.hi;
                    s_beta[1] = be.lo;
                }
            };
            if constexpr (kExact) {
                FF v[2] = {{rzk.s, rzk.c}, {rrk.s, rrk.c}};
                if (mixed_sum<2, true>(ms, ms.rz, 1, v, g, rank, ffred, reinterpret_cast<float2*>(part1),
                                 sync, finish, [] {}))
                    goto done;
            } else {
                FF v[2] = {rzk.result(), rrk.result()};
                group_publish_ff<2>(v, ffred, reinterpret_cast<float2*>(part1), rank);
                if (sync()) goto done;
                FF t[2];
                group_reduce0_ff<2, kRB>(reinterpret_cast<const float2*>(part1), G, t);
                if (threadIdx.x == 0) finish(t);
                __syncthreads();
            }
        }
        if (s_flag) {
            // reliable update: u += x in FP64, then r = b - A u in FP64
            const bool check = sc.may_end(a.max_iter);
            double2* const u = reinterpret_cast<double2*>(a.u);
            for (uint32_t s = s0 + warp; s < s1; s += nw) {
                const uint32_t i = s * 32 + lane, li = i - s0 * 32;
                if (i >= Nn) continue;
                const float4 xo = o.x[li];
                double2 ui = u[i];
                ui.x += (double)xo.x + (double)xo.z;
                ui.y += (double)xo.y + (double)xo.w;
                u[i] = ui;
                o.x[li] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            if (sync()) goto done;
            double rrl = 0.0, rpl = 0.0;
            FFAcc rzk{0.f, 0.f};
            true_residual<kThreads>(a, o, s0, s1, check, rrl, rzk, nullptr, &rpl, false);
            const FF t = rzk.result();
            double v[3] = {rrl, (double)t.hi + (double)t.lo, rpl};
            group_publish<3>(v, red, part2, rank);
            if (sync()) goto done;
            double tt[3];
            group_reduce0<3>(part2, G, tt);
            if (threadIdx.x == 0) {
                FF be;
                s_flag = sc.replaced(tt, check, a.max_iter, be);
                if (!s_flag) {
                    s_beta[0] = be.hi;
                    s_beta[1] = be.lo;
                }
            }
            __syncthreads();
            if (s_flag == 2) break;
        }
        {   // L3: p = z + beta p (own copy and the global one)
            const FF beta = {s_beta[0], s_beta[1]};
            for (uint32_t s = s0 + warp; s < s1; s += nw) {
                const uint32_t i = s * 32 + lane, li = i - s0 * 32;
                if (i >= Nn) continue;
                const float4 ri = o.r[li], p = o.p[li];
                const float2 di = o.dv[li];
                const FF n0 = ff_add(ff_mulf({ri.x, ri.z}, di.x), ff_mul(beta, {p.x, p.z}));
                const FF n1 = ff_add(ff_mulf({ri.y, ri.w}, di.y), ff_mul(beta, {p.y, p.w}));
                const float4 pn = make_float4(n0.hi, n1.hi, n0.lo, n1.lo);
                if (kRes) o.p[li] = pn;
                gp[i] = pn;
            }
        }
        if (sync()) goto done;
    }
    {   // b.u in FP64 (the compliance F^T u when b is the load vector).  part0
        // was last read before the L2 barrier of the last iteration.
        const double2* __restrict__ u = reinterpret_cast<const double2*>(a.u);
        const double2* __restrict__ b = reinterpret_cast<const double2*>(a.b);
        double bu = 0.0;
        for (uint32_t s = s0 + warp; s < s1; s += nw) {
            const uint32_t i = s * 32 + lane;
            if (i >= Nn) continue;
            const double2 ui = u[i], bi = b[i];
            bu = fma(bi.x, ui.x, fma(bi.y, ui.y, bu));
        }
        double v[1] = {bu};
        group_publish<1>(v, red, part0, rank);
        if (sync()) goto done;
        double J[1];
        group_reduce0<1>(part0, G, J);
        if (rank == 0 && threadIdx.x == 0) g.res[5] = J[0];
    }
done:
    if (rank == 0 && threadIdx.x == 0) {
        g.res[0] = (double)sc.k;
        g.res[1] = (double)sc.nupd;
        int st = ld_volatile(g.status);
        g.res[2] = st != 0 ? (double)st : (sc.converged ? 0.0 : 1.0);
        g.res[3] = sc.rr64;
        g.res[4] = sc.bb;
    }
}

// kOwn: the own-row vectors in dynamic shared memory (known at compile time,
// so their addresses are 32-bit shared ones).
template <int kOwn, bool kExact>
__global__ void __launch_bounds__(kMixThreads, kMixMinBlocks) k_cg_mixed(MixArgs a,
                                                                                Group g) {
    extern __shared__ __align__(16) unsigned char smem[];
    mixed_solve<kOwn, kMixThreads, kExact>(a, g, smem);
}

// Many independent systems stored in one block-diagonal layout, in one
// launch: block b works for system groups[block_of[b]].  A system has a few
// blocks: sums by partials.
template <int kOwn>
__global__ void __launch_bounds__(kBatThreads, kBatMinBlocks)
    k_cg_mixed_many(MixArgs a, const Group* __restrict__ groups,
                    const uint32_t* __restrict__ block_of) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Group sg;
    if (threadIdx.x == 0) sg = groups[block_of[blockIdx.x]];
    __syncthreads();
    mixed_solve<kOwn, kBatThreads, false>(a, sg, smem);
}

// The SpMV's matrix stream (FP32 values, remainders, columns: 32 B per block
// entry) in units of this device's L2; negative: not known.
double stream_over_l2(const nbg_bsr_t& A, double bytes_per_entry = 32.0) {
    int dev = 0, l2 = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) != cudaSuccess || l2 <= 0)
        return -1.0;
    return bytes_per_entry * (double)A.n_entries / l2;
}

// Share of the matrix stream marked evict_last (of 2^32): 45 % of L2 while the
// stream and the vectors are not much larger than it, falling to 30 % from 1.4
// times L2 on, where the rest of the stream pushes the vectors out.  Ghost
// form, us per iteration with 30 % everywhere and with this rule (best of a
// scan in steps of 50): 0.45 L2 14.7 and 14.4 (14.4), 0.57 18.1 and 17.3
// (17.3), 0.63 19.0 and 17.8 (17.8), 0.69 21.1 and 20.7 (20.5), 0.87 25.1 and
// 25.2 (25.1), 1.1 30.6 and 30.6 (30.6), 1.37 38.9 and 38.8 (38.5).  A stream of
// more than twice the L2 gains less from the kept part than its vectors lose
// (without and with: q4 with 2.1M dof 80.0 and 86.4, T3 with 2.6M dof 99.4 and
// 106.6, at 1.6 times the L2 53.8 and 52.2).
uint32_t keep_share(const nbg_bsr_t& A, double bytes_per_entry = 32.0) {
    const double x = stream_over_l2(A, bytes_per_entry);
    if (x <= 0.0 || x > 2.0) return 0;
    const double share = std::min(0.45, std::max(0.30, 0.45 - (x - 0.7) * (0.15 / 0.7)));
    return (uint32_t)(4294967295.0 * std::min(1.0, share / x));
}

// Vectors, partial sums, then what a launch needs at zero: barrier, status
// and result words and the records and words of the slice form's sums.
constexpr size_t kMixTail = 3 * 256 + kArBytes + 2 * kExactBytes;

size_t mixed_core_bytes(uint32_t N) {
    const size_t f = align256((size_t)N * 4), h = align256((size_t)N * 4);
    return 6 * f + 2 * h + align256(kMaxBlocks * 6 * 8) + kMixTail;
}

// The vector slots at the start of a workspace (indexed by node row, a
// float4 each): p, x, r, A p.
void carve_vectors(MixArgs& a, char* base, uint32_t N) {
    const size_t f = align256((size_t)N * 4);
    a.p = (float4*)base;
    a.x4 = (float4*)(base + 2 * f);
    a.r4 = (float4*)(base + 4 * f);
    a.w4 = (float4*)(base + 6 * f);
    a.ph = a.pl = nullptr;
}

// plus the permuted copies of b and x for a layout with a node order
size_t mixed_bytes(uint32_t N) { return mixed_core_bytes(N) + perm_tail_bytes(N); }

// The mixed solver's SpMV operator as its own launch: w = A p with the split
// matrix and float-float p, two lanes per node row, the solver's L2 policy
// (a share `keep` of the slices evict_last).  One block per
// SM, slices split evenly, as in the solver.
__global__ void __launch_bounds__(kMixThreads, kMixMinBlocks)
    k_spmv_mixed(MixArgs a, float2* __restrict__ wh, float2* __restrict__ wl) {
    uint32_t s0, s1;
    slice_range(a.A.n_slices, s0, s1);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nw = kMixThreads / 32, par = lane >> 4, nh = 2 * (s1 - s0);
    for (uint32_t h = warp; h < nh; h += nw) {
        const uint32_t s = s0 + (h >> 1), r = ((h & 1) << 4) | (lane & 15);
        const uint32_t i = s * 32 + r;
        if (s * 32 + ((h & 1) << 4) >= a.A.Nn) continue;
        FF y0, y1;
        const uint64_t pol = l2_policy(kept<kMixThreads>(a, s - s0, s1 - s0));
        spmv_half_split<true>(a, s, r, par, i < a.A.Nn, pol, y0, y1);
        if (par || i >= a.A.Nn) continue;
        wh[i] = make_float2(y0.hi, y1.hi);
        wl[i] = make_float2(y0.lo, y1.lo);
    }
}

// ---------------------------------------------------------------------------
// Ghost-node form of the single-system solver.
//
// A block's SpMV reads p at its own rows and at the rows of other blocks that
// its rows couple to, its ghosts (on the 1M-dof cantilever, a block's strip of
// about 3.4 grid rows has the two neighbouring grid rows as ghosts, 0.6 times
// its own row count).  This form keeps p for the block's own rows and for
// its ghosts in shared memory, with the layout's columns renumbered locally
// in 16 bits (own row slots first, then the ghosts in ascending node order),
// so the SpMV gathers from shared memory, not L2, and the matrix stream is
// 30 B per block entry instead of 32.  Owners publish their residual r
// (after L2 and after each reliable update); after the barrier that ends L2
// every block computes its ghosts' new p itself, with the owner's arithmetic
// on the owner's r and on its own copy of the ghost's previous p (the same
// bits, by induction from p = z at the start), so the third barrier of each
// iteration (the exchange of p) goes away.  The iterates equal those of the
// global-gather form bit for bit.  x moves to global memory to leave shared
// memory to the ghosts.
//
// At 1.05M dof an iteration (65 thousand cycles) was two thirds SpMV, at 70 to
// 78 % of DRAM's rate, then 5 to 6 thousand cycles for each sum, 6.5 for L2 and
// 4.3 for L3.  So x is updated while warp 0 sums (from when its fence is over:
// the fence, 2,000 cycles, waits for all the traffic before it), and L2 leaves
// z in A p's place, so that L3 reads the own rows from shared memory.
// Microseconds per iteration before and after: 314,000 dof 13.2 and 12.6,
// 482,000 18.8 and 18.1, 1.05M 31.9 and 30.7, 1.30M 40.4 and 38.9.
//
// The plan (ghost lists, local columns) depends on the launch's block
// partition and is rebuilt by a short kernel at the start of every solve.
// spmv_half_split with local columns and p (own rows and ghosts) in shared
// memory as float4 {hi of both dofs, lo of both dofs}; the same products and
// sums in the same order.
__device__ __forceinline__ void spmv_half_local(const MixArgs& a, const uint16_t* __restrict__ lcol,
                                                const float4* P, const uint32_t* so,
                                                uint32_t s, uint32_t r, uint32_t par, bool live,
                                                uint64_t pol, FF& y0, FF& y1) {
    const float4* __restrict__ bh = reinterpret_cast<const float4*>(a.A.b32);
    const uint2* __restrict__ bl = reinterpret_cast<const uint2*>(a.A.blo);
    const uint32_t* __restrict__ bx = reinterpret_cast<const uint32_t*>(a.A.bxt);
    FFAcc2 acc{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};  // rows 0 and 1
    // so: this block's slice offsets, so[0] that of its first slice
    const uint32_t k0 = so[s] + par, k1 = live ? so[s + 1] : 0;
#pragma unroll(kUnroll)
    for (uint32_t k = k0; k < k1; k += 2) {
        const size_t e = (size_t)k * 32 + r;
        const uint32_t c = ld_hint(lcol + e, pol);
        const float4 m = ld_hint(bh + e, pol);  // a00 a10 a01 a11
        const float4 sc = rem23_scale4(ld_hint(bl + e, pol), ld_hint(bx + e, pol));
        const float4 pv = P[c];
        acc.fma2s(make_float2(m.x, m.y), make_float2(sc.x, sc.y), pv.x, pv.z);
        acc.fma2s(make_float2(m.z, m.w), make_float2(sc.z, sc.w), pv.y, pv.w);
    }
    FF t[2] = {FFAcc{acc.s.x, acc.c.x}.result(), FFAcc{acc.s.y, acc.c.y}.result()};
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const float h = __shfl_xor_sync(0xffffffffu, t[j].hi, 16);
        const float l = __shfl_xor_sync(0xffffffffu, t[j].lo, 16);
        t[j] = ff_add(t[j], FF{h, l});
    }
    y0 = t[0];
    y1 = t[1];
}

// The ghost form keeps r and x in global memory (the workspace's x rows; r in
// its r and A p rows by turns: L2 reads one and writes the other, so that no
// block overwrites a row that another may still be reading as a ghost, and
// the sum between the two needs no fence).
__device__ __forceinline__ float4* ghost_r(const MixArgs& a, uint32_t turn) {
    return turn & 1 ? a.w4 : a.r4;
}
__device__ __forceinline__ float4* ghost_x(const MixArgs& a) { return a.x4; }

// true_residual for the ghost form: r (float-float) to global memory, where
// the owner keeps it and the blocks that hold this row as a ghost read it, z
// to Z.
template <int kThreads>
__device__ __forceinline__ void true_residual_ghost(const MixArgs& a, float4* r4, const float4* P,
                                                    float4* Z, uint32_t s0, uint32_t s1,
                                                    bool check, double& rr, FFAcc& rz,
                                                    double* bb, double* rp) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nw = kThreads / 32;
    const float2* __restrict__ dinv = reinterpret_cast<const float2*>(a.A.dinv32);
    for (uint32_t s = s0 + warp; s < s1; s += nw) {
        const uint32_t i = s * 32 + lane, li = i - s0 * 32;
        if (i >= a.A.Nn) continue;
        const double2 ri = row_residual(a, s, lane, check, rr, bb);
        if (rp) *rp = dot_with(ri.x, ri.y, P[li], *rp);
        const FF f0 = ff_from_double(ri.x), f1 = ff_from_double(ri.y);
        r4[i] = make_float4(f0.hi, f1.hi, f0.lo, f1.lo);
        const float2 di = dinv[i];
        const FF z0 = ff_mulf(f0, di.x), z1 = ff_mulf(f1, di.y);
        rz.fma2(f0.hi, f0.lo, z0.hi, z0.lo);
        rz.fma2(f1.hi, f1.lo, z1.hi, z1.lo);
        Z[li] = make_float4(z0.hi, z1.hi, z0.lo, z1.lo);
    }
}

template <int kThreads>
__device__ __forceinline__ void mixed_solve_ghost(const MixArgs& a, const Group& g,
                                                  const GhostArgs& gh, unsigned char* smem) {
    __shared__ double red[3 * 32];
    float2* const ffred = reinterpret_cast<float2*>(red);
    __shared__ float s_alpha[2], s_beta[2];
    __shared__ int s_flag;  // 0 iterate, 1 reliable update, 2 stop
    __shared__ MixScalars sc;  // thread 0 only, but for may_end()
    __shared__ MixSums ms;
    const unsigned G = g.g_size;
    const uint32_t rank = blockIdx.x - g.g_base;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nw = kThreads / 32;
    uint32_t s0, s1;
    group_slice_range(g.s_begin, g.s_end, rank, G, s0, s1);
    const uint32_t Nn = a.A.Nn, nslot = (s1 - s0) * 32;
    const uint32_t ng = gh.count[rank];
    float4* const P = reinterpret_cast<float4*>(smem);
    float4* const W = P + gh.pcap;  // A p, then z of the own rows {hi, hi, lo, lo}
    uint32_t* const GID = reinterpret_cast<uint32_t*>(W + gh.scap);
    // slice offsets of this block, indexed by s - s0
    uint32_t* const SO = GID + gh.gcap;
    float4* r4 = ghost_r(a, 0);  // the current residual
    uint32_t turn = 0;
    float4* __restrict__ x4 = ghost_x(a);
    const float2* __restrict__ dinv = reinterpret_cast<const float2*>(a.A.dinv32);
    double* const part0 = g.part;
    double* const part1 = g.part + g.pstride;
    double* const part2 = g.part + 3 * g.pstride;
#if NBG_BARRIER_COUNT
    unsigned bar_target = 0;
    auto sync = [&]() { return grid_barrier_count(g.bar, G, bar_target, g.status); };
#else
    auto sync = [&]() { return grid_barrier(g.bar, G, rank, g.status); };
#endif

    auto as4 = [](const FF2& v) { return make_float4(v.hi.x, v.hi.y, v.lo.x, v.lo.y); };
    auto from4 = [](float4 v) -> FF2 {
        return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
    };

    if (tid == 0) {
        sc.clear();
        ms.init(g.sums);
    }
    for (uint32_t j = tid; j < ng; j += kThreads) GID[j] = gh.ids[(size_t)rank * kGhostMax + j];
    for (uint32_t j = tid; j <= s1 - s0; j += kThreads) SO[j] = a.A.slice_off[s0 + j];
    {   // init: x = 0, r = b - A u (FP64), own p = z, r published
        for (uint32_t s = s0 + warp; s < s1; s += nw) {
            const uint32_t i = s * 32 + lane;
            if (i >= Nn) continue;
            x4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        double rrl = 0.0, bbl = 0.0;
        FFAcc rzk{0.f, 0.f};
        true_residual_ghost<kThreads>(a, r4, P, P, s0, s1, true, rrl, rzk, &bbl, nullptr);
        const FF t = rzk.result();
        double v[3] = {rrl, bbl, (double)t.hi + (double)t.lo};
        group_publish<3>(v, red, part2, rank);
    }
    if (sync()) goto done;
    {
        double t[3];
        group_reduce0<3>(part2, G, t);
        if (tid == 0) {
            s_flag = sc.start(t, a);
            ms.scale[1] = window_scale(sc.rz.hi);
            ms.scale[2] = window_scale((float)sc.rr64);
        }
        // ghosts start as their owners' p = z
        for (uint32_t j = tid; j < ng; j += kThreads) {
            const uint32_t c = GID[j];
            const float4 rc = r4[c];
            const float2 dc = dinv[c];
            const FF z0 = ff_mulf({rc.x, rc.z}, dc.x), z1 = ff_mulf({rc.y, rc.w}, dc.y);
            P[nslot + j] = make_float4(z0.hi, z1.hi, z0.lo, z1.lo);
        }
        __syncthreads();
    }
    while (s_flag != 2) {
        {   // L1: w = A p from shared memory, p.w (two lanes per node row)
            FFAcc pw{0.f, 0.f};
            const uint32_t par = lane >> 4, nh = 2 * (s1 - s0);
            for (uint32_t h = warp; h < nh; h += nw) {
                const uint32_t s = s0 + (h >> 1), r = ((h & 1) << 4) | (lane & 15);
                const uint32_t i = s * 32 + r, li = i - s0 * 32;
                if (s * 32 + ((h & 1) << 4) >= Nn) continue;
                FF y0, y1;
                const uint64_t pol = l2_policy(kept<kThreads>(a, s - s0, s1 - s0));
                spmv_half_local(a, gh.lcol, P, SO, s - s0, r, par, i < Nn, pol, y0, y1);
                if (par || i >= Nn) continue;
                W[li] = make_float4(y0.hi, y1.hi, y0.lo, y1.lo);
                const float4 p = P[li];
                pw.fma2(p.x, p.z, y0.hi, y0.lo);
                pw.fma2(p.y, p.w, y1.hi, y1.lo);
            }
            FF v[1] = {{pw.s, pw.c}};
            if (mixed_sum<1, false>(ms, ms.pw, 0, v, g, rank, ffred, reinterpret_cast<float2*>(part0), sync,
                             [&](const FF (&pws)[1]) {
                                 const FF al = sc.alpha(pws[0]);
                                 s_alpha[0] = al.hi;
                                 s_alpha[1] = al.lo;
                             }, [] {}))
                goto done;
        }
        {   // L2: r -= alpha w, z = r / Aii; r published; x += alpha p
            const FF alpha = {s_alpha[0], s_alpha[1]};
            FFAcc rzk{0.f, 0.f}, rrk{0.f, 0.f};
            float4* const rnew = ghost_r(a, ++turn);
            // both dofs of a row at once on the packed FP32x2 instructions
            // (the same roundings as the global-gather form's scalar code)
            const FF2 alpha2 = ff2_bcast(alpha);
            auto row = [&](uint32_t i, float4 ro, float2 di) {
                const uint32_t li = i - s0 * 32;
                const FF2 aw = ff2_mul(alpha2, from4(W[li]));
                const FF2 r = ff2_add(from4(ro), {f2neg(aw.hi), f2neg(aw.lo)});
                rnew[i] = as4(r);
                const FF2 z = ff2_mulf(r, di);
                W[li] = as4(z);  // for L3, in place of A p
                rzk.fma2(r.hi.x, r.lo.x, z.hi.x, z.lo.x);
                rzk.fma2(r.hi.y, r.lo.y, z.hi.y, z.lo.y);
                rrk.fma2(r.hi.x, r.lo.x, r.hi.x, r.lo.x);
                rrk.fma2(r.hi.y, r.lo.y, r.hi.y, r.lo.y);
            };
            // two slices per step, their global loads issued together (one
            // memory round trip for both); rows in the same order as one
            // slice per step, so the sums are unchanged
            for (uint32_t s = s0 + warp; s < s1; s += 2 * nw) {
                const uint32_t iA = s * 32 + lane, iB = iA + 32 * nw;
                if (iA >= Nn) continue;
                const bool vB = s + nw < s1 && iB < Nn;
                const float4 rA = r4[iA];
                const float2 dA = dinv[iA];
                float4 rB{};
                float2 dB{};
                if (vB) {
                    rB = r4[iB];
                    dB = dinv[iB];
                }
                row(iA, rA, dA);
                if (vB) row(iB, rB, dB);
            }
            // x += alpha p by the other warps while warp 0 sums: off the
            // critical path
            auto update_x = [&]() {
                const uint32_t step = 32 * (nw - 1);
                for (uint32_t iA = s0 * 32 + tid - 32; iA < s1 * 32 && iA < Nn; iA += 2 * step) {
                    const uint32_t iB = iA + step;
                    const bool vB = iB < s1 * 32 && iB < Nn;
                    const float4 xA = x4[iA], xB = vB ? x4[iB] : make_float4(0.f, 0.f, 0.f, 0.f);
                    x4[iA] = as4(ff2_add(from4(xA), ff2_mul(alpha2, from4(P[iA - s0 * 32]))));
                    if (vB) x4[iB] = as4(ff2_add(from4(xB), ff2_mul(alpha2, from4(P[iB - s0 * 32]))));
                }
            };
            r4 = rnew;
            FF v[2] = {{rzk.s, rzk.c}, {rrk.s, rrk.c}};
            if (mixed_sum<2, true>(ms, ms.rz, 1, v, g, rank, ffred, reinterpret_cast<float2*>(part1), sync,
                             [&](const FF (&t2)[2]) {
                                 FF be;
                                 s_flag = sc.step(t2[0], t2[1], a.max_iter, be);
                                 if (!s_flag) {
                                     s_beta[0] = be.hi;
                                     s_beta[1] = be.lo;
                                 }
                             }, update_x))
                goto done;
        }
        if (s_flag) {
            // reliable update: u += x in FP64, then r = b - A u in FP64
            const bool check = sc.may_end(a.max_iter);
            double2* const u = reinterpret_cast<double2*>(a.u);
            for (uint32_t s = s0 + warp; s < s1; s += nw) {
                const uint32_t i = s * 32 + lane;
                if (i >= Nn) continue;
                const float4 xo = x4[i];
                double2 ui = u[i];
                ui.x += (double)xo.x + (double)xo.z;
                ui.y += (double)xo.y + (double)xo.w;
                u[i] = ui;
                x4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            if (sync()) goto done;
            double rrl = 0.0, rpl = 0.0;
            FFAcc rzk{0.f, 0.f};
            true_residual_ghost<kThreads>(a, r4, P, W, s0, s1, check, rrl, rzk, nullptr, &rpl);
            const FF t = rzk.result();
            double v[3] = {rrl, (double)t.hi + (double)t.lo, rpl};
            group_publish<3>(v, red, part2, rank);
            if (sync()) goto done;
            double tt[3];
            group_reduce0<3>(part2, G, tt);
            if (tid == 0) {
                FF be;
                s_flag = sc.replaced(tt, check, a.max_iter, be);
                if (!s_flag) {
                    s_beta[0] = be.hi;
                    s_beta[1] = be.lo;
                }
            }
            __syncthreads();
            if (s_flag == 2) break;
        }
        {   // L3: p = z + beta p for the own rows and the ghosts (no barrier:
            // every p this block's next SpMV reads is in its shared memory)
            const FF beta = {s_beta[0], s_beta[1]};
            const FF2 beta2 = ff2_bcast(beta);
            auto pnew = [&](uint32_t l, const FF2& z) {
                P[l] = as4(ff2_add(z, ff2_mul(beta2, from4(P[l]))));
            };
            // the ghosts from their owners' r, two per step, the loads issued
            // together
            for (uint32_t j = tid; j < ng; j += 2 * kThreads) {
                const uint32_t jB = j + kThreads;
                const uint32_t cA = GID[j], cB = jB < ng ? GID[jB] : cA;
                const float4 rA = r4[cA], rB = r4[cB];
                const float2 dA = dinv[cA], dB = dinv[cB];
                pnew(nslot + j, ff2_mulf(from4(rA), dA));
                if (jB < ng) pnew(nslot + jB, ff2_mulf(from4(rB), dB));
            }
            // the own rows from z in shared memory
            for (uint32_t l = tid; l < nslot && s0 * 32 + l < Nn; l += kThreads)
                pnew(l, from4(W[l]));
            __syncthreads();
        }
    }
    {   // b.u in FP64 (the compliance F^T u when b is the load vector).  part0
        // was last read before the L2 barrier of the last iteration.
        const double2* __restrict__ u = reinterpret_cast<const double2*>(a.u);
        const double2* __restrict__ b = reinterpret_cast<const double2*>(a.b);
        double bu = 0.0;
        for (uint32_t s = s0 + warp; s < s1; s += nw) {
            const uint32_t i = s * 32 + lane;
            if (i >= Nn) continue;
            const double2 ui = u[i], bi = b[i];
            bu = fma(bi.x, ui.x, fma(bi.y, ui.y, bu));
        }
        double v[1] = {bu};
        group_publish<1>(v, red, part0, rank);
        if (sync()) goto done;
        double J[1];
        group_reduce0<1>(part0, G, J);
        if (rank == 0 && tid == 0) g.res[5] = J[0];
    }
done:
    if (rank == 0 && tid == 0) {
        g.res[0] = (double)sc.k;
        g.res[1] = (double)sc.nupd;
        int st = ld_volatile(g.status);
        g.res[2] = st != 0 ? (double)st : (sc.converged ? 0.0 : 1.0);
        g.res[3] = sc.rr64;
        g.res[4] = sc.bb;
    }
}

__global__ void __launch_bounds__(kMixThreads, kMixMinBlocks)
    k_cg_mixed_ghost(MixArgs a, Group g, GhostArgs gh) {
    extern __shared__ __align__(16) unsigned char smem[];
    mixed_solve_ghost<kMixThreads>(a, g, gh, smem);
}

#include "mixed_slice.cuh"

}  // namespace

extern "C" int nbg_spmv_bsr_mixed(const nbg_bsr_t* A, const float* ph, const float* pl,
                                  float* wh, float* wl, void* stream) {
    if (!A || !A->b32 || !A->blo || !A->bxt || !ph || !pl || !wh || !wl) return NBG_ERR_ARG;
    if (A->perm) return NBG_ERR_ARG;  // the operator alone is for layouts in mesh order
    if (A->Nn == 0) return NBG_OK;
    MixArgs a;
    memset(&a, 0, sizeof(a));
    a.A = *A;
    a.ph = ph;
    a.pl = pl;
    a.keep = keep_share(*A);
    unsigned G = 0;
    const int rc = coop_grid((const void*)k_spmv_mixed, A->n_slices, &G, kMixThreads);
    if (rc != NBG_OK) return rc;
    k_spmv_mixed<<<G, kMixThreads, 0, (cudaStream_t)stream>>>(
        a, reinterpret_cast<float2*>(wh), reinterpret_cast<float2*>(wl));
    NBG_CHECK(cudaGetLastError());
    return NBG_OK;
}



extern "C" size_t nbg_cg_mixed_workspace_bytes(uint32_t N) { return mixed_bytes(N); }

namespace {
thread_local int g_mixed_form = 0;  // form of this thread's last nbg_cg_mixed launch
}  // namespace

extern "C" int nbg_cg_mixed_last_form(void) { return g_mixed_form; }

extern "C" size_t nbg_cg_mixed_layout_workspace_bytes(const nbg_bsr_t* A) {
    return A ? mixed_bytes(A->N) + ghost_plan_bytes(*A) : 0;
}

namespace {
// The ghost-node form for a G-block partition: 1 and its launch data when the
// vectors fit in shared memory at one block per SM.
int ghost_setup(const nbg_bsr_t& A, unsigned G, char* plan, cudaStream_t s, GhostArgs* gh,
                size_t* dyn) {
    uint32_t widest;
    if (!ghost_plan(A, G, plan, s, gh, &widest)) return 0;
    const size_t bytes = 16 * (size_t)gh->pcap + 16 * (size_t)gh->scap + 4 * (size_t)gh->gcap +
                         4 * ((size_t)gh->scap / 32 + 1);
    if (!fits_smem((const void*)k_cg_mixed_ghost, kMixThreads, bytes, G)) return 0;
    *dyn = bytes;
    return 1;
}

// Blocks of the slice form, 0 when the system is too large for it (a block
// has at most 32 warps and the grid one block per SM).  Four slices per
// block, one warp per scheduler, while there are SMs: the sums cost about
// the same over 17 blocks as over 152, the SpMV's FP32 work grows with the
// warps that share a scheduler.  Microseconds per iteration with 2, 4, 8, 16
// and 24 slices per block, with sums that were polled at once (0.3 slower than
// with kLeadUp): 4,290 dof 4.5, 4.4, 4.4, 5.5, 8.5; 16,770 dof 4.5, 4.4, 4.9, 5.9,
// 8.9.
unsigned slice_grid(uint32_t n_slices, int nsm) {
    const unsigned most = exact_grid((unsigned)nsm);
    if (n_slices > most * (kMixThreads / 32)) return 0;
    return std::min(most, (n_slices + 3) / 4);
}

template <int kThreads>
const void* slice_kernel_of(bool ghost) {
    return ghost ? (const void*)k_cg_mixed_slice<true, kThreads>
                 : (const void*)k_cg_mixed_slice<false, kThreads>;
}

// The instance with the most registers for `threads`.
const void* slice_kernel(bool ghost, int threads) {
    return threads <= 512 ? slice_kernel_of<512>(ghost)
         : threads <= 896 ? slice_kernel_of<896>(ghost)
                          : slice_kernel_of<kMixThreads>(ghost);
}

// The slice form with ghosts for a G-block partition: as ghost_setup; the
// matrix takes what shared memory is left, *keep entries of every row.
int slice_setup(const nbg_bsr_t& A, unsigned G, int threads, char* plan, cudaStream_t s,
                GhostArgs* gh, uint32_t* keep, size_t* dyn) {
    uint32_t widest;
    if (!ghost_plan(A, G, plan, s, gh, &widest)) return 0;
    const size_t base = 16 * (size_t)gh->pcap + 16 * (size_t)gh->gcap +
                        4 * (size_t)((gh->gcap + 3) & ~3u);
    int dev = 0, optin = 0;
    cudaFuncAttributes fa;
    const void* fn = slice_kernel(true, threads);
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) !=
            cudaSuccess ||
        cudaFuncGetAttributes(&fa, fn) != cudaSuccess)
        return 0;
    if (base + fa.sharedSizeBytes > (size_t)optin) return 0;
    const size_t left = (size_t)optin - fa.sharedSizeBytes - base;
    const size_t column = slice_entry_bytes(threads) * (size_t)threads;
    *keep = (uint32_t)std::min<size_t>(widest, left / column);
    *dyn = base + column * *keep;
    return fits_smem(fn, threads, *dyn, G) ? 1 : 0;
}
}  // namespace

namespace {
// Whether the rows of a block, without any ghosts, would fit in the ghost-node
// form's shared memory (2.1M dof on 152 SMs).  Up to there the global-gather form
// sums in fixed point as that form does, so that both give the same bits with any
// workspace; past it by partials, its iterations being bound by DRAM (us with
// partials and in fixed point, own rows in global memory: 1.13M dof 44.4 and 44.9,
// 1.67M 63.6 and 64.7, 1.97M 72.1 and 72.5; the ghost-node form itself at 1.13M dof
// 37.6 and 34.5, at 1.28M 42.1 and 39.2).
bool ghost_sizes(uint32_t n_slices, int nsm) {
    size_t most = 0;
    const unsigned G = exact_grid((unsigned)nsm * kMixMinBlocks);
    return allow_smem((const void*)k_cg_mixed_ghost, &most) == cudaSuccess &&
           (n_slices + G - 1) / G * (size_t)(32 * 2 * sizeof(float4)) <= most;
}

const void* mixed_kernel(int own, bool exact) {
    return own == 3 ? (const void*)k_cg_mixed<3, true>
         : own == 2 ? (const void*)k_cg_mixed<2, true>
         : own == 1 ? (exact ? (const void*)k_cg_mixed<1, true> : (const void*)k_cg_mixed<1, false>)
                    : (const void*)k_cg_mixed<0, false>;
}

// slices per block of a batch's waves
constexpr uint32_t kSlicesFew = 16, kSlicesMost = 28;
const void* slices_kernel(int threads) {
    return threads <= 32 * (int)kSlicesFew ? (const void*)k_cg_mixed_slices<32 * kSlicesFew>
                                           : (const void*)k_cg_mixed_slices<32 * kSlicesMost>;
}

const void* batch_kernel(int own) {
    return own == 3 ? (const void*)k_cg_mixed_many<3>
         : own == 2 ? (const void*)k_cg_mixed_many<2>
         : own == 1 ? (const void*)k_cg_mixed_many<1>
                    : (const void*)k_cg_mixed_many<0>;
}
}  // namespace

extern "C" int nbg_cg_mixed(const nbg_bsr_t* A, const double* b, double* x, uint32_t max_iter,
                            double tol, double delta, unsigned flags, nbg_mixed_result_t* result,
                            void* ws, size_t ws_bytes, void* stream) {
    if (!result || !A) return NBG_ERR_ARG;
    *result = nbg_mixed_result_t{0, 0, 0, 0.0, 0.0};
    if (A->Nn == 0) return NBG_OK;
    if (!A->b64 || !A->b32 || !A->blo || !A->bxt || !A->dinv32 || !(delta > 0.0 && delta < 1.0))
        return NBG_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t need = mixed_bytes(A->N), plan_bytes = ghost_plan_bytes(*A);
    void* own = nullptr;
    if (!ws) {
        NBG_CHECK(cudaMalloc(&own, need + plan_bytes));
        ws = own;
        ws_bytes = need + plan_bytes;
    } else if (ws_bytes < need) {
        return NBG_ERR_ARG;
    }
    char* base = (char*)ws;
    // the ghost form when the workspace holds its plan
    char* const plan = plan_bytes && ws_bytes >= need + plan_bytes ? base + need : nullptr;
    const size_t f = align256((size_t)A->N * 4), h = align256((size_t)A->N * 4);
    MixArgs a;
    a.A = *A;
    a.b = b;
    a.u = x;
    carve_vectors(a, base, A->N);
    Group g;
    g.part = (double*)(base + 6 * f + 2 * h);
    char* tail = base + 6 * f + 2 * h + align256(kMaxBlocks * 6 * 8);
    g.bar = (unsigned*)tail;
    g.status = (int*)(tail + 256);
    g.res = (double*)(tail + 512);
    g.sums = (unsigned char*)tail + 3 * 256 + kArBytes;
    a.max_iter = max_iter;
    a.tol = tol;
    a.delta = delta;
    a.flags = flags;
    a.keep = keep_share(*A);
    int rc = NBG_OK;
    unsigned G = 1;
    size_t dyn = 0;
    double hr[5] = {0, 0, 0, 0, 0};
    cudaError_t e = cudaMemsetAsync(tail, 0, kMixTail, s);
    if (A->perm) {  // solve in the layout's node order
        double* bp = (double*)(base + mixed_core_bytes(A->N));
        double* xp = bp + align256((size_t)A->N * 8) / 8;
        if (e == cudaSuccess) e = perm_gather(A->Nn, A->perm, b, bp, s);
        if (e == cudaSuccess) e = perm_gather(A->Nn, A->perm, (const double*)x, xp, s);
        a.b = bp;
        a.u = xp;
    }
    GhostArgs gh;
    memset(&gh, 0, sizeof(gh));
    SliceArgs sl{0, 0, (unsigned char*)tail + 3 * 256};
    bool ghost = false;
    int dev = 0, nsm = 0, threads = kMixThreads;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const unsigned slice_g = NBG_MIXED_RESIDENT ? slice_grid(A->n_slices, nsm) : 0;
    const void* fn = nullptr;
    bool resident = slice_g != 0;  // the own rows' vectors on chip
    if (e == cudaSuccess && slice_g) {
        G = slice_g;
        threads = 32 * (int)((A->n_slices + G - 1) / G);
        ghost = plan && slice_setup(*A, G, threads, plan, s, &gh, &sl.keep, &dyn) == 1;
        if (!ghost) dyn = 0;
        (void)cudaGetLastError();  // a plan that could not run leaves the global-gather form
        fn = slice_kernel(ghost, threads);
    } else if (e == cudaSuccess && plan) {
        // one block per SM, as the resident global-gather form's first choice
        const unsigned want = (A->n_slices + kMixThreads / 32 - 1) / (kMixThreads / 32);
        G = std::max(1u, std::min(exact_grid((unsigned)nsm * kMixMinBlocks), want));
        ghost = ghost_setup(*A, G, plan, s, &gh, &dyn) == 1;
        (void)cudaGetLastError();
        if (ghost) fn = (const void*)k_cg_mixed_ghost;
    }
    if (e == cudaSuccess && !fn) {
        // as many of the own rows' vectors in shared memory as fit, at the
        // same grid: the rows of a block, and so the sums, are the same
        for (int own = NBG_MIXED_RESIDENT ? 3 : 0; own >= 0 && rc == NBG_OK && !fn; own--) {
            fn = mixed_kernel(own, ghost_sizes(A->n_slices, nsm));
            rc = coop_grid_resident(fn, A->n_slices, own_node_bytes(own) * 32, &G, &dyn, kMixThreads,
                                    kMixMinBlocks, kExactMaxBlocks);
            resident = own == 3;
            if (own > 0 && (dyn == 0 || (own < 3 && dyn > kOwnSmem))) fn = nullptr;
        }
    }
    g.s_begin = 0;
    g.s_end = A->n_slices;
    g.g_base = 0;
    g.g_size = G;
    g.pstride = kMaxBlocks;
    if (ghost) a.keep = keep_share(*A, 30.0);
    g_mixed_form = ghost      ? NBG_MIXED_GHOST
                 : resident ? NBG_MIXED_RESIDENT_ROWS
                            : NBG_MIXED_GLOBAL_ROWS;
    if (e == cudaSuccess && rc == NBG_OK) {
        void* args[] = {&a, &g, &gh, &sl};
        e = cudaLaunchCooperativeKernel(fn, dim3(G), dim3(threads), args, dyn, s);
        if (e == cudaSuccess && A->perm) e = perm_scatter(A->Nn, A->perm, (const double*)a.u, x, s);
    }
    if (e == cudaSuccess && rc == NBG_OK)
        e = cudaMemcpyAsync(hr, g.res, sizeof(hr), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && rc == NBG_OK) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) rc = nbg_cuda_error(e);
    if (rc == NBG_OK) {
        result->niter = (uint32_t)hr[0];
        result->n_updates = (uint32_t)hr[1];
        result->status = (int)hr[2];
        result->bnorm = sqrt(hr[4]);
        result->relres = hr[4] > 0 ? sqrt(hr[3] / hr[4]) : sqrt(hr[3]);
        rc = result->status;
    }
    if (own) cudaFree(own);
    return rc;
}

// ------------------------------------------------------------------ batch
// Many independent systems stored as one block-diagonal layout (each
// system's node rows start on a slice boundary) and solved by one
// cooperative launch of k_cg_mixed_many, replayed as a CUDA graph together
// with zeroing x and, optionally, the SIMP compliance sensitivities.

namespace {
// One launch of the slice form (k_cg_mixed_slices): systems side by side, one
// block per SM, a warp for each slice.
struct Wave {
    std::vector<uint32_t> systems, blocks;
    uint32_t first;  // blocks of the waves before it
    unsigned G;
    int threads;
};
}  // namespace

struct nbg_mixed_batch {
    nbg_bsr_t A;
    const double* b;
    double* x;
    uint32_t n_sys;
    std::vector<uint32_t> slice_ptr, blocks;
    uint32_t max_iter;
    double tol, delta, gamma;
    unsigned flags;
    cudaStream_t stream;
    void* ws;
    MixArgs args;  // settings shared by every system
    Group* d_groups;
    uint32_t* d_map;
    double* d_res;
    unsigned char* d_state;
    unsigned G;
    size_t dyn;
    int own;      // own-row vectors in shared memory (mixed_solve's kOwn), or kSliceForm
    std::vector<Wave> waves;  // slice form: its launches, one after the other
    unsigned char* d_sums;    // kBatchSums per system
    uint2* d_range;           // slices of each block
    char* d_plan;             // ghost plan; null: not for the slice form
    // compliance sensitivities after the solve (a = b = x)
    bool sens;
    uint32_t nen, N_elem;
    const double* nod;
    const uint32_t* conn;
    const double* rho;
    double* dJ;
    double nu, thickness, penal, E0, Emin;
    cudaGraph_t graph;
    cudaGraphExec_t exec;
};

namespace {

constexpr size_t kStateStride = 256;  // per system: barrier +0, status +128, plan failed +192
constexpr size_t kBatchSums = kArBytes + 2 * kExactBytes;  // per system, of the slice form
constexpr int kSliceForm = 4;  // nbg_mixed_batch::own
constexpr size_t kResStride = 8;      // doubles of result per system

size_t batch_bytes(uint32_t N, uint32_t n_sys) {
    return mixed_bytes(N) + align256((size_t)n_sys * kStateStride) +
           align256((size_t)n_sys * kResStride * 8) + align256((size_t)n_sys * sizeof(Group)) +
           align256((size_t)kMaxBlocks * 4);
}

double* part_slots(char* base, uint32_t N) {
    const size_t f = align256((size_t)N * 4), h = align256((size_t)N * 4);
    return (double*)(base + 6 * f + 2 * h);
}

// Blocks per system: one each (or enough for most_per_block slices), then one
// at a time to the system with the largest weight per block (weight =
// slices^gamma), never more than one per least_per_block slices.  Minimises
// the largest weight per block.
void share_blocks(const std::vector<uint32_t>& sp, double gamma, unsigned total,
                  uint32_t least_per_block, uint32_t most_per_block, std::vector<uint32_t>& out) {
    const size_t n = sp.size() - 1;
    std::vector<double> w(n);
    std::vector<uint32_t> cap(n);
    out.assign(n, 1);
    unsigned used = 0;
    for (size_t i = 0; i < n; i++) {
        const uint32_t S = sp[i + 1] - sp[i];
        w[i] = std::pow((double)std::max<uint32_t>(S, 1), gamma);
        cap[i] = std::max<uint32_t>(1, (S + least_per_block - 1) / least_per_block);
        if (most_per_block) out[i] = std::max<uint32_t>(1, (S + most_per_block - 1) / most_per_block);
        used += out[i];
    }
    for (unsigned left = total - used; left > 0; --left) {
        size_t best = n;
        double bw = -1.0;
        for (size_t i = 0; i < n; i++)
            if (out[i] < cap[i] && w[i] / out[i] > bw) {
                bw = w[i] / out[i];
                best = i;
            }
        if (best == n) break;
        out[best]++;
    }
}

uint32_t max_slices_per_block(const std::vector<uint32_t>& sp, const std::vector<uint32_t>& bl) {
    uint32_t m = 0;
    for (size_t i = 0; i + 1 < sp.size(); i++)
        m = std::max(m, (sp[i + 1] - sp[i] + bl[i] - 1) / bl[i]);
    return m;
}

// The systems in waves of at most `most` slices per block, as few as first-fit
// decreasing finds; the time that they take, in us per square root of slices (an
// iteration's time, and iterations grow with a mesh's length), or a negative
// number when a system is too large.  Measured us per iteration of a wave: 4.5
// with 4 slices per block, 5.6 with 16, the most that leaves a thread 128
// registers, 7.0 with 17, 8.9 with 27, 11.6 with 32 (which is not used).
double slice_waves(const std::vector<uint32_t>& sp, double gamma, unsigned total, uint32_t most,
                   std::vector<Wave>& waves) {
    const uint32_t n = (uint32_t)sp.size() - 1;
    auto slices = [&](uint32_t i) { return sp[i + 1] - sp[i]; };
    auto least = [&](uint32_t i) { return std::max(1u, (slices(i) + most - 1) / most); };
    std::vector<uint32_t> order(n);
    for (uint32_t i = 0; i < n; i++) order[i] = i;
    std::stable_sort(order.begin(), order.end(),
                     [&](uint32_t i, uint32_t j) { return slices(i) > slices(j); });
    waves.clear();
    if (least(order[0]) > total) return -1.0;
    for (uint32_t i : order) {
        auto w = std::find_if(waves.begin(), waves.end(),
                              [&](const Wave& v) { return v.G + least(i) <= total; });
        if (w == waves.end()) w = waves.insert(waves.end(), Wave{{}, {}, 0, 0, 0});
        w->systems.push_back(i);
        w->G += least(i);
    }
    double cost = 0.0;
    uint32_t first = 0;
    for (Wave& w : waves) {
        std::vector<uint32_t> own{0};
        for (uint32_t i : w.systems) own.push_back(own.back() + slices(i));
        share_blocks(own, gamma, total, kSlicesFew, most, w.blocks);
        const uint32_t per = std::max(1u, max_slices_per_block(own, w.blocks));
        w.threads = 32 * (int)per;
        w.first = first;
        w.G = 0;
        for (uint32_t v : w.blocks) w.G += v;
        first += w.G;
        cost += std::sqrt((double)slices(w.systems[0])) *
                (per <= kSlicesFew ? 4.2 + 0.085 * per : 7.0 + 0.18 * (per - kSlicesFew - 1));
    }
    return first <= kMaxBlocks ? cost : -1.0;
}

// The better of two packings, when it beats all systems side by side in the
// other form, whose iteration takes 8 us and 1.7 ns per slice: that is bound by
// DRAM once the systems are larger than L2, while a wave's matrices are in shared
// memory and L2; but a wave's block works for one system, however small.
// Milliseconds in the other form and in waves: 24 systems of 48 and 96
// elements' length 12.5 and 7.0, 6 of 96 and 192 25.0 and 11.1, 12 of 64 to 256
// 50.0 and 30.3, 24 of 48 to 192 40.0 and 33.6, 24 of 64 to 512 277 and 259 (254 now); 20 of
// 96 to 384, six of them of 2,323 slices, stay (180, in waves 196).
bool best_waves(const std::vector<uint32_t>& sp, double gamma, unsigned nsm,
                std::vector<Wave>& waves) {
    uint32_t largest = 0;
    for (size_t i = 0; i + 1 < sp.size(); i++) largest = std::max(largest, sp[i + 1] - sp[i]);
    double best = std::sqrt((double)largest) * (8.0 + 0.0017 * sp.back());
    waves.clear();
    for (uint32_t most : {kSlicesFew, kSlicesMost}) {
        std::vector<Wave> w;
        const double cost =
            NBG_MIXED_RESIDENT ? slice_waves(sp, gamma, exact_grid(nsm), most, w) : -1.0;
        if (cost >= 0.0 && cost < best) {
            best = cost;
            waves.swap(w);
        }
    }
    return !waves.empty();
}

inline int cu(cudaError_t e) { return e == cudaSuccess ? NBG_OK : nbg_cuda_error(e); }

void drop_graph(nbg_mixed_batch* m) {
    if (m->exec) cudaGraphExecDestroy(m->exec);
    if (m->graph) cudaGraphDestroy(m->graph);
    m->exec = nullptr;
    m->graph = nullptr;
}

// Block shares, launch size and the per-system argument table for `gamma`.
int batch_plan(nbg_mixed_batch* m, double gamma) {
    int dev = 0, nsm = 0;
    NBG_CHECK(cudaGetDevice(&dev));
    NBG_CHECK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const uint32_t n = m->n_sys;
    std::vector<uint32_t> bl;
    unsigned G = 0;
    size_t dyn = 0;
    int own = NBG_MIXED_RESIDENT ? 3 : 0;
    // a launch of per_sm blocks per SM that keeps `own` vectors of its rows in
    // shared memory, when it fits
    auto fits = [&](int per_sm) -> int {
        const void* fn = batch_kernel(own);
        size_t most = 0;
        NBG_CHECK(allow_smem(fn, &most));
        const unsigned total = std::min<unsigned>((unsigned)nsm * per_sm, kMaxBlocks);
        if (n > total) return NBG_OK;
        share_blocks(m->slice_ptr, gamma, total, kBatThreads / 32, 0, bl);
        const size_t bytes =
            (size_t)max_slices_per_block(m->slice_ptr, bl) * own_node_bytes(own) * 32;
        if (bytes > most || (own < 3 && bytes * per_sm > kOwnSmem)) return NBG_OK;
        int occ = 0;
        NBG_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kBatThreads, bytes));
        unsigned used = 0;
        for (uint32_t v : bl) used += v;
        if ((uint64_t)occ * (unsigned)nsm >= used) {
            G = used;
            dyn = bytes;
        }
        return NBG_OK;
    };
    // the resident block count of the form that takes any systems
    int occ0 = 0;
    NBG_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ0, batch_kernel(0), kBatThreads, 0));
    const unsigned total0 = std::min<unsigned>((unsigned)nsm * (unsigned)std::max(occ0, 1), kMaxBlocks);
    if (n > total0) return NBG_ERR_ARG;  // every system needs a co-resident block
    // the slice form where it takes the systems
    std::vector<Wave> waves;
    if (m->d_plan && best_waves(m->slice_ptr, gamma, (unsigned)nsm, waves)) {
        NBG_CHECK(cudaFuncSetAttribute((const void*)k_ghost_plan,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(kGhostKeys * 4)));
        own = kSliceForm;
        bl.assign(n, 0);
        for (const Wave& w : waves) {
            size_t most = 0;
            NBG_CHECK(allow_smem(slices_kernel(w.threads), &most));
            dyn = dyn ? std::min(dyn, most) : most;
            G += w.G;
            for (size_t k = 0; k < w.systems.size(); k++) bl[w.systems[k]] = w.blocks[k];
        }
    } else {
        waves.clear();
    }
    // all own rows in shared memory, with fewer blocks per SM if need be;
    // else at the full block count as many of the vectors as fit
    for (int per_sm = kBatMinBlocks; own == 3 && per_sm >= 1 && !G; --per_sm) {
        const int rc = fits(per_sm);
        if (rc != NBG_OK) return rc;
    }
    while (!G && own > 1) {
        own--;
        const int rc = fits(kBatMinBlocks);
        if (rc != NBG_OK) return rc;
    }
    if (!G) {
        own = 0;
        share_blocks(m->slice_ptr, gamma, total0, kBatThreads / 32, 0, bl);
        for (uint32_t v : bl) G += v;
        dyn = 0;
    }
    // shared settings, group table and block -> system map
    char* base = (char*)m->ws;
    MixArgs& a = m->args;
    memset(&a, 0, sizeof(a));
    a.A = m->A;
    a.b = m->b;
    a.u = m->x;
    carve_vectors(a, base, m->A.N);  // shared by every system, by the global node row
    a.max_iter = m->max_iter;
    a.tol = m->tol;
    a.delta = m->delta;
    a.flags = m->flags;
    // all of a batch's matrix or nothing: a system reads its part again only
    // after every other system's (24 systems, 252 MB: 337 ms with none kept,
    // 351 with a fifth; 12 systems, 41 MB: 33.2 ms with all, 34.2 with none)
    const double in_l2 = stream_over_l2(m->A);
    a.keep = own == kSliceForm || (in_l2 > 0.0 && in_l2 <= 0.30) ? 0xFFFFFFFFu : 0;
    m->own = own;
    std::vector<Group> groups(n);
    std::vector<uint32_t> map(G);
    double* part = part_slots(base, m->A.N);
    unsigned gb = 0;
    for (uint32_t i = 0; i < n; i++) {
        Group& g = groups[i];
        g.part = part + 6 * (size_t)gb;
        g.pstride = bl[i];
        g.bar = (unsigned*)(m->d_state + i * kStateStride);
        g.status = (int*)(m->d_state + i * kStateStride + 128);
        g.res = m->d_res + i * kResStride;
        g.sums = own == kSliceForm ? m->d_sums + i * kBatchSums + kArBytes : nullptr;
        g.s_begin = m->slice_ptr[i];
        g.s_end = m->slice_ptr[i + 1];
        g.g_base = gb;
        g.g_size = bl[i];
        for (uint32_t k = 0; k < bl[i]; k++) map[gb + k] = i;
        gb += bl[i];
    }
    std::vector<uint2> range(G);
    for (const Wave& w : waves) {  // blocks numbered within their wave
        uint32_t at = 0;
        for (uint32_t i : w.systems) {
            const uint64_t S = m->slice_ptr[i + 1] - m->slice_ptr[i];
            groups[i].g_base = at;
            for (uint32_t k = 0; k < bl[i]; k++) {  // as group_slice_range
                map[w.first + at + k] = i;
                range[w.first + at + k] = make_uint2(m->slice_ptr[i] + (uint32_t)(S * k / bl[i]),
                                                     m->slice_ptr[i] + (uint32_t)(S * (k + 1) / bl[i]));
            }
            at += bl[i];
        }
    }
    NBG_CHECK(cudaMemcpy(m->d_groups, groups.data(), n * sizeof(Group), cudaMemcpyHostToDevice));
    NBG_CHECK(cudaMemcpy(m->d_map, map.data(), G * 4, cudaMemcpyHostToDevice));
    if (own == kSliceForm)
        NBG_CHECK(cudaMemcpy(m->d_range, range.data(), G * sizeof(uint2), cudaMemcpyHostToDevice));
    m->waves = waves;
    m->blocks = bl;
    m->G = G;
    m->dyn = dyn;
    m->gamma = gamma;
    drop_graph(m);
    return NBG_OK;
}

// The work of one batch launch, enqueued on s (captured into the graph).
cudaError_t batch_enqueue(nbg_mixed_batch* m, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(m->x, 0, 8 * (size_t)m->A.N, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->d_state, 0, (size_t)m->n_sys * kStateStride, s);
    if (e != cudaSuccess) return e;
    const Group* groups = m->d_groups;
    const uint32_t* map = m->d_map;
    MixArgs args = m->args;
    cudaLaunchConfig_t cfg = {};
    cfg.dynamicSmemBytes = m->dyn;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (m->own != kSliceForm) {
        cfg.gridDim = dim3(m->G);
        cfg.blockDim = dim3(kBatThreads);
        void* params[] = {&args, &groups, &map};
        e = cudaLaunchKernelExC(&cfg, batch_kernel(m->own), params);
    } else {
        e = cudaMemsetAsync(m->d_sums, 0, (size_t)m->n_sys * kBatchSums, s);
    }
    for (const Wave& w : m->waves) {
        if (e != cudaSuccess) return e;
        // planned in each launch, from the columns that the layout has then
        GhostArgs gh;
        memset(&gh, 0, sizeof(gh));
        uint16_t* lcol;
        uint32_t *ids, *count;
        ghost_regions(m->A, w.G, m->d_plan, &lcol, &ids, &count);
        gh.lcol = lcol;
        gh.ids = ids;
        gh.count = count;
        map = m->d_map + w.first;
        const PlanBatch pb{m->d_range + w.first, map, m->dyn, (uint32_t)(kStateStride / 4)};
        k_ghost_plan<<<w.G, 1024, kGhostKeys * 4, s>>>(
            m->A, lcol, ids, count, (int*)(m->d_state + 128) + kNoPlan, pb);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        SliceArgs sl{0, (uint32_t)m->dyn, nullptr};
        cfg.gridDim = dim3(w.G);
        cfg.blockDim = dim3(w.threads);
        void* params[] = {&args, &groups, &map, &gh, &sl};
        e = cudaLaunchKernelExC(&cfg, slices_kernel(w.threads), params);
    }
    if (e != cudaSuccess || !m->sens) return e;
    const int rc = nbg_simp_sensitivity_f64(m->nen, m->N_elem, m->nod, m->conn, m->nu,
                                            m->thickness, m->rho, m->penal, m->E0, m->Emin, m->x,
                                            m->x, m->dJ, s);
    return rc == NBG_OK ? cudaSuccess : cudaErrorLaunchFailure;
}

int build_graph(nbg_mixed_batch* m) {
    cudaStream_t cap;
    NBG_CHECK(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
    cudaError_t e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        const cudaError_t e1 = batch_enqueue(m, cap);
        cudaGraph_t g = nullptr;
        const cudaError_t e2 = cudaStreamEndCapture(cap, &g);
        e = e1 != cudaSuccess ? e1 : e2;
        if (e == cudaSuccess) {
            m->graph = g;
            e = cudaGraphInstantiate(&m->exec, g, 0);
        } else if (g) {
            cudaGraphDestroy(g);
        }
    }
    cudaStreamDestroy(cap);
    if (e != cudaSuccess) {
        drop_graph(m);
        return nbg_cuda_error(e);
    }
    return NBG_OK;
}

}  // namespace

extern "C" int nbg_mixed_batch_create(nbg_mixed_batch_t** out, const nbg_bsr_t* A,
                                      const double* b, double* x, uint32_t n_sys,
                                      const uint32_t* slice_ptr, uint32_t max_iter, double tol,
                                      double delta, unsigned flags, void* stream) {
    if (!out || !A || A->perm) return NBG_ERR_ARG;  // instances own contiguous slices
    *out = nullptr;
    if (!A || !b || !x || !slice_ptr || n_sys == 0 || n_sys > kMaxBlocks || !A->b64 ||
        !A->b32 || !A->blo || !A->bxt || !A->dinv32 || !(delta > 0.0 && delta < 1.0))
        return NBG_ERR_ARG;
    if (slice_ptr[0] != 0 || slice_ptr[n_sys] != A->n_slices) return NBG_ERR_ARG;
    for (uint32_t i = 0; i < n_sys; i++)
        if (slice_ptr[i + 1] < slice_ptr[i]) return NBG_ERR_ARG;
    nbg_mixed_batch* m = new (std::nothrow) nbg_mixed_batch();
    if (!m) return NBG_ERR_NOMEM;
    m->A = *A;
    m->b = b;
    m->x = x;
    m->n_sys = n_sys;
    m->slice_ptr.assign(slice_ptr, slice_ptr + n_sys + 1);
    m->max_iter = max_iter;
    m->tol = tol;
    m->delta = delta;
    m->flags = flags;
    m->stream = (cudaStream_t)stream;
    std::vector<Wave> waves;
    int dev = 0, nsm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    bool slices = e == cudaSuccess && best_waves(m->slice_ptr, 1.5, (unsigned)nsm, waves);
    const size_t base_bytes = batch_bytes(A->N, n_sys), sums = align256((size_t)n_sys * kBatchSums),
                 ranges = align256(sizeof(uint2) * kMaxBlocks);
    const size_t need = base_bytes + (slices ? sums + ranges + ghost_plan_bytes(*A) : 0);
    if (e == cudaSuccess) e = cudaMalloc(&m->ws, need);
    if (e == cudaErrorMemoryAllocation && slices) {  // side by side needs no plan
        (void)cudaGetLastError();
        slices = false;
        e = cudaMalloc(&m->ws, base_bytes);
    }
    if (e != cudaSuccess) {
        delete m;
        return nbg_cuda_error(e);
    }
    char* p = (char*)m->ws + mixed_bytes(A->N);
    m->d_state = (unsigned char*)p;
    p += align256((size_t)n_sys * kStateStride);
    m->d_res = (double*)p;
    p += align256((size_t)n_sys * kResStride * 8);
    m->d_groups = (Group*)p;
    p += align256((size_t)n_sys * sizeof(Group));
    m->d_map = (uint32_t*)p;
    p = (char*)m->ws + base_bytes;
    m->d_sums = (unsigned char*)p;
    m->d_range = (uint2*)(p + sums);
    m->d_plan = slices ? p + sums + ranges : nullptr;
    // weights slices^1.5: CG's iterations grow with a mesh's length, so with
    // shares in proportion to the slices the small systems finish early and
    // their blocks idle (24 systems of 64 to 512 elements' length: 377 ms at
    // gamma 0.75, 332 at 1, 299 at 1.25, 281 at 1.5, 345 at 1.75; 20 of 96 to
    // 384: 210, 198, 193, 184, 185)
    int rc = batch_plan(m, 1.5);
    if (rc != NBG_OK) {
        nbg_mixed_batch_destroy(m);
        return rc;
    }
    *out = m;
    return NBG_OK;
}

extern "C" void nbg_mixed_batch_destroy(nbg_mixed_batch_t* m) {
    if (!m) return;
    drop_graph(m);
    if (m->ws) cudaFree(m->ws);
    delete m;
}

extern "C" int nbg_mixed_batch_plan(nbg_mixed_batch_t* m, double gamma) {
    if (!m || !(gamma >= 0.0 && gamma <= 4.0)) return NBG_ERR_ARG;
    return batch_plan(m, gamma);
}

extern "C" uint32_t nbg_mixed_batch_blocks(const nbg_mixed_batch_t* m, uint32_t* blocks,
                                           double* gamma) {
    if (!m) return 0;
    if (blocks) std::copy(m->blocks.begin(), m->blocks.end(), blocks);
    if (gamma) *gamma = m->gamma;
    return m->G;
}

// How the last launch ran, for checks: the return value is its waves of the slice
// form (0: all systems side by side, < 0: error), form[i] is NBG_MIXED_GHOST where
// system i had its ghosts in shared memory, else NBG_MIXED_RESIDENT_ROWS or
// NBG_MIXED_GLOBAL_ROWS.
extern "C" int nbg_mixed_batch_form(const nbg_mixed_batch_t* m, int* form) {
    if (!m || !form) return NBG_ERR_ARG;
    std::vector<unsigned char> state((size_t)m->n_sys * kStateStride);
    NBG_CHECK(cudaMemcpyAsync(state.data(), m->d_state, state.size(), cudaMemcpyDeviceToHost,
                              m->stream));
    NBG_CHECK(cudaStreamSynchronize(m->stream));
    for (uint32_t i = 0; i < m->n_sys; i++) {
        int failed;
        memcpy(&failed, &state[i * kStateStride + 128 + 4 * kNoPlan], sizeof(int));
        form[i] = m->own == kSliceForm && !failed ? NBG_MIXED_GHOST
                : m->own >= 3                     ? NBG_MIXED_RESIDENT_ROWS
                                                  : NBG_MIXED_GLOBAL_ROWS;
    }
    return (int)m->waves.size();
}

extern "C" int nbg_mixed_batch_set_sensitivity(nbg_mixed_batch_t* m, uint32_t nen,
                                               uint32_t N_elem, const double* nod,
                                               const uint32_t* conn, double nu, double thickness,
                                               const double* rho, double penal, double E0,
                                               double Emin, double* dJ) {
    if (!m || (nen != 3 && nen != 4) || (N_elem && (!nod || !conn || !rho || !dJ)))
        return NBG_ERR_ARG;
    m->sens = N_elem > 0;
    m->nen = nen;
    m->N_elem = N_elem;
    m->nod = nod;
    m->conn = conn;
    m->nu = nu;
    m->thickness = thickness;
    m->rho = rho;
    m->penal = penal;
    m->E0 = E0;
    m->Emin = Emin;
    m->dJ = dJ;
    drop_graph(m);
    return NBG_OK;
}

extern "C" int nbg_mixed_batch_launch(nbg_mixed_batch_t* m) {
    if (!m) return NBG_ERR_ARG;
    const int rc = m->exec ? NBG_OK : build_graph(m);
    if (rc != NBG_OK) return rc;
    NBG_CHECK(cudaGraphLaunch(m->exec, m->stream));
    return NBG_OK;
}

extern "C" int nbg_mixed_batch_results(nbg_mixed_batch_t* m, nbg_mixed_result_t* res,
                                       double* J) {
    if (!m) return NBG_ERR_ARG;
    std::vector<double> h((size_t)m->n_sys * kResStride);
    NBG_CHECK(cudaMemcpyAsync(h.data(), m->d_res, h.size() * 8, cudaMemcpyDeviceToHost,
                              m->stream));
    NBG_CHECK(cudaStreamSynchronize(m->stream));
    int worst = NBG_OK;
    for (uint32_t i = 0; i < m->n_sys; i++) {
        const double* r = &h[(size_t)i * kResStride];
        nbg_mixed_result_t t;
        t.niter = (uint32_t)r[0];
        t.n_updates = (uint32_t)r[1];
        t.status = (int)r[2];
        t.bnorm = std::sqrt(r[4]);
        t.relres = r[4] > 0 ? std::sqrt(r[3] / r[4]) : std::sqrt(r[3]);
        if (res) res[i] = t;
        if (J) J[i] = r[5];
        if (t.status < 0 && worst >= 0) worst = t.status;
        else if (t.status > 0 && worst == NBG_OK) worst = t.status;
    }
    return worst;
}

extern "C" int nbg_mixed_batch_tune(nbg_mixed_batch_t* m, uint32_t n_cand, const double* gammas,
                                    double* ms) {
    if (!m || !n_cand || !gammas) return NBG_ERR_ARG;
    cudaEvent_t t0, t1;
    NBG_CHECK(cudaEventCreate(&t0));
    NBG_CHECK(cudaEventCreate(&t1));
    int rc = NBG_OK;
    double best_ms = 0.0, best_g = gammas[0];
    for (uint32_t c = 0; c < n_cand && rc == NBG_OK; c++) {
        rc = nbg_mixed_batch_plan(m, gammas[c]);
        if (rc == NBG_OK) rc = nbg_mixed_batch_launch(m);  // builds the graph, warms up
        if (rc == NBG_OK) rc = cu(cudaEventRecord(t0, m->stream));
        if (rc == NBG_OK) rc = nbg_mixed_batch_launch(m);
        if (rc == NBG_OK) rc = cu(cudaEventRecord(t1, m->stream));
        if (rc == NBG_OK) rc = cu(cudaEventSynchronize(t1));
        float t = 0.f;
        if (rc == NBG_OK) rc = cu(cudaEventElapsedTime(&t, t0, t1));
        if (rc == NBG_OK) {
            const int st = nbg_mixed_batch_results(m, nullptr, nullptr);
            if (st < 0) rc = st;
        }
        if (ms) ms[c] = t;
        if (rc == NBG_OK && (c == 0 || t < best_ms)) {
            best_ms = t;
            best_g = gammas[c];
        }
    }
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    if (rc != NBG_OK) return rc;
    return nbg_mixed_batch_plan(m, best_g);
}
