// Grid-wide sums for the persistent solvers whose iterations are bound by
// latency.
//
// ExactSum: sums in fixed point, one hop.  Every value is cut into five
// 20-bit limbs below 2^20 times the sum's previous value; limbs are summed
// as integers, over a warp (redux), over the block's warps (redux again) and
// over the grid by one 64-bit reduction per limb at L2, whose top byte counts
// the blocks.  A block polls the words it added to until every count is
// complete: the sum arrives with the last poll, with no partials to publish
// before a barrier (whose release fence alone takes 800 cycles) and to load
// behind it.  152 blocks: 0.87 us against 1.57 us for the counting barrier
// with its partials, measured alone; the block sums take about 200 cycles
// instead of 1,000 to 1,500 for float-float (FP64: more) shuffle trees.  The
// words are never reset: each block subtracts their value at its last sum.
// Integer sums do not depend on their order, so the result is the same bits
// whatever the partition.  The window reaches from 2^20 above to 2^-80 below
// the previous value: the sum is exact but for each addend's bits below that,
// half a unit of 2^-80 times the previous value, within the bounds of float-float
// and FP64 adds.  Where the window does not serve (no previous value yet, an
// addend above it, infinities and NaN, a sum 2^24 times smaller than the last, a
// float-float sum below 2^-97) every block sees so, and the records sum the same
// values with float-float or FP64 adds instead.
//
// AllReduce: sums by records.  A record is 16 bytes, a 64-bit payload and a
// 64-bit epoch, written and read as one 128-bit access
// (ld/st.relaxed.gpu.b128: single-copy atomic).  A reader polls the record
// itself until its epoch is the one it waits for, so the payload needs no
// fence before it and no second load after it.  152 blocks polling the same
// records queue at the same L2 lines (2.5 us), so above 16 blocks the sum runs
// in two stages over a grid of groups (columns) and members (rows): the
// members of a group sum their group, then the blocks of a row sum the
// groups.  No record has more than 16 readers; the order is fixed.
#pragma once

#include "common.cuh"
#include "fixed_sum.cuh"

namespace nbg {

__device__ __forceinline__ void st_record(void* p, uint64_t v, uint64_t epoch) {
    asm volatile("{.reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t;}" ::"l"(p),
                 "l"(v), "l"(epoch)
                 : "memory");
}

__device__ __forceinline__ void ld_record(const void* p, uint64_t& v, uint64_t& epoch) {
    asm volatile("{.reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t;}"
                 : "=l"(v), "=l"(epoch)
                 : "l"(p)
                 : "memory");
}

__device__ __forceinline__ uint64_t ff_bits(float hi, float lo) {
    return (uint64_t)__float_as_uint(lo) << 32 | __float_as_uint(hi);
}

__device__ __forceinline__ FF bits_ff(uint64_t b) {
    return {__uint_as_float((uint32_t)b), __uint_as_float((uint32_t)(b >> 32))};
}

// Bounded wait of one poll loop: true when the caller must give up (the
// limit has passed, or another block has recorded an error).
struct PollLimit {
    uint64_t t0 = 0;
    unsigned it = 0;
    __device__ __forceinline__ bool expired(int* status) {
        if ((++it & 63u) != 0) return false;
        const uint64_t t = globaltimer();
        if (t0 == 0) t0 = t;
        if (t - t0 > kSpinLimitNs) {
            atomicCAS(status, 0, NBG_ERR_TIMEOUT);
            return true;
        }
        return ld_volatile(status) != 0;
    }
};

// How values of a type are summed: FP64 adds, or float-float pairs whose low
// parts are only renormalised at the end (the shuffle of the next level then
// waits for one add, not for the whole float-float sum).
struct SumF64 {
    using T = double;
    __device__ static uint64_t bits(T v) { return (uint64_t)__double_as_longlong(v); }
    __device__ static T from(uint64_t b) { return __longlong_as_double((long long)b); }
    __device__ static T zero() { return 0.0; }
    __device__ static T xor_add(T v, int o) { return v + __shfl_xor_sync(0xffffffffu, v, o); }
    __device__ static T finish(T v) { return v; }
};

struct SumFF {
    using T = FF;
    __device__ static uint64_t bits(T v) { return ff_bits(v.hi, v.lo); }
    __device__ static T from(uint64_t b) { return bits_ff(b); }
    __device__ static T zero() { return {0.f, 0.f}; }
    __device__ static T xor_add(T v, int o) {
        const float h = __shfl_xor_sync(0xffffffffu, v.hi, o);
        const float l = __shfl_xor_sync(0xffffffffu, v.lo, o);
        const FF t = two_sum(v.hi, h);
        return {t.hi, __fadd_rn(t.lo, __fadd_rn(v.lo, l))};
    }
    __device__ static T finish(T v) { return fast_two_sum(v.hi, v.lo); }
};

constexpr unsigned kArLanes = 16;                       // readers of a record
constexpr unsigned kArMaxBlocks = kArLanes * kArLanes;  // of one launch
// [2 epochs][2 stages][2 values][kArMaxBlocks] records; zero at launch
constexpr size_t kArBytes = 2 * 2 * 2 * kArMaxBlocks * 16;

// One launch's place in the sums: block `rank` of G <= kArMaxBlocks.
struct AllReduce {
    unsigned char* area;
    int* status;
    uint32_t groups, group, member, size, rows;
    uint64_t epoch;

    __device__ __forceinline__ void init(void* a, int* st, uint32_t G, uint32_t rank) {
        area = (unsigned char*)a;
        status = st;
        groups = (G + kArLanes - 1) / kArLanes;
        group = rank % groups;
        member = rank / groups;
        size = (G - group + groups - 1) / groups;  // members of this group
        rows = (G + groups - 1) / groups;          // of the largest group
        epoch = 0;
    }
    __device__ __forceinline__ unsigned char* slot(uint32_t stage, uint32_t value,
                                                   uint32_t at) const {
        return area +
               ((((uint32_t)(epoch & 1) * 2 + stage) * 2 + value) * kArMaxBlocks + at) * 16;
    }
    // Sum over the records at .. at + n of a stage, lanes 0-15 value 0 and
    // lanes 16-31 value 1; nonzero return: give up.
    template <class S, int NV>
    __device__ __forceinline__ int gather(uint32_t stage, uint32_t at, uint32_t n,
                                          typename S::T& out) const {
        const uint32_t lane = threadIdx.x & 31, m = lane & (kArLanes - 1), v = lane / kArLanes;
        const bool active = m < n && v < NV;
        const void* p = slot(stage, v < NV ? v : 0, at + m);
        uint64_t b = S::bits(S::zero());
        PollLimit lim;
        for (;;) {
            bool ok = true;
            if (active) {
                uint64_t e;
                ld_record(p, b, e);
                ok = e == epoch;
            }
            if (__all_sync(0xffffffffu, ok)) break;
            if (__any_sync(0xffffffffu, lim.expired(status))) return 1;
        }
        typename S::T t = active ? S::from(b) : S::zero();
#pragma unroll
        for (int o = kArLanes / 2; o > 0; o >>= 1) t = S::xor_add(t, o);
        out = S::finish(t);
        return 0;
    }
    // Grid-wide sums of NV (1 or 2) values, called by one whole warp whose
    // lanes all hold this block's values in v; on return (0) they hold the
    // sums.  Successive calls use the two halves of the area in turn: a block
    // enters call e + 2 only after every reader of its records of call e has
    // posted its record of call e + 1.
    template <class S, int NV>
    __device__ __forceinline__ int sum(typename S::T (&v)[NV]) {
        static_assert(NV == 1 || NV == 2, "one half-warp per value");
        epoch++;
        const uint32_t lane = threadIdx.x & 31, h = lane / kArLanes;
        if (lane < NV)
            st_record(slot(0, lane, group * kArLanes + member),
                      S::bits(NV == 2 && lane ? v[NV - 1] : v[0]), epoch);
        typename S::T t;
        if (gather<S, NV>(0, group * kArLanes, size, t)) return 1;
        if (groups > 1) {
            if ((lane & (kArLanes - 1)) == 0 && h < NV) {
                st_record(slot(1, h, member * kArLanes + group), S::bits(t), epoch);
                // a row that this group has no member in: its last one posts there too
                if (member + 1 == size && size < rows)
                    st_record(slot(1, h, size * kArLanes + group), S::bits(t), epoch);
            }
            if (gather<S, NV>(1, member * kArLanes, groups, t)) return 1;
        }
        v[0] = S::from(__shfl_sync(0xffffffffu, S::bits(t), 0));
        if (NV == 2) v[NV - 1] = S::from(__shfl_sync(0xffffffffu, S::bits(t), kArLanes));
        return 0;
    }
};

// Sum over a block: every warp's butterfly into sh[value * 32 + warp]
// (block_sum_begin, before a __syncthreads), then warp 0 adds the warps'
// sums and holds the total in every lane (block_sum_end).
template <class S, int NV>
__device__ __forceinline__ void block_sum_begin(typename S::T (&v)[NV], uint64_t* sh) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] = S::xor_add(v[k], o);
        if (lane == 0) sh[k * 32 + warp] = S::bits(S::finish(v[k]));
    }
}

template <class S, int NV>
__device__ __forceinline__ void block_sum_end(typename S::T (&v)[NV], const uint64_t* sh,
                                              uint32_t n_warps) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = lane < n_warps ? S::from(sh[k * 32 + lane]) : S::zero();
    if (n_warps > 1) {
        int top = 1;  // the smallest power of two >= n_warps
        while (top < (int)n_warps) top <<= 1;
        for (int o = top >> 1; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < NV; k++) v[k] = S::xor_add(v[k], o);
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] = S::finish(v[k]);
    }
    // lanes past the butterfly's width hold partial sums: take lane 0's
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = S::from(__shfl_sync(0xffffffffu, S::bits(v[k]), 0));
}

// ---------------------------------------------------------------- ExactSum
// words of one site: [2 epochs][2 values * kSumWords], each epoch a 128-byte
// line of its own; zero at launch
constexpr size_t kExactBytes = 2 * 128;
// The first poll of a sum, sent right behind the block's own adds, met none of
// a later block's, and the sum was seen a second way to L2 and back (700
// cycles) after it.  A block now waits before it by what it was ahead of the
// last block: kLeadUp cycles more after a poll that came too early, kLeadDown
// less after one that served.  Fixed waits were best at 200 cycles on 17 blocks
// and at 300 to 600 on 152, growing with the slices of a block; this follows
// them, for each sum and block.  Milliseconds without, with 32/8, 64/8, 64/4
// and 128/8: 64 x 32 mixed 1.95, 1.83, 1.83, 1.85, 1.91; 127 x 64 FP64 5.29,
// 5.08, 5.02, 4.98, 5.00; 512 x 256 mixed 38.8, 38.6, 38.2, 38.2, 38.4; the
// gradient at 255 x 128 10.65, 10.17, 9.95, 9.89, 10.10.  Two to four polls in
// flight were slower (5 to 30 %), and so was a second line for every other
// block's adds (0 to 5 %).
constexpr unsigned kLeadUp = 64, kLeadDown = 4, kLeadMost = 1000;

// A warp's limbs into sh[warp * 16 + value * kSumWords + limb], before a
// __syncthreads.
constexpr int kSumShared = 32 * 16;  // ints of sh
template <int NV, class V, class W>
__device__ __forceinline__ void exact_begin(const V (&v)[NV], const W (&window)[NV], int* sh) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        int l[kSumWords];
        limbs_of(v[k], window[k], l);
#pragma unroll
        for (int j = 0; j < kSumWords; j++) {
            const int t = __reduce_add_sync(0xffffffffu, l[j]);
            if (lane == 0) sh[warp * 16 + k * kSumWords + j] = t;
        }
    }
}

// Named barriers of the whole block (0 is __syncthreads).
__device__ __forceinline__ void bar_arrive(int id) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(blockDim.x) : "memory");
}
__device__ __forceinline__ void bar_sync(int id) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(blockDim.x) : "memory");
}

// One place in a kernel where sums are taken (in shared memory: only warp 0
// uses it).
struct ExactSum {
    unsigned long long* words;
    unsigned long long last[2][2 * kSumWords];  // the words at the end of the last sums
    unsigned half;
    unsigned lead;  // cycles between the block's adds and its first poll

    __device__ __forceinline__ void init(void* area) {  // by one thread
        words = (unsigned long long*)area;
        for (int k = 0; k < 4 * kSumWords; k++) last[k / (2 * kSumWords)][k % (2 * kSumWords)] = 0;
        half = lead = 0;
    }
    // The block's limbs are in sh; the sums of NV (1 or 2) values over the
    // grid's G <= 255 blocks, value 0 in the even lanes and value 1 in the odd
    // ones (one value: in every lane), as an integer x of 61 bits and an
    // exponent e: x 2^e (least: as in read_limbs).  kFence: the sum is also a barrier for the block's
    // plain loads and stores (release before it, acquire after it).  out() is
    // called when the block's part is on its way.  Returns 0, 1 (outside the
    // window: sum again by records) or 2 (give up).  Called by one whole warp.
    template <int NV, bool kFence, class Out>
    __device__ __forceinline__ int sum(const int* sh, uint32_t n_warps, uint32_t G, int* status,
                                       const int (&window)[NV], int least, long long& x, int& e,
                                       Out out) {
        const uint32_t lane = threadIdx.x & 31;
        constexpr uint32_t kW = NV * kSumWords;
        // lanes 0-15 add the even warps' words, lanes 16-31 the odd ones'
        const uint32_t word = lane & 15;
        int mine = 0;
        if (word < kW)
#pragma unroll 4
            for (uint32_t w = lane >> 4; w < n_warps; w += 2) mine += sh[w * 16 + word];
        mine += __shfl_down_sync(0xffffffffu, mine, 16);
        const unsigned h = half;
        unsigned long long* const p = words + 16 * h + lane;
        unsigned long long d = 0;
        const unsigned long long before = lane < kW ? last[h][lane] : 0;
        if (kFence) __threadfence();
        if (lane < kW) {
            const unsigned long long add = (1ull << 56) + (unsigned long long)(mine + (1ll << 32));
            asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(add) : "memory");
        }
        out();
        // no gain behind a fence (1M dof: 212.1 ms with and without)
        unsigned wait = kFence ? 0 : lead;
        for (const unsigned c0 = (unsigned)clock(); (unsigned)clock() - c0 < wait;) {}
        PollLimit lim;
        for (bool first = true;; first = false) {
            bool ok = true;
            if (lane < kW) {
                if (kFence)  // not a fence behind the loop: it would wait for stores too
                    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(d) : "l"(p) : "memory");
                else
                    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(d) : "l"(p) : "memory");
                ok = ((d - before) >> 56) == G;
            }
            if (__all_sync(0xffffffffu, ok)) {
                wait = first ? wait - min(wait, kLeadDown) : min(wait + kLeadUp, kLeadMost);
                break;
            }
            if (__any_sync(0xffffffffu, lim.expired(status))) return 2;
        }
        const long long t = (long long)((d - before) & ((1ull << 56) - 1)) - ((long long)G << 32);
        if (lane < kW) last[h][lane] = d;
        if (lane == 0) {
            half = h ^ 1;
            lead = wait;
        }
        // even lanes put value 0 together, odd ones value 1
        const uint32_t k = NV == 2 ? lane & 1 : 0;
        long long l[kSumWords];
#pragma unroll
        for (int j = 0; j < kSumWords; j++) l[j] = __shfl_sync(0xffffffffu, t, k * kSumWords + j);
        const bool bad = read_limbs(l, NV == 2 && k ? window[NV - 1] : window[0], least, x, e);
        return __any_sync(0xffffffffu, bad);
    }
    template <int NV>
    __device__ __forceinline__ int sum(const int* sh, uint32_t n_warps, uint32_t G, int* status,
                                       const int (&window)[NV], int least, long long& x, int& e) {
        return sum<NV, false>(sh, n_warps, G, status, window, least, x, e, [] {});
    }
};

}  // namespace nbg
