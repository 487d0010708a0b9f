// The ghost plan of a persistent solver on the 2x2-block SELL layout: for a
// partition of the slices over G blocks, each block's ghosts (the node rows of
// other blocks that its rows couple to) and the layout's columns renumbered
// within the block in 16 bits: own row slots first, then the ghosts in
// ascending node order.
#pragma once

#include <algorithm>
#include <vector>

#include "persist.cuh"

namespace {

using namespace nbg;

constexpr uint32_t kGhostMax = 16384;   // ghosts per block
constexpr uint32_t kGhostKeys = 32768;  // outside-column references per block the plan sorts

struct GhostArgs {
    const uint16_t* lcol;   // local column of every layout entry
    const uint32_t* ids;    // kGhostMax ghost node ids per block, ascending
    const uint32_t* count;  // ghosts per block, then the block's widest slice
    uint32_t scap;          // own row slots of the largest block
    uint32_t pcap;          // row slots + ghosts, largest over the blocks
    uint32_t gcap;          // ghosts, largest over the blocks
};

// One block per group of the solver's partition: its ghosts (the columns of
// its live rows outside its row slots, sorted and made unique in shared
// memory) and the local column of each of its entries.  *fail is set when a
// block has more outside references than kGhostKeys, more ghosts than
// kGhostMax, or more than 65535 local columns; the solver then keeps the
// global-gather form.  A batched launch: block b has the slices from
// pb.range[b].x to .y, belongs to system pb.system_of[b], whose own *fail is
// pb.fail_stride ints further on for each, and fails too when its rows and
// ghosts take more than pb.limit bytes at 16 per row and 36 per ghost.
struct PlanBatch {
    const uint2* range;
    const uint32_t* system_of;
    size_t limit;
    uint32_t fail_stride;
};
__global__ void __launch_bounds__(1024, 1) k_ghost_plan(nbg_bsr_t A, uint16_t* lcol,
                                                      uint32_t* ids, uint32_t* count,
                                                      int* fail, PlanBatch pb) {
    extern __shared__ __align__(16) uint32_t keys[];  // kGhostKeys
    __shared__ uint32_t s_n;
    __shared__ uint32_t s_scan[32];
    __shared__ uint32_t s_wide;  // widest slice
    const uint32_t tid = threadIdx.x, bd = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nw = bd >> 5;
    uint32_t s0, s1;
    slice_range(A.n_slices, s0, s1);
    if (pb.range) {
        s0 = pb.range[blockIdx.x].x;
        s1 = pb.range[blockIdx.x].y;
        fail += pb.system_of[blockIdx.x] * pb.fail_stride;
    }
    const uint32_t n0 = s0 * 32, nslot = (s1 - s0) * 32;
    if (tid == 0) s_n = s_wide = 0;
    __syncthreads();
    for (uint32_t s = s0 + warp; s < s1; s += nw) {
        const uint32_t i = s * 32 + lane;
        if (lane == 0) atomicMax(&s_wide, A.slice_off[s + 1] - A.slice_off[s]);
        if (i >= A.Nn) continue;
        for (uint32_t k = A.slice_off[s]; k < A.slice_off[s + 1]; k++) {
            const uint32_t c = A.bcol[(size_t)k * 32 + lane];
            if (c - n0 >= nslot) {
                const uint32_t pos = atomicAdd(&s_n, 1u);
                if (pos < kGhostKeys) keys[pos] = c;
            }
        }
    }
    __syncthreads();
    const uint32_t n = s_n;
    if (n > kGhostKeys) {  // the same n in every thread
        if (tid == 0) atomicExch(fail, 1);
        return;
    }
    uint32_t P2 = 1;
    while (P2 < n) P2 <<= 1;
    for (uint32_t j = n + tid; j < P2; j += bd) keys[j] = 0xffffffffu;
    __syncthreads();
    // bitonic sort of keys[0, P2)
    for (uint32_t size = 2; size <= P2; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint32_t t = tid; t < P2 / 2; t += bd) {
                const uint32_t lo = 2 * stride * (t / stride) + (t % stride), hi = lo + stride;
                const uint32_t x = keys[lo], y = keys[hi];
                if ((x > y) == ((lo & size) == 0)) {
                    keys[lo] = y;
                    keys[hi] = x;
                }
            }
            __syncthreads();
        }
    // unique: each thread counts the first occurrences in its chunk, an
    // exclusive block scan places them
    const uint32_t chunk = (n + bd - 1) / bd;
    const uint32_t j0 = min(tid * chunk, n), j1 = min(j0 + chunk, n);
    uint32_t cnt = 0;
    for (uint32_t j = j0; j < j1; j++) cnt += (j == 0 || keys[j] != keys[j - 1]);
    uint32_t v = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= (uint32_t)o) v += t;
    }
    if (lane == 31) s_scan[warp] = v;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < nw ? s_scan[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= (uint32_t)o) w += t;
        }
        s_scan[lane] = w;
    }
    __syncthreads();
    const uint32_t u = s_scan[nw - 1];
    if (u > kGhostMax || nslot + u > 65535u ||
        (pb.range && 16 * (size_t)nslot + 36 * (size_t)u + 16 > pb.limit)) {  // the same u in every thread
        if (tid == 0) atomicExch(fail, 1);
        return;
    }
    uint32_t* const my = ids + (size_t)blockIdx.x * kGhostMax;
    uint32_t pos = v - cnt + (warp ? s_scan[warp - 1] : 0);
    for (uint32_t j = j0; j < j1; j++)
        if (j == 0 || keys[j] != keys[j - 1]) my[pos++] = keys[j];
    __syncthreads();
    for (uint32_t j = tid; j < u; j += bd) keys[j] = my[j];
    if (tid == 0) {
        count[blockIdx.x] = u;
        count[gridDim.x + blockIdx.x] = s_wide;
    }
    __syncthreads();
    for (uint32_t s = s0 + warp; s < s1; s += nw) {
        const uint32_t i = s * 32 + lane;
        for (uint32_t k = A.slice_off[s]; k < A.slice_off[s + 1]; k++) {
            const size_t e = (size_t)k * 32 + lane;
            uint32_t lc = i - n0;  // rows past Nn (never read): their own slot
            if (i < A.Nn) {
                const uint32_t c = A.bcol[e];
                if (c - n0 < nslot) {
                    lc = c - n0;
                } else {
                    uint32_t lo = 0, hi = u;  // first ghost >= c (it is there)
                    while (lo < hi) {
                        const uint32_t mid = (lo + hi) >> 1;
                        if (keys[mid] < c) lo = mid + 1; else hi = mid;
                    }
                    lc = nslot + lo;
                }
            }
            lcol[e] = (uint16_t)lc;
        }
    }
}

// Workspace of the ghost plan for layout A on this device: local columns,
// ghost lists of up to one block per SM, counts, the failure flag.
size_t ghost_plan_bytes(const nbg_bsr_t& A) {
    int dev = 0, nsm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    const size_t G = (size_t)nsm;
    return align256(2 * (size_t)A.n_entries) + align256(G * kGhostMax * 4) + align256(G * 8) + 256;
}

// Where the plan of a G-block partition stands in its workspace region.
void ghost_regions(const nbg_bsr_t& A, unsigned G, char* plan, uint16_t** lcol, uint32_t** ids,
                   uint32_t** count) {
    *lcol = (uint16_t*)plan;
    *ids = (uint32_t*)(plan + align256(2 * (size_t)A.n_entries));
    *count = *ids + (size_t)G * kGhostMax;
}

// The ghost plan for a G-block partition of A and the sizes that its launch
// needs: returns 1 and fills gh and *widest (entries of the longest slice
// row), or 0 (the caller keeps a global-gather form).  plan: the
// workspace region of ghost_plan_bytes(A).
int ghost_plan(const nbg_bsr_t& A, unsigned G, char* plan, cudaStream_t s, GhostArgs* gh,
               uint32_t* widest) {
    uint16_t* lcol;
    uint32_t *ids, *count;
    ghost_regions(A, G, plan, &lcol, &ids, &count);
    int* fail = (int*)((char*)count + align256((size_t)G * 8));
    int dev = 0, nsm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    if (G > (unsigned)nsm) return 0;  // beyond the plan's space
    if (cudaFuncSetAttribute((const void*)k_ghost_plan,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(kGhostKeys * 4)) != cudaSuccess)
        return 0;
    if (cudaMemsetAsync(fail, 0, sizeof(int), s) != cudaSuccess) return 0;
    k_ghost_plan<<<G, 1024, kGhostKeys * 4, s>>>(A, lcol, ids, count, fail, PlanBatch{});
    if (cudaGetLastError() != cudaSuccess) return 0;
    std::vector<uint32_t> cnt(2 * (size_t)G);
    int hfail = 1;
    if (cudaMemcpyAsync(cnt.data(), count, 8 * (size_t)G, cudaMemcpyDeviceToHost, s) !=
            cudaSuccess ||
        cudaMemcpyAsync(&hfail, fail, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess || hfail)
        return 0;
    uint32_t scap = 0, pcap = 0, gcap = 0, ecap = 0;
    for (unsigned b = 0; b < G; b++) {
        const uint32_t s0 = (uint32_t)(((uint64_t)A.n_slices * b) / G);
        const uint32_t s1 = (uint32_t)(((uint64_t)A.n_slices * (b + 1)) / G);
        scap = std::max(scap, 32 * (s1 - s0));
        pcap = std::max(pcap, 32 * (s1 - s0) + cnt[b]);
        gcap = std::max(gcap, cnt[b]);
        ecap = std::max(ecap, cnt[G + b]);
    }
    gh->lcol = lcol;
    gh->ids = ids;
    gh->count = count;
    gh->scap = scap;
    gh->pcap = pcap;
    gh->gcap = gcap;
    *widest = ecap;
    return 1;
}

// Whether `bytes` of dynamic shared memory let G blocks of `fn` run at once.
bool fits_smem(const void* fn, int threads, size_t bytes, unsigned G) {
    int dev = 0, nsm = 0, occ = 0;
    size_t most = 0;
    return cudaGetDevice(&dev) == cudaSuccess &&
           cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
           allow_smem(fn, &most) == cudaSuccess && bytes <= most &&
           cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, threads, bytes) ==
               cudaSuccess &&
           (uint64_t)occ * (unsigned)nsm >= G;
}

}  // namespace
