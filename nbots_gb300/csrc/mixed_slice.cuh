// Slice form of the single-system mixed solver, for systems of at most one
// slice (32 node rows) per warp of the grid: 32 slices per block, one
// 1024-thread block per SM, 4,864 slices (311,000 dofs) on 152 SMs.  Included
// by mixed.cu, after the solver's types.
//
// Such a solve is bound by latency, not by bytes or issue: at 66,306 dof the
// ghost-node form took 13.2 us per iteration, of which its SpMV 5.5 (two half
// slices per warp, one after the other, each waiting twice for L2), the two
// barriers with the partial sums' loads behind them 4.2, the block sums 1.6
// and the reloads of x, r and 1/Aii 1.6.  Here
//   - warp w owns slice w of its block for the whole solve, lane l row l, so
//     x, r, z, A p and 1/Aii stay in registers;
//   - the first entries of every row, as many as fit, stay in shared memory
//     beside p of the rows and ghosts (all of them up to about 20 slices per
//     block; the loads of the others go out before the resident entries are
//     worked on, so that L2 answers meanwhile);
//   - sums over the grid are taken in fixed point in one hop
//     (allreduce.cuh);
//   - owners publish z = r / Aii as epoch-tagged records, so the update of
//     the ghosts' p needs no fence: the warps other than the one that sums
//     poll their block's ghosts meanwhile.
// An iteration has no barrier and no fence.  Microseconds per iteration, the
// ghost-node form (one 1024-thread block per 32 slices) before and this one:
// 4,290 dof 11.5 and 4.1, 66,306 dof 13.2 and 4.6, 91,204 dof (T3) 13.4 and
// 4.9, 263,682 dof 14.0 and 9.0.  At 66,306 dof the rest is the two sums (2.2
// to 2.8 thousand cycles each, of which about 1,500 are the way to L2 and
// back), the SpMV (2.1) and the two divisions (0.9).
//
// kGhost = false (a workspace without the ghost plan, or ghosts that do not
// fit): p is gathered from global memory and exchanged behind a barrier, the
// matrix comes from L2; the same arithmetic in the same order, so both give
// the same bits.

struct SliceArgs {
    uint32_t keep;  // entries of each row in shared memory (batched: as many as fit)
    uint32_t dyn;   // bytes of dynamic shared memory
    // the sums' records (kArBytes) and words (2 kExactBytes), zero at launch
    // (batched: the group's)
    unsigned char* ar;
};

// The resident entries of one row, those of the k-th column at [k * 32]
// (kDecoded: the remainders' scales ready for use in place of their counts,
// 34 instead of 30 B per entry).
struct SliceMatrix {
    const float4* hi;
    const float4* sc;
    const uint2* lo;
    const uint32_t* ext;
    const uint16_t* col;
};
__host__ __device__ constexpr bool slice_decoded(int threads) { return threads <= 512; }
__host__ __device__ constexpr size_t slice_entry_bytes(int threads) {
    return slice_decoded(threads) ? 34 : 30;
}

__device__ __forceinline__ void slice_entry(FFAcc2& acc, float4 m, float4 sc, float4 p) {
    acc.fma2s(make_float2(m.x, m.y), make_float2(sc.x, sc.y), p.x, p.z);
    acc.fma2s(make_float2(m.z, m.w), make_float2(sc.z, sc.w), p.y, p.w);
}

// One row of w = A p, all entries in one lane: n_res resident ones, then
// those at e0, e0 + 32, ... < e1 of the layout.
template <bool kGhost, bool kDecoded, int kUnrollRes, int kBatch>
__device__ __forceinline__ FF2 slice_row(const MixArgs& a, const GhostArgs& gh,
                                         const SliceMatrix& sm, uint32_t n_res, const float4* P,
                                         uint32_t e0, uint32_t e1, uint64_t pol) {
    const float4* __restrict__ bh = reinterpret_cast<const float4*>(a.A.b32);
    const uint2* __restrict__ bl = reinterpret_cast<const uint2*>(a.A.blo);
    const uint32_t* __restrict__ bx = reinterpret_cast<const uint32_t*>(a.A.bxt);
    FFAcc2 acc{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    bool first = true;
    do {
        uint32_t c[kBatch], ext[kBatch];
        float4 m[kBatch];
        uint2 lo[kBatch];
#pragma unroll
        for (int j = 0; j < kBatch; j++) {
            const uint32_t e = e0 + 32 * j;
            if (e < e1) {
                c[j] = kGhost ? ld_hint(gh.lcol + e, pol) : ld_hint(a.A.bcol + e, pol);
                m[j] = ld_hint(bh + e, pol);
                lo[j] = ld_hint(bl + e, pol);
                ext[j] = ld_hint(bx + e, pol);
            }
        }
        if (kGhost && first) {
#pragma unroll(kUnrollRes)
            for (uint32_t k = 0; k < n_res; k++)
                slice_entry(acc, sm.hi[k * 32],
                            kDecoded ? sm.sc[k * 32]
                                     : rem23_scale4(sm.lo[k * 32], sm.ext[k * 32]),
                            P[sm.col[k * 32]]);
            first = false;
        }
#pragma unroll
        for (int j = 0; j < kBatch; j++)
            if (e0 + 32 * j < e1)
                slice_entry(acc, m[j], rem23_scale4(lo[j], ext[j]), kGhost ? P[c[j]] : a.p[c[j]]);
        e0 += 32 * kBatch;
    } while (e0 < e1);
    const FF y0 = FFAcc{acc.s.x, acc.c.x}.result(), y1 = FFAcc{acc.s.y, acc.c.y}.result();
    return {make_float2(y0.hi, y1.hi), make_float2(y0.lo, y1.lo)};
}

// z of a node row as two records, one per dof, in an array each: a warp's
// records then fill whole sectors
__device__ __forceinline__ void publish_z(unsigned char* zx, unsigned char* zy, uint32_t i,
                                          const FF2& z, uint64_t epoch) {
    st_record(zx + (size_t)i * 16, ff_bits(z.hi.x, z.lo.x), epoch);
    st_record(zy + (size_t)i * 16, ff_bits(z.hi.y, z.lo.y), epoch);
}

// kThreads: the largest block; 512 threads leave 128 registers each.
// kBatch: one of several systems in the launch.
template <bool kGhost, bool kBatch, int kThreads>
__device__ __forceinline__ void slice_solve(const MixArgs& a, const Group& g, const GhostArgs& gh,
                                            const SliceArgs& sl, unsigned char* smem) {
    __shared__ double red[3 * 32];
    __shared__ int s_sum1[kSumShared], s_sum2[kSumShared];
    __shared__ uint64_t s_ff[2 * 32];
    __shared__ float s_alpha[2], s_beta[2];
    __shared__ float s_scale[3];  // windows of p.w, r.z, |r|^2
    __shared__ int s_flag;  // 0 iterate, 1 reliable update, 2 stop
    __shared__ int s_fail;   // a wait for ghosts or records ran out
    __shared__ int s_again;  // the fixed-point sum's status: 1 sum by records, 2 give up
    __shared__ MixScalars sc;  // thread 0 only, but for may_end()
    const unsigned G = kBatch ? g.g_size : gridDim.x;
    const uint32_t rank = kBatch ? blockIdx.x - g.g_base : blockIdx.x;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t bd = blockDim.x, nw = bd >> 5;
    uint32_t s0, s1;
    if (kBatch) group_slice_range(g.s_begin, g.s_end, rank, G, s0, s1);
    else slice_range(a.A.n_slices, s0, s1);
    const uint32_t Nn = a.A.Nn, nslot = (s1 - s0) * 32;
    const uint32_t s = s0 + warp, i = s * 32 + lane, li = warp * 32 + lane;
    const bool live = warp < s1 - s0 && i < Nn;
    const uint32_t ng = kGhost ? gh.count[blockIdx.x] : 0;
    const uint32_t pcap = kBatch ? nslot + ng : gh.pcap, gcap = kBatch ? ng : gh.gcap;
    // shared memory: p of rows and ghosts, z of the ghosts, ghost ids, matrix
    float4* const P = reinterpret_cast<float4*>(smem);
    float4* const ZG = P + pcap;
    uint32_t* const GID = reinterpret_cast<uint32_t*>(ZG + gcap);
    float4* const mat = reinterpret_cast<float4*>(GID + ((gcap + 3) & ~3u));
    const uint32_t keep =
        kBatch && kGhost ? (uint32_t)((sl.dyn - ((unsigned char*)mat - smem)) /
                                      (slice_entry_bytes(kThreads) * bd))
                         : sl.keep;
    const uint32_t cap = nw * keep * 32, m0 = warp * keep * 32 + lane;
    constexpr bool kDecoded = slice_decoded(kThreads);
    uint32_t* const mat2 = reinterpret_cast<uint32_t*>(mat + cap);
    const SliceMatrix sm = {mat + m0, mat + cap + m0, reinterpret_cast<const uint2*>(mat2) + m0,
                            mat2 + 2 * cap + m0,
                            reinterpret_cast<const uint16_t*>(mat2) + (kDecoded ? 8 : 6) * cap + m0};
    // z records of every node row, over the workspace's r and A p rows
    unsigned char* const zx = reinterpret_cast<unsigned char*>(a.r4);
    unsigned char* const zy = zx + (size_t)Nn * 16;
    double* const part0 = g.part;
    double* const part2 = g.part + 3 * g.pstride;
    double2* const u = reinterpret_cast<double2*>(a.u);
    const double2* __restrict__ b = reinterpret_cast<const double2*>(a.b);
    auto area = [&]() { return kBatch ? g.sums - kArBytes : sl.ar; };
    unsigned bar_target = 0;
    auto sync = [&]() { return grid_barrier_count(g.bar, G, bar_target, g.status); };
    __shared__ ExactSum sum1, sum2;  // p.w; r.z and |r|^2
    __shared__ uint64_t s_epoch;     // of the sums by records
    // sums of v by records, by warp 0; the totals in v
    auto by_records = [&](auto& v) {
        constexpr int kNV = sizeof(v) / sizeof(FF);
        AllReduce ar;
        ar.init(area(), g.status, G, rank);
        ar.epoch = s_epoch;
        block_sum_end<SumFF, kNV>(v, s_ff, nw);
        const int fail = ar.sum<SumFF, kNV>(v);
        if (lane == 0) {
            s_epoch = ar.epoch;
            s_fail = fail;
        }
    };
    uint64_t zepoch = 1;
    const uint64_t pol = l2_policy(kept_at(warp, a.keep));

    // the resident entries of this warp's slice, then the others [e0, e1);
    // rows past Nn hold no entries
    uint32_t e0 = 0, e1 = 0, n_res = 0;
    if (live) {
        const uint32_t k0 = a.A.slice_off[s], k1 = a.A.slice_off[s + 1];
        n_res = kGhost ? min(k1 - k0, keep) : 0;
        for (uint32_t k = 0; k < n_res; k++) {
            const uint32_t e = (k0 + k) * 32 + lane;
            const_cast<float4*>(sm.hi)[k * 32] = reinterpret_cast<const float4*>(a.A.b32)[e];
            const uint2 lo = reinterpret_cast<const uint2*>(a.A.blo)[e];
            const uint32_t ext = reinterpret_cast<const uint32_t*>(a.A.bxt)[e];
            if (kDecoded) {
                const_cast<float4*>(sm.sc)[k * 32] = rem23_scale4(lo, ext);
            } else {
                const_cast<uint2*>(sm.lo)[k * 32] = lo;
                const_cast<uint32_t*>(sm.ext)[k * 32] = ext;
            }
            const_cast<uint16_t*>(sm.col)[k * 32] = gh.lcol[e];
        }
        e0 = (k0 + n_res) * 32 + lane;
        e1 = k1 * 32 + lane;
    }

    // p of the row: in P with ghosts, else in registers
    const float2 zero2 = make_float2(0.f, 0.f);
    FF2 x{zero2, zero2}, r{zero2, zero2}, w{zero2, zero2}, p{zero2, zero2};
    // x of the row: in registers where there are enough, else in global
    // memory (it is read and written off the critical path)
    constexpr bool kXGlobal = kThreads > 512;
    const float2 di = live ? reinterpret_cast<const float2*>(a.A.dinv32)[i] : zero2;

    auto as4 = [](const FF2& v) { return make_float4(v.hi.x, v.hi.y, v.lo.x, v.lo.y); };
    auto from4 = [](float4 v) -> FF2 {
        return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
    };
    // r = b - A u for this lane's row (row_residual) as float-float, z = r / Aii;
    // |r|^2 in FP64, r.z; |b|^2, r.p
    auto true_residual = [&](bool check, double& rr, FFAcc& rz, double* bb, double* rp) {
        if (!live) return;
        const double2 ri = row_residual(a, s, lane, check, rr, bb);
        if (rp) *rp = dot_with(ri.x, ri.y, kGhost ? P[li] : as4(p), *rp);
        const FF f0 = ff_from_double(ri.x), f1 = ff_from_double(ri.y);
        r = {make_float2(f0.hi, f1.hi), make_float2(f0.lo, f1.lo)};
        const FF2 z = ff2_mulf(r, di);
        rz.fma2(r.hi.x, r.lo.x, z.hi.x, z.lo.x);
        rz.fma2(r.hi.y, r.lo.y, z.hi.y, z.lo.y);
    };
    // z of this block's ghosts into ZG, by the threads from `first` on (whole
    // warps): waits for the records of epoch zepoch
    auto poll_ghosts = [&](uint32_t first) {
        PollLimit lim;
        for (uint32_t j = tid - first; j < ng; j += bd - first) {
            const size_t at = (size_t)GID[j] * 16;
            uint64_t v0, v1, ea, eb;
            for (;;) {
                ld_record(zx + at, v0, ea);
                ld_record(zy + at, v1, eb);
                if (ea == zepoch && eb == zepoch) break;
                if (lim.expired(g.status)) {
                    s_fail = 1;
                    return;
                }
            }
            const FF f0 = bits_ff(v0), f1 = bits_ff(v1);
            ZG[j] = make_float4(f0.hi, f1.hi, f0.lo, f1.lo);
        }
    };

    if (tid == 0) {
        sc.clear();
        s_fail = 0;
        s_epoch = 0;
        sum1.init(area() + kArBytes);
        sum2.init(area() + kArBytes + kExactBytes);
    }
    if (kGhost) {
        for (uint32_t j = tid; j < ng; j += bd) GID[j] = gh.ids[(size_t)blockIdx.x * kGhostMax + j];
        // no record of an earlier solve may look current
        if (live) {
            st_record(zx + (size_t)i * 16, 0, 0);
            st_record(zy + (size_t)i * 16, 0, 0);
        }
    }
    {   // init: x = 0, r = b - A u (FP64), p = z
        double rrl = 0.0, bbl = 0.0;
        FFAcc rzk{0.f, 0.f};
        true_residual(true, rrl, rzk, &bbl, nullptr);
        p = ff2_mulf(r, di);
        if (kXGlobal && live) a.x4[i] = as4(x);
        if (kGhost) {
            if (warp < s1 - s0) P[li] = as4(p);
        } else if (live) {
            a.p[i] = as4(p);
        }
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
            s_scale[0] = 0.f;
            s_scale[1] = window_scale(sc.rz.hi);
            s_scale[2] = window_scale((float)sc.rr64);
        }
        if (kGhost) {  // ghosts start as their owners' p = z
            if (live) publish_z(zx, zy, i, ff2_mulf(r, di), zepoch);
            poll_ghosts(0);
            for (uint32_t j = tid; j < ng; j += bd) P[nslot + j] = ZG[j];
            zepoch++;
        }
        __syncthreads();
        if (s_fail) goto done;
    }
    while (s_flag != 2) {
        {   // L1: w = A p, p.w
            FFAcc pw{0.f, 0.f};
            if (live) {
                w = slice_row<kGhost, kDecoded, kThreads <= 512 ? 9 : 4, kThreads <= 512 ? 3 : 1>(
                    a, gh, sm, n_res, P, e0, e1, pol);
                if (kGhost) p = from4(P[li]);
                pw.fma2(p.hi.x, p.lo.x, w.hi.x, w.lo.x);
                pw.fma2(p.hi.y, p.lo.y, w.hi.y, w.lo.y);
            }
            FF v[1] = {{pw.s, pw.c}};
            const float scale[1] = {s_scale[0]};
            exact_begin<1>(v, scale, s_sum1);
            __syncthreads();
            auto finish = [&](FF pws) {
                s_scale[0] = window_scale(pws.hi);
                const FF al = sc.alpha(pws);
                s_alpha[0] = al.hi;
                s_alpha[1] = al.lo;
            };
            if (warp == 0) {
                long long xs;
                int es;
                const int st =
                    sum1.sum<1>(s_sum1, nw, G, g.status, {window_exponent(scale[0])}, kLeastFF, xs, es);
                if (tid == 0) {
                    s_again = st;
                    if (!st) finish(exact_ff(xs, es));
                }
            }
            __syncthreads();
            if (s_again) {
                if (s_again == 2) goto done;
                block_sum_begin<SumFF, 1>(v, s_ff);
                __syncthreads();
                if (warp == 0) {
                    by_records(v);
                    if (tid == 0) finish(v[0]);
                }
                __syncthreads();
                if (s_fail) goto done;
            }
        }
        {   // L2: x += alpha p, r -= alpha w, z = r / Aii, published
            const FF2 alpha = ff2_bcast(FF{s_alpha[0], s_alpha[1]});
            FFAcc rzk{0.f, 0.f}, rrk{0.f, 0.f};
            if (live) {
                const FF2 aw = ff2_mul(alpha, w);
                r = ff2_add(r, {f2neg(aw.hi), f2neg(aw.lo)});
                const FF2 z = ff2_mulf(r, di);
                if (kGhost) publish_z(zx, zy, i, z, zepoch);
                rzk.fma2(r.hi.x, r.lo.x, z.hi.x, z.lo.x);
                rzk.fma2(r.hi.y, r.lo.y, z.hi.y, z.lo.y);
                rrk.fma2(r.hi.x, r.lo.x, r.hi.x, r.lo.x);
                rrk.fma2(r.hi.y, r.lo.y, r.hi.y, r.lo.y);
            }
            FF v[2] = {{rzk.s, rzk.c}, {rrk.s, rrk.c}};
            const float scale[2] = {s_scale[1], s_scale[2]};
            exact_begin<2>(v, scale, s_sum2);
            __syncthreads();
            auto finish = [&](FF rzs, FF rrs) {
                s_scale[1] = window_scale(rzs.hi);
                s_scale[2] = window_scale(rrs.hi);
                FF be;
                s_flag = sc.step(rzs, rrs, a.max_iter, be);
                if (!s_flag) {
                    s_beta[0] = be.hi;
                    s_beta[1] = be.lo;
                }
            };
            if (warp == 0) {
                long long xs;
                int es;
                const int st = sum2.sum<2>(
                    s_sum2, nw, G, g.status,
                    {window_exponent(scale[0]), window_exponent(scale[1])}, kLeastFF, xs, es);
                const FF t = exact_ff(xs, es);  // r.z in lane 0, |r|^2 in lane 1
                const FF rrs = {__shfl_sync(0xffffffffu, t.hi, 1), __shfl_sync(0xffffffffu, t.lo, 1)};
                if (tid == 0) {
                    s_again = st;
                    if (!st) finish(t, rrs);
                }
            }
            // off the critical path: x, and the ghosts' z
            if (live) {
                if (kGhost) p = from4(P[li]);
                if (kXGlobal) x = from4(a.x4[i]);
                x = ff2_add(x, ff2_mul(alpha, p));
                if (kXGlobal) a.x4[i] = as4(x);
            }
            if (kGhost) {
                if (nw == 1) poll_ghosts(0);
                else if (warp) poll_ghosts(32);
                zepoch++;
            }
            __syncthreads();
            if (s_fail || s_again == 2) goto done;
            if (s_again) {
                block_sum_begin<SumFF, 2>(v, s_ff);
                __syncthreads();
                if (warp == 0) {
                    by_records(v);
                    if (tid == 0) finish(v[0], v[1]);
                }
                __syncthreads();
                if (s_fail) goto done;
            }
        }
        if (s_flag) {
            // reliable update: u += x in FP64, then r = b - A u in FP64
            const bool check = sc.may_end(a.max_iter);
            if (live) {
                if (kXGlobal) x = from4(a.x4[i]);
                double2 ui = u[i];
                ui.x += (double)x.hi.x + (double)x.lo.x;
                ui.y += (double)x.hi.y + (double)x.lo.y;
                u[i] = ui;
                x = {zero2, zero2};
                if (kXGlobal) a.x4[i] = as4(x);
            }
            if (sync()) goto done;
            double rrl = 0.0, rpl = 0.0;
            FFAcc rzk{0.f, 0.f};
            true_residual(check, rrl, rzk, nullptr, &rpl);
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
            if (kGhost) {
                if (live) publish_z(zx, zy, i, ff2_mulf(r, di), zepoch);
                poll_ghosts(0);
                zepoch++;
                __syncthreads();
                if (s_fail) goto done;
            }
        }
        {   // L3: p = z + beta p for the row, and for the block's ghosts
            const FF2 beta = ff2_bcast(FF{s_beta[0], s_beta[1]});
            if (live) {
                if (kGhost) p = from4(P[li]);
                p = ff2_add(ff2_mulf(r, di), ff2_mul(beta, p));
                if (kGhost) P[li] = as4(p);
                else a.p[i] = as4(p);
            }
            for (uint32_t j = tid; j < ng; j += bd)
                P[nslot + j] = as4(ff2_add(from4(ZG[j]), ff2_mul(beta, from4(P[nslot + j]))));
            if (kGhost) __syncthreads();
        }
        if (!kGhost && sync()) goto done;
    }
    {   // b.u in FP64 (the compliance F^T u when b is the load vector)
        double bu = 0.0;
        if (live) {
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

template <bool kGhost, int kThreads>
__global__ void __launch_bounds__(kThreads, 1)
    k_cg_mixed_slice(MixArgs a, Group g, GhostArgs gh, SliceArgs sl) {
    extern __shared__ __align__(16) unsigned char smem[];
    slice_solve<kGhost, false, kThreads>(a, g, gh, sl, smem);
}

// Batched: block b works for system groups[block_of[b]], with its ghosts where
// the plan found room for them in all of the system's blocks.
constexpr int kNoPlan = 16;  // ints from a system's status to its plan's failure flag
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 1)
    k_cg_mixed_slices(MixArgs a, const Group* __restrict__ groups,
                      const uint32_t* __restrict__ block_of, GhostArgs gh, SliceArgs sl) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Group sg;
    if (threadIdx.x == 0) sg = groups[block_of[blockIdx.x]];
    __syncthreads();
    if (sg.status[kNoPlan] == 0) slice_solve<true, true, kThreads>(a, sg, gh, sl, smem);
    else slice_solve<false, true, kThreads>(a, sg, gh, sl, smem);
}
