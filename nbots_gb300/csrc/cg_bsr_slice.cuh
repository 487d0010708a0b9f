// Slice form of the FP64 block CG, for systems of at most 32 slices (32 node
// rows each) per block of a one-block-per-SM grid: 311,000 dofs on 152 SMs.
// Included by cg_bsr.cu, after the solver's types.
//
// The global form below it spent 17.8 us per iteration on 16,770 dof: 17
// blocks of 16 warps, whose FP64 work shared 17 SMs' pipes (a warp issues one
// FP64 instruction in 65 cycles, 16 warps of an SM one each in 305), three
// grid barriers, and FP64 sums of 16 to 21 dependent adds per block and
// again per grid.  Here
//   - the slices spread over all SMs, and a warp owns its rows for the whole
//     solve, with x, g, A p and 1/Aii in registers.  kDofs = 1: a half slice,
//     lanes l and l + 16 share a node row, take alternate entries of it and
//     own one dof each; kDofs = 2: a slice, lane l owns both dofs of row l;
//   - p of the rows and of the block's ghosts and as many entries of each row
//     as fit stay in shared memory (ghost_plan.cuh);
//   - sums over the grid are taken in fixed point in one hop (allreduce.cuh),
//     off the FP64 pipe;
//   - owners publish q = g / Aii as epoch-tagged records, which the warps
//     that do not sum poll meanwhile; every block then updates its ghosts' p
//     itself, as mixed.cu's ghost-node form does.
// The iteration, its stop rules and the check on the true residual are those
// of the global form.  Microseconds per iteration, the global form and this
// one: 4,290 dof 15.7 and 4.9, 16,770 dof 17.8 and 4.9, 66,306 dof 18.0 and
// 6.9, 263,682 dof 27.2 and 16.1 (there FP64 issue bounds both).

struct BsrSliceArgs {
    GhostArgs gh;
    uint32_t keep;        // entries of each row in shared memory
    unsigned char* qrec;  // q records, 16 B per dof
    void* sums;           // records (kArBytes) and words (2 kExactBytes), zero at launch
};

template <bool JAC, bool LAGGED, int kDofs, int kThreads>
__global__ void __launch_bounds__(kThreads, 1) k_cg_bsr_slice(CgBsrArgs a, BsrSliceArgs sl) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double red[3 * 32];
    __shared__ int s_sum1[kSumShared], s_sum2[kSumShared];
    __shared__ uint64_t s_f64[2 * 32];
    __shared__ double s_coef;   // alpha, then beta
    __shared__ int s_win[3];    // windows of p.w, g.q, g.g
    __shared__ int s_stop;      // 0 iterate, 1 stop, 2 confirm on the true residual first
    __shared__ int s_fail;      // a wait for ghosts or records ran out
    __shared__ int s_again;     // the fixed-point sum's status: 1 sum by records, 2 give up
    __shared__ ExactSum sum1, sum2;
    __shared__ uint64_t s_epoch;
    __shared__ CgBsrScalars sc;  // thread 0 only
    const unsigned G = gridDim.x;
    const uint32_t rank = blockIdx.x;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t bd = blockDim.x, nw = bd >> 5;
    uint32_t s0, s1;
    slice_range(a.A.n_slices, s0, s1);
    const uint32_t Nn = a.A.Nn, nslot = (s1 - s0) * 32;
    // this lane's node row i (row r of slice s0 + ls) and dofs
    const uint32_t ls = kDofs == 2 ? warp : warp >> 1;
    const uint32_t par = kDofs == 2 ? 0 : lane >> 4;
    const uint32_t r = kDofs == 2 ? lane : ((warp & 1) << 4) | (lane & 15);
    const uint32_t i = (s0 + ls) * 32 + r, li = ls * 32 + r;
    const bool live = ls < s1 - s0 && i < Nn;
    const uint32_t ng = sl.gh.count[rank];
    double2* const P = reinterpret_cast<double2*>(smem);  // p of rows and ghosts
    double2* const QG = P + sl.gh.pcap;                   // q of the ghosts
    uint32_t* const GID = reinterpret_cast<uint32_t*>(QG + sl.gh.gcap);
    // resident entries: [slice][k][row], values by rows of the block
    const uint32_t per = sl.keep * 32, cap = (sl.gh.scap / 32) * per;
    double2* const M0 = reinterpret_cast<double2*>(GID + ((sl.gh.gcap + 3) & ~3u));
    double2* const M1 = M0 + cap;
    uint16_t* const MC = reinterpret_cast<uint16_t*>(M1 + cap);
    const uint32_t m0 = ls * per + r;
    const double2* __restrict__ b = reinterpret_cast<const double2*>(a.b);
    double2* const gx = reinterpret_cast<double2*>(a.x);  // read here, written through a.x
    unsigned bar_target = 0;
    auto sync = [&]() { return grid_barrier_count(a.bar, G, bar_target, a.status); };
    uint64_t qepoch = 1;
    double* const part2 = a.part + 3 * kMaxBlocks;

    uint32_t k0 = 0, width = 0, n_res = 0;
    double x[kDofs], g[kDofs], w[kDofs], di[kDofs];
#pragma unroll
    for (int d = 0; d < kDofs; d++) x[d] = g[d] = w[d] = di[d] = 0.0;
    auto dof = [&](double2 v, int d) { return kDofs == 2 ? (d ? v.y : v.x) : (par ? v.y : v.x); };
    if (live) {
        k0 = a.A.slice_off[s0 + ls];
        width = a.A.slice_off[s0 + ls + 1] - k0;
        n_res = min(width, sl.keep);
        const double2* __restrict__ bv = reinterpret_cast<const double2*>(a.A.b64);
        for (uint32_t k = par; k < n_res; k += kDofs == 2 ? 1 : 2) {
            const size_t e = (size_t)(k0 + k) * 32 + r;
            M0[m0 + k * 32] = bv[2 * e];
            M1[m0 + k * 32] = bv[2 * e + 1];
            MC[m0 + k * 32] = sl.gh.lcol[e];
        }
        const double2 xi = gx[i];
        const double2 dv = JAC ? reinterpret_cast<const double2*>(a.A.dinv64)[i]
                               : make_double2(1.0, 1.0);
#pragma unroll
        for (int d = 0; d < kDofs; d++) {
            x[d] = dof(xi, d);
            di[d] = dof(dv, d);
        }
    }
    // A v for this lane's dofs: v in shared memory by local column (kLocal), or
    // global by node.  Every lane of a warp whose rows are live or not calls it.
    auto multiply = [&](auto kLocal, const double2* v, double (&y)[kDofs]) {
        constexpr uint32_t kStep = kDofs == 2 ? 1 : 2;
        const double2* __restrict__ bv = reinterpret_cast<const double2*>(a.A.b64);
        const uint64_t pol = l2_policy(false);
        double y0 = 0.0, y1 = 0.0;
        auto entry = [&](double2 top, double2 bot, double2 p) {
            y0 = fma(top.x, p.x, y0);
            y1 = fma(bot.x, p.x, y1);
            y0 = fma(top.y, p.y, y0);
            y1 = fma(bot.y, p.y, y1);
        };
        uint32_t k = par;
        if (decltype(kLocal)::value) {
#pragma unroll 3
            for (; k < n_res; k += kStep) entry(M0[m0 + k * 32], M1[m0 + k * 32], v[MC[m0 + k * 32]]);
        }
#pragma unroll 2
        for (; k < width; k += kStep) {
            const size_t e = (size_t)(k0 + k) * 32 + r;
            const uint32_t c = decltype(kLocal)::value ? ld_hint(sl.gh.lcol + e, pol)
                                                       : ld_hint(a.A.bcol + e, pol);
            const double2 top = ld_hint(bv + 2 * e, pol), bot = ld_hint(bv + 2 * e + 1, pol);
            entry(top, bot, v[c]);
        }
        if (kDofs == 2) {
            y[0] = y0;
            y[kDofs - 1] = y1;
        } else {  // the lane of dof `par` takes its partner's half of that dof
            const double other = __shfl_xor_sync(0xffffffffu, par ? y0 : y1, 16);
            y[0] = (par ? y1 : y0) + other;
        }
    };
    // g = A x - b from global x, q = g / Aii: sums of g.q, g.g, b.b
    auto true_residual = [&](double (&v)[3]) {
        double ax[kDofs];
        multiply(FalseType{}, gx, ax);
        if (!live) return;
        const double2 bi = b[i];
#pragma unroll
        for (int d = 0; d < kDofs; d++) {
            const double bd_ = dof(bi, d);
            g[d] = ax[d] - bd_;
            v[0] = fma(g[d], g[d] * di[d], v[0]);
            v[1] = fma(g[d], g[d], v[1]);
            v[2] = fma(bd_, bd_, v[2]);
        }
    };
    // this lane's entry of p
    auto own_p = [&](int d) -> double& {
        return reinterpret_cast<double*>(P + li)[kDofs == 2 ? d : par];
    };
    auto publish_q = [&]() {
        if (live)
#pragma unroll
            for (int d = 0; d < kDofs; d++)
                st_record(sl.qrec + ((size_t)(kDofs == 2 ? d : par) * Nn + i) * 16,
                          (uint64_t)__double_as_longlong(g[d] * di[d]), qepoch);
    };
    // q of the ghosts into QG by the threads from `first` (whole warps) on
    auto poll_ghosts = [&](uint32_t first) {
        PollLimit lim;
        for (uint32_t j = tid - first; j < ng; j += bd - first) {
            const unsigned char* q = sl.qrec + (size_t)GID[j] * 16;
            uint64_t v0, v1, ea, eb;
            for (;;) {
                ld_record(q, v0, ea);
                ld_record(q + (size_t)Nn * 16, v1, eb);
                if (ea == qepoch && eb == qepoch) break;
                if (lim.expired(a.status)) {
                    s_fail = 1;
                    return;
                }
            }
            QG[j] = make_double2(__longlong_as_double((long long)v0),
                                 __longlong_as_double((long long)v1));
        }
    };
    // sums of v by records, by warp 0; the totals in v
    auto by_records = [&](auto& v) {
        constexpr int kNV = sizeof(v) / sizeof(double);
        AllReduce ar;
        ar.init(sl.sums, a.status, G, rank);
        ar.epoch = s_epoch;
        block_sum_end<SumF64, kNV>(v, s_f64, nw);
        const int fail = ar.sum<SumF64, kNV>(v);
        if (lane == 0) {
            s_epoch = ar.epoch;
            s_fail = fail;
        }
    };

    if (tid == 0) {
        sc.clear();
        s_fail = 0;
        s_epoch = 0;
        sum1.init((unsigned char*)sl.sums + kArBytes);
        sum2.init((unsigned char*)sl.sums + kArBytes + kExactBytes);
    }
    for (uint32_t j = tid; j < ng; j += bd) GID[j] = sl.gh.ids[(size_t)rank * kGhostMax + j];
    // no record of an earlier solve may look current
    if (live)
#pragma unroll
        for (int d = 0; d < kDofs; d++)
            st_record(sl.qrec + ((size_t)(kDofs == 2 ? d : par) * Nn + i) * 16, 0, 0);
    {   // init: g = A x - b, q = g / Aii, p = -q
        double v[3] = {0.0, 0.0, 0.0};
        true_residual(v);
        if (live)
#pragma unroll
            for (int d = 0; d < kDofs; d++) own_p(d) = -(g[d] * di[d]);
        group_publish<3>(v, red, part2, rank);
    }
    if (sync()) goto done;
    {
        double t[3];
        group_reduce0<3>(part2, G, t);
        if (tid == 0) {
            s_stop = sc.start(t, a);
            s_win[0] = kNoWindow;
            s_win[1] = window_f64(sc.gq);
            s_win[2] = window_f64(sc.gg);
        }
        publish_q();
        poll_ghosts(0);
        for (uint32_t j = tid; j < ng; j += bd) P[nslot + j] = make_double2(-QG[j].x, -QG[j].y);
        qepoch++;
        __syncthreads();
        if (s_fail) goto done;
    }
    while (!s_stop) {
        {   // L1: w = A p, p.w
            multiply(TrueType{}, P, w);
            double v[1] = {0.0};
            if (live)
#pragma unroll
                for (int d = 0; d < kDofs; d++) v[0] = fma(own_p(d), w[d], v[0]);
            const int win[1] = {s_win[0]};
            exact_begin<1>(v, win, s_sum1);
            __syncthreads();
            auto finish = [&](double pw) {
                s_win[0] = window_f64(pw);
                s_coef = sc.gq / pw;
            };
            if (warp == 0) {
                long long xs;
                int es;
                const int st = sum1.sum<1>(s_sum1, nw, G, a.status, win, kLeastF64, xs, es);
                if (tid == 0) {
                    s_again = st;
                    if (!st) finish(exact_f64(xs, es));
                }
            }
            __syncthreads();
            if (s_again) {
                if (s_again == 2) goto done;
                block_sum_begin<SumF64, 1>(v, s_f64);
                __syncthreads();
                if (warp == 0) {
                    by_records(v);
                    if (tid == 0) finish(v[0]);
                }
                __syncthreads();
                if (s_fail) goto done;
            }
        }
        {   // L2: g += alpha w, q = g / Aii, published; x += alpha p
            const double alpha = s_coef;
            double v[2] = {0.0, 0.0};
            if (live) {
#pragma unroll
                for (int d = 0; d < kDofs; d++) {
                    g[d] = fma(alpha, w[d], g[d]);
                    v[0] = fma(g[d], g[d] * di[d], v[0]);
                    v[1] = fma(g[d], g[d], v[1]);
                }
            }
            publish_q();
            const int win[2] = {s_win[1], s_win[2]};
            exact_begin<2>(v, win, s_sum2);
            __syncthreads();
            auto finish = [&](double gq, double gg) {
                s_win[1] = window_f64(gq);
                s_win[2] = window_f64(gg);
                s_coef = sc.step<LAGGED>(gq, gg, a, s_stop);
            };
            if (warp == 0) {
                long long xs;
                int es;
                const int st = sum2.sum<2>(s_sum2, nw, G, a.status, win, kLeastF64, xs, es);
                const double t = exact_f64(xs, es);  // g.q in lane 0, g.g in lane 1
                const double gg = __shfl_sync(0xffffffffu, t, 1);
                if (tid == 0) {
                    s_again = st;
                    if (!st) finish(t, gg);
                }
            }
            // off the critical path: x, and the ghosts' q
            if (live)
#pragma unroll
                for (int d = 0; d < kDofs; d++) x[d] = fma(alpha, own_p(d), x[d]);
            if (nw == 1) poll_ghosts(0);
            else if (warp) poll_ghosts(32);
            qepoch++;
            __syncthreads();
            if (s_fail || s_again == 2) goto done;
            if (s_again) {
                block_sum_begin<SumF64, 2>(v, s_f64);
                __syncthreads();
                if (warp == 0) {
                    by_records(v);
                    if (tid == 0) finish(v[0], v[1]);
                }
                __syncthreads();
                if (s_fail) goto done;
            }
        }
        if (!LAGGED && s_stop == 2) {
            // confirm on the true residual
            if (live)
#pragma unroll
                for (int d = 0; d < kDofs; d++) a.x[2 * (size_t)i + (kDofs == 2 ? d : par)] = x[d];
            if (sync()) goto done;
            double v[3] = {0.0, 0.0, 0.0};
            true_residual(v);
            group_publish<3>(v, red, part2, rank);
            if (sync()) goto done;
            double t[3];
            group_reduce0<3>(part2, G, t);
            if (tid == 0) s_coef = sc.checked(t[0], t[1], a, s_stop);
            __syncthreads();
            if (s_stop) break;
            publish_q();
            poll_ghosts(0);
            qepoch++;
            __syncthreads();
            if (s_fail) goto done;
        }
        if (s_stop) break;
        {   // L3: p = -q + beta p, for the rows and the ghosts
            const double beta = s_coef;
            if (live)
#pragma unroll
                for (int d = 0; d < kDofs; d++) own_p(d) = fma(beta, own_p(d), -(g[d] * di[d]));
            for (uint32_t j = tid; j < ng; j += bd) {
                const double2 q = QG[j], p = P[nslot + j];
                P[nslot + j] = make_double2(fma(beta, p.x, -q.x), fma(beta, p.y, -q.y));
            }
            __syncthreads();
        }
    }
done:
    if (live)
#pragma unroll
        for (int d = 0; d < kDofs; d++) a.x[2 * (size_t)i + (kDofs == 2 ? d : par)] = x[d];
    if (rank == 0 && tid == 0) sc.report_to(a);
}

// The instance for `threads` threads, one (kDofs = 1) or two dofs per lane.
template <bool JAC, bool LAGGED>
const void* bsr_slice_kernel_of(int dofs, int threads) {
    if (dofs == 1) return (const void*)k_cg_bsr_slice<JAC, LAGGED, 1, 256>;
    return threads <= 512 ? (const void*)k_cg_bsr_slice<JAC, LAGGED, 2, 512>
         : threads <= 896 ? (const void*)k_cg_bsr_slice<JAC, LAGGED, 2, 896>
                          : (const void*)k_cg_bsr_slice<JAC, LAGGED, 2, 1024>;
}

// Workspace of the slice form's plan; none for a system that is too large for it.
size_t slice_plan_bytes(const nbg_bsr_t& A) {
    int dev = 0, nsm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    return A.n_slices > 32 * exact_grid((unsigned)nsm) ? 0 : ghost_plan_bytes(A);
}

// Launch data of the slice form: 1, or 0 (the global form runs).  Two slices
// per block, one warp per scheduler, while there are SMs (4,290 dof: 4.9 us
// per iteration with 2 slices, 5.5 with 4; 16,770 dof: 5.1 and 5.7).  A lane
// per dof up to four slices per block, where the FP64 latency of a row counts
// (16,770 dof: 5.1 us against 6.2 with a lane per row); above, its rounding up
// of odd entry counts costs more FP64 issue than it saves (66,306 dof: 7.5
// against 7.2, T3 with 91,204 dof: 9.1 against 8.3).  These with sums that were
// polled at once, 0.1 to 0.3 us slower than with kLeadUp (allreduce.cuh).
int bsr_slice_setup(const nbg_bsr_t& A, bool jac, bool lagged, char* plan, cudaStream_t s,
                    BsrSliceArgs* sl, const void** fn, unsigned* G, int* threads, size_t* dyn) {
    int dev = 0, nsm = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) !=
            cudaSuccess)
        return 0;
    const unsigned most = exact_grid((unsigned)nsm);
    if (A.n_slices > 32 * most) return 0;
    *G = std::min(most, (A.n_slices + 1) / 2);
    const unsigned spb = (A.n_slices + *G - 1) / *G;
    const int dofs = spb <= 4 ? 1 : 2;
    *threads = 32 * (int)(dofs == 1 ? 2 * spb : spb);
    *fn = jac ? (lagged ? bsr_slice_kernel_of<true, true>(dofs, *threads)
                        : bsr_slice_kernel_of<true, false>(dofs, *threads))
              : (lagged ? bsr_slice_kernel_of<false, true>(dofs, *threads)
                        : bsr_slice_kernel_of<false, false>(dofs, *threads));
    uint32_t widest;
    if (!ghost_plan(A, *G, plan, s, &sl->gh, &widest)) return 0;
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, *fn) != cudaSuccess) return 0;
    const size_t base = 16 * (size_t)sl->gh.pcap + 16 * (size_t)sl->gh.gcap +
                        4 * (size_t)((sl->gh.gcap + 3) & ~3u);
    if (base + fa.sharedSizeBytes > (size_t)optin) return 0;
    const size_t left = (size_t)optin - fa.sharedSizeBytes - base;
    const size_t column = 34 * (size_t)sl->gh.scap;
    sl->keep = (uint32_t)std::min<size_t>(widest, left / column);
    *dyn = base + column * sl->keep;
    return fits_smem(*fn, *threads, *dyn, *G) ? 1 : 0;
}
