// FEM assembly kernels: element stiffness, deterministic row-gather into the
// nbots CSR pattern, load increments, Dirichlet elimination, strain, stress.
//
// Parity: every floating-point step repeats nbots' operation order with
// explicitly rounded operations (no FMA), so K, F, strain and stress equal
// the reference's bits.  The gather visits, for each CSR 2x2 node block, the
// elements shared by its two nodes in ascending element id: that is the
// order in which nbots' serial element loop adds into each slot
// (pde_bot/finite_element/solid_mechanics/pipeline.c:60-69), so no float
// atomics and no colouring are needed for bitwise determinism.
#include <cstdint>

#include "common.cuh"

using namespace nbg;

namespace {

// nbots' element tables (pde_bot/finite_element/element.c:54-121), Q4 with
// its 12-significant-digit truncation; node-major [node * N_gp + gp].
#define QA 0.622008467928
#define QB 0.166666666667
#define QC 0.044658198739
#define QD 0.394337567297
#define QE 0.105662432703
__constant__ double c_q4_N[16] = {QA, QB, QC, QB, QB, QA, QB, QC, QC, QB, QA, QB, QB, QC, QB, QA};
__constant__ double c_t3_N[3] = {1.0 / 3.0, 1.0 / 3.0, 1.0 / 3.0};

template <int NN> struct Tab;
template <> struct Tab<4> {
    static constexpr int NGP = 4;
    __device__ static double N(int i, int g) { return c_q4_N[i * 4 + g]; }
    __device__ static double w(int) { return 1.0; }
};
template <> struct Tab<3> {
    static constexpr int NGP = 1;
    __device__ static double N(int i, int g) { return c_t3_N[i]; }
    __device__ static double w(int) { return 0.5; }
};

// The derivative tables as compile-time factors: |dpsi|, |deta| of a Q4 node
// are QD or QE, so the products with a coordinate (or an inverse Jacobian
// entry) are two per operand, with their signs, instead of one per node and
// point (k_strain at 1M dof: 0.50 to 0.38 ms).
template <int NN> struct Grad;
template <> struct Grad<4> {
    static constexpr double kBig = QD, kSmall = QE;
    // sign * (1 big, 2 small) of the node-major tables above
    __device__ static constexpr int psi(int i, int g) {
        constexpr int t[16] = {-1, -1, -2, -2, 1, 1, 2, 2, 2, 2, 1, 1, -2, -2, -1, -1};
        return t[i * 4 + g];
    }
    __device__ static constexpr int eta(int i, int g) {
        constexpr int t[16] = {-1, -2, -2, -1, -2, -1, -1, -2, 2, 1, 1, 2, 1, 2, 2, 1};
        return t[i * 4 + g];
    }
};
template <> struct Grad<3> {  // 0 stands for the factor 0.0
    static constexpr double kBig = 1.0, kSmall = 0.0;
    __device__ static constexpr int psi(int i, int) { return i == 0 ? -1 : i == 1 ? 1 : 2; }
    __device__ static constexpr int eta(int i, int) { return i == 0 ? -1 : i == 1 ? 2 : 1; }
};

__device__ __forceinline__ double pick(int f, double big, double small) {
    const double v = f == 1 || f == -1 ? big : small;
    return f < 0 ? -v : v;  // (-t) v is -(t v) bit for bit
}

// nb_fem_get_jacobian + nb_fem_get_derivatives (utils.c:9-60) with the shared
// products: xb = big x, xs = small x per coordinate (16 of each element instead
// of 16 of each Gauss point).
template <int NN>
__device__ __forceinline__ double shape_derivs_shared(const double (&xb)[NN], const double (&xs)[NN],
                                                      const double (&yb)[NN],
                                                      const double (&ys)[NN], int gp,
                                                      double (&dx)[NN], double (&dy)[NN]) {
    double dx_dpsi = 0.0, dy_dpsi = 0.0, dx_deta = 0.0, dy_deta = 0.0;
#pragma unroll
    for (int i = 0; i < NN; i++) {
        const int p = Grad<NN>::psi(i, gp), e = Grad<NN>::eta(i, gp);
        dx_dpsi = add(dx_dpsi, pick(p, xb[i], xs[i]));
        dx_deta = add(dx_deta, pick(e, xb[i], xs[i]));
        dy_dpsi = add(dy_dpsi, pick(p, yb[i], ys[i]));
        dy_deta = add(dy_deta, pick(e, yb[i], ys[i]));
    }
    const double detJ = sub(mul(dx_dpsi, dy_deta), mul(dy_dpsi, dx_deta));
    const double j[4] = {dvd(dy_deta, detJ), dvd(-dy_dpsi, detJ), dvd(-dx_deta, detJ),
                         dvd(dx_dpsi, detJ)};
    double jb[4], js[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        jb[k] = mul(j[k], Grad<NN>::kBig);
        js[k] = mul(j[k], Grad<NN>::kSmall);
    }
#pragma unroll
    for (int i = 0; i < NN; i++) {
        const int p = Grad<NN>::psi(i, gp), e = Grad<NN>::eta(i, gp);
        dx[i] = add(pick(p, jb[0], js[0]), pick(e, jb[1], js[1]));
        dy[i] = add(pick(p, jb[2], js[2]), pick(e, jb[3], js[3]));
    }
    return detJ;
}

// Node blocks of an element matrix, i <= j: block t holds {a00 a01 a10 a11}.
template <int NN>
__host__ __device__ constexpr int n_blocks() { return NN * (NN + 1) / 2; }
template <int NN>
__device__ __forceinline__ int block_at(int i, int j) {  // i <= j
    return i * NN - i * (i - 1) / 2 + (j - i);
}

// One node block: a 32-byte sector.
__device__ __forceinline__ void st_block(double* p, const double (&t)[4]) {
    asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p), "d"(t[0]), "d"(t[1]), "d"(t[2]),
                 "d"(t[3])
                 : "memory");
}

__device__ __forceinline__ void ld_block(const double* p, double (&t)[4]) {
    asm("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];"
        : "=d"(t[0]), "=d"(t[1]), "=d"(t[2]), "=d"(t[3])
        : "l"(p));
}

// Ke and Fe of one element per thread.  FP64 issue bounds it (GB300: about
// 1.7 FP64 operations per SM and clock), so everything that repeats is
// computed once: Ke is exactly symmetric in nbots' arithmetic (the mirrored
// entry multiplies the same factors), the four entries of a node block share
// their four products, products with the tables are shared as above, and
// factors of exactly 1 (the Q4 weights, a unit thickness: kUnit) and the load
// of a massless element are left out: about 1,130 operations per Q4 element,
// 1.16 ms for the 1M-dof cantilever's 524,288 (1.76 ms before, entry by entry).
// kBlocks: the element's node blocks one after the other (Ke[(e n_blocks +
// t) 4 ..], 32 B each, what k_gather_blocks reads) and one double of Fe
// without self weight (0, or NaN where the element has none); else
// entry-major: Ke[(a * 2NN + b) * N_elem + e], Fe[a * N_elem + e].
template <int NN, bool kBlocks, bool kUnit>
__global__ void __launch_bounds__(128) k_element(uint32_t N_elem, const double* __restrict__ nod,
                                                 const uint32_t* __restrict__ conn,
                                                 const double* __restrict__ E, double nu, double th,
                                                 double density, int self_weight, double gx,
                                                 double gy, const uint8_t* __restrict__ enabled,
                                                 const double* __restrict__ dmg,
                                                 double* __restrict__ Ke, double* __restrict__ Fe,
                                                 uint32_t* distorted) {
    constexpr int ND = 2 * NN;
    constexpr int NGP = Tab<NN>::NGP;
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= N_elem) return;
    double xb[NN], xs[NN], yb[NN], ys[NN];
#pragma unroll
    for (int i = 0; i < NN; i++) {
        const uint32_t n = conn[(size_t)e * NN + i];
        const double2 v = kBlocks ? reinterpret_cast<const double2*>(nod)[n]
                                  : make_double2(nod[2 * (size_t)n], nod[2 * (size_t)n + 1]);
        xb[i] = mul(Grad<NN>::kBig, v.x);
        xs[i] = mul(Grad<NN>::kSmall, v.x);
        yb[i] = mul(Grad<NN>::kBig, v.y);
        ys[i] = mul(Grad<NN>::kSmall, v.y);
    }
    // assemble_element (pipeline.c:93-98) and set_plane_stress (formulas.c:48-54)
    double D0 = 1e-6, D1 = 1e-6, D3 = 1e-6, dens = 1e-6;  // D2 = D0
    if (enabled == nullptr || enabled[e]) {
        double Ee = E[e];
        D0 = dvd(Ee, sub(1.0, mul(nu, nu)));
        D1 = mul(nu, D0);
        D3 = dvd(Ee, mul(2.0, add(1.0, nu)));
        dens = density;
    }
    double fx = 0.0, fy = 0.0;
    if (self_weight) {
        fx = mul(gx, dens);
        fy = mul(gy, dens);
    }
    double k[n_blocks<NN>()][4];
    double f[ND];
#pragma unroll
    for (int t = 0; t < n_blocks<NN>(); t++) k[t][0] = k[t][1] = k[t][2] = k[t][3] = 0.0;
#pragma unroll
    for (int i = 0; i < ND; i++) f[i] = 0.0;
#pragma unroll
    for (int gp = 0; gp < NGP; gp++) {
        double dx[NN], dy[NN];
        const double detJ = shape_derivs_shared<NN>(xb, xs, yb, ys, gp, dx, dy);
        if (detJ < 0) {
            atomicMin(distorted, e);
            return;
        }
        // detJ * t * w of a term
        auto weigh = [&](double v) {
            v = mul(v, detJ);
            if (!kUnit) v = mul(v, th);
            return NN == 4 ? v : mul(v, Tab<NN>::w(gp));  // w = 1 for Q4
        };
        // DMG_pipeline_assemble_system (static_damage2D.c:527-534): each
        // Gauss point scales D by (1 - damage) first
        double G0 = D0, G1 = D1, G3 = D3;
        if (dmg != nullptr) {
            const double keep = sub(1.0, dmg[(size_t)e * NGP + gp]);
            G0 = mul(D0, keep);
            G1 = mul(D1, keep);
            G3 = mul(D3, keep);
        }
        // pipeline_sum_gauss_point (pipeline.c:197-212)
        int t = 0;
#pragma unroll
        for (int i = 0; i < NN; i++) {
#pragma unroll
            for (int j = i; j < NN; j++) {
                const double xx = mul(dx[i], dx[j]), yy = mul(dy[i], dy[j]);
                const double xy = mul(dx[i], dy[j]), yx = i == j ? xy : mul(dy[i], dx[j]);
                k[t][0] = add(k[t][0], weigh(add(mul(xx, G0), mul(yy, G3))));
                k[t][1] = add(k[t][1], weigh(add(mul(xy, G1), mul(yx, G3))));
                if (i != j) k[t][2] = add(k[t][2], weigh(add(mul(yx, G1), mul(xy, G3))));
                k[t][3] = add(k[t][3], weigh(add(mul(yy, G0), mul(xx, G3))));
                t++;
            }
        }
        if (self_weight || !kBlocks) {
#pragma unroll
            for (int i = 0; i < NN; i++) {
                double integral = mul(Tab<NN>::N(i, gp), detJ);
                if (!kUnit) integral = mul(integral, th);
                if (NN != 4) integral = mul(integral, Tab<NN>::w(gp));
                f[2 * i] = add(f[2 * i], mul(integral, fx));
                f[2 * i + 1] = add(f[2 * i + 1], mul(integral, fy));
            }
        } else {  // zero loads: 0, but NaN where the Jacobian is not finite
            f[0] = add(f[0], mul(kUnit ? detJ : mul(detJ, th), 0.0));
        }
    }
    int t = 0;
#pragma unroll
    for (int i = 0; i < NN; i++) {
#pragma unroll
        for (int j = i; j < NN; j++) {
            if (i == j) k[t][2] = k[t][1];
            if (kBlocks) {
                st_block(Ke + ((size_t)e * n_blocks<NN>() + t) * 4, k[t]);
            } else {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int a = 2 * i + (q >> 1), b = 2 * j + (q & 1);
                    Ke[(size_t)(a * ND + b) * N_elem + e] = k[t][q];
                    if (i != j) Ke[(size_t)(b * ND + a) * N_elem + e] = k[t][q];
                }
            }
            t++;
        }
    }
    if (kBlocks && !self_weight) {
        Fe[e] = f[0];
        return;
    }
#pragma unroll
    for (int i = 0; i < ND; i++) Fe[(size_t)i * N_elem + e] = f[i];
}

// K and F of one node (its two CSR rows share one sorted column list made of
// (2w, 2w+1) pairs, sparse.c:36-52, so each pair is one 2x2 block) by merging
// the incidence lists of its row and column nodes.  block(i, j, e, v) gives
// the node block (i, j) of element e.  Returns the pairs found.
template <class Block>
__device__ __forceinline__ unsigned long long gather_node(
    uint32_t v, const uint32_t* __restrict__ inc_ptr, const uint32_t* __restrict__ inc_elem,
    const uint8_t* __restrict__ inc_local, const uint32_t* __restrict__ rp,
    const uint32_t* __restrict__ ci, double* __restrict__ K, Block block) {
    const uint32_t a0 = inc_ptr[v], a1 = inc_ptr[v + 1];
    const uint32_t r0 = rp[2 * v], r1 = rp[2 * v + 1], len = r1 - r0;
    unsigned long long cnt = 0;
    for (uint32_t kk = 0; kk < len; kk += 2) {
        const uint32_t c = ci[r0 + kk];
        const uint32_t w = c >> 1;
        const bool paired = !(c & 1) && kk + 1 < len && ci[r0 + kk + 1] == c + 1;
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        uint32_t ia = a0, ib = inc_ptr[w];
        const uint32_t ib1 = inc_ptr[w + 1];
        while (paired && ia < a1 && ib < ib1) {
            const uint32_t ea = inc_elem[ia], eb = inc_elem[ib];
            if (ea < eb) { ia++; continue; }
            if (eb < ea) { ib++; continue; }
            double t[4];
            block(inc_local[ia], inc_local[ib], ea, t);
#pragma unroll
            for (int q = 0; q < 4; q++) s[q] = add(s[q], t[q]);
            cnt++;
            ia++;
            ib++;
        }
        if (!paired) {
            // not a node block: nbots' pattern never makes one; leave the
            // slot at zero and make the pair count disagree
            K[r0 + kk] = 0.0;
            K[r1 + kk] = 0.0;
            cnt += 1ull << 40;
            kk -= 1;  // advance by one column only
            continue;
        }
        K[r0 + kk] = s[0];
        K[r0 + kk + 1] = s[1];
        K[r1 + kk] = s[2];
        K[r1 + kk + 1] = s[3];
    }
    return cnt;
}

// The gather from entry-major element matrices, one thread per node.
template <int NN>
__global__ void __launch_bounds__(128) k_gather(uint32_t N_nod, uint32_t N_elem,
                                                const uint32_t* __restrict__ inc_ptr,
                                                const uint32_t* __restrict__ inc_elem,
                                                const uint8_t* __restrict__ inc_local,
                                                const uint32_t* __restrict__ rp,
                                                const uint32_t* __restrict__ ci,
                                                const double* __restrict__ Ke,
                                                const double* __restrict__ Fe,
                                                double* __restrict__ K, double* __restrict__ F,
                                                unsigned long long* matched) {
    constexpr int ND = 2 * NN;
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= N_nod) return;
    const size_t P = N_elem;
    const unsigned long long cnt = gather_node(
        v, inc_ptr, inc_elem, inc_local, rp, ci, K, [&](int i, int j, uint32_t e, double (&t)[4]) {
#pragma unroll
            for (int q = 0; q < 4; q++)
                t[q] = Ke[(size_t)((2 * i + (q >> 1)) * ND + 2 * j + (q & 1)) * P + e];
        });
    double f0 = 0.0, f1 = 0.0;
    for (uint32_t ia = inc_ptr[v]; ia < inc_ptr[v + 1]; ia++) {
        const uint32_t e = inc_elem[ia];
        const int i = inc_local[ia];
        f0 = add(f0, Fe[(size_t)(2 * i) * P + e]);
        f1 = add(f1, Fe[(size_t)(2 * i + 1) * P + e]);
    }
    F[2 * v] = f0;
    F[2 * v + 1] = f1;
    if (cnt) atomicAdd(matched, cnt);
}

// The gather from element node blocks.  A node walks its elements in
// ascending order (nbots' order of addition into every slot) and adds each
// one's row of blocks to the row's columns in shared memory: one 32-byte load
// per block, no merging of incidence lists; a warp then writes its nodes' rows
// with coalesced stores.  Rows of more than kGatherCols columns, columns that
// are not node blocks and elements that list a node twice go through
// gather_node, which finds (and misses) the same pairs.  1M dof: 0.26 ms
// against 0.55 for merging per block on entry-major matrices (64 entries per
// Q4 element instead of 10 blocks); its bytes would take 0.06.
constexpr int kGatherCols = 12, kGatherThreads = 64;

// 0.0 + v
__device__ __forceinline__ double plus_zero(double v) {
    return __double_as_longlong(v) == (long long)(1ull << 63) ? 0.0 : v;
}

template <int NN>
__global__ void __launch_bounds__(kGatherThreads)
    k_gather_blocks(uint32_t N_nod, uint32_t N_elem, const uint32_t* __restrict__ inc_ptr,
                    const uint32_t* __restrict__ inc_elem, const uint8_t* __restrict__ inc_local,
                    const uint32_t* __restrict__ rp, const uint32_t* __restrict__ ci,
                    const uint32_t* __restrict__ conn, const double* __restrict__ Ke,
                    const double* __restrict__ Fe, int self_weight, double* __restrict__ K,
                    double* __restrict__ F, unsigned long long* matched,
                    const uint32_t* distorted) {
    __shared__ double acc[4 * kGatherCols][kGatherThreads + 1];
    // assembly stops at a distorted element: K and F stay as they are
    if (*distorted != 0xffffffffu) return;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const uint32_t v = blockIdx.x * kGatherThreads + tid;
    const bool valid = v < N_nod;
    uint32_t r0 = 0, len = 0, a0 = 0, a1 = 0;
    if (valid) {
        r0 = rp[2 * v];
        len = rp[2 * v + 1] - r0;
        a0 = inc_ptr[v];
        a1 = inc_ptr[v + 1];
    }
    bool fast = valid && len <= 2 * kGatherCols && !(len & 1);
    uint32_t col[kGatherCols];  // column nodes, ascending
#pragma unroll
    for (int p = 0; p < kGatherCols; p++) {
        col[p] = 0xffffffffu;
        if (fast && 2u * p < len) {
            const uint32_t c = ci[r0 + 2 * p];
            if ((c & 1) || ci[r0 + 2 * p + 1] != c + 1 || (p && col[p - 1] >= c >> 1)) fast = false;
            col[p] = c >> 1;
#pragma unroll
            for (int q = 0; q < 4; q++) acc[4 * p + q][tid] = 0.0;
        }
    }
    auto block = [&](int i, int j, uint32_t e, double (&t)[4]) {
        ld_block(Ke + ((size_t)e * n_blocks<NN>() + block_at<NN>(min(i, j), max(i, j))) * 4, t);
        if (i > j) {
            const double s = t[1];
            t[1] = t[2];
            t[2] = s;
        }
    };
    unsigned long long cnt = 0;
    double f0 = 0.0, f1 = 0.0;
    uint32_t last = 0xffffffffu, touched = 0;
    // four elements at a time, their loads issued together
    for (uint32_t ia = a0; ia < a1; ia += 4) {
        const uint32_t n = min(4u, a1 - ia);
        uint32_t el[4], node[4][NN];
        int loc[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            el[c] = c < n ? inc_elem[ia + c] : 0;
            loc[c] = c < n ? inc_local[ia + c] : 0;
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
            if (c >= n) continue;
            if (NN == 4) {
                const uint4 t = reinterpret_cast<const uint4*>(conn)[el[c]];
                node[c][0] = t.x;
                node[c][1] = t.y;
                node[c][2] = t.z;
                node[c][NN - 1] = t.w;
            } else {
#pragma unroll
                for (int j = 0; j < NN; j++) node[c][j] = conn[(size_t)el[c] * NN + j];
            }
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
            if (c >= n) continue;
            const uint32_t e = el[c];
            const int i = loc[c];
            if (self_weight) {
                f0 = add(f0, Fe[(size_t)(2 * i) * N_elem + e]);
                f1 = add(f1, Fe[(size_t)(2 * i + 1) * N_elem + e]);
            } else {
                f0 = add(f0, Fe[e]);
            }
            if (e == last) fast = false;
            last = e;
#pragma unroll
            for (int j = 0; j < NN; j++)
#pragma unroll
                for (int q = 0; q < j; q++)
                    if (node[c][q] == node[c][j]) fast = false;
            if (!fast) continue;
            double t[NN][4];
#pragma unroll
            for (int j = 0; j < NN; j++) block(i, j, e, t[j]);
#pragma unroll
            for (int j = 0; j < NN; j++) {
                int at = 0;
                bool found = false;
#pragma unroll
                for (int p = 0; p < kGatherCols; p++) {
                    at += col[p] < node[c][j];
                    found |= col[p] == node[c][j];
                }
                if (!found) continue;
                // the first term of a slot is added to 0.0: itself, but 0.0 for
                // -0.0 (no FP64 addition: they bound this kernel)
                const bool first = !(touched >> at & 1);
                touched |= 1u << at;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    double& slot = acc[4 * at + q][tid];
                    slot = first ? plus_zero(t[j][q]) : add(slot, t[j][q]);
                }
                cnt++;
            }
        }
    }
    if (valid) {
        F[2 * v] = f0;
        F[2 * v + 1] = self_weight ? f1 : f0;
        if (!fast) cnt = gather_node(v, inc_ptr, inc_elem, inc_local, rp, ci, K, block);
    }
    // the warp's rows, one node at a time
    __syncwarp();
    const uint32_t n_fast = fast ? len : 0;
    for (int n = 0; n < 32; n++) {
        const uint32_t l = __shfl_sync(0xffffffffu, n_fast, n);
        const uint32_t base = __shfl_sync(0xffffffffu, r0, n);
        for (uint32_t t = lane; t < 2 * l; t += 32) {
            const uint32_t row = t >= l, q = t - row * l;
            K[base + t] = acc[2 * (q & ~1u) + 2 * row + (q & 1)][(tid & ~31u) + n];
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    if (lane == 0 && cnt) atomicAdd(matched, cnt);
}

__global__ void k_increments(uint32_t n_groups, const uint32_t* __restrict__ idx,
                             const uint32_t* __restrict__ gptr, const double* __restrict__ inc,
                             double* __restrict__ F) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n_groups) return;
    double f = F[idx[g]];
    for (uint32_t k = gptr[g]; k < gptr[g + 1]; k++) f = add(f, inc[k]);
    F[idx[g]] = f;
}

__global__ void k_pick_nodes(uint32_t n, const uint32_t* __restrict__ ids,
                             const double2* __restrict__ nod, double2* __restrict__ xy) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) xy[k] = nod[ids[k]];
}

// Offsets of every dof's events in the list sorted by dof (a binary search
// each: 10 steps for a clamped edge of 500 nodes).
__global__ void k_event_ptr(uint32_t N, uint32_t n_ev, const uint32_t* __restrict__ ev_dof,
                            uint32_t* __restrict__ ev_ptr) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > N) return;
    uint32_t lo = 0, hi = n_ev;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (ev_dof[mid] < i) lo = mid + 1; else hi = mid;
    }
    ev_ptr[i] = lo;
}

constexpr int kMaxRowEvents = 96;

// Thread per row j: replay, in global event order, every Dirichlet event
// that touches row j: its own (row reset to the identity, F[j] = value) and
// those of the dofs in its columns (K[j][d] = 0, F[j] -= K[j][d] * value).
__global__ void __launch_bounds__(128) k_dirichlet(uint32_t N, const uint32_t* __restrict__ rp,
                                                   const uint32_t* __restrict__ ci,
                                                   double* __restrict__ K, double* __restrict__ F,
                                                   const uint32_t* __restrict__ ev_ptr,
                                                   const uint32_t* __restrict__ ev_of,
                                                   const double* __restrict__ ev_val, int* status) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= N) return;
    uint32_t evn[kMaxRowEvents];
    uint32_t pos[kMaxRowEvents];  // CSR slot of the column, or UINT32_MAX for the row's own event
    int n = 0;
    const uint32_t b = rp[j], e = rp[j + 1];
    for (uint32_t k = b; k < e; k++) {
        const uint32_t c = ci[k];
        for (uint32_t t = ev_ptr[c]; t < ev_ptr[c + 1]; t++) {
            if (n == kMaxRowEvents) {
                atomicCAS(status, 0, NBG_ERR_ARG);
                return;
            }
            evn[n] = ev_of[t];
            pos[n] = c == j ? 0xffffffffu : k;
            n++;
        }
    }
    if (n == 0) return;
    for (int a = 1; a < n; a++) {  // insertion sort by event number
        uint32_t ke = evn[a], kp = pos[a];
        int q = a - 1;
        while (q >= 0 && evn[q] > ke) {
            evn[q + 1] = evn[q];
            pos[q + 1] = pos[q];
            q--;
        }
        evn[q + 1] = ke;
        pos[q + 1] = kp;
    }
    double f = F[j];
    for (int a = 0; a < n; a++) {
        const double val = ev_val[evn[a]];
        if (pos[a] == 0xffffffffu) {
            for (uint32_t k = b; k < e; k++) K[k] = ci[k] == j ? 1.0 : 0.0;
            f = val;
        } else {
            const double var = K[pos[a]];
            K[pos[a]] = 0.0;
            f = sub(f, mul(var, val));
        }
    }
    F[j] = f;
}

template <int NN>
__global__ void __launch_bounds__(128) k_strain(uint32_t N_elem, const double* __restrict__ nod,
                                                const uint32_t* __restrict__ conn,
                                                const double* __restrict__ u,
                                                double* __restrict__ strain) {
    constexpr int NGP = Tab<NN>::NGP;
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= N_elem) return;
    double xb[NN], xs[NN], yb[NN], ys[NN], ux[NN], uy[NN];
#pragma unroll
    for (int i = 0; i < NN; i++) {
        uint32_t n = conn[(size_t)e * NN + i];
        const double x = nod[2 * (size_t)n], y = nod[2 * (size_t)n + 1];
        xb[i] = mul(Grad<NN>::kBig, x);
        xs[i] = mul(Grad<NN>::kSmall, x);
        yb[i] = mul(Grad<NN>::kBig, y);
        ys[i] = mul(Grad<NN>::kSmall, y);
        ux[i] = u[2 * (size_t)n];
        uy[i] = u[2 * (size_t)n + 1];
    }
    bool stop = false;
#pragma unroll
    for (int gp = 0; gp < NGP; gp++) {
        double s0 = 0.0, s1 = 0.0, s2 = 0.0;
        if (!stop) {
            double dx[NN], dy[NN];
            const double detJ = shape_derivs_shared<NN>(xb, xs, yb, ys, gp, dx, dy);
            if (detJ < 0) {
                stop = true;  // get_element_strain leaves the remaining points at zero
            } else {
#pragma unroll
                for (int i = 0; i < NN; i++) {
                    s0 = add(s0, mul(dx[i], ux[i]));
                    s1 = add(s1, mul(dy[i], uy[i]));
                    s2 = add(s2, add(mul(dy[i], ux[i]), mul(dx[i], uy[i])));
                }
            }
        }
        const size_t id = (size_t)e * NGP + gp;
        strain[id * 3] = s0;
        strain[id * 3 + 1] = s1;
        strain[id * 3 + 2] = s2;
    }
}

__global__ void k_stress(uint32_t N_elem, int ngp, const double* __restrict__ E, double nu,
                         const uint8_t* __restrict__ enabled, const double* __restrict__ strain,
                         double* __restrict__ stress) {
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= N_elem) return;
    double D0 = 1e-6, D1 = 1e-6, D2 = 1e-6, D3 = 1e-6;
    if (enabled == nullptr || enabled[e]) {
        D0 = dvd(E[e], sub(1.0, mul(nu, nu)));
        D1 = mul(nu, D0);
        D2 = D0;
        D3 = dvd(E[e], mul(2.0, add(1.0, nu)));
    }
    for (int g = 0; g < ngp; g++) {
        const size_t id = (size_t)e * ngp + g;
        const double e0 = strain[id * 3], e1 = strain[id * 3 + 1], e2 = strain[id * 3 + 2];
        stress[id * 3] = add(mul(e0, D0), mul(e1, D1));
        stress[id * 3 + 1] = add(mul(e0, D1), mul(e1, D2));
        stress[id * 3 + 2] = mul(e2, D3);
    }
}

// Principal stresses per Gauss point (pipeline.c:321-340): the mean of the
// normal stresses plus and minus the radius of Mohr's circle, nbots'
// operation order without contraction and a correctly rounded square root.
__global__ void k_main_stress(uint32_t n, const double* __restrict__ stress,
                              double* __restrict__ main_stress) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double sx = stress[(size_t)i * 3], sy = stress[(size_t)i * 3 + 1];
    const double txy = stress[(size_t)i * 3 + 2];
    const double avg = mul(0.5, add(sx, sy));
    const double d = sub(sx, sy);
    const double R = __dsqrt_rn(add(mul(0.25, mul(d, d)), mul(txy, txy)));
    main_stress[(size_t)i * 2] = add(avg, R);
    main_stress[(size_t)i * 2 + 1] = sub(avg, R);
}

inline unsigned nblk(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

extern "C" int nbg_main_stress_f64(uint32_t nen, uint32_t N_elem, const double* stress,
                                   double* main_stress, void* stream) {
    if (nen != 3 && nen != 4) return NBG_ERR_ARG;
    const uint64_t n = (uint64_t)N_elem * (nen == 4 ? 4 : 1);
    if (n == 0) return NBG_OK;
    if (n > UINT32_MAX) return NBG_ERR_ARG;
    k_main_stress<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>((uint32_t)n, stress,
                                                                  main_stress);
    NBG_CHECK(cudaGetLastError());
    return NBG_OK;
}

namespace {
template <bool kBlocks>
int launch_elements(uint32_t nen, uint32_t N_elem, const double* nod, const uint32_t* conn,
                    const double* E, double nu, double th, double density, int self_weight,
                    double gx, double gy, const uint8_t* enabled, const double* damage, double* Ke,
                    double* Fe, uint32_t* distorted, cudaStream_t s) {
    const unsigned g = nblk(N_elem, 128);
    auto go = [&](auto kernel) {
        kernel<<<g, 128, 0, s>>>(N_elem, nod, conn, E, nu, th, density, self_weight, gx, gy,
                                 enabled, damage, Ke, Fe, distorted);
    };
    const bool unit = th == 1.0;
    if (nen == 4) {
        if (unit) go(k_element<4, kBlocks, true>);
        else go(k_element<4, kBlocks, false>);
    } else if (nen == 3) {
        if (unit) go(k_element<3, kBlocks, true>);
        else go(k_element<3, kBlocks, false>);
    } else {
        return NBG_ERR_ARG;
    }
    NBG_CHECK(cudaGetLastError());
    return NBG_OK;
}
}  // namespace

extern "C" int nbg_element_stiffness_damage_f64(uint32_t nen, uint32_t N_elem, const double* nod,
                                                const uint32_t* conn, const double* E, double nu,
                                                double thickness, double density,
                                                int self_weight, double gx, double gy,
                                                const uint8_t* enabled, const double* damage,
                                                double* Ke, double* Fe, uint32_t* distorted,
                                                void* stream) {
    if (N_elem == 0) return NBG_OK;
    return launch_elements<false>(nen, N_elem, nod, conn, E, nu, thickness, density, self_weight,
                                  gx, gy, enabled, damage, Ke, Fe, distorted,
                                  (cudaStream_t)stream);
}

// The FEM system's pair of kernels (host/fem_internal.h): element node blocks
// and their gather.
extern "C" size_t nbg_fem_element_bytes(uint32_t nen) {
    return 32 * (size_t)(nen == 4 ? n_blocks<4>() : n_blocks<3>());
}

extern "C" int nbg_fem_element_blocks(uint32_t nen, uint32_t N_elem, const double* nod,
                                      const uint32_t* conn, const double* E, double nu,
                                      double thickness, double density, int self_weight, double gx,
                                      double gy, const uint8_t* enabled, const double* damage,
                                      double* Ke, double* Fe, uint32_t* distorted, void* stream) {
    if (N_elem == 0) return NBG_OK;
    return launch_elements<true>(nen, N_elem, nod, conn, E, nu, thickness, density, self_weight, gx,
                                 gy, enabled, damage, Ke, Fe, distorted, (cudaStream_t)stream);
}

extern "C" int nbg_fem_pick_nodes(uint32_t n, const uint32_t* ids, const double* nod, double* xy,
                                  void* stream) {
    if (n == 0) return NBG_OK;
    k_pick_nodes<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(
        n, ids, reinterpret_cast<const double2*>(nod), reinterpret_cast<double2*>(xy));
    NBG_CHECK(cudaGetLastError());
    return NBG_OK;
}

extern "C" int nbg_fem_event_ptr(uint32_t N, uint32_t n_ev, const uint32_t* ev_dof,
                                 uint32_t* ev_ptr, void* stream) {
    k_event_ptr<<<nblk((uint64_t)N + 1, 256), 256, 0, (cudaStream_t)stream>>>(N, n_ev, ev_dof,
                                                                             ev_ptr);
    NBG_CHECK(cudaGetLastError());
    return NBG_OK;
}

extern "C" int nbg_fem_gather_blocks(uint32_t nen, uint32_t N_nod, uint32_t N_elem,
                                     const uint32_t* inc_ptr, const uint32_t* inc_elem,
                                     const uint8_t* inc_local, const uint32_t* row_ptr,
                                     const uint32_t* col_idx, const uint32_t* conn,
                                     const double* Ke, const double* Fe, int self_weight, double* K,
                                     double* F, unsigned long long* matched,
                                     const uint32_t* distorted, void* stream) {
    if (N_nod == 0) return NBG_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned g = nblk(N_nod, kGatherThreads);
    if (nen == 4)
        k_gather_blocks<4><<<g, kGatherThreads, 0, s>>>(N_nod, N_elem, inc_ptr, inc_elem, inc_local,
                                                        row_ptr, col_idx, conn, Ke, Fe, self_weight,
                                                        K, F, matched, distorted);
    else if (nen == 3)
        k_gather_blocks<3><<<g, kGatherThreads, 0, s>>>(N_nod, N_elem, inc_ptr, inc_elem, inc_local,
                                                        row_ptr, col_idx, conn, Ke, Fe, self_weight,
                                                        K, F, matched, distorted);
    else
        return NBG_ERR_ARG;
    NBG_CHECK(cudaGetLastError());
    return NBG_OK;
}

extern "C" int nbg_element_stiffness_f64(uint32_t nen, uint32_t N_elem, const double* nod,
                                         const uint32_t* conn, const double* E, double nu,
                                         double thickness, double density, int self_weight,
                                         double gx, double gy, const uint8_t* enabled, double* Ke,
                                         double* Fe, uint32_t* distorted, void* stream) {
    return nbg_element_stiffness_damage_f64(nen, N_elem, nod, conn, E, nu, thickness, density,
                                            self_weight, gx, gy, enabled, nullptr, Ke, Fe,
                                            distorted, stream);
}

extern "C" int nbg_gather_assemble_f64(uint32_t nen, uint32_t N_nod, uint32_t N_elem,
                                       const uint32_t* inc_ptr, const uint32_t* inc_elem,
                                       const uint8_t* inc_local, const uint32_t* row_ptr,
                                       const uint32_t* col_idx, const double* Ke, const double* Fe,
                                       double* K, double* F, unsigned long long* matched,
                                       void* stream) {
    if (N_nod == 0) return NBG_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (nen == 4)
        k_gather<4><<<nblk(N_nod, 128), 128, 0, s>>>(N_nod, N_elem, inc_ptr, inc_elem, inc_local,
                                                     row_ptr, col_idx, Ke, Fe, K, F, matched);
    else if (nen == 3)
        k_gather<3><<<nblk(N_nod, 128), 128, 0, s>>>(N_nod, N_elem, inc_ptr, inc_elem, inc_local,
                                                     row_ptr, col_idx, Ke, Fe, K, F, matched);
    else
        return NBG_ERR_ARG;
    NBG_CHECK(cudaGetLastError());
    return NBG_OK;
}

extern "C" int nbg_apply_increments_f64(uint32_t n_groups, const uint32_t* idx_of_group,
                                        const uint32_t* group_ptr, const double* inc, double* F,
                                        void* stream) {
    if (n_groups == 0) return NBG_OK;
    k_increments<<<nblk(n_groups, 128), 128, 0, (cudaStream_t)stream>>>(n_groups, idx_of_group,
                                                                       group_ptr, inc, F);
    NBG_CHECK(cudaGetLastError());
    return NBG_OK;
}

extern "C" int nbg_dirichlet_f64(uint32_t N, const uint32_t* row_ptr, const uint32_t* col_idx,
                                 double* K, double* F, const uint32_t* ev_ptr,
                                 const uint32_t* ev_of, const double* ev_val, int* status,
                                 void* stream) {
    if (N == 0) return NBG_OK;
    k_dirichlet<<<nblk(N, 128), 128, 0, (cudaStream_t)stream>>>(N, row_ptr, col_idx, K, F, ev_ptr,
                                                               ev_of, ev_val, status);
    NBG_CHECK(cudaGetLastError());
    return NBG_OK;
}

extern "C" int nbg_strain_f64(uint32_t nen, uint32_t N_elem, const double* nod,
                              const uint32_t* conn, const double* u, double* strain,
                              void* stream) {
    if (N_elem == 0) return NBG_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (nen == 4)
        k_strain<4><<<nblk(N_elem, 128), 128, 0, s>>>(N_elem, nod, conn, u, strain);
    else if (nen == 3)
        k_strain<3><<<nblk(N_elem, 128), 128, 0, s>>>(N_elem, nod, conn, u, strain);
    else
        return NBG_ERR_ARG;
    NBG_CHECK(cudaGetLastError());
    return NBG_OK;
}

extern "C" int nbg_stress_f64(uint32_t nen, uint32_t N_elem, const double* E, double nu,
                              const uint8_t* enabled, const double* strain, double* stress,
                              void* stream) {
    if (N_elem == 0) return NBG_OK;
    if (nen != 3 && nen != 4) return NBG_ERR_ARG;
    k_stress<<<nblk(N_elem, 128), 128, 0, (cudaStream_t)stream>>>(N_elem, nen == 4 ? 4 : 1, E, nu,
                                                                 enabled, strain, stress);
    NBG_CHECK(cudaGetLastError());
    return NBG_OK;
}
