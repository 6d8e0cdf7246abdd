// s-step preconditioner of the CG sweep (precond_hprsdft with IPC = 4,
// cgpc_hprsdft_module.f90:126-348, in the Chebyshev-basis form described in
// cgvec.cuh) and the search-direction update folded into it
// (cg_module.f90:232-261).
#include <algorithm>
#include <type_traits>

#include "cgvec.cuh"
#include "kernels.cuh"
#include "tma.cuh"
#include "tmap.cuh"
#include "vec16.cuh"

namespace rsdft {

// Basis vector w_K (K = 0: r0 = g - A g, the reference's first residual) and
// its D dots: D >= 2, write w_K with <w_K, w_{K-1}> (K = 0: <g, w_0>), <w_K, w_K>
// and, with D = 3 (K >= 2), <w_K, w_{K-2}>; D = 1 (K = mloop), only
// <S w_{K-1}, w_{K-1}> with S = B for K = 1 and 2 B above.
template <typename T, int K, int D>
__global__ void __launch_bounds__(VT) k_ss_basis(const T* g, SSVec<T> sv, long ld, long n, PcArgs pa,
                                                 double* __restrict__ part, const int* active) {
    grid_dependency();
    constexpr bool STORE = D > 1;
    __shared__ double sh[D * (VT / 32)];
    const int b = blockIdx.y;
    if (active && !active[b]) return;
    const int items = vec_items(n);
    const long off = (long)b * ld, base = (long)blockIdx.x * (VT * items);
    const T* src = K == 0 ? g + off : sv.w[K > 0 ? K - 1 : 0] + off;
    const T inv_d = (T)(1.0 / pa.d);
    double acc[D];
#pragma unroll
    for (int k = 0; k < D; ++k) acc[k] = 0.0;
    int i1, i2, i3;
    pc_coords(base + threadIdx.x, pa, i1, i2, i3);
#pragma unroll 4
    for (int it = 0; it < items; ++it) {
        const long i = base + it * VT + threadIdx.x;
        if (i < n) {
            const T si = src[i];
            T wk;
            if constexpr (K == 0) {
                wk = si - pc_apply<T>(src, i, i1, i2, i3, pa);
            } else if constexpr (K == 1) {
                wk = pc_offdiag<T>(src, i, i1, i2, i3, pa) * inv_d;
            } else {
                wk = (T)2 * pc_offdiag<T>(src, i, i1, i2, i3, pa) * inv_d;
                if constexpr (STORE) {
                    const T w2 = sv.w[K >= 2 ? K - 2 : 0][off + i];
                    wk -= w2;
                    if constexpr (D == 3) acc[2] = fma((double)wk, (double)w2, acc[2]);
                }
            }
            acc[0] = fma((double)wk, (double)si, acc[0]);
            if constexpr (STORE) {
                sv.w[K < SS_MAXM ? K : 0][off + i] = wk;
                acc[1] = fma((double)wk, (double)wk, acc[1]);
            }
        }
        pc_step(pa, i1, i2, i3);
    }
    block_sum_n<VT, D>(acc, sh);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < D; ++k) part[((long)b * gridDim.x + blockIdx.x) * D + k] = acc[k];
    }
}

// Per band, one warp: sum the basis passes' partials (fixed order), expand
// them into the Gram matrix, run the reference's preconditioner recurrences
// on coefficient vectors (early exit when |r0|^2 < 1e-24,
// cgpc_hprsdft_module.f90:186), then rb = dV <Pg|g> = rb + dV sum_j cz_j
// <w_j|g> and the search-direction scalars bk = rb / gkgk, gkgk = rb
// (cg_module.f90:232-250).
//
// A basis pass dots what it has in hand: w_k with itself, with its source
// w_{k-1} and, in FP64 and on small FP32 grids, with w_{k-2}.  The rest of the Gram matrix
// follows from w_k = 2 B w_{k-1} - w_{k-2} with B symmetric, B w_0 = w_1 and
// 2 B w_j = w_{j+1} + w_{j-1}:
//   <w_k, w_j> = <w_{k-1}, w_{j+1}> + <w_{k-1}, w_{j-1}> - <w_{k-2}, w_j>,
//   <w_k, w_0> = 2 <w_{k-1}, w_1> - <w_{k-2}, w_0>,
// and, with B g = ((1 - d) g - w_0) / d (from w_0 = g - A g, A = d (I + B)),
//   <g, w_1> = ((1 - d) <g, w_0> - <w_0, w_0>) / d,
//   <g, w_{j+1}> = 2 ((1 - d) <g, w_j> - <w_0, w_j>) / d - <g, w_{j-1}>.
// The last pass needs one dot of its source, <S w_{m-1}, w_{m-1}>: it reads one
// vector where dots with all of w_0 .. w_{m-1} and g read mloop + 1.
// The order m is a template parameter, so that the small arrays stay in
// registers (6.3 us a launch; 14.8 with run-time loops over local memory).
template <int m>
__global__ void __launch_bounds__(128) s_sstep(CGScal s, SSPart pt, double* __restrict__ cz_out, int nb, double d,
                                               double dV, int first) {
    grid_dependency();
    const int b = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (b >= nb || !s.active[b]) return;  // uniform per warp
    double S[m + 1][3];
#pragma unroll
    for (int k = 0; k <= m; ++k) {
        const int D = pt.dots[k];
        const double* p = pt.part[k] + (long)b * pt.nch[k] * D;
#pragma unroll
        for (int q = 0; q < 3; ++q) S[k][q] = q < D ? warp_strided_sum(p + q, pt.nch[k], D, lane) : 0.0;
    }
    if (lane != 0) return;
    double G[m + 1][m + 1] = {}, gd[m] = {};
    G[0][0] = S[0][1];
#pragma unroll
    for (int k = 1; k <= m; ++k) {
        G[k][k] = S[k][1];
#pragma unroll
        for (int j = k - 1; j >= 0; --j) {
            double v;
            if (j == k - 1)  // the last pass leaves <S w_{m-1}, w_{m-1}>
                v = k == m && k >= 2 ? S[k][0] - G[k >= 2 ? k - 2 : 0][j] : S[k][0];
            else if (j == k - 2 && pt.dots[k] == 3)
                v = S[k][2];
            else if (j == 0)
                v = 2.0 * G[k - 1][1] - G[k >= 2 ? k - 2 : 0][0];
            else
                v = G[k - 1][j + 1] + G[k - 1][j > 0 ? j - 1 : 0] - G[k >= 2 ? k - 2 : 0][j];
            G[k][j] = G[j][k] = v;
        }
    }
    gd[0] = S[0][0];
#pragma unroll
    for (int j = 1; j < m; ++j) {
        const double t = ((1.0 - d) * gd[j - 1] - G[0][j - 1]) / d;
        gd[j] = j == 1 ? t : 2.0 * t - gd[j >= 2 ? j - 2 : 0];
    }
    double cz[m + 1] = {};
    double rr = G[0][0];
    if (!(rr < 1e-24)) {
        double r[m + 1] = {}, q[m + 1] = {}, ft[m + 1];
        r[0] = q[0] = 1.0;
#pragma unroll
        for (int il = 1; il <= m; ++il) {
            // ft = A q in the basis
#pragma unroll
            for (int i = 0; i <= m; ++i) ft[i] = d * q[i];
            ft[1] += d * q[0];
#pragma unroll
            for (int j = 1; j < m; ++j) {
                ft[j + 1] += 0.5 * d * q[j];
                ft[j - 1] += 0.5 * d * q[j];
            }
            double pAp = 0.0;
#pragma unroll
            for (int i = 0; i <= m; ++i)
#pragma unroll
                for (int j = 0; j <= m; ++j) pAp += q[i] * G[i][j] * ft[j];
            const double a = rr / pAp;
#pragma unroll
            for (int i = 0; i <= m; ++i) cz[i] += a * q[i];
            if (il == m) break;
#pragma unroll
            for (int i = 0; i <= m; ++i) r[i] -= a * ft[i];
            double rn = 0.0;
#pragma unroll
            for (int i = 0; i <= m; ++i)
#pragma unroll
                for (int j = 0; j <= m; ++j) rn += r[i] * G[i][j] * r[j];
            const double bb = rn / rr;
            rr = rn;
#pragma unroll
            for (int i = 0; i <= m; ++i) q[i] = r[i] + bb * q[i];
        }
    }
    double gz = 0.0;
#pragma unroll
    for (int j = 0; j < m; ++j) gz += cz[j] * gd[j];
    const double rb = s.rb[b] + dV * gz;
    s.rb[b] = rb;
    s.bk[b] = first ? 0.0 : rb / s.gkgk[b];
    s.gkgk[b] = rb;
#pragma unroll
    for (int j = 0; j < SS_MAXM; ++j) cz_out[(long)b * SS_MAXM + j] = j < m ? cz[j < m ? j : 0] : 0.0;
}

// p = g + sum_j cz_j w_j (+ bk p after the first step), the previous step's x
// update, and the line search's five dots of x, p and g (cg_module.f90:
// 268-297): <x|x>, <p|x>, <p|p>, <x|g>, <p|g>.  All three vectors are in
// registers here, so the dots cost no memory traffic; with g = -2 (H x - E x)
// they give <x|Hx> = E <x|x> - <x|g> / 2 and <p|Hx> = E <p|x> - <p|g> / 2,
// and <p|H p> comes from the H p kernels.  In the first step (hx given) the
// last two dots are <x|Hx> and <p|Hx> themselves: x may come in unnormalised,
// E is then no Rayleigh quotient and the identity would cancel (1.7e-12 in
// the residuals of a band of norm 27, against 1e-15 this way).
template <typename T, int M, int IT>
__global__ void __launch_bounds__(VT) k_ss_p(const T* __restrict__ g, const T* __restrict__ hx, SSVec<T> sv,
                                             T* __restrict__ p, T* __restrict__ x, long ld, long n, const double* cz,
                                             const double* bk_,
                                             const int* active, const int* pend,
                                             const double* u11_, const double* u21_,
                                             double* __restrict__ part, int vec) {
    grid_dependency();
    using G = Grp16<T>;
    constexpr int W = G::W;
    __shared__ double sh[5 * (VT / 32)];
    const int b = blockIdx.y;
    const bool act = active[b];
    const bool upd = pend && pend[b];  // the previous step's x update, which needs the old p
    if (!act && !upd) return;
    const int items = vec_items<IT>(n);
    const long off = (long)b * ld, base = (long)blockIdx.x * (VT * items);
    T c[M];
#pragma unroll
    for (int j = 0; j < M; ++j) c[j] = (T)cz[(long)b * SS_MAXM + j];
    const T bk = (T)bk_[b];
    const T u11 = upd ? (T)u11_[b] : (T)0, u21 = upd ? (T)u21_[b] : (T)0;
    const bool first = hx != nullptr, old = upd || !first;
    double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    auto elem = [&](T& xv, T& pv, T gv, T hv, const T* w) {
        if (upd) xv = cg_upd2_elem(xv, pv, u11, u21);
        T pg = gv;
#pragma unroll
        for (int j = 0; j < M; ++j) pg += c[j] * w[j];
        pv = first ? pg : pg + bk * pv;
        const double xd = (double)xv, pd = (double)pv, gd = (double)(first ? hv : gv);
        acc[0] = fma(xd, xd, acc[0]);
        acc[1] = fma(pd, xd, acc[1]);
        acc[2] = fma(pd, pd, acc[2]);
        acc[3] = fma(xd, gd, acc[3]);
        acc[4] = fma(pd, gd, acc[4]);
    };
#pragma unroll 2
    for (int it = 0; it < items / W; ++it) {
        const long i = base + ((long)it * VT + threadIdx.x) * W;
        if (vec && i + W <= n) {
            T pv[W], xv[W];
#pragma unroll
            for (int q = 0; q < W; ++q) pv[q] = (T)0;
            if (old) G::load(p + off + i, pv);
            G::load(x + off + i, xv);
            if (!act) {
#pragma unroll
                for (int q = 0; q < W; ++q) xv[q] = cg_upd2_elem(xv[q], pv[q], u11, u21);
                G::store(x + off + i, xv);
                continue;
            }
            T gv[W], hv[W], wv[M][W];
            G::load(g + off + i, gv);
#pragma unroll
            for (int q = 0; q < W; ++q) hv[q] = (T)0;
            if (first) G::load(hx + off + i, hv);
#pragma unroll
            for (int j = 0; j < M; ++j) G::load(sv.w[j] + off + i, wv[j]);
#pragma unroll
            for (int q = 0; q < W; ++q) {
                T w[M];
#pragma unroll
                for (int j = 0; j < M; ++j) w[j] = wv[j][q];
                elem(xv[q], pv[q], gv[q], hv[q], w);
            }
            if (upd) G::store(x + off + i, xv);
            G::store(p + off + i, pv);
        } else {
            for (int q = 0; q < W && i + q < n; ++q) {
                const long k = off + i + q;
                T pv = old ? p[k] : (T)0, xv = x[k];
                if (!act) {
                    x[k] = cg_upd2_elem(xv, pv, u11, u21);
                    continue;
                }
                T w[M];
#pragma unroll
                for (int j = 0; j < M; ++j) w[j] = sv.w[j][k];
                elem(xv, pv, g[k], first ? hx[k] : (T)0, w);
                if (upd) x[k] = xv;
                p[k] = pv;
            }
        }
    }
    if (!act) return;
    block_sum_n<VT, 5>(acc, sh);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < 5; ++k) part[((long)b * gridDim.x + blockIdx.x) * 5 + k] = acc[k];
    }
}

// element-wise basis step K with `dots` dots (one in the last pass)
template <typename T>
static int launch_ss_basis(int K, int dots, dim3 vg, cudaStream_t st, const T* g, SSVec<T> sv, long ld, long n,
                           const PcArgs& pa, double* part, const int* act) {
    // FP64 takes three dots from K = 2 on (sstep_precond)
#define RS_SS_CASE(KK, DD)                                                                    \
    if constexpr (sizeof(T) == 4 || KK < 2 || DD != 2) {                                      \
        if (K == KK && dots == DD) {                                                          \
            launch(k_ss_basis<T, KK, DD>, vg, VT, 0, st, g, sv, ld, n, pa, part, act);        \
            return RSDFT_OK;                                                                  \
        }                                                                                     \
    }
    RS_SS_CASE(0, 2)
    RS_SS_CASE(1, 2)
    RS_SS_CASE(2, 2)
    RS_SS_CASE(3, 2)
    RS_SS_CASE(2, 3)
    RS_SS_CASE(3, 3)
    RS_SS_CASE(1, 1)
    RS_SS_CASE(2, 1)
    RS_SS_CASE(3, 1)
    RS_SS_CASE(4, 1)
#undef RS_SS_CASE
    set_error("s-step basis index %d", K);
    return RSDFT_EUNSUP;
}

// ------------------------------------------- TMA z-march basis kernel
// One basis step as a z march over the 7-point operator, the hpsi stencil's
// pattern with Md = 1: a CTA owns TY full-width rows of one band; a producer
// warp streams each source plane (TY + 2 rows, periodic y wrap split into
// boxes) into a ring of S shared-memory stages, together with the TY-row tile
// of w_{K-2} at the plane that completes there (K >= 2, not the last step).  Consumer threads own VX x 2
// points, push the z contributions into 3 rotating accumulators, and at the
// completed plane form w_K, store it and add the step's dot products; the
// CTA's dot partials are summed in a fixed order at the end.  Every vector
// element is read once from memory.
struct PcMaps {
    CUtensorMap full, edge, mid, wrap;  // source boxes of TY + 2, TY + 1, TY, 1 rows
    CUtensorMap aux[1];                 // epilogue operand, TY rows
};

template <int K, int D>
struct PcStep {
    static constexpr int NA = (D > 1 && K >= 2) ? 1 : 0;  // w_{K-2}
    // CTAs per SM: two (<= 85 registers, half the stage ring each); one with three
    // dots, which spill at 80 registers (48^3 x 160 FP64 103 us a pass with two,
    // 88 with one; 72^3 x 480 695 and 643)
    static constexpr int CTAS = D == 3 ? 1 : 2;
};

__device__ __forceinline__ int pc_pwrap(int i, int n) {
    i %= n;
    return i < 0 ? i + n : i;
}

template <typename T, int K, int D>
__global__ void __launch_bounds__(384, PcStep<K, D>::CTAS) k_pc_tma(const __grid_constant__ PcMaps maps,
                                                                      T* __restrict__ wout,
                                                   StencilCoef cf, int n1, int n2, int n3, long ld, int zlen0,
                                                   int nzc, int TY, int RS, int S, int ncw,
                                                   double* __restrict__ part, const int* active,
                                                   int* __restrict__ err) {
    grid_dependency();
    using VT = Vec16<T>;
    using V = typename VT::t;
    constexpr int VX = 16 / (int)sizeof(T);
    constexpr int BY = 2;
    constexpr int NP = VX * BY;
    constexpr int NV = 3;  // x window: x - VX .. x + 2 VX - 1
    constexpr int NA = PcStep<K, D>::NA;
    constexpr bool STORE = D > 1;
    extern __shared__ __align__(128) unsigned char smem[];
    const int ROWS = TY + 2;
    const int SE = (ROWS + NA * TY) * RS;
    T* stages = reinterpret_cast<T*>(smem);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)S * SE * sizeof(T));
    uint64_t* empty = full + S;
    double* red = reinterpret_cast<double*>(empty + S);  // ncw x D

    const int t = threadIdx.x;
    const int warp = t >> 5, lane = t & 31;
    const int band = blockIdx.y / nzc;
    const int zc = blockIdx.y - band * nzc;
    if (active && !active[band]) return;  // uniform per CTA
    const int y0 = blockIdx.x * TY;
    const int zs = zc * zlen0;
    const int zlen = min(zs + zlen0, n3) - zs;
    const int nk = zlen + 2;  // arrival k <-> source plane zs - 1 + k
    const long plane = (long)n1 * n2;

    if (t == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], ncw);
        }
        mbar_fence_init();
    }
    __syncthreads();

    if (warp == ncw) {
        // ------------------------------------------------------ producer
        bool ok = true;
        if (lane == 0) {
            const uint32_t b_tile = (uint32_t)((size_t)TY * RS * sizeof(T));
            const uint32_t b_src = (uint32_t)((size_t)ROWS * RS * sizeof(T));
            for (int k = 0; k < nk; ++k) {
                const int s = k % S;
                if (k >= S && !mbar_wait(&empty[s], ((k / S) - 1) & 1)) ok = false;
                T* dst = stages + (size_t)s * SE;
                const int zp = pc_pwrap(zs - 1 + k, n3);
                const bool inner = k >= 1 && k < 1 + zlen;
                const bool aux = k >= 2;
                fence_proxy_async_smem();
                mbar_arrive_expect_tx(&full[s], (inner ? b_src : b_tile) + (aux ? NA * b_tile : 0u));
                if (!inner) {
                    tma_load_4d(dst + RS, &maps.mid, 0, y0, zp, band, &full[s]);
                } else if (y0 - 1 >= 0 && y0 + TY + 1 <= n2) {
                    tma_load_4d(dst, &maps.full, 0, y0 - 1, zp, band, &full[s]);
                } else if (TY == n2) {
                    tma_load_4d(dst, &maps.wrap, 0, n2 - 1, zp, band, &full[s]);
                    tma_load_4d(dst + RS, &maps.mid, 0, 0, zp, band, &full[s]);
                    tma_load_4d(dst + (1 + TY) * RS, &maps.wrap, 0, 0, zp, band, &full[s]);
                } else if (y0 - 1 < 0) {
                    tma_load_4d(dst, &maps.wrap, 0, n2 - 1, zp, band, &full[s]);
                    tma_load_4d(dst + RS, &maps.edge, 0, 0, zp, band, &full[s]);
                } else {
                    tma_load_4d(dst, &maps.edge, 0, y0 - 1, zp, band, &full[s]);
                    tma_load_4d(dst + (TY + 1) * RS, &maps.wrap, 0, 0, zp, band, &full[s]);
                }
                if (aux) {
#pragma unroll
                    for (int a = 0; a < NA; ++a)
                        tma_load_4d(dst + (ROWS + a * TY) * RS, &maps.aux[a], 0, y0, zs + k - 2, band, &full[s]);
                }
            }
        }
        __syncwarp();
        if (!ok) atomicExch(err, 1);
        return;
    }

    // ---------------------------------------------------------- consumers
    const int nxv = n1 / VX;
    const int ncons = nxv * (TY / BY);
    const bool thr = t < ncons;
    const int px = thr ? t % nxv : 0, py = thr ? t / nxv : 0;
    const int x = VX * px, yl = BY * py;
    const int xw = x - VX;
    T* __restrict__ ob = STORE ? wout + (long)band * ld + (long)n1 * (y0 + yl) + x : nullptr;
    const T c0 = (T)cf.c0, cx = (T)cf.cx[0], cy = (T)cf.cy[0], cz = (T)cf.cz[0];

    T acc[3][NP], cprev[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        acc[0][i] = acc[1][i] = acc[2][i] = (T)0;
        cprev[i] = (T)0;
    }
    double dots[D];
#pragma unroll
    for (int k = 0; k < D; ++k) dots[k] = 0.0;

    bool ok = true;
    int s = 0, u = 0;
    uint32_t ph = 0;
    for (int k = 0; k < nk; ++k) {
        if (!mbar_wait(&full[s], ph)) ok = false;
        const T* st = stages + (size_t)s * SE;
        const bool inner = k >= 1 && k < 1 + zlen;  // uniform
        T c[NP], in[NP];
        if (inner) {
            const T* sp = st + yl * RS + x;
#pragma unroll
            for (int i = 0; i < NP; ++i) in[i] = (T)0;
#pragma unroll
            for (int j = 0; j < BY + 2; ++j) {
                T v[VX];
                VT::get(*reinterpret_cast<const V*>(sp + j * RS), v);
#pragma unroll
                for (int r = 0; r < BY; ++r) {
                    const int m = j - 1 - r;
                    if (m == 0) {
#pragma unroll
                        for (int e = 0; e < VX; ++e) c[r * VX + e] = v[e];
                    } else if (m == 1 || m == -1) {
#pragma unroll
                        for (int e = 0; e < VX; ++e) in[r * VX + e] += cy * v[e];
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < BY; ++r) {
                const T* rp = st + (1 + yl + r) * RS;
                T w[NV * VX];
#pragma unroll
                for (int j = 0; j < NV; ++j) {
                    if (j == 1) {
                        // the centre vector: the row's own, read with the y window
#pragma unroll
                        for (int e = 0; e < VX; ++e) w[VX + e] = c[r * VX + e];
                        continue;
                    }
                    int xx = xw + VX * j;
                    xx += xx < 0 ? n1 : (xx >= n1 ? -n1 : 0);
                    VT::get(*reinterpret_cast<const V*>(rp + xx), w + j * VX);
                }
#pragma unroll
                for (int e = 0; e < VX; ++e) in[r * VX + e] += cx * (w[VX + e - 1] + w[VX + e + 1]);
            }
#pragma unroll
            for (int i = 0; i < NP; ++i) in[i] += c0 * c[i];
        } else {
#pragma unroll
            for (int r = 0; r < BY; ++r)
                VT::get(*reinterpret_cast<const V*>(st + (1 + yl + r) * RS + x), c + r * VX);
        }
        // z pushes: output k + 1 (first touch) and k - 1 (last touch); slot = arrival mod 3
        T o[NP];
#define RS_PC_PUSH(U)                                                  \
    {                                                                  \
        _Pragma("unroll") for (int i = 0; i < NP; ++i) {               \
            acc[(U + 1) % 3][i] = cz * c[i];                           \
            acc[(U + 2) % 3][i] += cz * c[i];                          \
            if (inner) acc[U][i] += in[i];                             \
            o[i] = acc[(U + 2) % 3][i];                                \
        }                                                              \
    }
        if (u == 0)
            RS_PC_PUSH(0)
        else if (u == 1)
            RS_PC_PUSH(1)
        else
            RS_PC_PUSH(2)
#undef RS_PC_PUSH
        if (k >= 2) {
            // plane zs + k - 2 is complete: o = operator part of w_K there
            const long zo = plane * (zs + k - 2);
#pragma unroll
            for (int r = 0; r < BY; ++r) {
                T av[NA > 0 ? NA : 1][VX];
#pragma unroll
                for (int a = 0; a < NA; ++a)
                    VT::get(*reinterpret_cast<const V*>(st + (ROWS + a * TY + yl + r) * RS + x), av[a]);
                T wk[VX];
#pragma unroll
                for (int e = 0; e < VX; ++e) {
                    const int i = r * VX + e;
                    if constexpr (K == 0)
                        wk[e] = -o[i];
                    else if constexpr (K == 1 || !STORE)
                        wk[e] = o[i];
                    else
                        wk[e] = o[i] - av[0][e];
                    const double wd = (double)wk[e];
                    dots[0] = fma(wd, (double)cprev[i], dots[0]);
                    if constexpr (STORE) dots[1] = fma(wd, wd, dots[1]);
                    if constexpr (D == 3) dots[2] = fma(wd, (double)av[0][e], dots[2]);
                }
                if constexpr (STORE) {
                    if (thr) *reinterpret_cast<V*>(ob + zo + (long)r * n1) = VT::make(wk);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NP; ++i) cprev[i] = c[i];
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);  // this warp is done with the stage
        if (++s == S) {
            s = 0;
            ph ^= 1u;
        }
        if (++u == 3) u = 0;
    }
    // fixed-order reduction of the dot partials over the consumer warps
#pragma unroll
    for (int k = 0; k < D; ++k) {
        double v = thr ? dots[k] : 0.0;
#pragma unroll
        for (int o2 = 16; o2 > 0; o2 >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o2);
        if (lane == 0) red[warp * D + k] = v;
    }
    asm volatile("bar.sync 1, %0;" ::"r"(ncw * 32) : "memory");
    if (t == 0) {
        const int nchunk = gridDim.x * nzc;
        const int chunk = zc * gridDim.x + blockIdx.x;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            double v = 0.0;
            for (int w = 0; w < ncw; ++w) v += red[w * D + k];
            part[((long)band * nchunk + chunk) * D + k] = v;
        }
    }
    if (!ok) atomicExch(err, 1);
}

// Geometry of k_pc_tma: TY (even, divides n2, n2 == TY or n2 >= TY + 1), row
// pitch RS (n1 rounded up to 128 bytes), ring depth S (2..8), consumer warps
// and the z split.  Chosen by march_cost as for the H psi stencil.
struct PcGeom {
    int TY = 0, RS = 0, S = 0, ncw = 0, threads = 0, nzc = 1;
    size_t smem = 0;
};

template <typename T>
static PcGeom pc_geometry(int n1, int n2, int n3, int mb, int sms, int part_cap, int na, int d, int ctas) {
    PcGeom best;
    constexpr int VX = 16 / (int)sizeof(T);
    const int RS = (int)((((size_t)n1 * sizeof(T) + 127) / 128) * 128 / sizeof(T));
    if (n1 % VX != 0 || n1 < VX || RS > 256 || n2 < 2) return best;
    double best_cost = 0.0;
    for (int TY = 2; TY <= std::min(n2, 254); TY += 2) {
        if (n2 % TY != 0 || !(TY == n2 || n2 >= TY + 1)) continue;
        const int ncw = ((n1 / VX) * (TY / 2) + 31) / 32;
        const int threads = 32 * (ncw + 1);
        if (threads > 384) continue;
        const size_t stage = (size_t)(TY + 2 + na * TY) * RS * sizeof(T);
        const size_t fixed = (size_t)ncw * d * sizeof(double);
        const size_t budget = (ctas > 1 ? 110 : 220) * 1024;
        if (budget <= fixed) continue;
        const int S = (int)std::min<size_t>((budget - fixed) / (stage + 16), 8);
        if (S < 2) continue;
        const int tiles = n2 / TY;
        const int zmax = std::min({std::max(1, n3 / 4), 65535 / mb, part_cap / tiles});
        int nzc = 1;
        if (zmax < 1) continue;
        // cycles per plane: shared-memory wavefronts (window and epilogue
        // loads, TMA fill) or the SM's share of HBM, times the CTAs sharing it
        const double row = RS * sizeof(T);
        const double lds = 1.1 * (ncw * 4.0 * (8 + 2 * na) + (TY + 2 + na * TY) * row / 128.0);
        const double hbm = (TY + 2 + (na + 1) * TY) * row / 23.0;
        const double t = 400.0 + ctas * std::max(lds, hbm);
        const double cost = march_cost((long)tiles * mb, n3, 2, zmax, (long)ctas * sms, t, 0.3 * t, &nzc);
        if (best.TY == 0 || cost <= 1.05 * best_cost) {  // the taller tile at a near tie
            best_cost = best.TY == 0 ? cost : std::min(cost, best_cost);
            best.TY = TY;
            best.RS = RS;
            best.S = S;
            best.ncw = ncw;
            best.threads = threads;
            best.nzc = nzc;
            best.smem = (size_t)S * stage + (size_t)S * 16 + fixed;
        }
    }
    return best;
}

// Launch basis step K through k_pc_tma; *used = false when the shape or the
// pointers do not suit it (the caller then takes the element-wise kernels).
template <typename T, int K, int D>
static int pc_tma_step(const T* src, const T* const* aux, T* wout, const PcArgs& pa, long ld, int mb,
                       int plan_mb, const int* active, double* part, int part_cap, int* nchunk, bool* used) {
    Context& c = ctx();
    *used = false;
    constexpr int NA = PcStep<K, D>::NA;
    constexpr bool STORE = D > 1;
    const int n1 = pa.n1, n2 = pa.n2, n3 = pa.n3;
    const int sms = c.num_sms > 0 ? c.num_sms : 148;
    const PcGeom g = pc_geometry<T>(n1, n2, n3, plan_mb, sms, part_cap, NA, D, PcStep<K, D>::CTAS);
    if (g.TY == 0 || (ld * sizeof(T)) % 16 != 0) return RSDFT_OK;
    if (STORE && reinterpret_cast<uintptr_t>(wout) % 16 != 0) return RSDFT_OK;
    const int zlen = div_up(n3, g.nzc);
    const int nzc = div_up(n3, zlen);
    PcMaps maps;
    const CUtensorMapDataType dt = sizeof(T) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    const unsigned long long dims[4] = {(unsigned long long)n1, (unsigned long long)n2, (unsigned long long)n3,
                                        (unsigned long long)mb};
    const unsigned long long strides[3] = {(unsigned long long)n1 * sizeof(T),
                                           (unsigned long long)n1 * n2 * sizeof(T),
                                           (unsigned long long)ld * sizeof(T)};
    const unsigned int RS = (unsigned)g.RS, TY = (unsigned)g.TY;
    const unsigned int bf[4] = {RS, TY + 2, 1, 1}, be[4] = {RS, TY + 1, 1, 1}, bm[4] = {RS, TY, 1, 1},
                       bw[4] = {RS, 1, 1, 1};
    if (encode_tmap_4d(&maps.full, dt, src, dims, strides, bf) != RSDFT_OK ||
        encode_tmap_4d(&maps.edge, dt, src, dims, strides, be) != RSDFT_OK ||
        encode_tmap_4d(&maps.mid, dt, src, dims, strides, bm) != RSDFT_OK ||
        encode_tmap_4d(&maps.wrap, dt, src, dims, strides, bw) != RSDFT_OK)
        return RSDFT_OK;
    for (int a = 0; a < NA; ++a)
        if (encode_tmap_4d(&maps.aux[a], dt, aux[a], dims, strides, bm) != RSDFT_OK) return RSDFT_OK;
    RS_CHECK(set_smem_optin((const void*)k_pc_tma<T, K, D>, 220 * 1024 + 8 * 16));
    // coefficients of the operator part: (A - I) for w_0, B = offdiag / d for
    // w_1, 2 B for the later steps
    StencilCoef cf{};
    const double sc = K == 0 ? 1.0 : (K == 1 ? 1.0 / pa.d : 2.0 / pa.d);
    cf.c0 = K == 0 ? pa.d - 1.0 : 0.0;
    cf.cx[0] = sc * pa.c1;
    cf.cy[0] = sc * pa.c2;
    cf.cz[0] = sc * pa.c3;
    dim3 grid(n2 / g.TY, (unsigned)(mb * nzc));
    launch(k_pc_tma<T, K, D>, grid, g.threads, g.smem, c.stream, maps, wout, cf, n1, n2, n3, ld, zlen, nzc,
           g.TY, g.RS, g.S, g.ncw, part, active, c.err_flag);
    RS_LAUNCH();
    *nchunk = (n2 / g.TY) * nzc;
    *used = true;
    return RSDFT_OK;
}

// basis step K of the s-step form through the TMA kernel (runtime K)
template <typename T>
static int pc_tma_dispatch(int K, int dots, const T* g, const SSVec<T>& sv, const PcArgs& pa, long ld, int mb,
                           int plan_mb, const int* active, double* part, int part_cap, int* nchunk, bool* used) {
    const T* src = K == 0 ? g : sv.w[K - 1];
    const T* aux[1] = {K >= 2 ? sv.w[K - 2] : nullptr};
    T* wout = dots > 1 ? sv.w[K] : nullptr;
#define RS_PC_CASE(KK, DD)                                                                                  \
    if constexpr (sizeof(T) == 4 || KK < 2 || DD != 2) {                                                    \
        if (K == KK && dots == DD)                                                                          \
            return pc_tma_step<T, KK, DD>(src, aux, wout, pa, ld, mb, plan_mb, active, part, part_cap, nchunk, \
                                          used);                                                            \
    }
    RS_PC_CASE(0, 2)
    RS_PC_CASE(1, 2)
    RS_PC_CASE(2, 2)
    RS_PC_CASE(3, 2)
    RS_PC_CASE(2, 3)
    RS_PC_CASE(3, 3)
    RS_PC_CASE(1, 1)
    RS_PC_CASE(2, 1)
    RS_PC_CASE(3, 1)
    RS_PC_CASE(4, 1)
#undef RS_PC_CASE
    *used = false;
    return RSDFT_OK;
}

template <typename T>
int sstep_precond(const T* g, const T* hx, const SSVec<T>& sv, T* p, T* x, long ld, int mb, int plan_mb, int mloop,
                  const CGScal& s, double* cz, double* part, int part_cap, double* dots, const PcArgs& pa, double dV) {
    const Context& c = ctx();
    cudaStream_t st = c.stream;
    const long n = c.ml;
    const int nchunk = vec_chunks(n, plan_mb, c.num_sms > 0 ? c.num_sms : 148);
    const dim3 vg(nchunk, mb);
    // <w_k, w_{k-2}> as a dot or from the recurrence (s_sstep): w_0 .. w_2 of a
    // smooth residual are nearly parallel, and the recurrence holds for the
    // stored vectors to their rounding, whose effect on a dot falls as
    // 1 / sqrt(n).  Residuals against 64 bits, FP64 48^3: 6.1e-14 by the
    // recurrence, 3.8e-14 by the dot (85 | 88 us a pass at 160 bands).  FP32, time of
    // a sweep and error of its residuals by the recurrence | by the dot: 24^3 x 32
    // 329 us, 1.8e-6 | 335, 1.9e-6; 36^3 x 80 752, 1.6e-6 | 774, 1.4e-6; 48^3 x 160
    // 2231, 1.6e-6 | 2283, 1.5e-6; 64^3 x 300 8127, 1.2e-6 | 8295, 1.2e-6: within the
    // scatter of the errors, so only small grids, where it is cheap, keep the dot.
    const bool third = sizeof(T) == 8 || n <= 65536;
    SSPart pt{};
    // basis steps: TMA z march where the shape allows, element-wise otherwise
    for (int k = 0; k <= mloop; ++k) {
        const int D = k == mloop ? 1 : (k >= 2 && third ? 3 : 2);
        double* out = part + (size_t)k * 3 * part_cap * mb;
        bool used = false;
        int nch = 0;
        RS_CHECK(pc_tma_dispatch<T>(k, D, g, sv, pa, ld, mb, plan_mb, s.active, out, part_cap, &nch, &used));
        if (!used) {
            RS_CHECK(launch_ss_basis<T>(k, D, vg, st, g, sv, ld, n, pa, out, s.active));
            nch = nchunk;
        }
        pt.part[k] = out;
        pt.nch[k] = nch;
        pt.dots[k] = D;
    }
    const int gv = grp16_ok<T>(ld, {g, hx, p, x, sv.w[0], sv.w[1], sv.w[2], sv.w[3]}) ? 1 : 0;
    auto launch_p = [&](auto M) {
        constexpr int MM = decltype(M)::value;
        launch(s_sstep<MM>, div_up(mb, 4), 128, 0, st, s, pt, cz, mb, pa.d, dV, hx ? 1 : 0);
        launch(vec_full(n, nchunk) ? k_ss_p<T, MM, 32> : k_ss_p<T, MM, 0>, vg, VT, 0, st, g, hx, sv, p, x, ld, n, (const double*)cz,
               (const double*)s.bk, (const int*)s.active, (const int*)(hx ? nullptr : s.pend),
               (const double*)s.u11, (const double*)s.u21, dots, gv);
    };
    switch (mloop) {
        case 1: launch_p(std::integral_constant<int, 1>{}); break;
        case 2: launch_p(std::integral_constant<int, 2>{}); break;
        case 3: launch_p(std::integral_constant<int, 3>{}); break;
        case 4: launch_p(std::integral_constant<int, 4>{}); break;
        default: set_error("s-step mloop %d", mloop); return RSDFT_EUNSUP;
    }
    RS_LAUNCH();
    return RSDFT_OK;
}

template int sstep_precond<double>(const double*, const double*, const SSVec<double>&, double*, double*, long, int,
                                   int, int, const CGScal&, double*, double*, int, double*, const PcArgs&, double);
template int sstep_precond<float>(const float*, const float*, const SSVec<float>&, float*, float*, long, int, int, int,
                                  const CGScal&, double*, double*, int, double*, const PcArgs&, double);

}  // namespace rsdft
