// Nonlocal force and the adjoint of hpsi.
//
// Force (calc_force_ps_nloc2, ps_nloc2_module.f90:1601-1654, :1760-1773):
//   w0 = iuV (-2 occ_n dV^2) sum_j uV(j) psi_n(JJP(j))
//   wk = sum_j duVdR_k(j) psi_n(JJP(j))
//   F(k, a) += w0 wk   over bands n with occ_n != 0 and projectors lma in a.
// Adjoint of y = H psi for a cotangent chi (the vector-Jacobian product):
//   dL/dV(r)  = sum_n chi_n(r) psi_n(r)                 (op_localpot)
//   dL/dR_ak  = sum_n sum_{lma in a} iuV dV [(chi.dk uV)(uV.psi) + (chi.uV)(dk uV.psi)]
// With chi_n = occ_n dV psi_n the second line is dE/dR = -F.
//
// k_nl_grad takes a sphere group (up to 4 projectors on one point list) x
// FG_BANDS bands per CTA: the group's point indices and 16 values per point
// (uV and its three derivatives of each projector) are staged in shared
// memory once and every warp gathers two vectors at a time (two bands, or one
// band and its cotangent) against them, 32 dot products in registers.  A
// butterfly leaves dot product i in lane i, so the products t d and the sum
// over the warp's bands need no further reduction.  Warps, band chunks and
// the projectors of an atom are added in a fixed order: bit-reproducible.
// The bound is the gather of psi (a sphere's rows are ~9 points, so it pulls
// most of the array's lines).  216-atom cell, 480 bands: 857 us per call with
// one CTA per sphere (216 CTAs, the 16 values re-read from L2 for every
// band), 258 us this way.
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"

namespace rsdft {

constexpr int FW = 8;         // warps per CTA
constexpr int FG_BANDS = 32;  // bands per CTA
constexpr int FG_CH = 512;    // sphere points staged at a time

// part[chunk][lma * 3 + k] = the chunk's band sum of each projector
template <bool CHI>
__global__ void __launch_bounds__(FW * 32) k_nl_grad(const double* psi, const double* chi,
                                                     long ld, int nb, const double* occ, double cscale,
                                                     const int* __restrict__ grp_lma0, const int* __restrict__ grp_cnt,
                                                     const int* __restrict__ lma_ptr, const int* __restrict__ jjp,
                                                     const double* __restrict__ uv, const double* __restrict__ duv,
                                                     const int* __restrict__ iuv, double dV, int nzlma,
                                                     double* __restrict__ part, int* __restrict__ err) {
    grid_dependency();
    extern __shared__ __align__(16) double fg_sm[];  // 16 x FG_CH values, FG_CH indices
    double(*s_c)[FG_CH] = reinterpret_cast<double(*)[FG_CH]>(fg_sm);
    int* s_j = reinterpret_cast<int*>(fg_sm + 16 * FG_CH);
    __shared__ double sh[FW][16];
    constexpr int BPW = CHI ? 1 : 2;  // bands a warp takes at a time
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = blockIdx.x;
    const int l0 = grp_lma0[g], cnt = grp_cnt[g];
    const int js = lma_ptr[l0], n = lma_ptr[l0 + 1] - js;
    long off[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) off[q] = q < cnt ? lma_ptr[l0 + q] : js;
    const int b0 = blockIdx.y * FG_BANDS, b1 = min(nb, b0 + FG_BANDS);
    const int nrep = (FG_BANDS + FW * BPW - 1) / (FW * BPW);
    // dot product i = 16 w + 4 q + c of vector w: c = 0 uV, c = 1..3 its
    // derivatives, projector q; lane i owns it after the reduction
    double tot = 0.0;
    int staged = -1;
    for (int r = 0; r < nrep; ++r) {
        const int bw = b0 + (r * FW + warp) * BPW;
        const double* v[2];
        bool act[2];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const int b = CHI ? bw : bw + w;
            act[w] = b < b1 && (CHI || !occ || occ[b] != 0.0);
            v[w] = (CHI && w == 1 ? chi : psi) + (long)(act[w] ? b : 0) * ld;
        }
        double acc[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = 0.0;
        for (int c0 = 0; c0 < n; c0 += FG_CH) {
            const int m = min(FG_CH, n - c0);
            if (staged != c0) {  // the same for every thread
                __syncthreads();
                for (int i = threadIdx.x; i < m; i += FW * 32) {
                    s_j[i] = jjp[js + c0 + i];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const long e = off[q] + c0 + i;
                        s_c[4 * q][i] = q < cnt ? uv[e] : 0.0;
#pragma unroll
                        for (int k = 0; k < 3; ++k) s_c[4 * q + 1 + k][i] = q < cnt ? duv[3 * e + k] : 0.0;
                    }
                }
                __syncthreads();
                staged = c0;
            }
#pragma unroll 2
            for (int j = lane; j < m; j += 32) {
                const int jj = s_j[j];
                const bool in = RS_DCHECK(jj >= 0 && jj < ld, CK_NL_GRAD_POINT, jj, err);
                double x[2];
#pragma unroll
                for (int w = 0; w < 2; ++w) x[w] = act[w] && in ? v[w][jj] : 0.0;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const double u = s_c[i][j];
                    acc[i] = fma(u, x[0], acc[i]);
                    acc[16 + i] = fma(u, x[1], acc[16 + i]);
                }
            }
        }
        // 32 sums over 32 lanes: at each step a lane keeps the half of the
        // values whose index has its own bit, so lane i ends with sum i
#pragma unroll
        for (int s = 16; s >= 1; s >>= 1) {
            const bool upper = (lane & s) != 0;
#pragma unroll
            for (int j = 0; j < s; ++j) {
                const double give = upper ? acc[j] : acc[j + s], keep = upper ? acc[j + s] : acc[j];
                acc[j] = keep + __shfl_xor_sync(0xffffffffu, give, s);
            }
        }
        const double d = acc[0];
        const int q = (lane >> 2) & 3;
        const double wq = q < cnt ? iuv[l0 + q] * dV : 0.0;
        double c;
        if (CHI) {  // (chi.duV)(uV.psi) + (chi.uV)(duV.psi), one half per lane half
            c = wq * d * __shfl_sync(0xffffffffu, d, (lane ^ 16) & ~3);
        } else {
            const int b = bw + (lane >> 4);
            const double t = __shfl_sync(0xffffffffu, d, lane & ~3);
            c = b < b1 && occ[b] != 0.0 ? cscale * occ[b] * wq * t * d : 0.0;
        }
        c += __shfl_xor_sync(0xffffffffu, c, 16);
        if (bw < b1) tot += c;
    }
    if (lane < 16) sh[warp][lane] = tot;
    __syncthreads();
    if (threadIdx.x < 16 && (threadIdx.x & 3) != 0) {
        const int q = threadIdx.x >> 2, k = (threadIdx.x & 3) - 1;
        if (q < cnt) {
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < FW; ++w) s += sh[w][threadIdx.x];
            part[((long)blockIdx.y * nzlma + l0 + q) * 3 + k] = s;
        }
    }
}

// f(3 a + k): the projectors of atom a in order, each over its band chunks in
// order; one warp per atom component (the lanes take the chunks)
__global__ void k_atom_sum(const double* part, int nchunk, int nzlma, const int* __restrict__ atom_ptr,
                           const int* __restrict__ atom_lma, int natom, double* __restrict__ f) {
    grid_dependency();
    const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= natom * 3) return;
    const int a = i / 3, k = i % 3;
    double s = 0.0;
    for (int e = atom_ptr[a]; e < atom_ptr[a + 1]; ++e)
        for (int y = lane; y < nchunk; y += 32) s += part[((long)y * nzlma + atom_lma[e]) * 3 + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) f[i] = s;
}

// dL/dV(r) = sum_n chi_n(r) psi_n(r), chi_n = occ_n dV psi_n when chi == NULL
// A thread takes W consecutive points (16-byte loads when the layout allows).
// The bands that take part (occ != 0; all of them with chi) are listed in
// shared memory first, so that a trip over four of them is four independent
// loads with no branch between them; their terms are added in band order.
constexpr int VA_LIST = 1024;  // bands listed at a time

template <int W, bool CHI>
__global__ void __launch_bounds__(256) k_vloc_adjoint(const double* psi, const double* chi,
                                                      long ld, int nb, const double* occ, double dV,
                                                      long n, double* __restrict__ out) {
    grid_dependency();
    __shared__ int s_b[VA_LIST];
    __shared__ double s_o[VA_LIST];
    __shared__ int s_n;
    const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * W;
    const bool in = i < n;  // n is a multiple of W
    constexpr int U = 4;
    double s[W];
#pragma unroll
    for (int e = 0; e < W; ++e) s[e] = 0.0;
    auto load = [](const double* p, double (&v)[W]) {
        if constexpr (W == 2) {
            const double2 t = *reinterpret_cast<const double2*>(p);
            v[0] = t.x;
            v[1] = t.y;
        } else {
            v[0] = *p;
        }
    };
    for (int b0 = 0; b0 < nb; b0 += VA_LIST) {
        __syncthreads();
        if (threadIdx.x < 32) {  // one warp lists the bands in order
            int cnt = 0;
            for (int b = b0; b < min(nb, b0 + VA_LIST); b += 32) {
                const int bb = b + (int)threadIdx.x;
                const double o = bb < nb ? (CHI ? 1.0 : occ[bb]) : 0.0;
                const unsigned m = __ballot_sync(0xffffffffu, o != 0.0);
                if (o != 0.0) {
                    const int at = cnt + __popc(m & ((1u << threadIdx.x) - 1u));
                    s_b[at] = bb;
                    s_o[at] = o * dV;
                }
                cnt += __popc(m);
            }
            if (threadIdx.x == 0) s_n = cnt;
        }
        __syncthreads();
        if (!in) continue;
        const int cnt = s_n;
        int q = 0;
        auto trip = [&](auto NU) {
            constexpr int N = decltype(NU)::value;
            double v[N][W], x[N][W];
#pragma unroll
            for (int u = 0; u < N; ++u) {
                load(psi + (long)s_b[q + u] * ld + i, v[u]);
                if (CHI) load(chi + (long)s_b[q + u] * ld + i, x[u]);
            }
#pragma unroll
            for (int u = 0; u < N; ++u)
#pragma unroll
                for (int e = 0; e < W; ++e)
                    s[e] = CHI ? fma(x[u][e], v[u][e], s[e]) : fma(s_o[q + u] * v[u][e], v[u][e], s[e]);
        };
        for (; q + U <= cnt; q += U) trip(std::integral_constant<int, U>{});
        for (; q < cnt; ++q) trip(std::integral_constant<int, 1>{});
    }
    if (!in) return;
#pragma unroll
    for (int e = 0; e < W; ++e) out[i + e] = s[e];
}

static int vloc_adjoint(const double* psi, const double* chi, long ld, int nb, const double* occ, double dV, long n,
                        double* out) {
    cudaStream_t st = ctx().stream;
    const bool vec = n % 2 == 0 && ld % 2 == 0 && reinterpret_cast<uintptr_t>(psi) % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(chi) % 16 == 0;
    auto kern = vec ? (chi ? k_vloc_adjoint<2, true> : k_vloc_adjoint<2, false>)
                    : (chi ? k_vloc_adjoint<1, true> : k_vloc_adjoint<1, false>);
    launch(kern, div_up(n, (vec ? 2 : 1) * 256L), 256, 0, st, psi, chi, ld, nb, occ, dV, n, out);
    RS_LAUNCH();
    return RSDFT_OK;
}

static int nl_grad(const double* psi, const double* chi, long ld, int nb, const double* occ, double cscale,
                   double* f_dev) {
    Context& c = ctx();
    const int nchunk = div_up(nb, FG_BANDS);
    double* part = nullptr;
    RS_CHECK(workspace_t("force_part", (size_t)c.nzlma * 3 * nchunk, &part));
    const size_t smem = FG_CH * (16 * sizeof(double) + sizeof(int));
    auto kern = chi ? k_nl_grad<true> : k_nl_grad<false>;
    RS_CHECK(set_smem_optin((const void*)kern, (int)smem));
    launch(kern, dim3(c.ngroup, nchunk), FW * 32, smem, c.stream, psi, chi, ld, nb, occ, cscale,
           (const int*)c.grp_lma0, (const int*)c.grp_cnt, (const int*)c.lma_ptr, (const int*)c.jjp,
           (const double*)c.uv, (const double*)c.duv, (const int*)c.iuv, c.dV, c.nzlma, part, c.err_flag);
    RS_LAUNCH();
    launch(k_atom_sum, div_up(c.natom * 3, 4), 128, 0, c.stream, (const double*)part, nchunk, c.nzlma,
           (const int*)c.atom_ptr, (const int*)c.atom_lma, c.natom, f_dev);
    RS_LAUNCH();
    return RSDFT_OK;
}

}  // namespace rsdft

using namespace rsdft;

extern "C" {

int rsdft_gpu_force_nloc(int mi, const double* unk, long ld, int mb, const double* occ, double* force2) {
    RS_ENTRY();
    RS_CHECK(require_grid());
    Context& c = ctx();
    if (!c.nl_set || !c.duv) {
        set_error("force_nloc: nonlocal tables with duvdr are not set");
        return RSDFT_ENOTINIT;
    }
    if (mi != c.natom || ld < c.ml || mb < 1 || !occ || !force2) {
        set_error("force_nloc: bad arguments (MI=%d natom=%d)", mi, c.natom);
        return RSDFT_EINVAL;
    }
    double *d, *docc, *f;
    bool st;
    RS_CHECK(wf_acquire(unk, ld, mb, "force_unk", &d, &st));
    RS_CHECK(stage_in(occ, sizeof(double) * mb, "force_occ", (void**)&docc));
    RS_CHECK(workspace_t("force_out", (size_t)3 * mi, &f));
    if (c.nzlma > 0) {
        // w0 wk with w0 = iuV (-2 occ dV^2) t: cscale * occ * (iuV dV) * t * d
        RS_CHECK(nl_grad(d, nullptr, ld, mb, docc, -2.0 * c.dV, f));
    } else {
        RS_CUDA(cudaMemsetAsync(f, 0, sizeof(double) * 3 * mi, c.stream));
    }
    RS_CHECK(stage_out(force2, f, sizeof(double) * 3 * mi));
    return RSDFT_OK;
}

int rsdft_gpu_hpsi_adjoint(const double* psi, const double* chi, long ld, int nb, const double* occ, double* dl_dv,
                           double* dl_dr) {
    RS_ENTRY();
    RS_CHECK(require_grid());
    Context& c = ctx();
    if (ld < c.ml || nb < 1 || (!chi && !occ) || (!dl_dv && !dl_dr)) {
        set_error("hpsi_adjoint: bad arguments");
        return RSDFT_EINVAL;
    }
    if (dl_dr && (!c.nl_set || !c.duv)) {
        set_error("hpsi_adjoint: position gradient needs nonlocal tables with duvdr");
        return RSDFT_ENOTINIT;
    }
    double *dp, *dc = nullptr, *docc = nullptr, *gv = nullptr, *gr = nullptr;
    bool sp, sc = false;
    RS_CHECK(wf_acquire(psi, ld, nb, "adj_psi", &dp, &sp));
    if (chi) RS_CHECK(wf_acquire(chi, ld, nb, "adj_chi", &dc, &sc));
    if (occ) RS_CHECK(stage_in(occ, sizeof(double) * nb, "adj_occ", (void**)&docc));
    if (dl_dv) {
        RS_CHECK(workspace_t("adj_dv", (size_t)c.ml, &gv));
        RS_CHECK(vloc_adjoint(dp, dc, ld, nb, docc, c.dV, c.ml, gv));
        RS_CHECK(stage_out(dl_dv, gv, sizeof(double) * c.ml));
    }
    if (dl_dr) {
        RS_CHECK(workspace_t("adj_dr", (size_t)3 * c.natom, &gr));
        if (c.nzlma > 0) {
            // chi = occ dV psi: dE/dR = sum 2 occ dV (iuV dV) t d
            RS_CHECK(nl_grad(dp, dc, ld, nb, docc, 2.0 * c.dV, gr));
        } else {
            RS_CUDA(cudaMemsetAsync(gr, 0, sizeof(double) * 3 * c.natom, c.stream));
        }
        RS_CHECK(stage_out(dl_dr, gr, sizeof(double) * 3 * c.natom));
    }
    (void)sp;
    (void)sc;
    return RSDFT_OK;
}

int rsdft_gpu_calc_density(const double* unk, long ld, int mb, const double* occ, double* rho) {
    RS_ENTRY();
    RS_CHECK(require_grid());
    Context& c = ctx();
    if (ld < c.ml || mb < 1 || !occ || !rho) {
        set_error("calc_density: bad arguments");
        return RSDFT_EINVAL;
    }
    double *dp, *docc = nullptr, *dr = nullptr;
    bool sp;
    RS_CHECK(wf_acquire(unk, ld, mb, "adj_psi", &dp, &sp));
    RS_CHECK(stage_in(occ, sizeof(double) * mb, "adj_occ", (void**)&docc));
    RS_CHECK(workspace_t("adj_dv", (size_t)c.ml, &dr));
    // the V-part adjoint with unit volume element: sum_n occ_n psi_n^2
    RS_CHECK(vloc_adjoint(dp, nullptr, ld, mb, docc, 1.0, c.ml, dr));
    RS_CHECK(stage_out(rho, dr, sizeof(double) * c.ml));
    (void)sp;
    return RSDFT_OK;
}

}  // extern "C"
