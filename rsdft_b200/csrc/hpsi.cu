// hpsi on sm_100a: H psi = T psi + Vloc psi + V_nl psi for a batch of bands.
//
//  1. k_nl_project: uVunk(lma, b) = iuV dV sum_j uV(j) psi(JJP(j), b)
//     (ps_nloc2_op_module.f90:161-175), one sphere group x 32 bands per CTA.
//  2. k_stencil_tma: the Md-order periodic FD Laplacian (kinetic_sol_module.
//     f90:72-77, 129-149) fused with the Vloc multiply (localpot_module.f90:
//     73): TMA-fed plane ring, z "push" march with register accumulators.
//  3. k_nl_scatter: the nonlocal scatter-add (ps_nloc2_op_module.f90:
//     255-263) turned into a per-point gather over a point-major CSR, so every
//     sum is deterministic.
//  Row widths that tiled TMA cannot address run k_stencil_row, the same march
//  fed by cp.async; what neither takes runs k_stencil, a register-queue kernel
//  with per-plane halo loads and the scatter fused in its epilogue.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kernels.cuh"
#include "tma.cuh"
#include "tmap.cuh"
#include "vec16.cuh"

namespace rsdft {

__device__ __forceinline__ int pwrap(int i, int n) {
    i %= n;
    return i < 0 ? i + n : i;
}

// ------------------------------------------------------------ projection
// A CTA takes one sphere group (up to 4 projectors sharing a point list) and
// PJ_WARPS x PJ_BW bands (16: two per warp, measured faster than four at
// Si216 480 bands, where more CTAs hide the gather latency better).  The
// group's point indices and projector values are staged in shared memory a
// chunk at a time; each lane strides the points and issues its warp's bands'
// gathers together.  Per (band, projector) the lanes sum points lane,
// lane+32, ... in order, then a fixed xor-shuffle tree.
constexpr int PJ_BW = 2;    // bands per warp
constexpr int PJ_WARPS = 8;
constexpr int PJ_CH = 512;  // sphere points staged per pass (multiple of 32)

template <typename T>
__global__ void __launch_bounds__(256) k_nl_project(const T* __restrict__ psi, long ld, int nb,
                                                    const int* __restrict__ grp_lma0,
                                                    const int* __restrict__ grp_cnt,
                                                    const int* __restrict__ lma_ptr,
                                                    const int* __restrict__ jjp,
                                                    const double* __restrict__ uv,
                                                    const int* __restrict__ iuv, double dV,
                                                    double* __restrict__ uvunk, int nzlma,
                                                    const int* band_active, int* __restrict__ err) {
    grid_dependency();
    __shared__ int s_j[PJ_CH];
    __shared__ double s_u[4][PJ_CH];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = blockIdx.x;
    const int l0 = grp_lma0[g], cnt = grp_cnt[g];
    const int js = lma_ptr[l0], n = lma_ptr[l0 + 1] - js;
    int off[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) off[q] = q < cnt ? lma_ptr[l0 + q] : js;
    const int bw0 = (blockIdx.y * PJ_WARPS + warp) * PJ_BW;
    bool act[PJ_BW];
    const T* p[PJ_BW];
#pragma unroll
    for (int w = 0; w < PJ_BW; ++w) {
        const int b = bw0 + w;
        act[w] = b < nb && (!band_active || band_active[b]);
        p[w] = psi + (long)(act[w] ? b : 0) * ld;
    }
    double acc[PJ_BW][4];
#pragma unroll
    for (int w = 0; w < PJ_BW; ++w)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[w][q] = 0.0;
    for (int c0 = 0; c0 < n; c0 += PJ_CH) {
        const int m = min(PJ_CH, n - c0);
        __syncthreads();
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            s_j[i] = jjp[js + c0 + i];
#pragma unroll
            for (int q = 0; q < 4; ++q) s_u[q][i] = q < cnt ? uv[off[q] + c0 + i] : 0.0;
        }
        __syncthreads();
#pragma unroll 2
        for (int j = lane; j < m; j += 32) {
            const int jj = s_j[j];
            const bool in = RS_DCHECK(jj >= 0 && jj < ld, CK_NL_PROJECT_POINT, jj, err);
            double v[PJ_BW];
#pragma unroll
            for (int w = 0; w < PJ_BW; ++w) v[w] = act[w] && in ? (double)__ldg(p[w] + jj) : 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (q < cnt) {
                    const double u = s_u[q][j];
#pragma unroll
                    for (int w = 0; w < PJ_BW; ++w) acc[w][q] = fma(u, v[w], acc[w][q]);
                }
            }
        }
    }
#pragma unroll
    for (int w = 0; w < PJ_BW; ++w)
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) acc[w][q] += __shfl_xor_sync(0xffffffffu, acc[w][q], s);
    if (lane == 0) {
#pragma unroll
        for (int w = 0; w < PJ_BW; ++w) {
            if (!act[w]) continue;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q < cnt) uvunk[(long)(bw0 + w) * nzlma + l0 + q] = iuv[l0 + q] * dV * acc[w][q];
        }
    }
}

template <typename T>
static int launch_project(const T* psi, long ld, int nb, double* uvunk, const int* band_active, cudaStream_t st) {
    const Context& c = ctx();
    dim3 grid(c.ngroup, div_up(nb, PJ_WARPS * PJ_BW));
    launch_ordinary(k_nl_project<T>, grid, 256, 0, st, psi, ld, nb, c.grp_lma0, c.grp_cnt, c.lma_ptr, c.jjp, c.uv, c.iuv,
           c.dV, uvunk, c.nzlma, band_active, c.err_flag);
    RS_LAUNCH();
    return RSDFT_OK;
}

// -------------------------------------------------------------- stencil
template <typename T>
struct StencilArgs {
    const T* psi;
    T* hpsi;
    long ld;
    int n1, n2, n3;
    int zlen, nzc;
    int z0, nzo;  // output planes [z0, z0 + nzo) (0, n3 when nzo = 0)
    const T* vloc;
    const int* pt_ptr;
    const int* pt_lma;
    const T* pt_uv;
    const double* uvunk;
    int nzlma;
    const int* band_active;
    const int* band_map;  // optional: launch band -> data band
    const int* gpt_ptr;   // point-major CSR over sphere groups
    const int* gpt_grp;
    const T* gpt_uv4;
    double* dot;          // optional: [band][ndot] partial sums of <psi|H psi> over the CTAs of a band
    int ndot;
};

template <typename T, int MD, int TX>
__global__ void __launch_bounds__(TX * 16) k_stencil(StencilArgs<T> a, StencilCoef cf) {
    grid_dependency();
    constexpr int TY = 16, SX = TX + 2 * MD, SY = TY + 2 * MD, NT = TX * TY;
    __shared__ T tile[SY * SX];
    const int t = threadIdx.x;
    const int tx = t % TX, ty = t / TX;
    const int nzc = a.nzc;
    int band = blockIdx.z / nzc;
    const int zc = blockIdx.z - band * nzc;
    if (a.band_map) band = a.band_map[band];
    if (a.band_active && !a.band_active[band]) return;  // uniform per CTA
    const int n1 = a.n1, n2 = a.n2, n3 = a.n3;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
    const int x = x0 + tx, y = y0 + ty;
    const bool act = (x < n1) && (y < n2);
    const long plane = (long)n1 * n2;
    const T* __restrict__ p = a.psi + (long)band * a.ld;
    T* __restrict__ h = a.hpsi + (long)band * a.ld;
    const int zs = a.z0 + zc * a.zlen;
    const int ze = min(zs + a.zlen, a.z0 + a.nzo);
    const long col = act ? (long)x + (long)n1 * y : 0;

    T cx[MD], cy[MD], cz[MD];
#pragma unroll
    for (int m = 0; m < MD; ++m) {
        cx[m] = (T)cf.cx[m];
        cy[m] = (T)cf.cy[m];
        cz[m] = (T)cf.cz[m];
    }
    const T c0 = (T)cf.c0;

    double dot = 0.0;
    T q[2 * MD + 1];
#pragma unroll
    for (int k = 0; k < 2 * MD; ++k) q[k] = act ? __ldg(p + col + plane * pwrap(zs - MD + k, n3)) : (T)0;

    for (int z = zs; z < ze; ++z) {
        q[2 * MD] = act ? __ldg(p + col + plane * pwrap(z + MD, n3)) : (T)0;
        __syncthreads();
        if (act) tile[(ty + MD) * SX + tx + MD] = q[MD];
        const T* pz = p + plane * z;
        for (int c = t; c < SY * SX; c += NT) {
            const int sy = c / SX, sx = c - sy * SX;
            const int otx = sx - MD, oty = sy - MD;
            const bool interior = (otx >= 0 && otx < TX && oty >= 0 && oty < TY && x0 + otx < n1 && y0 + oty < n2);
            if (!interior) {
                const int gx = pwrap(x0 + otx, n1), gy = pwrap(y0 + oty, n2);
                tile[c] = __ldg(pz + gx + (long)n1 * gy);
            }
        }
        __syncthreads();
        if (act) {
            const T* row = tile + (ty + MD) * SX + tx + MD;
            T v = c0 * q[MD];
#pragma unroll
            for (int m = 1; m <= MD; ++m) {
                v = v + cx[m - 1] * (row[-m] + row[m]) + cy[m - 1] * (row[-m * SX] + row[m * SX]) +
                    cz[m - 1] * (q[MD - m] + q[MD + m]);
            }
            const long j = col + plane * z;
            v = v + __ldg(a.vloc + j) * q[MD];
            if (a.pt_ptr) {
                const int s = __ldg(a.pt_ptr + j), e = __ldg(a.pt_ptr + j + 1);
                const double* un = a.uvunk + (long)band * a.nzlma;
                for (int k = s; k < e; ++k) v = v + __ldg(a.pt_uv + k) * (T)__ldg(un + __ldg(a.pt_lma + k));
            }
            h[j] = v;
            dot = fma((double)q[MD], (double)v, dot);
        }
#pragma unroll
        for (int k = 0; k < 2 * MD; ++k) q[k] = q[k + 1];
    }
    if (a.dot) {
        __shared__ double red[NT / 32];
        dot = block_sum<NT>(dot, red);
        if (t == 0)
            a.dot[(long)band * a.ndot + (long)zc * gridDim.x * gridDim.y + blockIdx.y * gridDim.x + blockIdx.x] = dot;
    }
}

struct TmaMaps {
    CUtensorMap full, edge, mid, wrap;  // psi boxes of height TY + 2 Md, TY + Md, TY, Md
    CUtensorMap vloc;                   // Vloc box of height TY
};

// Stencil coefficients in the kernel's arithmetic type, so every FMA takes
// its coefficient straight from the parameter bank (no per-use conversion).
template <typename T>
struct CoefT {
    T c0;
    T c0x, c0yz;  // c0 = c0x + c0yz exactly: x's own share of it, rounded to half the digits
    T cx[MAXMD], cy[MAXMD], cz[MAXMD];
};

template <typename T>
static CoefT<T> coef_as(const StencilCoef& cf) {
    CoefT<T> o{};
    o.c0 = (T)cf.c0;
    for (int m = 0; m < MAXMD; ++m) {
        o.cx[m] = (T)cf.cx[m];
        o.cy[m] = (T)cf.cy[m];
        o.cz[m] = (T)cf.cz[m];
    }
    double share = 0.0;
    for (int m = 0; m < MAXMD; ++m) share -= 2.0 * cf.cx[m];
    int e = 0;
    const double f = std::frexp(share, &e);
    constexpr int half = sizeof(T) == 8 ? 24 : 11;
    o.c0x = (T)std::ldexp(std::rint(std::ldexp(f, half)), e - half);
    o.c0yz = o.c0 - o.c0x;
    return o;
}

// Arithmetic lanes of the TMA stencil: one double, or two floats through the
// packed FP32 instructions of sm_100 (__ffma2_rn and friends: two
// independent IEEE operations per instruction, bitwise the same results as
// the scalar ones, half the issue slots).  A 16-byte shared-memory vector
// holds two packs in both cases.
template <typename T>
struct Pk;
template <>
struct Pk<double> {
    using t = double;
    static constexpr int W = 1;
    __device__ static __forceinline__ t fma(t a, t b, t c) { return __fma_rn(a, b, c); }
    __device__ static __forceinline__ t add(t a, t b) { return __dadd_rn(a, b); }
    __device__ static __forceinline__ t mul(t a, t b) { return __dmul_rn(a, b); }
    __device__ static __forceinline__ t splat(double v) { return v; }
    __device__ static __forceinline__ void dot(t a, t b, double& s) { s = __fma_rn(a, b, s); }
    __device__ static __forceinline__ t of(const double* p) { return p[0]; }
    __device__ static __forceinline__ void get2(const double2& v, t* o) {
        o[0] = v.x;
        o[1] = v.y;
    }
    __device__ static __forceinline__ double2 put2(const t* o) { return make_double2(o[0], o[1]); }
    __device__ static __forceinline__ void unpack2(const t* c, double* o) {
        o[0] = c[0];
        o[1] = c[1];
    }
};
template <>
struct Pk<float> {
    using t = float2;
    static constexpr int W = 2;
    __device__ static __forceinline__ t fma(t a, t b, t c) { return __ffma2_rn(a, b, c); }
    __device__ static __forceinline__ t add(t a, t b) { return __fadd2_rn(a, b); }
    __device__ static __forceinline__ t mul(t a, t b) { return __fmul2_rn(a, b); }
    __device__ static __forceinline__ t splat(float v) { return make_float2(v, v); }
    __device__ static __forceinline__ void dot(t a, t b, double& s) {
        s = __fma_rn((double)a.x, (double)b.x, s);
        s = __fma_rn((double)a.y, (double)b.y, s);
    }
    __device__ static __forceinline__ t of(const float* p) { return make_float2(p[0], p[1]); }
    __device__ static __forceinline__ void get2(const float4& v, t* o) {
        o[0] = make_float2(v.x, v.y);
        o[1] = make_float2(v.z, v.w);
    }
    __device__ static __forceinline__ float4 put2(const t* o) { return make_float4(o[0].x, o[0].y, o[1].x, o[1].y); }
    __device__ static __forceinline__ void unpack2(const t* c, float* o) {
        o[0] = c[0].x;
        o[1] = c[0].y;
        o[2] = c[1].x;
        o[3] = c[1].y;
    }
};

// One arrival's z pushes for accumulator slot U (compile time): outputs
// U + m (first touch at m = Md) and U - m get cz_m c, slot U gets the in-plane
// part when the plane is one of the tile's own, and slot U + Md + 1 (the
// output completed by this arrival) is written when hp is set.  NK packs per
// thread, two per row, written as one 16-byte vector, or (ROW: rows of any
// width) pack by pack, npk of each of the first nrow rows.
//
// DOT adds this plane's share of <psi|(T + Vloc) psi>.  Slot U holds
// sum_m cz_m psi(P - m) when plane P arrives; over the periodic grid the pairs
// (P, P - m) and (P, P + m) give equal sums, so the z part is twice
// psi(P) acc[U] and the dot needs no value that is not in registers here.
template <typename T, int MD, int NK, int BY, bool DOT, bool ROW, int U>
__device__ __forceinline__ void push_body(typename Pk<T>::t (&acc)[2 * MD + 1][NK], const typename Pk<T>::t* c,
                                          const typename Pk<T>::t* in, bool inner, const CoefT<T>& cf, T* hp,
                                          int n1, double& dot, int nrow, int npk) {
    using P = Pk<T>;
    constexpr int Q = 2 * MD + 1;
    if constexpr (DOT) {
        if (inner) {
#pragma unroll
            for (int i = 0; i < NK; ++i)
                if (!ROW || (i / 2 < nrow && i % 2 < npk)) P::dot(c[i], P::fma(P::splat((T)2), acc[U][i], in[i]), dot);
        }
    }
#pragma unroll
    for (int i = 0; i < NK; ++i) {
        acc[(U + MD) % Q][i] = P::mul(P::splat(cf.cz[MD - 1]), c[i]);
#pragma unroll
        for (int m = 1; m < MD; ++m) acc[(U + m) % Q][i] = P::fma(P::splat(cf.cz[m - 1]), c[i], acc[(U + m) % Q][i]);
#pragma unroll
        for (int m = 1; m <= MD; ++m)
            acc[(U + Q - m) % Q][i] = P::fma(P::splat(cf.cz[m - 1]), c[i], acc[(U + Q - m) % Q][i]);
        if (inner) acc[U][i] = P::add(acc[U][i], in[i]);
    }
    if (hp) {
#pragma unroll
        for (int r = 0; r < BY; ++r) {
            const typename P::t* o = &acc[(U + MD + 1) % Q][2 * r];
            if constexpr (!ROW) {
                *reinterpret_cast<typename Vec16<T>::t*>(hp + (long)r * n1) = P::put2(o);
            } else if (r < nrow) {
                *reinterpret_cast<typename P::t*>(hp + (long)r * n1) = o[0];
                if (npk > 1) *reinterpret_cast<typename P::t*>(hp + (long)r * n1 + P::W) = o[1];
            }
        }
    }
}

// Runtime slot -> compile-time slot: only the short push runs per case, so
// the loop body is not replicated 2 Md + 1 times.
template <typename T, int MD, int NK, int BY, bool DOT, bool ROW>
__device__ __forceinline__ void push_slot(int u, typename Pk<T>::t (&acc)[2 * MD + 1][NK], const typename Pk<T>::t* c,
                                          const typename Pk<T>::t* in, bool inner, const CoefT<T>& cf, T* hp,
                                          int n1, double& dot, int nrow = BY, int npk = 2) {
    constexpr int Q = 2 * MD + 1;
#define RS_PUSH_CASE(K)                                                                             \
    case K:                                                                                         \
        if constexpr (K < Q)                                                                        \
            push_body<T, MD, NK, BY, DOT, ROW, K>(acc, c, in, inner, cf, hp, n1, dot, nrow, npk);   \
        break;
    switch (u) {
        RS_PUSH_CASE(0) RS_PUSH_CASE(1) RS_PUSH_CASE(2) RS_PUSH_CASE(3) RS_PUSH_CASE(4) RS_PUSH_CASE(5)
        RS_PUSH_CASE(6) RS_PUSH_CASE(7) RS_PUSH_CASE(8) RS_PUSH_CASE(9) RS_PUSH_CASE(10) RS_PUSH_CASE(11)
        RS_PUSH_CASE(12) RS_PUSH_CASE(13) RS_PUSH_CASE(14) RS_PUSH_CASE(15) RS_PUSH_CASE(16)
        default: break;
    }
#undef RS_PUSH_CASE
}

// Threads of a march CTA: the register budget of the 2 Md + 1 accumulators (168
// per thread; three rows per thread take up to 255)
constexpr int march_threads(int by) { return by == 3 ? 256 : 384; }

// Order of the in-plane terms.  FP32: the y rows from the outermost inwards, x
// likewise, the centre last, so that few roundings are at the size of the large
// terms: the bands of a CG sweep (FP32, against FP64) at 24^3 were 4.4e-7 off
// with the terms in the order the rows lie in and 3.9e-7 this way, at 26^3 4.1e-7
// and 3.7e-7.  FP64 keeps the rows' order (72^3 x 480: 1625 us against 1667, and
// H psi of smooth bands no better).
template <typename T>
__device__ __forceinline__ constexpr int term_order(int i, int n) {
    return sizeof(T) == 8 ? i : (i % 2 == 0 ? i / 2 : n - 1 - i / 2);
}

// hpsi stencil + Vloc, TMA pipeline with a z "push" march.  A CTA owns TY
// full-width rows of one band and marches along z over planes zs-Md ..
// ze+Md-1.  One producer warp streams each plane (TY + 2 Md rows with the
// periodic y wrap split into boxes, plus the Vloc rows of the tile) into a
// ring of S shared-memory stages.  Each consumer thread owns VX (16 bytes)
// x BY points.  When plane P lands the thread
//  * forms the in-plane part of H psi at P (centre, Md x and y neighbours,
//    the x window read with periodic offsets, Vloc),
//  * adds cz_m psi(P) to the accumulators of the outputs P -+ m (m = 1..Md),
//  * and writes output P - Md, which is then complete.
// The 2 Md + 1 accumulators rotate through registers with compile-time
// indices (a switch on the slot selects the push), so a stage is read only
// while its own plane is current and the ring can stay shallow.
template <typename T, int MD, int BY, bool DOT>
__global__ void __launch_bounds__(march_threads(BY), 1)
    k_stencil_tma(const __grid_constant__ TmaMaps maps, StencilArgs<T> a, const CoefT<T> cf, int TY, int RS, int S,
                  int ncw, int* __restrict__ err) {
    grid_dependency();
    using VT = Vec16<T>;
    using V = typename VT::t;
    constexpr int VX = 16 / (int)sizeof(T);
    constexpr int MDX = (MD + VX - 1) / VX * VX;  // x window half-width, whole vectors
    constexpr int NV = 1 + 2 * MDX / VX;           // vectors in the x window
    constexpr int Q = 2 * MD + 1;                  // accumulator ring
    constexpr int NP = VX * BY;                    // points per thread
    extern __shared__ __align__(128) unsigned char smem[];
    const int n1 = a.n1, n2 = a.n2, n3 = a.n3;
    const int ROWS = TY + 2 * MD;
    const int SE = (ROWS + TY) * RS;  // elements per stage: psi rows, then Vloc rows
    T* stages = reinterpret_cast<T*>(smem);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)S * SE * sizeof(T));
    uint64_t* empty = full + S;

    const int t = threadIdx.x;
    const int warp = t >> 5, lane = t & 31;
    const int nzc = a.nzc;
    const int band = blockIdx.y / nzc;
    const int zc = blockIdx.y - band * nzc;
    if (a.band_active && !a.band_active[band]) return;  // uniform per CTA
    const int y0 = blockIdx.x * TY;
    const int zs = a.z0 + zc * a.zlen;
    const int zlen = min(zs + a.zlen, a.z0 + a.nzo) - zs;
    const int nk = zlen + 2 * MD;  // arrival k <-> plane zs - Md + k
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
            const uint32_t b_in = (uint32_t)((size_t)(ROWS + TY) * RS * sizeof(T));
            const uint32_t b_out = (uint32_t)((size_t)TY * RS * sizeof(T));
            for (int k = 0; k < nk; ++k) {
                const int s = k % S;
                if (k >= S && !mbar_wait(&empty[s], ((k / S) - 1) & 1)) ok = false;
                T* dst = stages + (size_t)s * SE;
                const int zp = pwrap(zs - MD + k, n3);
                const bool inner = k >= MD && k < MD + zlen;
                fence_proxy_async_smem();
                mbar_arrive_expect_tx(&full[s], inner ? b_in : b_out);
                if (!inner) {
                    // halo planes only feed the z accumulators: the TY own rows
                    tma_load_4d(dst + MD * RS, &maps.mid, 0, y0, zp, band, &full[s]);
                    continue;
                }
                if (y0 - MD >= 0 && y0 + TY + MD <= n2) {
                    tma_load_4d(dst, &maps.full, 0, y0 - MD, zp, band, &full[s]);
                } else if (TY == n2) {
                    tma_load_4d(dst, &maps.wrap, 0, n2 - MD, zp, band, &full[s]);
                    tma_load_4d(dst + MD * RS, &maps.mid, 0, 0, zp, band, &full[s]);
                    tma_load_4d(dst + (MD + TY) * RS, &maps.wrap, 0, 0, zp, band, &full[s]);
                } else if (y0 - MD < 0) {
                    tma_load_4d(dst, &maps.wrap, 0, n2 - MD, zp, band, &full[s]);
                    tma_load_4d(dst + MD * RS, &maps.edge, 0, 0, zp, band, &full[s]);
                } else {
                    tma_load_4d(dst, &maps.edge, 0, y0 - MD, zp, band, &full[s]);
                    tma_load_4d(dst + (TY + MD) * RS, &maps.wrap, 0, 0, zp, band, &full[s]);
                }
                tma_load_4d(dst + ROWS * RS, &maps.vloc, 0, y0, zp, 0, &full[s]);
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
    const int xw = x - MDX;  // first x of the periodic window
    T* __restrict__ hb = a.hpsi + (long)band * a.ld + (long)n1 * (y0 + yl) + x;
    using P = Pk<T>;
    using PT = typename P::t;
    constexpr int W = P::W;
    constexpr int NK = NP / W;  // packs per thread, two per row

    PT acc[Q][NK];
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int i = 0; i < NK; ++i) acc[q][i] = P::splat((T)0);

    bool ok = true;
    double dot = 0.0;
    int s = 0, u = 0;
    uint32_t ph = 0;
    for (int k = 0; k < nk; ++k) {
        if (!mbar_wait(&full[s], ph)) ok = false;
        const T* st = stages + (size_t)s * SE;
        const bool inner = k >= MD && k < MD + zlen;  // uniform
        PT c[NK], in[NK];
        if (inner) {
            const T* sp = st + yl * RS + x;
#pragma unroll
            for (int i = 0; i < NK; ++i) in[i] = P::splat((T)0);
            // y neighbours (the window also holds the thread's own rows)
#pragma unroll
            for (int jj = 0; jj < BY + 2 * MD; ++jj) {
                const int j = term_order<T>(jj, BY + 2 * MD);
                PT v[2];
                P::get2(*reinterpret_cast<const V*>(sp + j * RS), v);
#pragma unroll
                for (int r = 0; r < BY; ++r) {
                    const int m = j - MD - r;
                    if (m == 0) {
                        c[2 * r] = v[0];
                        c[2 * r + 1] = v[1];
                    } else if (m >= -MD && m <= MD) {
                        const PT cy = P::splat(cf.cy[(m > 0 ? m : -m) - 1]);
#pragma unroll
                        for (int e = 0; e < 2; ++e) in[2 * r + e] = P::fma(cy, v[e], in[2 * r + e]);
                    }
                }
            }
            // x neighbours from the periodic window of each own row (its
            // centre vector is the row's own, already read with the y window)
#pragma unroll
            for (int r = 0; r < BY; ++r) {
                const T* rp = st + (MD + yl + r) * RS;
                T w[NV * VX];
#pragma unroll
                for (int j = 0; j < NV; ++j) {
                    if (j == MDX / VX) {
                        P::unpack2(c + 2 * r, w + j * VX);
                        continue;
                    }
                    int xx = xw + VX * j;
                    xx += xx < 0 ? n1 : (xx >= n1 ? -n1 : 0);
                    VT::get(*reinterpret_cast<const V*>(rp + xx), w + j * VX);
                }
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int i = 1; i <= MD; ++i) {
                        const int m = sizeof(T) == 8 ? i : MD + 1 - i;
                        in[2 * r + e] = P::fma(P::splat(cf.cx[m - 1]),
                                               P::add(P::of(w + MDX + W * e - m), P::of(w + MDX + W * e + m)),
                                               in[2 * r + e]);
                    }
            }
            // centre and local potential
#pragma unroll
            for (int r = 0; r < BY; ++r) {
                PT vl[2];
                P::get2(*reinterpret_cast<const V*>(sp + (ROWS + r) * RS), vl);
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    in[2 * r + e] = P::fma(P::add(P::splat(cf.c0), vl[e]), c[2 * r + e], in[2 * r + e]);
            }
        } else {
#pragma unroll
            for (int r = 0; r < BY; ++r) P::get2(*reinterpret_cast<const V*>(st + (MD + yl + r) * RS + x), c + 2 * r);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);  // this warp is done with the stage
        // z pushes into the accumulator ring (slot = output arrival mod Q)
        // and, from arrival 2 Md on, the write of the completed output k - Md
        T* hp = (k >= 2 * MD && thr) ? hb + plane * (zs + k - 2 * MD) : nullptr;
        push_slot<T, MD, NK, BY, DOT, false>(u, acc, c, in, inner, cf, hp, n1, dot);
        if (++s == S) {
            s = 0;
            ph ^= 1u;
        }
        if (++u == Q) u = 0;
    }
    if constexpr (DOT) {
        // fixed-order sum over the consumer warps
        double* red = reinterpret_cast<double*>(empty + S);
        if (!thr) dot = 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (lane == 0) red[warp] = dot;
        asm volatile("bar.sync 1, %0;" ::"r"(ncw * 32) : "memory");
        if (t == 0) {
            double v = 0.0;
            for (int w = 0; w < ncw; ++w) v += red[w];
            a.dot[(long)band * a.ndot + zc * gridDim.x + blockIdx.x] = v;
        }
    }
    if (!ok) atomicExch(err, 1);
}

// The same z march for row widths that tiled TMA cannot address (strides that
// are no multiple of 16 bytes: odd widths in FP64, odd multiples of 2 in
// FP32).  Planes come in by 8-byte cp.async of all threads, one barrier per
// plane, into 16-byte aligned rows with the periodic x neighbours beside them,
// so every window load is a vector at a constant offset; y and z wrap where the
// rows are fetched, any n2 and n3.  The last vector of a row may stand half
// outside the grid; what lies there is computed and not stored.
//
// Order of the sum: symmetric pairs from the outermost inwards, x with its own
// share of the centre weight and Vloc, y with the rest of it, so that the large
// terms cancel before the sums meet.  Relative error of H psi against 80 bits,
// smooth bands at 45^3, Md = 6: 7.7e-16 with k_stencil (pairs, the innermost
// first), 6.6e-16 this way, 1.5e-15 with the y rows one by one and c0 + Vloc as one
// factor.
//
// Bound, as the TMA kernel's, by the shared-memory window loads and, with 10 to
// 12 warps per SM, their latency.  H psi at 45^3 x 101 FP64: 394 us with
// k_stencil (16 x 32 tiles re-reading their halo every plane, a quarter of the
// tiles' points outside the grid), 245 us with a thread on one x column (8-byte
// loads, 17 per point against 7 here of 16 bytes), 220 us this way.
constexpr int RS_STAGES = 3;  // planes of k_stencil_row's ring

template <typename T, int MD, int BY, bool DOT>
__global__ void __launch_bounds__(192, 2) k_stencil_row(StencilArgs<T> a, const CoefT<T> cf, int TY) {
    grid_dependency();
    using P = Pk<T>;
    using PT = typename P::t;
    using VT = Vec16<T>;
    using V = typename VT::t;
    constexpr int W = P::W;
    constexpr int VX = 2 * W;                      // values per 16-byte vector
    constexpr int HX = (MD + VX - 1) / VX * VX;    // x halo, whole vectors
    constexpr int NV = 1 + 2 * HX / VX;            // vectors in the x window
    constexpr int Q = 2 * MD + 1;
    constexpr int S = RS_STAGES;
    extern __shared__ __align__(128) unsigned char smem[];
    const int n1 = a.n1, n2 = a.n2, n3 = a.n3;
    const int nxv = (n1 + VX - 1) / VX;
    const int PX = nxv * VX + 2 * HX;
    const int ROWS = TY + 2 * MD;
    const int SE = (ROWS + TY) * PX;  // elements per stage: psi rows, then Vloc rows
    T* stages = reinterpret_cast<T*>(smem);
    const int t = threadIdx.x;
    const int nzc = a.nzc;
    const int band = blockIdx.y / nzc;
    const int zc = blockIdx.y - band * nzc;
    if (a.band_active && !a.band_active[band]) return;  // uniform per CTA
    const int y0 = blockIdx.x * TY;
    const int ny = min(TY, n2 - y0);
    const int zs = a.z0 + zc * a.zlen;
    const int zlen = min(zs + a.zlen, a.z0 + a.nzo) - zs;
    const int nk = zlen + 2 * MD;  // arrival k <-> plane zs - Md + k
    const long plane = (long)n1 * n2;
    const T* __restrict__ src = a.psi + (long)band * a.ld;
    const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(stages));
    // where each pack of a stage lies in its plane (the same for every plane;
    // -1: not used), so that a plane's copies cost a table look-up each
    int* goff = reinterpret_cast<int*>(smem + (size_t)S * SE * sizeof(T));
    for (int e = t; e < SE / W; e += blockDim.x) {
        const int r = e * W / PX, x = e * W - r * PX - HX;
        int g = -1;
        if (r < ROWS) {
            if (r < ny + 2 * MD) g = n1 * pwrap(y0 - MD + r, n2) + pwrap(x, n1);
        } else if (r - ROWS < ny && x >= 0 && x < n1) {
            g = n1 * (y0 + r - ROWS) + x;
        }
        goff[e] = g;
    }
    // columns no copy ever fills (Vloc past the grid) hold zeros, not NaNs
    for (int e = t; e < S * SE; e += blockDim.x) stages[e] = (T)0;
    __syncthreads();
    auto load_plane = [&](int k) {
        if (k < nk) {
            const uint32_t st = sbase + (uint32_t)((k % S) * SE) * (uint32_t)sizeof(T);
            const int zp = pwrap(zs - MD + k, n3);
            const bool inner = k >= MD && k < MD + zlen;
            const T *pz = src + plane * zp, *vz = a.vloc + plane * zp;
            // halo planes only feed the z accumulators: the own rows
            const int e0 = inner ? 0 : MD * PX / W, e1 = inner ? SE / W : (MD + ny) * PX / W, ev = ROWS * PX / W;
#pragma unroll 4
            for (int e = e0 + t; e < e1; e += blockDim.x) {
                const int g = goff[e];
                if (g >= 0)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(st + (uint32_t)e * 8u),
                                 "l"((e < ev ? pz : vz) + g)
                                 : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const bool thr = t < nxv * (TY / BY);
    const int px = thr ? t % nxv : 0, py = thr ? t / nxv : 0;
    const int x = VX * px, yl = BY * py;
    const int nrow = thr ? max(0, min(BY, ny - yl)) : 0;  // rows of this thread inside the grid
    const int npk = x + W < n1 ? 2 : 1;                    // packs of its vector inside the grid
    T* __restrict__ hb = a.hpsi + (long)band * a.ld + (long)n1 * (y0 + yl) + x;

    constexpr int NK = 2 * BY;
    PT acc[Q][NK];
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int i = 0; i < NK; ++i) acc[q][i] = P::splat((T)0);
    double dot = 0.0;
    // two planes in flight while one is used
    load_plane(0);
    load_plane(1);
    int u = 0;
    for (int k = 0; k < nk; ++k) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();  // plane k has landed for everyone; plane k - 1's stage is free
        load_plane(k + 2);
        const T* st = stages + (size_t)(k % S) * SE;
        const bool inner = k >= MD && k < MD + zlen;  // uniform
        const T* sp = st + (MD + yl) * PX + HX + x;    // the thread's first row
        PT c[NK], in[NK];
#pragma unroll
        for (int r = 0; r < BY; ++r) P::get2(*reinterpret_cast<const V*>(sp + r * PX), c + 2 * r);
        if (inner) {
            // y pairs (row r - m + row r + m), each row loaded where the order
            // first meets it
            PT v[BY + 2 * MD][2];
            auto row = [&](int j, bool first, int e) -> PT {
                if (j >= 0 && j < BY) return c[2 * (j >= 0 && j < BY ? j : 0) + e];
                if (first && e == 0) P::get2(*reinterpret_cast<const V*>(sp + j * PX), v[j + MD]);
                return v[j + MD][e];
            };
#pragma unroll
            for (int i = 0; i < NK; ++i) in[i] = P::splat((T)0);
#pragma unroll
            for (int m = MD; m >= 1; --m)
#pragma unroll
                for (int r = 0; r < BY; ++r)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const PT lo = row(r - m, r == BY - 1 || m == MD, e), hi = row(r + m, r == 0 || m == MD, e);
                        in[2 * r + e] = P::fma(P::splat(cf.cy[m - 1]), P::add(lo, hi), in[2 * r + e]);
                    }
#pragma unroll
            for (int r = 0; r < BY; ++r) {
                T w[NV * VX];
#pragma unroll
                for (int j = 0; j < NV; ++j) {
                    if (j == HX / VX)
                        P::unpack2(c + 2 * r, w + j * VX);
                    else
                        VT::get(*reinterpret_cast<const V*>(sp + r * PX - HX + VX * j), w + j * VX);
                }
                PT vl[2];
                P::get2(*reinterpret_cast<const V*>(sp + (ROWS - MD + r) * PX), vl);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    PT ix = P::splat((T)0);
#pragma unroll
                    for (int m = MD; m >= 1; --m)
                        ix = P::fma(P::splat(cf.cx[m - 1]), P::add(P::of(w + HX + W * e - m), P::of(w + HX + W * e + m)),
                                    ix);
                    ix = P::fma(vl[e], c[2 * r + e], P::fma(P::splat(cf.c0x), c[2 * r + e], ix));
                    in[2 * r + e] = P::add(ix, P::fma(P::splat(cf.c0yz), c[2 * r + e], in[2 * r + e]));
                }
            }
        }
        T* hp = (k >= 2 * MD && nrow > 0) ? hb + plane * (zs + k - 2 * MD) : nullptr;
        push_slot<T, MD, NK, BY, DOT, true>(u, acc, c, in, inner, cf, hp, n1, dot, nrow, npk);
        if (++u == Q) u = 0;
    }
    if constexpr (DOT) {
        __shared__ double red[6];
        const int warp = t >> 5, lane = t & 31, nw = blockDim.x >> 5;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (lane == 0) red[warp] = dot;
        __syncthreads();
        if (t == 0) {
            double v = 0.0;
            for (int w = 0; w < nw; ++w) v += red[w];
            a.dot[(long)band * a.ndot + zc * gridDim.x + blockIdx.x] = v;
        }
    }
}

// Nonlocal scatter after the stencil: hpsi(p, b) += sum over the sphere
// groups g covering p of sum_q uV(p, g, q) uVunk(g + q, b)
// (ps_nloc2_op_module.f90:255-263), one thread per covered point and a chunk
// of bands, SC_BU bands in flight at once (2: measured faster than 4 and 8).
// A point's entries are taken in projector order, so every sum has a fixed
// order.  Launched as a dependent of the stencil, whose H psi it reads through a
// plain pointer; uVunk is the projection's, complete before the stencil began.
constexpr int SC_BU = 2;

template <typename T>
__global__ void __launch_bounds__(128) k_nl_scatter(T* hpsi, long ld, int nb, int bchunk,
                                                   const int* __restrict__ nl_pts, const int* __restrict__ nl_ptr,
                                                   int npt, const int* __restrict__ gpt_grp,
                                                   const T* __restrict__ gpt_uv4, const double* __restrict__ uvunk,
                                                   int nzlma, const int* __restrict__ band_active,
                                                   int* __restrict__ err) {
    grid_dependency();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npt) return;
    const int p = nl_pts[i];
    if (!RS_DCHECK(p >= 0 && p < ld, CK_NL_SCATTER_POINT, p, err)) return;
    const int e0 = nl_ptr[i], e1 = nl_ptr[i + 1];
    const int b0 = blockIdx.y * bchunk, b1 = min(nb, b0 + bchunk);
    for (int b = b0; b < b1; b += SC_BU) {
        bool act[SC_BU];
        T o[SC_BU];
#pragma unroll
        for (int u = 0; u < SC_BU; ++u) {
            const int bb = b + u;
            act[u] = bb < b1 && (!band_active || band_active[bb]);
            o[u] = act[u] ? hpsi[(long)bb * ld + p] : (T)0;
        }
        for (int e = e0; e < e1; ++e) {
            // a group holds 1..4 projectors; missing ones have zero values
            // and must not be read past the end of uVunk
            const int g = __ldg(gpt_grp + e);
            if (!RS_DCHECK(g >= 0 && g < nzlma, CK_NL_SCATTER_GROUP, g, err)) continue;
            T uq[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) uq[q] = __ldg(gpt_uv4 + 4L * e + q);
#pragma unroll
            for (int u = 0; u < SC_BU; ++u) {
                if (!act[u]) continue;
                const double* un = uvunk + (long)(b + u) * nzlma;
                T c = uq[0] * (T)__ldg(un + g);
#pragma unroll
                for (int q = 1; q < 4; ++q)
                    if (g + q < nzlma) c += uq[q] * (T)__ldg(un + g + q);
                o[u] += c;
            }
        }
#pragma unroll
        for (int u = 0; u < SC_BU; ++u)
            if (act[u]) hpsi[(long)(b + u) * ld + p] = o[u];
    }
}

// Bands per scatter thread: 32, so that a point's entries are read from L1 for
// 15 of 16 band pairs, and fewer for a small block, down to one pair, until
// there are eight CTAs per SM (a thread's pairs are a serial chain: 24^3 x 32
// takes 16.6 us at 32 bands per thread, 2.8 us at 4).
static int scatter_chunk(int nb) {
    const Context& c = ctx();
    const long sms = c.num_sms > 0 ? c.num_sms : 148;
    int bch = 32;
    while (bch > SC_BU && (long)div_up(c.nl_npt, 128) * div_up(nb, bch) < 8 * sms) bch /= 2;
    return bch;
}

// Whether the stencil is launched as a dependent of the projection (of which
// it reads nothing): where the spheres are of ordinary size, so that the
// projection is short.  Behind a long one the waiting stencil CTAs' shared memory
// costs it its L1.  24^3 x 32, about 500 points per sphere:
// 24.6 us without; 256^3 x 1 band in an 8-atom cell, 57,000 points: 6070 us
// without, 6580 with.
static bool stencil_dependent() {
    const Context& c = ctx();
    return c.nl_set && c.nnz <= 1024L * c.nzlma;
}

template <typename T, int MD, int TX>
static void launch_stencil_tx(const StencilArgs<T>& a, const StencilCoef& cf, int nb, cudaStream_t st) {
    dim3 grid(div_up(a.n1, TX), div_up(a.n2, 16), nb * a.nzc);
    launch_ordinary(k_stencil<T, MD, TX>, grid, TX * 16, 0, st, a, cf);
}

template <typename T, int MD>
static void launch_stencil_md(const StencilArgs<T>& a, const StencilCoef& cf, int nb, cudaStream_t st) {
    if (a.n1 % 32 == 0 || a.n1 > 24)
        launch_stencil_tx<T, MD, 32>(a, cf, nb, st);
    else if (a.n1 % 24 == 0)
        launch_stencil_tx<T, MD, 24>(a, cf, nb, st);
    else
        launch_stencil_tx<T, MD, 16>(a, cf, nb, st);
}

// Geometry of k_stencil_tma: tile height TY (multiple of BY, divides n2,
// >= Md, and n2 == TY or n2 >= TY + Md), shared-memory row pitch RS (n1
// rounded up to 128 bytes; the columns past n1 arrive as zeros and are never
// read), ring depth S >= 3, consumer warps ncw, one producer warp, at most
// 384 threads (the register budget of the 2 Md + 1 accumulators).
struct TmaGeom {
    int TY = 0, RS = 0, S = 0, ncw = 0, threads = 0, nzc = 1;
    size_t smem = 0;
    double cost = 0.0;
};

// The tile height and z split of least march_cost.  A plane costs about 500
// cycles of latency plus 1.1 x its shared-memory wavefronts (window loads and
// TMA fill); a halo plane, which feeds the z accumulators only, a quarter.
// That reproduces 2140 cycles per plane at 72^3 FP64 (TY = 18) and 1940 FP32
// (TY = 36), and 26 us for 24^3 x 32 bands in one z chunk (measured 27.6),
// which the split takes to 12.5 us.
template <typename T, int MD, int BY>
static TmaGeom tma_geometry(int n1, int n2, int nz, int nb, int sms, int dot_cap) {
    TmaGeom best;
    constexpr int VX = 16 / (int)sizeof(T);
    constexpr int MDX = (MD + VX - 1) / VX * VX;
    const int RS = (int)((((size_t)n1 * sizeof(T) + 127) / 128) * 128 / sizeof(T));
    if (n1 % VX != 0 || n1 < MDX || RS > 256 || n2 < MD) return best;
    const size_t budget = 220 * 1024;
    double best_cost = 0.0;
    for (int TY = BY; TY <= std::min(n2, 256 - 2 * MD); TY += BY) {
        if (n2 % TY != 0 || TY < MD || !(TY == n2 || n2 >= TY + MD)) continue;
        const int ncw = ((n1 / VX) * (TY / BY) + 31) / 32;
        const int threads = 32 * (ncw + 1);
        if (threads > march_threads(BY)) continue;
        const size_t stage = (size_t)(2 * TY + 2 * MD) * RS * sizeof(T);
        const int S = (int)std::min<size_t>(budget / (stage + 16), 8);
        if (S < 3) continue;
        const int tiles = n2 / TY;
        const int zmax = std::min({std::max(1, nz / 4), 65535 / nb, dot_cap / tiles});
        if (zmax < 1) continue;
        // window loads per thread: BY + 2 Md rows, 2 MDX / VX vectors of each
        // own row, Vloc
        const double loads = BY + 2 * MD + BY * (2.0 * MDX / VX) + BY;
        const double t = 500.0 + 1.1 * (4.0 * loads * ncw + (2.0 * TY + 2 * MD) * RS * sizeof(T) / 128.0);
        int nzc = 1;
        const double cost = march_cost((long)tiles * nb, nz, 2 * MD, zmax, sms, t, 0.25 * t, &nzc);
        if (best.TY == 0 || cost <= 1.05 * best_cost) {  // the taller tile at a near tie
            best_cost = best.TY == 0 ? cost : std::min(cost, best_cost);
            best.TY = TY;
            best.RS = RS;
            best.S = S;
            best.ncw = ncw;
            best.threads = threads;
            best.nzc = nzc;
            best.cost = cost;
            best.smem = (size_t)S * stage + (size_t)S * 16 + 12 * sizeof(double);
        }
    }
    return best;
}

template <typename T, int MD, int BY, bool DOT>
static int launch_tma_dot(const TmaMaps& maps, const StencilArgs<T>& a, const StencilCoef& cf, int nb,
                          const TmaGeom& g, cudaStream_t st) {
    RS_CHECK(set_smem_optin((const void*)k_stencil_tma<T, MD, BY, DOT>, 220 * 1024 + 8 * 16 + 12 * 8));
    dim3 grid(a.n2 / g.TY, (unsigned)(nb * a.nzc));
    launch_as(stencil_dependent(), k_stencil_tma<T, MD, BY, DOT>, grid, g.threads, g.smem, st, maps, a, coef_as<T>(cf),
              g.TY, g.RS, g.S, g.ncw, ctx().err_flag);
    RS_LAUNCH();
    return RSDFT_OK;
}

template <typename T, int MD, int BY>
static int launch_tma(StencilArgs<T> a, const StencilCoef& cf, int nb, cudaStream_t st, HpsiDot* dot,
                      const TmaGeom& g, bool* used) {
    Context& c = ctx();
    *used = false;
    if (g.TY == 0) return RSDFT_OK;
    if (reinterpret_cast<uintptr_t>(a.hpsi) % 16 != 0 || (a.ld * sizeof(T)) % 16 != 0) return RSDFT_OK;
    a.zlen = div_up(a.nzo, g.nzc);
    a.nzc = div_up(a.nzo, a.zlen);
    if (dot) a.ndot = (a.n2 / g.TY) * a.nzc;
    TmaMaps maps;
    const CUtensorMapDataType dt = sizeof(T) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    const unsigned long long dims[4] = {(unsigned long long)a.n1, (unsigned long long)a.n2,
                                        (unsigned long long)a.n3, (unsigned long long)nb};
    const unsigned long long strides[3] = {(unsigned long long)a.n1 * sizeof(T),
                                           (unsigned long long)a.n1 * a.n2 * sizeof(T),
                                           (unsigned long long)a.ld * sizeof(T)};
    const unsigned long long vdims[4] = {(unsigned long long)a.n1, (unsigned long long)a.n2,
                                         (unsigned long long)a.n3, 1ull};
    const unsigned long long vstrides[3] = {strides[0], strides[1], (unsigned long long)a.n1 * a.n2 * a.n3 * sizeof(T)};
    const unsigned int RS = (unsigned)g.RS, TY = (unsigned)g.TY;
    const unsigned int bf[4] = {RS, TY + 2 * MD, 1, 1}, be[4] = {RS, TY + MD, 1, 1}, bm[4] = {RS, TY, 1, 1},
                       bw[4] = {RS, (unsigned)MD, 1, 1};
    if (encode_tmap_4d(&maps.full, dt, a.psi, dims, strides, bf) != RSDFT_OK ||
        encode_tmap_4d(&maps.edge, dt, a.psi, dims, strides, be) != RSDFT_OK ||
        encode_tmap_4d(&maps.mid, dt, a.psi, dims, strides, bm) != RSDFT_OK ||
        encode_tmap_4d(&maps.wrap, dt, a.psi, dims, strides, bw) != RSDFT_OK ||
        encode_tmap_4d(&maps.vloc, dt, a.vloc, vdims, vstrides, bm) != RSDFT_OK)
        return RSDFT_OK;  // not usable for this shape: the caller takes the general kernel
    if (dot) {
        dot->nch = a.ndot;
        dot->with_nl = false;
        a.dot = dot->part;
        RS_CHECK((launch_tma_dot<T, MD, BY, true>(maps, a, cf, nb, g, st)));
    } else {
        RS_CHECK((launch_tma_dot<T, MD, BY, false>(maps, a, cf, nb, g, st)));
    }
    *used = true;
    return RSDFT_OK;
}

// k_stencil_row: rows of whole packs (8 bytes), up to 192 vectors of 16, and
// 8-byte aligned arrays.
//
// The tile height and z split of least modelled time.  A plane takes 1350 plus
// 31 per copy a thread issues plus 0.8 per shared-memory wavefront (window loads
// and fill) of the CTAs that share the SM; a halo plane 0.23 of that; a CTA 1740
// plus 410 per copy to set up its offsets; whole waves.  Fitted (in SM cycles)
// to the times of all tiles and splits of 9^3 .. 111^3, 1 to 640 bands, Md 4, 6,
// 8: the choice is within 1.4 % (rms) of the best.  Two CTAs per SM throughout and
// no term for the copies, as suits the TMA march, splits small blocks into tiles
// of two rows and few z chunks: 45^3 x 1 band 30.3 us against 23.4, Md = 8 x 8
// bands 49.4 against 33.3 (projectors aside).
template <typename T, int MD, int BY>
static int launch_row(StencilArgs<T> a, const StencilCoef& cf, int nb, cudaStream_t st, HpsiDot* dot, bool* used) {
    *used = false;
    constexpr int W = Pk<T>::W, VX = 2 * W, S = RS_STAGES, HX = (MD + VX - 1) / VX * VX;
    const int nxv = div_up(a.n1, VX);
    if (a.n1 % W != 0 || nxv > 192) return RSDFT_OK;
    if (W > 1 && (reinterpret_cast<uintptr_t>(a.psi) % 8 != 0 || reinterpret_cast<uintptr_t>(a.hpsi) % 8 != 0 ||
                  reinterpret_cast<uintptr_t>(a.vloc) % 8 != 0 || a.ld % W != 0))
        return RSDFT_OK;
    const Context& c = ctx();
    const int sms = c.num_sms > 0 ? c.num_sms : 148;
    const double row = (nxv * VX + 2 * HX) * sizeof(T);
    const int plan = dot && dot->plan_nb ? dot->plan_nb : nb;
    int TY = 0, nzc = 1;
    double best = 0.0;
    for (int ty = BY; ty < a.n2 + BY; ty += BY) {
        const int threads = (nxv * (ty / BY) + 31) / 32 * 32;
        if (threads > 192) break;
        if ((2 * ty + 2 * MD) * row * (S + 0.5) > 110.0 * 1024) break;
        const int tiles = div_up(a.n2, ty);
        const int zmax = std::min({std::max(1, a.nzo / 4), 65535 / plan, (dot ? dot->cap : 1 << 20) / tiles});
        if (zmax < 1) continue;
        const double loads = BY + 2 * MD + BY * (2.0 * HX / VX) + BY;
        const double lds = 4.0 * loads * (threads / 32) + 2.0 * (2.0 * ty + 2 * MD) * row / 128.0;
        const double copies = (2.0 * ty + 2 * MD) * row / 8.0 / threads;
        const double smem = (2.0 * ty + 2 * MD) * row * (S + 0.5);
        const int per_sm = std::max(1, (int)std::min(227.0 * 1024 / (smem + 1024), 65536.0 / (168 * threads)));
        for (int z = 1; z <= zmax; ++z) {
            const int zlen = div_up(a.nzo, z), n = div_up(a.nzo, zlen);
            const long ctas = (long)tiles * plan * n;
            const int share = (int)std::min<long>(per_sm, (ctas + sms - 1) / sms);
            const double t = 1350.0 + 31.0 * copies + 0.8 * share * lds;
            const double cost = (double)((ctas + (long)per_sm * sms - 1) / ((long)per_sm * sms)) *
                                (zlen * t + 2 * MD * 0.23 * t + 1740.0 + 410.0 * copies);
            if (TY == 0 || cost < best || (ty > TY && cost <= 1.02 * best)) {  // the taller tile at a near tie
                best = TY == 0 ? cost : std::min(cost, best);
                TY = ty;
                nzc = n;
            }
        }
    }
    if (TY == 0) return RSDFT_OK;
    a.zlen = div_up(a.nzo, nzc);
    a.nzc = div_up(a.nzo, a.zlen);
    const int tiles = div_up(a.n2, TY), threads = (nxv * (TY / BY) + 31) / 32 * 32;
    const size_t se = (size_t)(2 * TY + 2 * MD) * (nxv * VX + 2 * HX);
    const size_t smem = se * (S * sizeof(T) + sizeof(int) / W);
    auto kern = dot ? k_stencil_row<T, MD, BY, true> : k_stencil_row<T, MD, BY, false>;
    RS_CHECK(set_smem_optin((const void*)kern, (int)smem));
    if (dot) {
        dot->nch = a.ndot = tiles * a.nzc;
        dot->with_nl = false;
        a.dot = dot->part;
    }
    launch_as(stencil_dependent(), kern, dim3(tiles, (unsigned)(nb * a.nzc)), threads, smem, st, a, coef_as<T>(cf), TY);
    RS_LAUNCH();
    *used = true;
    return RSDFT_OK;
}

template <typename T, int MD>
static int launch_stencil_md2(StencilArgs<T> a, const StencilCoef& cf, int nb, cudaStream_t st, HpsiDot* dot) {
    const Context& c = ctx();
    bool used = false;
    // Rows per thread: two up to Md = 6, one above, where the 2 Md + 1
    // accumulators of two rows no longer fit the register budget.  In FP64 also
    // three (246 registers, 7 instead of 11 warps at 72^3): the window loads per
    // point drop from 7 to 6, the stencil of 72^3 x 480 from 1113 to 1018 us.
    // Only on the same tiles, for the long windows (Md >= 5) and with six warps
    // left: 42^3 x 351 at Md = 4 took 283 us against 250.  H psi at Md = 6, two |
    // three rows, us: same tiles 36^3 x 320 211 | 192, 48^3 404 | 393, 54^3 584 | 585,
    // 72^3 x 240 888 | 823, 96^3 x 101 911 | 872; other tiles 60^3 x 320 711 | 780, 84^3
    // 962 | 980, 90^3 993 | 1096 (42^3 385 | 326: the cost, fitted to two rows, does
    // not tell these apart).  In FP32, where a load
    // serves twice the points and the warps' latency counts more, three rows
    // took 660 us against 646.
    constexpr int BY = MD <= 6 ? 2 : 1;
    const int plan = dot && dot->plan_nb ? dot->plan_nb : nb, cap = dot ? dot->cap : 1 << 20;
    const int nsm = c.num_sms > 0 ? c.num_sms : 148;
    const TmaGeom g = tma_geometry<T, MD, BY>(a.n1, a.n2, a.nzo, plan, nsm, cap);
    if constexpr (sizeof(T) == 8 && (MD == 5 || MD == 6)) {
        const TmaGeom g3 = tma_geometry<T, MD, 3>(a.n1, a.n2, a.nzo, plan, nsm, cap);
        if (g.TY != 0 && g3.TY == g.TY && g3.ncw >= 6 && g3.cost < 0.93 * g.cost)
            RS_CHECK((launch_tma<T, MD, 3>(a, cf, nb, st, dot, g3, &used)));
    }
    if (!used) RS_CHECK((launch_tma<T, MD, BY>(a, cf, nb, st, dot, g, &used)));
    if (!used) RS_CHECK((launch_row<T, MD, (MD <= 6 ? 2 : 1)>(a, cf, nb, st, dot, &used)));
    if (used) {
        if (a.gpt_ptr && c.nl_npt > 0) {
            const int bch = scatter_chunk(nb);
            dim3 grid(div_up(c.nl_npt, 128), div_up(nb, bch));
            launch(k_nl_scatter<T>, grid, 128, 0, st, a.hpsi, a.ld, nb, bch, (const int*)c.nl_pts,
                   (const int*)c.nl_ptr, c.nl_npt, a.gpt_grp, a.gpt_uv4, a.uvunk, a.nzlma, a.band_active,
                   c.err_flag);
            RS_LAUNCH();
        }
        return RSDFT_OK;
    }
    // rows beyond both z marches (odd FP32 widths, more than 192 vectors):
    // register-queue kernel with per-plane halo loads and the nonlocal scatter
    // fused
    const int tx = (a.n1 % 32 == 0 || a.n1 > 24) ? 32 : (a.n1 % 24 == 0 ? 24 : 16);
    const long base = (long)div_up(a.n1, tx) * div_up(a.n2, 16) * (dot && dot->plan_nb ? dot->plan_nb : nb);
    const long want = 8L * (c.num_sms > 0 ? c.num_sms : 148);
    int nzc = (int)std::min<long>(std::max<long>(1, (want + base - 1) / base), std::max(1, a.nzo / 8));
    const int nxy = div_up(a.n1, tx) * div_up(a.n2, 16);
    while (((long)nb * nzc > 65535 || (dot && nxy * nzc > dot->cap)) && nzc > 1) --nzc;
    a.zlen = div_up(a.nzo, nzc);
    a.nzc = div_up(a.nzo, a.zlen);
    if (dot) {
        if (nxy * a.nzc > dot->cap) {
            set_error("hpsi: %d partial sums per band exceed %d", nxy * a.nzc, dot->cap);
            return RSDFT_EINVAL;
        }
        dot->nch = a.ndot = nxy * a.nzc;
        dot->with_nl = true;
        a.dot = dot->part;
    }
    launch_stencil_md<T, MD>(a, cf, nb, st);
    RS_LAUNCH();
    return RSDFT_OK;
}

template <typename T>
static int launch_stencil(StencilArgs<T> a, const StencilCoef& cf, int md, int nb, cudaStream_t st,
                          HpsiDot* dot = nullptr) {
    if (a.nzo <= 0) {
        a.z0 = 0;
        a.nzo = a.n3;
    }
    switch (md) {
        case 1: return launch_stencil_md2<T, 1>(a, cf, nb, st, dot);
        case 2: return launch_stencil_md2<T, 2>(a, cf, nb, st, dot);
        case 3: return launch_stencil_md2<T, 3>(a, cf, nb, st, dot);
        case 4: return launch_stencil_md2<T, 4>(a, cf, nb, st, dot);
        case 5: return launch_stencil_md2<T, 5>(a, cf, nb, st, dot);
        case 6: return launch_stencil_md2<T, 6>(a, cf, nb, st, dot);
        case 7: return launch_stencil_md2<T, 7>(a, cf, nb, st, dot);
        case 8: return launch_stencil_md2<T, 8>(a, cf, nb, st, dot);
        default: set_error("Md=%d unsupported", md); return RSDFT_EUNSUP;
    }
}

template <typename T>
int hpsi_device(const T* psi, T* hpsi, long ld, int nb, int spin, const int* band_active, HpsiDot* dot) {
    Context& c = ctx();
    if (nb <= 0) return RSDFT_OK;
    if (nb > 65535) {
        set_error("hpsi: nb=%d exceeds 65535", nb);
        return RSDFT_EINVAL;
    }
    if (!c.vloc || c.vloc_ml != c.ml) {
        set_error("hpsi: rsdft_gpu_set_vloc has not been called for the current grid");
        return RSDFT_ENOTINIT;
    }
    const bool nl = c.nl_set && c.nzlma > 0;
    double* uvunk = nullptr;
    if (nl) {
        RS_CHECK(workspace_t("hpsi_uvunk", (size_t)nb * c.nzlma, &uvunk));
        RS_CHECK(launch_project<T>(psi, ld, nb, uvunk, band_active, c.stream));
    }
    StencilArgs<T> a{};
    a.psi = psi;
    a.hpsi = hpsi;
    a.ld = ld;
    a.n1 = c.n1;
    a.n2 = c.n2;
    a.n3 = c.n3;
    a.vloc = (const T*)(sizeof(T) == 8 ? (const void*)(c.vloc + (long)(spin - 1) * c.ml)
                                       : (const void*)(c.vloc32 + (long)(spin - 1) * c.ml));
    a.pt_ptr = nl ? c.pt_ptr : nullptr;
    a.pt_lma = c.pt_lma;
    a.pt_uv = (const T*)(sizeof(T) == 8 ? (const void*)c.pt_uv : (const void*)c.pt_uv32);
    a.uvunk = uvunk;
    a.nzlma = c.nzlma;
    a.band_active = band_active;
    a.band_map = nullptr;
    a.gpt_ptr = nl ? c.gpt_ptr : nullptr;
    a.gpt_grp = c.gpt_grp;
    a.gpt_uv4 = (const T*)(sizeof(T) == 8 ? (const void*)c.gpt_uv4 : (const void*)c.gpt_uv4_32);
    if (dot) dot->uvunk = uvunk;
    return launch_stencil<T>(a, c.sc, c.md, nb, c.stream, dot);
}

template int hpsi_device<double>(const double*, double*, long, int, int, const int*, HpsiDot*);
template int hpsi_device<float>(const float*, float*, long, int, int, const int*, HpsiDot*);

}  // namespace rsdft

using namespace rsdft;

extern "C" int rsdft_gpu_hamiltonian(int k, int s, const double* tpsi, double* htpsi, int n1, int n2, int ib1,
                                     int ib2) {
    RS_ENTRY();
    RS_CHECK(require_grid());
    Context& c = ctx();
    if (k != 1) {
        set_error("hamiltonian: k=%d, only the Gamma point (k=1) is supported", k);
        return RSDFT_EUNSUP;
    }
    if (s < 1 || s > c.nspin) {
        set_error("hamiltonian: s=%d outside 1..%d", s, c.nspin);
        return RSDFT_EINVAL;
    }
    const long ld = (long)n2 - n1 + 1;
    const int nb = ib2 - ib1 + 1;
    if (ld != c.ml || nb < 1) {
        set_error("hamiltonian: n2-n1+1=%ld must equal ML=%ld and ib2>=ib1", ld, c.ml);
        return RSDFT_EINVAL;
    }
    double *dpsi, *dh;
    bool sp, sh;
    RS_CHECK(wf_acquire(tpsi, ld, nb, "ham_in", &dpsi, &sp));
    RS_CHECK(wf_acquire(htpsi, ld, nb, "ham_out", &dh, &sh, false));
    RS_CHECK(hpsi_device<double>(dpsi, dh, ld, nb, s, nullptr));
    RS_CHECK(wf_release(htpsi, dh, ld, nb, sh));
    return RSDFT_OK;
}

// ----------------------------------------------------- the three operators
// hamiltonian applies op_kinetic, op_localpot and op_nonlocal in turn
// (hamiltonian_module.f90:42-58).  A domain-decomposed caller needs them
// apart: the kinetic + local part on a slab extended by its halo planes, and
// the nonlocal part as projection partial sums over the slab's own points,
// which the ranks add up before the scatter (ps_nloc2_op_module.f90:
// 161-250).  These entries give those pieces on the context's grid and
// projector tables.
namespace rsdft {
namespace {

int check_block(const char* who, int s, long ld, int nb) {
    Context& c = ctx();
    if (s < 1 || s > c.nspin) {
        set_error("%s: s=%d outside 1..%d", who, s, c.nspin);
        return RSDFT_EINVAL;
    }
    if (ld < c.ml || nb < 1 || nb > 65535) {
        set_error("%s: ld=%ld (ML=%ld), nb=%d", who, ld, c.ml, nb);
        return RSDFT_EINVAL;
    }
    return RSDFT_OK;
}

}  // namespace
}  // namespace rsdft

extern "C" int rsdft_gpu_op_local(int s, const double* tpsi, double* htpsi, long ld, int nb, int z0, int nz) {
    RS_ENTRY();
    RS_CHECK(require_grid());
    Context& c = ctx();
    RS_CHECK(check_block("op_local", s, ld, nb));
    if (z0 < 0 || nz < 1 || z0 + nz > c.n3) {
        set_error("op_local: planes [%d, %d) outside 0..%d", z0, z0 + nz, c.n3);
        return RSDFT_EINVAL;
    }
    if (!c.vloc || c.vloc_ml != c.ml) {
        set_error("op_local: rsdft_gpu_set_vloc has not been called for the current grid");
        return RSDFT_ENOTINIT;
    }
    double *dpsi, *dh;
    bool sp, sh;
    RS_CHECK(wf_acquire(tpsi, ld, nb, "ham_in", &dpsi, &sp));
    RS_CHECK(wf_acquire(htpsi, ld, nb, "ham_out", &dh, &sh, false));
    StencilArgs<double> a{};
    a.psi = dpsi;
    a.hpsi = dh;
    a.ld = ld;
    a.n1 = c.n1;
    a.n2 = c.n2;
    a.n3 = c.n3;
    a.vloc = c.vloc + (long)(s - 1) * c.ml;
    a.nzlma = c.nzlma;
    a.z0 = z0;
    a.nzo = nz;
    RS_CHECK(launch_stencil<double>(a, c.sc, c.md, nb, c.stream));
    RS_CHECK(wf_release(htpsi, dh, ld, nb, sh));
    return RSDFT_OK;
}

extern "C" int rsdft_gpu_op_nonlocal_project(const double* tpsi, long ld, int nb, double* uvunk) {
    RS_ENTRY();
    RS_CHECK(require_grid());
    Context& c = ctx();
    RS_CHECK(check_block("op_nonlocal_project", 1, ld, nb));
    if (!uvunk) {
        set_error("op_nonlocal_project: NULL uvunk");
        return RSDFT_EINVAL;
    }
    if (!c.nl_set || c.nzlma == 0) return RSDFT_OK;
    double* dpsi;
    bool sp;
    RS_CHECK(wf_acquire(tpsi, ld, nb, "ham_in", &dpsi, &sp));
    double* du = nullptr;
    RS_CHECK(workspace_t("op_uvunk", (size_t)c.nzlma * nb, &du));
    RS_CHECK(launch_project<double>(dpsi, ld, nb, du, nullptr, c.stream));
    RS_CHECK(stage_out(uvunk, du, sizeof(double) * (size_t)c.nzlma * nb));
    return RSDFT_OK;
}

extern "C" int rsdft_gpu_op_nonlocal_add(const double* uvunk, double* htpsi, long ld, int nb) {
    RS_ENTRY();
    RS_CHECK(require_grid());
    Context& c = ctx();
    RS_CHECK(check_block("op_nonlocal_add", 1, ld, nb));
    if (!uvunk) {
        set_error("op_nonlocal_add: NULL uvunk");
        return RSDFT_EINVAL;
    }
    if (!c.nl_set || c.nzlma == 0 || c.nl_npt == 0) return RSDFT_OK;
    void* du = nullptr;
    RS_CHECK(stage_in(uvunk, sizeof(double) * (size_t)c.nzlma * nb, "op_uvunk_in", &du));
    double* dh;
    bool sh;
    RS_CHECK(wf_acquire(htpsi, ld, nb, "ham_out", &dh, &sh));
    const int bch = scatter_chunk(nb);
    dim3 grid(div_up(c.nl_npt, 128), div_up(nb, bch));
    launch_ordinary(k_nl_scatter<double>, grid, 128, 0, c.stream, dh, ld, nb, bch, (const int*)c.nl_pts, (const int*)c.nl_ptr,
           c.nl_npt, (const int*)c.gpt_grp, (const double*)c.gpt_uv4, (const double*)du, c.nzlma, (const int*)nullptr,
           c.err_flag);
    RS_LAUNCH();
    RS_CHECK(wf_release(htpsi, dh, ld, nb, sh));
    return RSDFT_OK;
}

// ------------------------------------------------- allocation-free hamiltonian
// rsdft_gpu_hamiltonian_noalloc: the same H psi, for callers that must not
// allocate device memory during the call.  Its only scratch, the projection
// coefficients uVunk(nzlma, nb), lives in the file-scope array below, which
// every GPU that loads this library holds until the process exits.  In host
// code the array's name is a host-side stand-in, not a device address, so the
// kernel is given the address cudaGetSymbolAddress returns for the bound
// device.  rsdft_gpu_init looks it up (with that device current) and the
// context keeps it, so a finalize / device reset / init sequence looks it up
// again instead of reusing an address from an earlier context.
namespace rsdft {

static __device__ __align__(256) double g_hpsi_noalloc_uvunk[RSDFT_NOALLOC_SCRATCH_VALUES];

int noalloc_bind_scratch() {
    Context& c = ctx();
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_hpsi_noalloc_uvunk);
    if (e != cudaSuccess || !p) {
        set_error("cudaGetSymbolAddress of the static hamiltonian_noalloc scratch failed on device %d: %s", c.device,
                  cudaGetErrorString(e));
        return RSDFT_ECUDA;
    }
    c.noalloc_scratch = static_cast<double*>(p);
    return RSDFT_OK;
}

namespace {

int noalloc_scratch(double** out) {
    int dev = -1;
    RS_CUDA(cudaGetDevice(&dev));
    if (dev != ctx().device) {
        set_error("hamiltonian_noalloc: current device %d is not the device %d given to rsdft_gpu_init", dev,
                  ctx().device);
        return RSDFT_EINVAL;
    }
    if (!ctx().noalloc_scratch) {
        set_error("hamiltonian_noalloc: the static scratch has no device address (rsdft_gpu_init did not bind it)");
        return RSDFT_ENOTINIT;
    }
    *out = ctx().noalloc_scratch;
    return RSDFT_OK;
}

// H psi on device-visible blocks with uVunk in the static scratch.  The
// projection kernel writes every uVunk(lma, b) of the call before the stencil
// reads it, so nothing left from an earlier call is ever read.
int hpsi_static_scratch(const double* psi, double* hpsi, long ld, int nb, int spin) {
    Context& c = ctx();
    if (!c.vloc || c.vloc_ml != c.ml) {
        set_error("hamiltonian_noalloc: rsdft_gpu_set_vloc has not been called for the current grid");
        return RSDFT_ENOTINIT;
    }
    const bool nl = c.nl_set && c.nzlma > 0;
    double* uvunk = nullptr;
    if (nl) {
        RS_CHECK(noalloc_scratch(&uvunk));
        RS_CHECK(launch_project<double>(psi, ld, nb, uvunk, nullptr, c.stream));
    }
    StencilArgs<double> a{};
    a.psi = psi;
    a.hpsi = hpsi;
    a.ld = ld;
    a.n1 = c.n1;
    a.n2 = c.n2;
    a.n3 = c.n3;
    a.vloc = c.vloc + (long)(spin - 1) * c.ml;
    a.pt_ptr = nl ? c.pt_ptr : nullptr;
    a.pt_lma = c.pt_lma;
    a.pt_uv = c.pt_uv;
    a.uvunk = uvunk;
    a.nzlma = c.nzlma;
    a.gpt_ptr = nl ? c.gpt_ptr : nullptr;
    a.gpt_grp = c.gpt_grp;
    a.gpt_uv4 = c.gpt_uv4;
    return launch_stencil<double>(a, c.sc, c.md, nb, c.stream);
}

}  // namespace
}  // namespace rsdft

extern "C" int rsdft_gpu_hamiltonian_noalloc(int k, int s, const double* tpsi, double* htpsi, int n1, int n2,
                                             int ib1, int ib2) {
    RS_ENTRY();
    RS_CHECK(require_grid());
    Context& c = ctx();
    if (k != 1) {
        set_error("hamiltonian_noalloc: k=%d, only the Gamma point (k=1) is supported", k);
        return RSDFT_EUNSUP;
    }
    if (s < 1 || s > c.nspin) {
        set_error("hamiltonian_noalloc: s=%d outside 1..%d", s, c.nspin);
        return RSDFT_EINVAL;
    }
    const long ld = (long)n2 - n1 + 1;
    const int nb = ib2 - ib1 + 1;
    if (ld != c.ml || nb < 1 || nb > 65535) {
        set_error("hamiltonian_noalloc: n2-n1+1=%ld must equal ML=%ld and 1 <= ib2-ib1+1 <= 65535", ld, c.ml);
        return RSDFT_EINVAL;
    }
    if (c.nl_set && (long)nb * c.nzlma > RSDFT_NOALLOC_SCRATCH_VALUES) {
        set_error("hamiltonian_noalloc: %d bands x %d projectors = %ld scratch values exceed the static maximum "
                  "%ld (%ld MiB); call it on at most %ld bands at a time",
                  nb, c.nzlma, (long)nb * c.nzlma, (long)RSDFT_NOALLOC_SCRATCH_VALUES,
                  (long)RSDFT_NOALLOC_SCRATCH_VALUES * 8 / (1 << 20), (long)RSDFT_NOALLOC_SCRATCH_VALUES / c.nzlma);
        return RSDFT_EINVAL;
    }
    void *dpsi = nullptr, *dh = nullptr;
    const size_t span = sizeof(double) * (size_t)ld * (size_t)nb;
    const int rp = resolve(tpsi, span, &dpsi);
    if (rp < 0) return rp;
    const int rh = resolve(htpsi, span, &dh);
    if (rh < 0) return rh;
    if (!rp || !rh) {
        set_error("hamiltonian_noalloc: tpsi and htpsi must be device memory or lie in a registered wavefunction "
                  "(this entry point stages nothing)");
        return RSDFT_EINVAL;
    }
    return hpsi_static_scratch(static_cast<const double*>(dpsi), static_cast<double*>(dh), ld, nb, s);
}
