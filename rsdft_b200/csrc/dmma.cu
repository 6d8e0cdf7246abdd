// FP64 contractions of the plain form on the FP64 tensor cores of sm_100a
// (mma.sync.m8n8k4 .f64, the DMMA path; tcgen05 has no FP64 kind).
//
// One kernel, k_dmma, computes tiles of C'(m, n) = sum_k A'(m, k) B'(k, n)
// for the two shapes of the eigensolver and every small product of the
// Rayleigh-Ritz step:
//   * Gram matrices psi^T Y (gram_schmidt_t_module.f90:187,
//     subspace_diag_la_module.f90:96, subspace_mate_sl_module.f90:27-366):
//     A' = psi^T, B' = Y, K = the grid; split-K over the grid, each CTA's
//     tile sum written whole, the splits added in a fixed order by
//     k_dmma_reduce (bit-reproducible);
//   * rotations psi V (gram_schmidt_t_module.f90:198, subspace_diag_la_module
//     .f90:200, subspace_rotv_sl_module.f90:92): computed transposed,
//     (psi V)^T = V^T psi^T, so that both tensor-core operands are read from
//     shared memory in the layout the grid dimension arrives in;
//   * the small dense NN / TN products of the Rayleigh-Ritz step and of the
//     eigensolver's Newton-Schulz steps.
// A' is always staged k-contiguous ([m][k] rows of BK + 4 doubles, so the
// eight rows a fragment load touches fall on distinct 32-byte bank groups);
// B' is staged [n][k] when the caller's B is k-contiguous and [k][n] when it
// is n-contiguous (rows of BN + 8 doubles).  Operand tiles arrive through
// 8-byte cp.async copies (any leading dimension), three stages deep.
#include <algorithm>

#include "common.cuh"
#include "dmma.cuh"

namespace rsdft {

namespace {

struct DmmaArgs {
    const double* A;  // A'(m, k) = A[m * lda + k]
    long lda;
    const double* B;  // B'(k, n) = B[k + n * ldb] (KMAJOR) or B[k * ldb + n]
    long ldb;
    double* C;        // C'(m, n) = C[m * ldcm + n * ldcn]
    long ldcm, ldcn;
    int M, N;
    long K;
    long kchunk;      // K values per split (blockIdx.y), a multiple of DM_BK
    double alpha, beta;
    double* partial;  // split-K: raw tile sums [split][tile][BM][BN], C unused; null: C written
    int sym;          // only tiles tm <= tn (a symmetric product)
    int ntm, ntiles;
    const int* only_if;  // run only if this device flag is set (null: always)
    const int* need;     // else the row tiles with need[tm] (null: none); need[ntm]: any
};

constexpr int DM_BK = 16;  // K per stage (four m8n8k4 steps)
constexpr int DM_NS = 3;   // cp.async stages

__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = valid ? 8 : 0;  // 0 source bytes: the 8 destination bytes are zero-filled
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async16(double* dst, const double* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// D (8x8) += A (8x4, row) B (4x8, col); per lane: a = A[lane/4][lane%4],
// b = B[lane%4][lane/4], d = D[lane/4][2 (lane%4) + {0, 1}]
__device__ __forceinline__ void dmma_884(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ void tile_of(const DmmaArgs& g, int t, int& tm, int& tn) {
    if (!g.sym) {
        tm = t % g.ntm;
        tn = t / g.ntm;
        return;
    }
    tn = 0;  // upper triangle, column by column: (0,0), (0,1), (1,1), (0,2), ...
    while (t > tn) {
        t -= tn + 1;
        ++tn;
    }
    tm = t;
}

template <int BM, int BN, int WM, int WN, bool KMAJOR, bool VEC, int CPS>
__global__ void __launch_bounds__(32 * WM * WN, CPS) k_dmma(DmmaArgs g) {
    grid_dependency();
    constexpr int BK = DM_BK, NS = DM_NS, NT = 32 * WM * WN;
    constexpr int SA = BK + 4;
    constexpr int SB = KMAJOR ? BK + 4 : BN + 8;
    constexpr int AST = BM * SA;
    constexpr int BST = KMAJOR ? BN * SB : BK * SB;
    constexpr int TM = BM / WM / 8, TN = BN / WN / 8;  // 8x8 tiles per warp
    static_assert(TM >= 1 && TN >= 1 && BM % (8 * WM) == 0 && BN % (8 * WN) == 0, "warp tiling");
    extern __shared__ __align__(16) double dsm[];
    const bool all = !g.only_if || *g.only_if;
    if (!all && !(g.need && g.need[g.ntm])) return;
    double* As = dsm;
    double* Bs = dsm + NS * AST;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm0 = (warp % WM) * (BM / WM), wn0 = (warp / WM) * (BN / WN);
    // one tile per CTA; a conditional launch, which as a rule does nothing,
    // comes with a small grid that walks the tiles
    for (int tile = blockIdx.x; tile < g.ntiles; tile += gridDim.x) {
        if (tile != (int)blockIdx.x) __syncthreads();  // the last tile's stages are still read
        int tm, tn;
        tile_of(g, tile, tm, tn);
        if (!all && !g.need[tm]) continue;  // the same for the CTA
        const int m0 = tm * BM, n0 = tn * BN;
        const long k0 = (long)blockIdx.y * g.kchunk;
        const long k1 = min(g.K, k0 + g.kchunk);
        const int nkb = k1 > k0 ? (int)((k1 - k0 + BK - 1) / BK) : 0;

        // operand tiles: 8-byte copies, or 16-byte ones (pairs of doubles along
        // the contiguous dimension) when every row start is 16-byte aligned and
        // the pair is wholly inside or outside the valid range (K, M, N even)
        auto load_stage = [&](int s, int kb) {
            const long kb0 = k0 + (long)kb * BK;
            double* as = As + s * AST;
            constexpr int V = VEC ? 2 : 1;
            for (int e = threadIdx.x; e < BM * BK / V; e += NT) {
                const int r = e / (BK / V), kk = (e % (BK / V)) * V;
                const long k = kb0 + kk;
                const bool ok = m0 + r < g.M && k < k1;
                const double* src = ok ? g.A + (long)(m0 + r) * g.lda + k : g.A;
                if (VEC) cp_async16(as + r * SA + kk, src, ok);
                else cp_async8(as + r * SA + kk, src, ok);
            }
            double* bs = Bs + s * BST;
            if (KMAJOR) {
                for (int e = threadIdx.x; e < BN * BK / V; e += NT) {
                    const int r = e / (BK / V), kk = (e % (BK / V)) * V;
                    const long k = kb0 + kk;
                    const bool ok = n0 + r < g.N && k < k1;
                    const double* src = ok ? g.B + k + (long)(n0 + r) * g.ldb : g.B;
                    if (VEC) cp_async16(bs + r * SB + kk, src, ok);
                    else cp_async8(bs + r * SB + kk, src, ok);
                }
            } else {
                for (int e = threadIdx.x; e < BN * BK / V; e += NT) {
                    const int kk = e / (BN / V), c = (e % (BN / V)) * V;
                    const long k = kb0 + kk;
                    const bool ok = n0 + c < g.N && k < k1;
                    const double* src = ok ? g.B + k * g.ldb + (n0 + c) : g.B;
                    if (VEC) cp_async16(bs + kk * SB + c, src, ok);
                    else cp_async8(bs + kk * SB + c, src, ok);
                }
            }
        };

        double acc[TM][TN][2];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

#pragma unroll
        for (int s = 0; s < NS - 1; ++s) {
            if (s < nkb) load_stage(s, s);
            cp_async_commit();
        }
        const int fr = lane >> 2, fc = lane & 3;
        for (int kb = 0; kb < nkb; ++kb) {
            cp_async_wait<NS - 2>();
            __syncthreads();  // stage kb has landed; every warp is done with stage kb - 1
            if (kb + NS - 1 < nkb) load_stage((kb + NS - 1) % NS, kb + NS - 1);
            cp_async_commit();
            const double* as = As + (kb % NS) * AST + (wm0 + fr) * SA + fc;
            const double* bs = Bs + (kb % NS) * BST + (KMAJOR ? (wn0 + fr) * SB + fc : fc * SB + wn0 + fr);
#pragma unroll
            for (int ks = 0; ks < BK; ks += 4) {
                double a[TM], b[TN];
#pragma unroll
                for (int i = 0; i < TM; ++i) a[i] = as[8 * i * SA + ks];
#pragma unroll
                for (int j = 0; j < TN; ++j) b[j] = KMAJOR ? bs[8 * j * SB + ks] : bs[ks * SB + 8 * j];
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) dmma_884(acc[i][j], a[i], b[j]);
            }
        }
        cp_async_wait<0>();

        if (g.partial) {
            double* P = g.partial + ((size_t)blockIdx.y * g.ntiles + tile) * (size_t)(BM * BN);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const int r = wm0 + 8 * i + fr, c = wn0 + 8 * j + 2 * fc;
                    *reinterpret_cast<double2*>(P + (size_t)r * BN + c) = make_double2(acc[i][j][0], acc[i][j][1]);
                }
            continue;
        }
        const bool pair = g.ldcn == 1 && (g.ldcm % 2) == 0 && (reinterpret_cast<uintptr_t>(g.C) % 16) == 0;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int m = m0 + wm0 + 8 * i + fr, n = n0 + wn0 + 8 * j + 2 * fc;
                if (m >= g.M) continue;
                double* o = g.C + (long)m * g.ldcm + (long)n * g.ldcn;
                if (pair && n + 1 < g.N) {
                    double2 v = make_double2(g.alpha * acc[i][j][0], g.alpha * acc[i][j][1]);
                    if (g.beta != 0.0) {
                        const double2 old = *reinterpret_cast<const double2*>(o);
                        v.x = fma(g.beta, old.x, v.x);
                        v.y = fma(g.beta, old.y, v.y);
                    }
                    *reinterpret_cast<double2*>(o) = v;
                    continue;
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (n + e < g.N) {
                        double* oe = o + (long)e * g.ldcn;
                        const double v = g.alpha * acc[i][j][e];
                        *oe = g.beta == 0.0 ? v : fma(g.beta, *oe, v);
                    }
                }
            }
    }
}

// C(i, j) = alpha * sum over splits of the raw tile sums; a symmetric product
// holds the tiles on and above the diagonal and the mirror image is written
// along with them; symmetrize returns alpha/2 (G + G^T).  A block takes 32
// elements along a tile's contiguous dimension; each of its 32 warps adds every
// 32nd split and the warps' sums are added in order (24^3 x 32: 61 us when a
// thread added 296 splits by itself with its neighbours a tile row apart,
// about 5 us this way).
template <int BT>
__global__ void __launch_bounds__(1024) k_dmma_reduce(const double* P, int nsplit, int ntiles, int ntm,
                                                      int sym, int m, int n, double alpha, int symmetrize,
                                                      double* __restrict__ C, long ldc, const int* only_if) {
    grid_dependency();
    __shared__ double sh[2][32][33];
    if (only_if && !*only_if) return;
    constexpr int CB = BT / 32;  // column blocks of a tile
    const int cx = threadIdx.x, y = threadIdx.y;
    for (int blk = blockIdx.x; blk < ntiles * BT * CB; blk += gridDim.x) {
        const int t = blk / (BT * CB), rest = blk % (BT * CB);
        const int r = rest / CB, c = rest % CB * 32 + cx;
        int tm, tn;
        if (sym) {
            tn = 0;
            for (int u = t; u > tn; ++tn) u -= tn + 1;
            tm = t - tn * (tn + 1) / 2;
        } else {
            tm = t % ntm;
            tn = t / ntm;
        }
        const int i = tm * BT + r, j = tn * BT + c;
        if (i >= m || j - cx >= n) continue;  // uniform: the whole block is outside
        // the transposed element is another one only on a diagonal tile of a
        // symmetric product, or anywhere in a full one
        const bool both = symmetrize && (!sym || tm == tn);
        const size_t zs = (size_t)ntiles * (BT * BT);
        const double* p = P + (size_t)t * (BT * BT) + (size_t)r * BT + c;
        const double* q = P + (size_t)(sym ? t : tn + tm * ntm) * (BT * BT) + (size_t)c * BT + r;
        double s = 0.0, u = 0.0;
#pragma unroll 4
        for (int z = y; z < nsplit; z += 32) {
            s += p[z * zs];
            if (both) u += q[z * zs];
        }
        __syncthreads();
        sh[0][y][cx] = s;
        sh[1][y][cx] = u;
        __syncthreads();
        if (y > 0 || j >= n) continue;
        const int nz = min(nsplit, 32);
        double v = 0.0, w = 0.0;
        for (int z = 0; z < nz; ++z) {
            v += sh[0][z][cx];
            w += sh[1][z][cx];
        }
        if (both) v = 0.5 * (v + w);
        v *= alpha;
        C[(long)j * ldc + i] = v;
        if (sym && tm < tn) C[(long)i * ldc + j] = v;
    }
}

template <int BM, int BN, int WM, int WN, bool KMAJOR, int CPS>
int launch_dmma(const DmmaArgs& g, int nsplit, bool vec) {
    constexpr int SA = DM_BK + 4;
    constexpr int SB = KMAJOR ? DM_BK + 4 : BN + 8;
    constexpr size_t smem = (size_t)DM_NS * (BM * SA + (KMAJOR ? BN * SB : DM_BK * SB)) * sizeof(double);
    const void* fn = vec ? (const void*)k_dmma<BM, BN, WM, WN, KMAJOR, true, CPS>
                         : (const void*)k_dmma<BM, BN, WM, WN, KMAJOR, false, CPS>;
    RS_CHECK(set_smem_optin(fn, (int)smem));
    const int sms = ctx().num_sms > 0 ? ctx().num_sms : 148;
    const dim3 grid(g.only_if ? std::min(g.ntiles, 4 * sms) : g.ntiles, nsplit);
    if (vec)
        launch(k_dmma<BM, BN, WM, WN, KMAJOR, true, CPS>, grid, 32 * WM * WN, smem, ctx().stream, g);
    else
        launch(k_dmma<BM, BN, WM, WN, KMAJOR, false, CPS>, grid, 32 * WM * WN, smem, ctx().stream, g);
    RS_LAUNCH();
    return RSDFT_OK;
}

// 16-byte operand copies are exact when both operands' bases and leading
// dimensions keep every row start 16-byte aligned and the K, M, N limits
// are even (a pair of doubles is then wholly valid or wholly out of range)
bool vec_ok(const DmmaArgs& g) {
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) % 16) == 0; };
    return al(g.A) && al(g.B) && g.lda % 2 == 0 && g.ldb % 2 == 0 && g.K % 2 == 0 && g.M % 2 == 0 && g.N % 2 == 0 &&
           g.kchunk % 2 == 0;
}

}  // namespace

// One Gram product with BT x BT tiles, at most `slots` CTAs resident.
template <int BT, int WM, int WN, int CPS>
static int gram_tiles(DmmaArgs g, double alpha, int symmetrize, double* C, long ldc) {
    Context& c = ctx();
    g.ntm = div_up(g.M, BT);
    g.ntiles = g.sym ? g.ntm * (g.ntm + 1) / 2 : g.ntm * div_up(g.N, BT);
    // whole waves of CTAs: the largest split count with tiles x splits <= two
    // waves, at least eight K blocks each (a CTA's pipeline fill), K split
    // evenly
    const long slots = (long)CPS * (c.num_sms > 0 ? c.num_sms : 148);
    const long kblocks = (g.K + DM_BK - 1) / DM_BK;
    int nsplit = (int)std::max<long>(1, std::min<long>((kblocks + 7) / 8, 2 * slots / g.ntiles));
    g.kchunk = ((kblocks + nsplit - 1) / nsplit) * DM_BK;
    nsplit = (int)((g.K + g.kchunk - 1) / g.kchunk);
    RS_CHECK(workspace_t("dmma_partials", (size_t)nsplit * g.ntiles * BT * BT, &g.partial));
    RS_CHECK((launch_dmma<BT, BT, WM, WN, true, CPS>(g, nsplit, vec_ok(g))));
    const int nblk = g.ntiles * BT * (BT / 32);
    launch(k_dmma_reduce<BT>, g.only_if ? std::min(nblk, 512) : nblk, dim3(32, 32), 0, c.stream, (const double*)g.partial,
           nsplit, g.ntiles, g.ntm, g.sym, g.M, g.N, alpha, symmetrize, C, ldc, g.only_if);
    RS_LAUNCH();
    return RSDFT_OK;
}

// Tall Gram: C (m x n, column-major, ldc) = alpha A^T B for A (K x m), B
// (K x n) column-major with leading dimension ld, K = kdim (the grid).
int dmma_gram(const double* A, const double* B, long ld, long kdim, int m, int n, double alpha, int symmetrize,
              double* C, long ldc, bool symmetric_product, const int* only_if) {
    DmmaArgs g{};
    g.only_if = only_if;
    g.A = A;
    g.lda = ld;
    g.B = B;
    g.ldb = ld;
    g.M = m;
    g.N = n;
    g.K = kdim;
    // upper tiles only for a symmetric product: A^T A, or A^T (H A) of a
    // symmetric operator (its lower tiles equal the upper ones to rounding;
    // the diagonal tiles are symmetrised by the reduction)
    g.sym = (m == n && (A == B || (symmetric_product && symmetrize))) ? 1 : 0;
    // Tile edge: the work is the tiles' area, padding included, and 64 x 64
    // tiles (half the reuse of an operand in registers) run at about 0.85 of
    // the rate of 128 x 128 ones: 160 bands, symmetric, take 3 tiles of 128^2
    // or 6 of 64^2, 390 us and 185 us.  Up to 32 bands one 32 x 32 tile does.
    const int mx = std::max(m, n);
    if (mx <= 32) return gram_tiles<32, 2, 2, 4>(g, alpha, symmetrize, C, ldc);
    auto area = [&](long t) {
        const long a = div_up(m, t), b = div_up(n, t);
        return (double)(g.sym ? a * (a + 1) / 2 : a * b) * t * t;
    };
    if (area(64) < 0.85 * area(128)) return gram_tiles<64, 2, 4, 2>(g, alpha, symmetrize, C, ldc);
    return gram_tiles<128, 4, 4, 1>(g, alpha, symmetrize, C, ldc);
}

// General product C = alpha op(A) B + beta C (column-major; op = A or A^T),
// C m x n, inner dimension k.  Computed as C^T = B^T op(A)^T, so the tensor-
// core A operand is B^T (k-contiguous in memory) and the B operand op(A)^T,
// which is k-contiguous for op = T ([n][k] staging) and row-contiguous for
// op = N ([k][n] staging).
int dmma_gemm(bool transA, long m, int n, int k, double alpha, const double* A, long lda, const double* B, long ldb,
              double beta, double* C, long ldc, const int* only_if, const int* need) {
    DmmaArgs g{};
    g.only_if = only_if;
    g.A = B;  // A'(j, kk) = B[kk + j ldb]
    g.lda = ldb;
    g.B = A;  // B'(kk, i) = op(A)(i, kk)
    g.ldb = lda;
    g.C = C;  // C'(j, i) = C[i + j ldc]
    g.ldcm = ldc;
    g.ldcn = 1;
    g.M = n;
    g.K = k;
    g.alpha = alpha;
    g.beta = beta;
    g.kchunk = ((long)k + DM_BK - 1) / DM_BK * DM_BK;
    if (m > 1L << 30) {
        set_error("dmma_gemm: m = %ld too large", m);
        return RSDFT_EINVAL;
    }
    g.N = (int)m;
    const bool vec = vec_ok(g);
    if (m >= 4096) {
        // tall output (a rotation psi V): 128 bands x 64 grid points per
        // CTA, eight warps of 32 x 32, two CTAs per SM so that one CTA's
        // operand prologue and store epilogue overlap the other's MMAs
        constexpr int BM = 128, BN = 64;
        g.ntm = div_up(n, BM);
        g.ntiles = g.ntm * div_up(m, BN);
        g.need = need;
        return transA ? launch_dmma<BM, BN, 4, 2, true, 2>(g, 1, vec) : launch_dmma<BM, BN, 4, 2, false, 2>(g, 1, vec);
    }
    // small dense products: 32 x 32 tiles, four warps
    constexpr int BM = 32, BN = 32;
    g.ntm = div_up(n, BM);
    g.ntiles = g.ntm * div_up(m, BN);
    return transA ? launch_dmma<BM, BN, 2, 2, true, 4>(g, 1, vec) : launch_dmma<BM, BN, 2, 2, false, 4>(g, 1, vec);
}

}  // namespace rsdft
