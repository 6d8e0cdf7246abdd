// The plain form's FP64 contractions on the 5th-generation tensor cores
// (tcgen05 kind::i8): an error-free splitting of FP64 operands into INT8
// slices whose products are exact in INT32 (the scheme of Ootomo, Ozaki and
// Yokota, "DGEMM on integer matrix multiplication unit", 2024).
//
// A vector (a band, or a column of the rotation matrix) is scaled by a power
// of two to 62-bit integers, q = rint(x 2^(62 - e)) with |x| < 2^e, and q is
// written in eight balanced base-256 digits, q = sum_s d_s 256^(7 - s), each
// an int8, the first at most 64.  A product of two values is the sum of the
// digit products d_s d'_t with s + t <= 7.  Digit products of equal s + t share
// an INT32 accumulator: at most (6 x 2^14 + 2 x 2^13) x 16,384 terms < 2^31, so a
// chain of IM_SEG K blocks is exact, after which the eight accumulators are
// folded into FP64.
//
// Precision.  An element is held to 2^-63 of its vector's largest, and the
// products left out come to 2^-62 of the largest (rms) per term, so the error of
// a sum of k terms is at most about 2^-60 k of the vectors' largest values, where
// FP64 arithmetic gives 2^-53 of each partial sum.  It is the smaller one as long
// as the terms reach 2^-9 or so of the largest, but unlike FP64's it does not
// shrink with them: where a band decays (vacuum, a localised band) its tail
// would lose digits.  So k_imma_slice looks for points at which 64 bands, and
// stretches of 32 points over which one band, stay below 2^-12 of their largest:
//   the first, or a band below 2^-20 over such a stretch: the whole block goes to
//     the FP64 tensor pipe;
//   a tail band between 2^-12 and 2^-20 (the lowest bands of the 216-atom cell reach
//     2^-13): the Gram products stay (sums over the whole grid, good to 2^-60 of the
//     norms, FP64's bound being 2^-53 x points x the overlap of the moduli), and of a
//     rotation the columns made up of tail bands (k_imma_slice_v) go to the FP64
//     pipe, in tiles of 128.
// What is left are isolated values near a band's nodes, good to 2^-60 of its
// largest.
//
// Why: the FP64 tensor pipe gives 37 TFLOP/s, the INT8 pipe 36 digit products
// per FP64 product at 3.2 to 3.4 POP/s measured, an FP64 rate of about 90 TFLOP/s.
// 72^3 x 480, psi^T psi: 1255 us against 4365 us (DMMA, upper tiles); psi V: 2090 us
// against 6360 us; slicing psi for both 1040 us (exponents included).  With seven
// digits, 34 products, 1170, 2000 and 960 us.
//
// k_imma, one CTA per 128 x 64 tile of D(m, n) = sum_k A(m, k) B(n, k):
//   warp 0    TMA producer: per K block of 64 the eight slices of both tiles
//             (64-byte swizzle), one box each, into a ring of IM_NS stages;
//   warp 1    allocates TMEM; one lane issues the MMAs.  The eight slices of B
//             lie one after the other in shared memory and the accumulators
//             of s + t = 0..7 one after the other in TMEM, so A's slice s
//             meets B's slices t, t + 1, .. as one MMA of N = 64 x (slices),
//             at most 256: 12 MMAs per K step instead of 36, and A is read
//             from shared memory once per MMA (36 MMAs of N = 64 would be
//             bound by that, 48 cycles of shared memory for 32 of MMA);
//   warps 2-9 fold the accumulators (two warps per TMEM lane quadrant).
// What bounds the Gram form is the tensor pipe (88 to 93 % active at 110,592 x 480).
// The rotation's reaches 75 %: its tiles are nb / 64 K blocks long, and the next
// one's MMAs wait for the fold's TMEM reads, the accumulators taking all of TMEM.
#include <algorithm>
#include <climits>

#include "common.cuh"
#include "imma.cuh"
#include "tmap.cuh"
#include "umma.cuh"

namespace rsdft {

namespace {

constexpr int IM_S = 8;        // slices
constexpr int IM_M = 128;      // tile rows (TMEM lanes)
constexpr int IM_N = 64;       // tile columns
constexpr int IM_K = 64;       // K block: one 64-byte row
constexpr int IM_NS = 2;       // stages
constexpr int IM_SEG = 16384 / IM_K;  // K blocks per exact INT32 chain
constexpr int IM_ABYTES = IM_M * IM_K, IM_BBYTES = IM_N * IM_K;
constexpr int IM_STAGE = IM_S * (IM_ABYTES + IM_BBYTES);
constexpr int IM_EPI = 8;      // epilogue warps
constexpr int IM_THREADS = 32 * (2 + IM_EPI);
constexpr int IM_D = 8;        // accumulators, s + t = 0 .. 7
constexpr int IM_TCOLS = IM_D * IM_N;  // all of TMEM
static_assert(IM_S == IM_D, "slice 0 of A opens every accumulator");
constexpr int IM_BITS = 62;    // integer bits of a scaled value
constexpr int IM_TINY = 12;    // values below 2^-IM_TINY of the largest: singly, or the band is a tail band
constexpr int IM_DEEP = 20;    // below 2^-IM_DEEP: singly only
constexpr int IM_OWN = 10;     // a column whose other weights are below 2^-IM_OWN of its tail bands' is theirs
// exponents beyond which 2^(IM_BITS - e) or the products leave the range
constexpr int IM_EMAX = 400;

// ------------------------------------------------------------------ slicing
// exps[b] = max over the band of the exponent e with |x| < 2^e (frexp's), by
// integer maximum, so the order does not matter; zero bands keep the initial
// value.
__global__ void __launch_bounds__(256) k_imma_exp(const double* A, long ld, long ml,
                                                  int* exps, int* bad) {
    grid_dependency();
    const double* p = A + (long)blockIdx.y * ld;
    const long per = (ml + gridDim.x - 1) / gridDim.x;
    const long i1 = min(ml, (blockIdx.x + 1) * per);
    double m = 0.0;
    bool fin = true;
#pragma unroll 8
    for (long i = blockIdx.x * per + threadIdx.x; i < i1; i += 256) {
        const double v = fabs(p[i]);
        fin = fin && v <= 1.7976931348623157e308;  // false for a NaN too
        m = fmax(m, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ double sh[8];
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    const bool all = __syncthreads_and(fin);
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) m = fmax(m, sh[w]);
        int e = 0;
        if (all && m > 0.0) {
            frexp(m, &e);
            atomicMax(exps + blockIdx.y, e);
        }
        if (!all || e > IM_EMAX) *bad = 1;
    }
}

// A zero vector has every digit zero whatever its exponent (-IM_EMAX marks it);
// a tiny one is out of range.  Also clears the tail and column flags.
__global__ void k_imma_exp_check(int* exps, int n, int* tail, int nflags, int* bad) {
    grid_dependency();
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < nflags) tail[b] = 0;
    if (b >= n) return;
    if (exps[b] < -100000)
        exps[b] = -IM_EMAX;
    else if (exps[b] <= -IM_EMAX)
        *bad = 1;
}

// the eight digits of x: lo holds the bytes of slices 7, 6, 5, 4, hi those of
// 3, 2, 1, 0
__device__ __forceinline__ void imma_digits(double x, double scale, uint32_t& lo, uint32_t& hi) {
    const unsigned long long q = (unsigned long long)__double2ll_rn(x * scale) + 0x8080808080808080ull;
    lo = (uint32_t)q ^ 0x80808080u;
    hi = (uint32_t)(q >> 32) ^ 0x80808080u;
}

// 4 x 4 byte transpose: row j of the result holds byte j of a, b, c, d
__device__ __forceinline__ void byte_transpose(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t (&o)[4]) {
    const uint32_t ab0 = __byte_perm(a, b, 0x5140), ab1 = __byte_perm(a, b, 0x7362);
    const uint32_t cd0 = __byte_perm(c, d, 0x5140), cd1 = __byte_perm(c, d, 0x7362);
    o[0] = __byte_perm(ab0, cd0, 0x5410);
    o[1] = __byte_perm(ab0, cd0, 0x7632);
    o[2] = __byte_perm(ab1, cd1, 0x5410);
    o[3] = __byte_perm(ab1, cd1, 0x7632);
}

// A 64-band x 64-point block per CTA; a thread slices 4 bands x 4 points and
// transposes the digits in registers both ways, and each layout goes out
// through shared memory in 16-byte stores.  rows: [s][kb][nb][64 points]; cols:
// [s][mb][ml][64 bands].
//
// Looks for decaying bands (file header): *bad when at one of the CTA's points all
// its bands (if at least 32) are below 2^-IM_TINY of their largest, or over 32
// aligned points one band below 2^-IM_DEEP; tail[band] when it is below 2^-IM_TINY
// there.  Bands that are zero throughout are left out.
__global__ void __launch_bounds__(256) k_imma_slice(const double* A, long ld, long ml, int nb, int nkb,
                                                    const int* exps, int8_t* __restrict__ rows,
                                                    int8_t* __restrict__ cols, int* tail, int* bad, int vec) {
    grid_dependency();
    // pitch 17: the transposed words of a half warp (rows 4 apart) fall on 8
    // banks (at a pitch of 20, which 16-byte reads want, on 2: 872 us per
    // 72^3 x 480 block instead of 753)
    __shared__ uint32_t sm[IM_S][64][17];
    __shared__ uint32_t s_row[8][4];  // per warp: the points (16 x 4) where its 8 bands are tiny
    if (__syncthreads_or(*bad)) return;  // one answer for the CTA: another may set it meanwhile
    const int p = threadIdx.x & 15, q = threadIdx.x >> 4;
    const int kb = blockIdx.x, mb = blockIdx.y;
    const long i0 = (long)kb * 64 + 4 * p;
    const int b0 = mb * 64 + 4 * q;
    uint32_t lo[4][4], hi[4][4];  // [band][point]
    uint32_t tiny = 0, run = 0;   // bit 4 r + e: tiny or no value; bit r (4 + r): four tiny (deep) values
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int b = b0 + r;
        double x[4] = {0.0, 0.0, 0.0, 0.0};
        double scale = 0.0;
        uint32_t floor_hi = 0xffffffffu;  // no value: below any
        if (b < nb) {
            const int ex = exps[b];
            scale = scalbn(1.0, IM_BITS - ex);
            if (ex != -IM_EMAX) floor_hi = (uint32_t)(ex - IM_TINY + 1023) << 20;
            const double* src = A + (long)b * ld + i0;
            if (vec && i0 + 4 <= ml) {
                const double2 u = *reinterpret_cast<const double2*>(src), v = *reinterpret_cast<const double2*>(src + 2);
                x[0] = u.x;
                x[1] = u.y;
                x[2] = v.x;
                x[3] = v.y;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (i0 + e < ml) x[e] = src[e];
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            imma_digits(x[e], scale, lo[r][e], hi[r][e]);
            if ((uint32_t)(__double2hiint(x[e]) & 0x7fffffff) < floor_hi) tiny |= 1u << (4 * r + e);
        }
        if (floor_hi != 0xffffffffu && ((tiny >> (4 * r)) & 15u) == 15u && i0 + 4 <= ml) {
            run |= 1u << r;
            uint32_t big = 0;
#pragma unroll
            for (int e = 0; e < 4; ++e) big = max(big, (uint32_t)(__double2hiint(x[e]) & 0x7fffffff));
            if (big < floor_hi - ((uint32_t)(IM_DEEP - IM_TINY) << 20)) run |= 16u << r;
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // bits 0, 8 (16, 24): a run of eight lanes' points of the half warp's band
    auto runs_of = [&](int bit) {
        uint32_t n = __ballot_sync(0xffffffffu, (run >> bit) & 1u);
        n &= n >> 4;
        n &= n >> 2;
        return n & (n >> 1) & 0x01010101u;
    };
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        uint32_t m = __ballot_sync(0xffffffffu, ((tiny >> e) & 0x1111u) == 0x1111u && i0 + e < ml);
        m &= m >> 16;
        if (lane == 0) s_row[warp][e] = m & 0xffffu;
        const uint32_t n = runs_of(e);  // here e is the band
        if (n) {                        // the same for the warp
            if ((lane & 15) == 0 && ((n >> lane) & 0x0101u)) tail[b0 + e] = 1;
            if (runs_of(4 + e) && lane == 0) *bad = 1;
        }
    }
    auto check_rows = [&] {
        if (threadIdx.x < 4 && nb - mb * 64 >= 32) {
            uint32_t m = 0xffffu;
#pragma unroll
            for (int w = 0; w < 8; ++w) m &= s_row[w][threadIdx.x];
            if (m) *bad = 1;
        }
    };
    if (rows) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            uint32_t tl[4], th[4];
            byte_transpose(lo[r][0], lo[r][1], lo[r][2], lo[r][3], tl);
            byte_transpose(hi[r][0], hi[r][1], hi[r][2], hi[r][3], th);
#pragma unroll
            for (int s = 0; s < IM_S; ++s) sm[s][4 * q + r][p] = s < 4 ? th[3 - s] : tl[7 - s];
        }
        __syncthreads();
        check_rows();
        for (int t = threadIdx.x; t < IM_S * 64 * 4; t += 256) {
            const int s = t >> 8, r = (t >> 2) & 63, w = t & 3;
            if (mb * 64 + r < nb)
                *reinterpret_cast<uint4*>(rows + (((size_t)s * nkb + kb) * nb + mb * 64 + r) * 64 + 16 * w) =
                    make_uint4(sm[s][r][4 * w], sm[s][r][4 * w + 1], sm[s][r][4 * w + 2], sm[s][r][4 * w + 3]);
        }
        __syncthreads();
    }
    if (!cols) return;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        uint32_t tl[4], th[4];
        byte_transpose(lo[0][e], lo[1][e], lo[2][e], lo[3][e], tl);
        byte_transpose(hi[0][e], hi[1][e], hi[2][e], hi[3][e], th);
#pragma unroll
        for (int s = 0; s < IM_S; ++s) sm[s][4 * p + e][q] = s < 4 ? th[3 - s] : tl[7 - s];
    }
    __syncthreads();
    if (!rows) check_rows();
    const int nmb = gridDim.y;
    for (int t = threadIdx.x; t < IM_S * 64 * 4; t += 256) {
        const int s = t >> 8, i = (t >> 2) & 63, w = t & 3;
        const long gi = (long)kb * 64 + i;
        if (gi < ml)
            *reinterpret_cast<uint4*>(cols + (((size_t)s * nmb + mb) * ml + gi) * 64 + 16 * w) =
                make_uint4(sm[s][i][4 * w], sm[s][i][4 * w + 1], sm[s][i][4 * w + 2], sm[s][i][4 * w + 3]);
    }
}

// V'(m, n) = V(m, n) 2^exps[m] per column n: its exponent e, as the product's
// scale 2^(e - 12), and its slices [s][mb][n][64], one warp per column.  need[n /
// 128] (and need[all groups]) is set for a column whose weights on other than tail
// bands are below 2^-IM_OWN of its largest: it may come out as a tail.
__global__ void __launch_bounds__(128) k_imma_slice_v(const double* V, int ldv, int nb, int nmb,
                                                      const int* exps, const int* tail, int* need,
                                                      double* __restrict__ vscale, int8_t* __restrict__ out, int* bad) {
    grid_dependency();
    const int n = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (n >= nb || __any_sync(0xffffffffu, *bad)) return;
    const double* v = V + (long)n * ldv;
    int e = INT_MIN, eo = INT_MIN;  // largest exponent over all bands, over those without tails
    bool fin = true;
    for (int m = lane; m < nb; m += 32) {
        const double x = fabs(v[m]);
        fin = fin && x <= 1.7976931348623157e308;
        int k = 0;
        if (fin && x > 0.0) {
            frexp(x, &k);
            e = max(e, k + exps[m]);
            if (!tail[m]) eo = max(eo, k + exps[m]);
        }
    }
    e = __reduce_max_sync(0xffffffffu, e);
    eo = __reduce_max_sync(0xffffffffu, eo);
    fin = __all_sync(0xffffffffu, fin);
    if (e == INT_MIN) e = eo = 0;
    if (!fin || e > IM_EMAX || e < -IM_EMAX) {
        if (lane == 0) *bad = 1;
        return;
    }
    if (lane == 0 && (eo == INT_MIN || eo < e - IM_OWN)) {
        need[n / 128] = 1;
        need[(nb + 127) / 128] = 1;
    }
    if (lane == 0) vscale[n] = scalbn(1.0, e - 12);
    for (int m = lane; m < nmb * 64; m += 32) {
        const double x = m < nb ? scalbn(v[m], exps[m] - e) : 0.0;
        uint32_t lo, hi;
        imma_digits(x, scalbn(1.0, IM_BITS), lo, hi);
        int8_t* o = out + ((size_t)(m >> 6) * nb + n) * 64 + (m & 63);
        const size_t ss = (size_t)nmb * nb * 64;
#pragma unroll
        for (int s = 0; s < IM_S; ++s)
            o[s * ss] = (int8_t)((s < 4 ? hi >> (8 * (3 - s)) : lo >> (8 * (7 - s))) & 255u);
    }
}

// ----------------------------------------------------------------- products
struct ImmaMaps {
    CUtensorMap a, b;  // {64, rows, K blocks, slices}
};

struct ImmaArgs {
    int kblocks, kb_per_split;
    int ntm, ntn, ntiles;
    int sym;           // GRAM: only tiles with 128 tm <= 64 tn + 63
    double* partial;   // GRAM: [split][tile][64][128]
    double* out;       // rotation: out[n * ldo + m]
    long ldo;
    long mrows;
    int nrows;
    const double* vscale;  // rotation: 2^(exponent of V's column - 12)
    const int* bad;
    int* err;
};

__device__ __forceinline__ void imma_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

// instruction descriptor, kind::i8: D = S32 (2), A = B = signed 8-bit (1),
// both K-major, M = 128
__host__ __device__ constexpr uint32_t imma_idesc(int N) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(IM_M >> 4) << 24);
}

// tile of a symmetric Gram product: column tiles in order, each with the row
// tiles 0 .. tn / 2
__host__ __device__ inline void imma_sym_tile(int t, int& tm, int& tn) {
    tn = 0;
    while (t > tn / 2) {
        t -= tn / 2 + 1;
        ++tn;
    }
    tm = t;
}

template <bool GRAM>
__global__ void __launch_bounds__(IM_THREADS, 1) k_imma(const __grid_constant__ ImmaMaps maps, ImmaArgs g) {
    grid_dependency();
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)IM_NS * IM_STAGE);
    uint64_t* empty = full + IM_NS;
    uint64_t* accf = empty + IM_NS;
    uint64_t* acce = accf + 1;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(acce + 1);
    if (*g.bad) return;  // uniform over the grid
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // work units, each one exact chain: GRAM, the segments of this CTA's tile
    // and K range; rotation, the tiles blockIdx.x, blockIdx.x + gridDim.x, ..
    // (n fastest, so that CTAs running together share A tiles in L2)
    int tm0 = 0, tn0 = 0, kb0 = 0, kb1 = g.kblocks, nunits;
    if (GRAM) {
        if (g.sym) {
            imma_sym_tile(blockIdx.x, tm0, tn0);
        } else {
            tm0 = blockIdx.x % g.ntm;
            tn0 = blockIdx.x / g.ntm;
        }
        kb0 = blockIdx.y * g.kb_per_split;
        kb1 = min(kb0 + g.kb_per_split, g.kblocks);
        nunits = (max(kb1 - kb0, 0) + IM_SEG - 1) / IM_SEG;
    } else {
        nunits = (int)blockIdx.x < g.ntiles ? (g.ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    }
    auto unit = [&](int u, int& tm, int& tn, int& ka, int& kz) {
        if (GRAM) {
            tm = tm0;
            tn = tn0;
            ka = kb0 + u * IM_SEG;
            kz = min(ka + IM_SEG, kb1);
        } else {
            const int t = (int)blockIdx.x + u * (int)gridDim.x;
            tm = t / g.ntn;
            tn = t % g.ntn;
            ka = 0;
            kz = g.kblocks;
        }
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < IM_NS; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(accf, 1);
        mbar_init(acce, IM_EPI);
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tslot, IM_TCOLS);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = *tslot;
    bool ok = true;

    if (warp == 0) {
        // ------------------------------------------------------ TMA producer
        if (lane == 0) {
            int it = 0;
            for (int u = 0; u < nunits && ok; ++u) {
                int tm, tn, ka, kz;
                unit(u, tm, tn, ka, kz);
                for (int kb = ka; kb < kz; ++kb, ++it) {
                    const int s = it % IM_NS;
                    if (it >= IM_NS && !mbar_wait(&empty[s], ((it / IM_NS) - 1) & 1)) {
                        ok = false;
                        break;
                    }
                    unsigned char* st = smem + (size_t)s * IM_STAGE;
                    mbar_arrive_expect_tx(&full[s], IM_STAGE);
                    tma_load_4d(st, &maps.a, 0, tm * IM_M, kb, 0, &full[s]);
                    tma_load_4d(st + IM_S * IM_ABYTES, &maps.b, 0, tn * IM_N, kb, 0, &full[s]);
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------- MMA issuer
        if (lane == 0) {
            int it = 0;
            for (int u = 0; u < nunits && ok; ++u) {
                int tm, tn, ka, kz;
                unit(u, tm, tn, ka, kz);
                if (u >= 1 && !mbar_wait(acce, (u - 1) & 1)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                for (int kb = ka; kb < kz; ++kb, ++it) {
                    const int s = it % IM_NS;
                    if (!mbar_wait(&full[s], (it / IM_NS) & 1)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = smem_u32(smem + (size_t)s * IM_STAGE);
                    const uint32_t sb = sa + IM_S * IM_ABYTES;
#pragma unroll
                    for (int kk = 0; kk < 2; ++kk) {  // two K steps of 32 bytes
#pragma unroll
                        for (int i = 0; i < IM_S; ++i) {
                            const uint64_t ad = umma_desc_sw64(sa + i * IM_ABYTES + kk * 32);
                            // slices t of B with s + t <= 7, four at a time
#pragma unroll
                            for (int j = 0; j < IM_D - i; j += 4) {
                                const int nj = IM_D - i - j < 4 ? IM_D - i - j : 4;
                                const uint64_t bd = umma_desc_sw64(sb + j * IM_BBYTES + kk * 32);
                                // a chain's first products, slice 0 with all, overwrite
                                const uint32_t acc = (kb == ka && kk == 0 && i == 0) ? 0u : 1u;
                                imma_mma(tbase + (uint32_t)((i + j) * IM_N), ad, bd, imma_idesc(IM_N * nj), acc);
                            }
                        }
                    }
                    umma_commit(&empty[s]);
                }
                umma_commit(accf);
            }
        }
    } else {
        // ---------------------------------------------------------- epilogue
        const int q = warp & 3;            // TMEM lane quadrant
        const int h = (warp - 2) >> 2;     // column half
        const int row = 32 * q + lane;
        const uint32_t tq = tbase + ((uint32_t)(32 * q) << 16) + (uint32_t)(h * 32);
        double acc[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) acc[c] = 0.0;
        for (int u = 0; u < nunits; ++u) {
            int tm, tn, ka, kz;
            unit(u, tm, tn, ka, kz);
            if (!mbar_wait(accf, u & 1)) {
                ok = false;
                break;
            }
            tc_fence_after();
            // sum_d D_d 256^-d from two exact 64-bit sums, D_0..D_3 and D_4..D_7.
            // The MMAs of the next tile wait for these reads (the accumulators
            // take all of TMEM), so four loads are issued per wait.
#pragma unroll
            for (int c0 = 0; c0 < 32; c0 += 16) {
                double v[16];
#pragma unroll
                for (int d0 = 0; d0 < IM_D; d0 += 4) {
                    uint32_t r[4][16];
#pragma unroll
                    for (int d = 0; d < 4; ++d) tmem_ld_x16(tq + (uint32_t)((d0 + d) * IM_N + c0), r[d]);
                    tmem_ld_wait();
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        const long long t = (((long long)(int)r[0][c] * 256 + (int)r[1][c]) * 256 + (int)r[2][c]) * 256 +
                                            (int)r[3][c];
                        if (d0 == 0)
                            v[c] = (double)t * 5.9604644775390625e-08;  // 256^-3
                        else
                            v[c] = fma((double)t, 1.3877787807814457e-17, v[c]);  // 256^-7
                    }
                }
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    if (GRAM)
                        acc[c0 + c] += v[c];
                    else
                        acc[c0 + c] = v[c];
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acce);
            if (!GRAM) {
                const long m = (long)tm * IM_M + row;
                const int n0 = tn * IM_N + h * 32;
                if (m < g.mrows) {
                    double* o = g.out + (size_t)n0 * g.ldo + m;
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        if (n0 + c < g.nrows) o[(size_t)c * g.ldo] = acc[c] * __ldg(g.vscale + n0 + c);
                }
            }
        }
        if (GRAM && ok) {
            double* P = g.partial + ((size_t)blockIdx.y * g.ntiles + blockIdx.x) * (size_t)(IM_M * IM_N);
#pragma unroll
            for (int c = 0; c < 32; ++c) P[(size_t)(h * 32 + c) * IM_M + row] = acc[c];
        }
    }
    if (!ok) atomicExch(g.err, 3);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tbase, IM_TCOLS);
    }
}

// C(i, j) = alpha 2^(ea(i) + eb(j) - 12) x the splits' sum (fixed order), one
// block per 32 rows x 8 columns of a tile; a symmetric product writes the
// mirror image of what lies above the 128 x 128 diagonal blocks, and inside
// those averages the two halves when symmetrize is set.
__global__ void __launch_bounds__(256) k_imma_reduce(const double* P, int nsplit, int ntiles, int nb,
                                                     const int* ea, const int* eb,
                                                     double alpha, int symmetrize, const int* bad,
                                                     double* __restrict__ C, long ldc) {
    grid_dependency();
    if (*bad) return;
    const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y;
    if (i >= nb || j >= nb) return;
    const int tm = i / IM_M, tn = j / IM_N;
    if (tm > tn / 2) return;  // below the diagonal blocks: mirrored
    auto sum = [&](int r, int c) {
        const int a = r / IM_M, b = c / IM_N;
        // tiles before column tile b: sum_{v < b} (v / 2 + 1)
        const int t = (b / 2) * (b / 2 + 1) + (b % 2) * (b / 2 + 1) + a;
        const double* p = P + (size_t)t * (IM_M * IM_N) + (size_t)(c - b * IM_N) * IM_M + (r - a * IM_M);
        double s = 0.0;
#pragma unroll 4
        for (int z = 0; z < nsplit; ++z) s += p[(size_t)z * ntiles * (IM_M * IM_N)];
        return s * scalbn(1.0, ea[r] + eb[c] - 12);
    };
    double v = sum(i, j);
    const bool diag = tm == j / IM_M;
    if (diag && symmetrize) v = 0.5 * (v + sum(j, i));
    v *= alpha;
    C[(long)j * ldc + i] = v;
    if (!diag) C[(long)i * ldc + j] = v;
}

int imma_map(CUtensorMap* mp, const int8_t* base, long rows, int nkb, int box_rows) {
    const unsigned long long r = (unsigned long long)rows;
    const unsigned long long dims[4] = {64ull, r, (unsigned long long)nkb, (unsigned long long)IM_S};
    const unsigned long long strides[3] = {64ull, r * 64, r * 64 * nkb};
    const unsigned int box[4] = {64u, (unsigned)box_rows, 1u, (unsigned)IM_S};
    return encode_tmap_4d(mp, CU_TENSOR_MAP_DATA_TYPE_UINT8, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B);
}

template <bool GRAM>
int launch_imma(const ImmaMaps& maps, const ImmaArgs& g, dim3 grid) {
    const size_t smem = (size_t)IM_NS * IM_STAGE + 128;
    RS_CHECK(set_smem_optin((const void*)k_imma<GRAM>, (int)smem));
    // not a dependent: V's scales come from the launch before, through __ldg (plain
    // loads wait for the stores of the column before: 137 us against 127 at 48^3 x 160)
    launch_ordinary(k_imma<GRAM>, grid, IM_THREADS, smem, ctx().stream, maps, g);
    RS_LAUNCH();
    return RSDFT_OK;
}

}  // namespace

// A rotation runs over all bands in one chain, which is exact up to IM_SEG K
// blocks; a larger set takes the DMMA form, as it did before there were slices.
//
// Below, the lower end: the slicing, the reductions and the conditional launches
// behind (40 to 60 us an operation, slices 8 us per 10^6 values) against what the
// faster products save.  DMMA | INT8, us, Gram-Schmidt: 24^3 x 160 507 | 507, x 192
// 591 | 568, 20^3 x 192 532 | 530, 30^3 x 128 436 | 459, x 144 602 | 561, 42^3 x 128
// 640 | 637, 48^3 x 96 672 | 663, x 64 413 | 438; subspace_diag: 24^3 x 160 813 | 826,
// x 192 954 | 956, x 256 1270 | 1246, 36^3 x 128 761 | 782, x 160 1074 | 1019, 48^3 x 96
// 884 | 883.  Up to 128 bands the DMMA form has 64 x 64 tiles to match.
bool imma_suits(long ml, int nb) {
    return ml >= 4096 && (double)ml * nb * nb >= 5e8 && (nb > 128 || (nb >= 96 && ml >= 100000)) && nb <= IM_SEG * IM_K;
}

int imma_slice(const double* A, long ld, long ml, int nb, const char* ws, bool need_rows, bool need_cols, int* bad,
               ImmaSlices* out) {
    Context& c = ctx();
    const int nkb = div_up(ml, 64), nmb = div_up(nb, 64);
    int8_t *rows = nullptr, *cols = nullptr;
    int* exps = nullptr;
    const int nflags = nb + div_up(nb, 128) + 1;  // tail bands, column groups
    const std::string name(ws);
    if ((need_rows && workspace_optional_t((name + "_r").c_str(), (size_t)IM_S * nkb * nb * 64, &rows) != RSDFT_OK) ||
        (need_cols && workspace_optional_t((name + "_c").c_str(), (size_t)IM_S * nmb * ml * 64, &cols) != RSDFT_OK) ||
        workspace_optional_t((name + "_e").c_str(), (size_t)nb + nflags, &exps) != RSDFT_OK) {
        // one layout without the other is of no use
        release_optional((name + "_r").c_str());
        release_optional((name + "_c").c_str());
        return RSDFT_ENOMEM;
    }
    RS_CUDA(cudaMemsetAsync(exps, 0x80, sizeof(int) * nb, c.stream));
    const int sms = c.num_sms > 0 ? c.num_sms : 148;
    const int chunks = (int)std::max<long>(1, std::min<long>(div_up(ml, 4096), div_up(16L * sms, nb) + 7));
    launch(k_imma_exp, dim3(chunks, nb), 256, 0, c.stream, A, ld, ml, exps, bad);
    int* tail = exps + nb;
    launch(k_imma_exp_check, div_up(nflags, 128), 128, 0, c.stream, exps, nb, tail, nflags, bad);
    const int vec = (ld % 2 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0) ? 1 : 0;
    launch(k_imma_slice, dim3(nkb, nmb), 256, 0, c.stream, A, ld, ml, nb, nkb, (const int*)exps, rows, cols,
           tail, bad, vec);
    RS_LAUNCH();
    *out = ImmaSlices{rows, cols, exps, tail, tail + nb, nb, ml};
    return RSDFT_OK;
}

int imma_gram(const ImmaSlices& a, const ImmaSlices& b, double alpha, int symmetrize, const int* bad, double* C,
              long ldc) {
    Context& c = ctx();
    const int nb = a.nb, nkb = div_up(a.ml, 64);
    ImmaMaps maps;
    RS_CHECK(imma_map(&maps.a, a.rows, nb, nkb, IM_M));
    RS_CHECK(imma_map(&maps.b, b.rows, nb, nkb, IM_N));
    ImmaArgs g{};
    g.kblocks = nkb;
    g.ntm = div_up(nb, IM_M);
    g.ntn = div_up(nb, IM_N);
    g.sym = 1;
    for (int tn = 0; tn < g.ntn; ++tn) g.ntiles += tn / 2 + 1;
    // one CTA per SM; K split so that the CTAs fill whole waves
    const int sms = c.num_sms > 0 ? c.num_sms : 148;
    int nsplit = std::max(1, std::min(nkb, sms / g.ntiles));
    g.kb_per_split = div_up(nkb, nsplit);
    nsplit = div_up(nkb, g.kb_per_split);
    RS_CHECK(workspace_optional_t("imma_part", (size_t)nsplit * g.ntiles * IM_M * IM_N, &g.partial));
    g.bad = bad;
    g.err = c.err_flag;
    RS_CHECK(launch_imma<true>(maps, g, dim3(g.ntiles, nsplit)));
    launch(k_imma_reduce, dim3(div_up(nb, 32), div_up(nb, 8)), dim3(32, 8), 0, c.stream, (const double*)g.partial,
           nsplit, g.ntiles, nb, a.exps, b.exps, alpha, symmetrize, bad, C, ldc);
    RS_LAUNCH();
    return RSDFT_OK;
}

int imma_slice_v(const ImmaSlices& a, const double* V, int ldv, int* bad, ImmaV* out) {
    Context& c = ctx();
    const int nb = a.nb, nmb = div_up(nb, 64);
    int8_t* sv = nullptr;
    double* vscale = nullptr;
    RS_CHECK(workspace_optional_t("imma_v", (size_t)IM_S * nmb * nb * 64, &sv));
    RS_CHECK(workspace_optional_t("imma_vscale", (size_t)nb, &vscale));
    launch(k_imma_slice_v, div_up(nb, 4), 128, 0, c.stream, V, ldv, nb, nmb, a.exps, a.tail, a.need, vscale, sv, bad);
    RS_LAUNCH();
    *out = ImmaV{sv, vscale};
    return RSDFT_OK;
}

int imma_rotate(const ImmaSlices& a, const ImmaV& v, const int* bad, double* out, long ld) {
    Context& c = ctx();
    const int nb = a.nb, nmb = div_up(nb, 64);
    ImmaMaps maps;
    RS_CHECK(imma_map(&maps.a, a.cols, a.ml, nmb, IM_M));
    RS_CHECK(imma_map(&maps.b, v.slices, nb, nmb, IM_N));
    ImmaArgs g{};
    g.kblocks = nmb;
    g.ntm = div_up(a.ml, IM_M);
    g.ntn = div_up(nb, IM_N);
    g.ntiles = g.ntm * g.ntn;
    g.out = out;
    g.ldo = ld;
    g.mrows = a.ml;
    g.nrows = nb;
    g.vscale = v.scale;
    g.bad = bad;
    g.err = c.err_flag;
    const int sms = c.num_sms > 0 ? c.num_sms : 148;
    return launch_imma<false>(maps, g, dim3((unsigned)std::min(g.ntiles, sms)));
}

}  // namespace rsdft
