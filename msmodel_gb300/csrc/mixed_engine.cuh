// mixed_engine.cuh -- device side of the mixed-precision engine, shared by
// mixed.cu (host side, launches) and the mixed_k*.cu (a CTA per matrix) and
// mixed_t*.cu (a cluster per matrix) units, each of which defines
// MSG_MIXED_KERNEL_BODY and instantiates one (kind, d = 3 only) variant of
// k_engine_mixed, so that the twelve variants compile in parallel.
#pragma once
// The mixed-precision engine: the LU trailing updates run on the
// tcgen05 tensor cores as exact products of bf16 slices, everything else in
// double-float (FP32 hi + lo) on the FP32 pipe: the panel with its pivots'
// reciprocals, the TRSM, the epilogue and, for d = 3 and d = 2, the matrix
// assembly.  In FP64: the elements on the diagonal, those of other dimensions, the
// reciprocals of U's diagonal in the solves, the refinement's residuals and ln.
//
// Trailing update C -= A B (A: m x K panel, B: K x nn rows, K <= 32, complex):
//  * every row of A (column of B) is scaled by a power of two so its largest
//    |Re|, |Im| lies in [1/2, 1), then cut into NS integer slices
//    x 2^(8-e) = s0 + s1 2^-9 + ... + s_{NS-1} 2^-9(NS-1) (|s_k| <= 256);
//    slice k is stored as the bf16 value s_k 2^-9k, which is exact (NS = 4:
//    35 bits; NS = 6: 53 bits, the whole double-float);
//  * the slice pairs (i, j) with i + j < NS are multiplied; level l = i + j is
//    accumulated in its own TMEM accumulator for l < NG - 1 and the rest in
//    one shared accumulator.  Levels below NG - 1 are sums of at most
//    3 x 64 integer products below 2^16, hence integers below 2^24 and exact
//    whatever order and rounding the tensor core's FP32 adder uses;
//  * the slice count is chosen per item from the span of its matrix entries
//    (largest over smallest |entry|): NS = 4 (tile 128 x 32, NG = 3) while the
//    span is below 2^8, else NS = 6 (tile 128 x 16, NG = 4); dlogf items
//    always take six.  The per-row scale makes the error of a product grow
//    with the spread of magnitudes inside a row of L or a column of U: at
//    d = 3, Im k = -0.05, N = 1024 (span 2^6) four slices keep ln det within
//    ~1.4e-9 of FP64, while at d = 2, Im k = -0.3, N = 2048 (span 2^19, the
//    exponential growth e^{|Im k| r} over a disk of radius 25) they leave
//    ~1e-5 and six slices are needed;
//  * a complex product is three MMAs with four slices, A_re (Re B, Im B) together,
//    A_im Im B with the negate-B bit of the instruction descriptor and A_im Re B, into
//    2 NG TN = 192 TMEM columns; with six slices two, A_re and A_im with (Re B, Im B),
//    into 4 NG TN = 256;
//  * epilogue: C (double-float, global) -= 2^(ea+eb-16) (sum of the levels).
// Operand slices are written to global images in the tensor core's
// core-matrix layout and moved to shared memory by bulk copies (TMA engine).
#include <cuda_bf16.h>
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include "engine_internal.h"
#include "lu64.cuh"
#include "df.cuh"
#include "umma.cuh"
#include "green_df.cuh"
#include "green_df2.cuh"

namespace msg {

constexpr int MT_M = 128;               // tile rows = TMEM lanes
constexpr int A_SUB = MT_M * NB * 2;    // one 128 x 32 bf16 operand tile: 8 KB
constexpr int TMEM_COLS = 256;          // accumulators: 192 (four slices) or 256 columns; two CTAs share the SM's 512
constexpr float RANGE_LIMIT = 1.0e18f;  // larger entries leave the safe FP32 exponent range
constexpr float SPAN_WIDE = 256.0f;     // entry span above which an item is sliced six ways
// amplitude items (iterative refinement to an FP64 residual): the LU only has to
// make the refinement contract, so four slices serve up to a far larger span
constexpr float SPAN_WIDE_REFINED = 1048576.0f;

// slice configurations: NS slices per operand, TN tile columns, NG TMEM accumulator groups
template <int NS> struct SliceCfg;
// and TMEM columns per group: Re, Im of A B for four slices; for six, whose MMAs are
// what bounds a tile (126 of them 6.6k of its 15.4k cycles), A_re (Re B, Im B) and
// A_im (Re B, Im B) apart, two MMAs a complex product and the sums in the epilogue:
// 304 ln det at d = 2, n = 2048 561 -> 512 ms, 512 dlogf at n = 300 23.0 -> 21.8
template <> struct SliceCfg<4> { static constexpr int TN = 32, NG = 3, GC = 2 * 32; };
template <> struct SliceCfg<6> { static constexpr int TN = 16, NG = 4, GC = 4 * 16; };
static_assert(SliceCfg<4>::NG * SliceCfg<4>::GC <= TMEM_COLS && SliceCfg<6>::NG * SliceCfg<6>::GC <= TMEM_COLS,
              "the accumulators fit the allocation");
template <int NS> __host__ __device__ constexpr int a_band() { return 2 * NS * A_SUB; }  // NS slices x {Re, Im}
// A B tile's operand rows, per slice: Re, Im of its columns, so that A_re times
// (Re, Im) is one MMA of N = 2 TN.  304 ln det at d = 2, n = 2048: 647 ms with four
// MMAs a complex product, 605 with three (before six slices took two); 512 dlogf 10% less.  (A third block of
// rows, -Im, makes it two, but the shared memory comes out of the L1 cache: 2% slower
// at n = 64, and no room for two CTAs per SM with six slices.)
template <int NS> __host__ __device__ constexpr int b_rows() { return 2 * SliceCfg<NS>::TN; }
template <int NS> __host__ __device__ constexpr int b_sub() { return b_rows<NS>() * NB * 2; }
template <int NS> __host__ __device__ constexpr int b_band() { return NS * b_sub<NS>(); }
constexpr int EB_BYTES = 128;  // a tile's column scales, behind its slices in the image
// shared-memory operand buffer: A band then B band (NS = 4: 64 + 16 KB; NS = 6: 96 + 12 KB)
constexpr int GEMM_BYTES = a_band<6>() + b_band<6>() > a_band<4>() + b_band<4>() ? a_band<6>() + b_band<6>()
                                                                                   : a_band<4>() + b_band<4>();
// global image bytes per 128 rows of A and per column of B, the larger of the two configurations
constexpr int A_IMG_BAND = a_band<6>();
constexpr int B_IMG_COL = std::max((b_band<6>() + EB_BYTES) / SliceCfg<6>::TN, (b_band<4>() + EB_BYTES) / SliceCfg<4>::TN);

// per-phase cycle accounting (thread 0, only when X.stats is set)
enum { PH_ASSEMBLE = 0, PH_PANEL, PH_TRSM, PH_SLICE, PH_TILES, PH_SOLVE, PH_ITEMS, PH_N };

struct MixPanel {
    float4 T[NB][NB + 1];
    float4 T2[NB][NB + 1];
    float4 urow[NB];
    // assembly of d = 3 and d = 2: sin/cos/2^x tables, coordinates of the tile's atoms as
    // double-floats, and (d = 2) the item's K_nu constants
    Df3Tables tab;
    float4 ci[NB], cj[NB];  // x.h x.l y.h y.l
    float2 ciz[NB], cjz[NB];
    Df2Item d2;
    // assembly of d != 3: pair lists of the K_nu regime grouping
    unsigned short list[3 * 1024];
    int cnt[4];
};
struct MixGemm {
    uint8_t buf[GEMM_BYTES];  // A band at 0, B band at a_band<NS>()
};
// The operand buffers come last: a launch that never slices six ways (no item
// of its job can need it) allocates only the four-slice part of the union and
// leaves the rest of the SM's 256 KB of shared memory to the L1 cache.
struct MixSmem {
    static constexpr int NTH = NT;  // threads of the CTA (the block reductions of lu64.cuh)
    uint64_t bar_a, bar_b, bar_mma;
    uint32_t tmem;
    int err;
    int mma_stuck;        // an MMA completion wait ran out: 1 + the parity it waited on
    zc diag[3];
    double red_v[NT / 32];
    int red_i[NT / 32];
    int red_k[2][NT / 32], red_p[2][NT / 32];
    float4 rpiv;          // reciprocal of the panel's pivot
    alignas(16) float eb[2][EB_BYTES / 4];  // column scales of this tile and the next
    int nz;
    int rng[2];           // the item's entry range, this CTA's part (float bits), and every CTA's of the team
    int team_rng[16][2];
    int team_bad[16];     // every CTA's flag of a wait that ran out (a word of its own: a CTA ahead of the
                          // others writes it while they may still read the ranges)
    double team_max[16];
    double red_s[3][NT / 32];
    int info, bcast_i, item;
    unsigned long long stat[PH_N];
    long long t0;
    union alignas(128) {
        MixGemm g;
        MixPanel p;
        LuSmem lu;  // the FP64 assembly of the refinement's copy of M
    } u;
};
// dynamic shared memory of a launch with and without room for six slices
constexpr size_t MIX_SMEM_WIDE = sizeof(MixSmem) + 128;
constexpr size_t MIX_SMEM_NARROW =
    offsetof(MixSmem, u) + std::max({(size_t)(a_band<4>() + b_band<4>()), sizeof(MixPanel), sizeof(LuSmem)}) + 128;

__device__ __forceinline__ void stat_start(MixSmem& s) {
    if (threadIdx.x == 0) s.t0 = clock64();
}
__device__ __forceinline__ void stat_add(MixSmem& s, int ph) {
    if (threadIdx.x == 0) {
        long long t = clock64();
        s.stat[ph] += (unsigned long long)(t - s.t0);
        s.t0 = t;
    }
}

// per-CTA global scratch of the mixed engine
struct MixScratch {
    uint8_t* imgA;   // ceil(nmax/128) * A_IMG_BAND per CTA
    uint8_t* imgB;   // (ceil(nmax/32) * 32) * B_IMG_COL per CTA
    float* ea;       // row scales 2^(e-8) of the sliced A operand, padded
    float* eb;       // column scales (four slices; six keep them in the image)
    size_t a_stride, b_stride, e_stride;
    int* err;        // device flag: 1 = an mbarrier wait timed out
    unsigned long long* stats;  // per-phase SM cycles summed over CTAs, or nullptr
    int first_wait;  // poll limit of the first operand wait of each trailing update (WAIT_LIMIT
                     // unless a test shortens it to make that wait run out)
};


struct Phases {
    uint32_t a, b, mma;
};

// ---------------------------------------------------------------- slicing
// NS pre-scaled bf16 slices of the double-float x (hi, lo) for row exponent e:
// x 2^(8-e) = s0 + s1 2^-9 + ... with integers |s_k| <= 256 (bf16 holds every
// integer up to 256 exactly); 8 + 9 (NS - 1) significant bits
template <int NS>
__device__ __forceinline__ void slice_n(float h, float l, int e, float* o) {
    float xh = ldexpf(h, 8 - e), xl = ldexpf(l, 8 - e);
    float s0 = rintf(xh);
    df r = two_sum(__fsub_rn(xh, s0), xl);
    o[0] = s0;
    float sc = 1.0f / 512.0f;
#pragma unroll
    for (int k = 1; k < NS; ++k) {
        float rh = __fmul_rn(r.h, 512.0f), rl = __fmul_rn(r.l, 512.0f);
        float sk = rintf(rh);
        r = two_sum(__fsub_rn(rh, sk), rl);
        o[k] = sk * sc;
        sc *= 1.0f / 512.0f;
    }
}

__device__ __forceinline__ int row_exponent(float mx) {
    int e = 0;
    if (mx > 0.0f) frexpf(mx, &e);
    return e;
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}

// One operand row of K <= 32 complex values (stride `st` in float4) -> put(slice,
// 0 Re / 1 Im, first k, 8 bf16); exponent returned.
template <int NS, class Put>
__device__ __forceinline__ int slice_operand_row(const float4* src, size_t st, int K, Put put) {
    float mx = 0.0f;
    for (int kk = 0; kk < K; ++kk) {
        float4 v = src[kk * st];
        mx = fmaxf(mx, fmaxf(fabsf(v.x), fabsf(v.z)));
    }
    const int e = row_exponent(mx);
    for (int kb = 0; kb < NB / 8; ++kb) {
        uint32_t w[2 * NS][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float re[2][NS], im[2][NS];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int kk = kb * 8 + 2 * q + t;
                if (kk < K) {
                    float4 v = src[kk * st];
                    slice_n<NS>(v.x, v.y, e, re[t]);
                    slice_n<NS>(v.z, v.w, e, im[t]);
                } else {
#pragma unroll
                    for (int sl = 0; sl < NS; ++sl) re[t][sl] = im[t][sl] = 0.0f;
                }
            }
#pragma unroll
            for (int sl = 0; sl < NS; ++sl) {
                w[2 * sl][q] = pack2(re[0][sl], re[1][sl]);
                w[2 * sl + 1][q] = pack2(im[0][sl], im[1][sl]);
            }
        }
#pragma unroll
        for (int sub = 0; sub < 2 * NS; ++sub)
            put(sub >> 1, sub & 1, kb * 8, make_uint4(w[sub][0], w[sub][1], w[sub][2], w[sub][3]));
    }
    return e;
}

// A operand: rows [0, m) of the m x K panel P (column-major, ld), all bands;
// ea[i] = 2^(e_i - 8), the row's scale
template <int NS, class Team>
static __device__ void slice_panel_rows(const float4* P, int ld, int m, int K, uint8_t* img, float* ea, const Team& tm) {
    const int mp = (m + MT_M - 1) / MT_M * MT_M;
    for (int i = tm.rank * NT + threadIdx.x; i < mp; i += NT * tm.size) {
        uint8_t* band = img + (size_t)(i / MT_M) * a_band<NS>();
        const int r = i % MT_M;
        if (i < m) {
            ea[i] = ldexpf(1.0f, slice_operand_row<NS>(P + i, (size_t)ld, K, [&](int sl, int c, int k, uint4 w) {
                               *reinterpret_cast<uint4*>(band + (2 * sl + c) * A_SUB + cm_offset(r, k, MT_M)) = w;
                           }) - 8);
        } else {
            ea[i] = 0.0f;
            for (int kb = 0; kb < NB / 8; ++kb)
                for (int sub = 0; sub < 2 * NS; ++sub)
                    *reinterpret_cast<uint4*>(band + sub * A_SUB + cm_offset(r, kb * 8, MT_M)) = make_uint4(0, 0, 0, 0);
        }
    }
}

// B operand: columns [0, nn) of the K x nn block Bp (column-major, ld); eb[j] = 2^(e_j - 8)
template <int NS, class Team>
static __device__ void slice_block_cols(const float4* Bp, int ld, int nn, int K, uint8_t* img, float* geb, const Team& tm) {
    constexpr int TN = SliceCfg<NS>::TN;
    const int np = (nn + TN - 1) / TN * TN;
    for (int j = tm.rank * NT + threadIdx.x; j < np; j += NT * tm.size) {
        uint8_t* band = img + (size_t)(j / TN) * (b_band<NS>() + EB_BYTES);
        const int r = j % TN;
        float* eb = NS == 6 ? reinterpret_cast<float*>(band + b_band<NS>()) + r : geb + j;
        auto put = [&](int sl, int c, int k, uint4 w) {
            *reinterpret_cast<uint4*>(band + sl * b_sub<NS>() + cm_offset(c * TN + r, k, b_rows<NS>())) = w;
        };
        if (j < nn) {
            *eb = ldexpf(1.0f, slice_operand_row<NS>(Bp + (size_t)j * ld, 1, K, put) - 8);
        } else {
            *eb = 0.0f;
            for (int k = 0; k < NB; k += 8)
                for (int sl = 0; sl < NS; ++sl)
                    for (int c = 0; c < 2; ++c) put(sl, c, k, make_uint4(0, 0, 0, 0));
        }
    }
}

// ---------------------------------------------------------------- tensor-core update
// Accumulator group g (TMEM columns GC g ..: Re, Im, or the two pairs)
// holds slice level l = g for g < NG - 1 and levels >= NG - 1 in the last
// group, so that the low levels stay exact whatever the tensor core's FP32
// summation order and rounding.
// Issued by warp 0 as a whole (lead: its elected lane): with the branch uniform
// 304 ln det at d = 2, n = 2048 take 647 ms against 706 ms issued by one thread,
// 512 dlogf of n = 100..600 55.5 against 62.1, 300 ln det at d = 3, n = 1024 10% less.
template <int NS>
__device__ __forceinline__ void issue_tile_mmas(uint32_t a0, uint32_t b0, uint64_t* bar, uint32_t tmem, uint32_t lead) {
    constexpr int TN = SliceCfg<NS>::TN, NG = SliceCfg<NS>::NG;
    const uint32_t id2 = idesc_bf16(MT_M, 2 * TN), idp = idesc_bf16(MT_M, TN), idn = idesc_bf16(MT_M, TN, false, true);
    // core-matrix strides: K direction (LBO) R/8*128, row direction (SBO) 128; a K step of 16 is
    // R*32 bytes; a descriptor's start address counts 16-byte units
    const uint64_t da0 = sdesc(a0, MT_M * 16, 128), db0 = sdesc(b0, b_rows<NS>() * 16, 128);
    auto dA = [&](int k, int c, int ks) { return da0 + ((k * 2 + c) * A_SUB + ks * (MT_M * 32)) / 16; };
    auto dB = [&](int k, int row, int ks) { return db0 + (k * b_sub<NS>() + ks * (b_rows<NS>() * 32) + row * 16) / 16; };
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
#pragma unroll
        for (int l = 0; l < NS; ++l) {
            const int g = l < NG - 1 ? l : NG - 1;
#pragma unroll
            for (int i = 0; i <= l; ++i) {
                const int j = l - i;
                const uint32_t acc = (ks == 0 && i == 0 && l == g) ? 0u : 1u;  // first product of group g
                const uint32_t tre = tmem + SliceCfg<NS>::GC * g, tim = tre + TN;
                umma_bf16_lead(tre, dA(i, 0, ks), dB(j, 0, ks), id2, acc, lead);
                if (NS == 6) {
                    umma_bf16_lead(tre + 2 * TN, dA(i, 1, ks), dB(j, 0, ks), id2, acc, lead);
                } else {
                    umma_bf16_lead(tre, dA(i, 1, ks), dB(j, TN, ks), idn, 1, lead);
                    umma_bf16_lead(tim, dA(i, 1, ks), dB(j, 0, ks), idp, 1, lead);
                }
            }
        }
    }
    umma_commit_lead(bar, lead);
}

// c - (L0 + L1 + ... ): the exact levels enter by two-sums, the last group and
// every error term gather in one FP32 accumulator, one renormalisation
template <int NG>
__device__ __forceinline__ df df_sub_levels(df c, const float* lv) {
    df t = two_sum(c.h, -lv[0]);
    float lo = __fadd_rn(c.l, t.l);
#pragma unroll
    for (int g = 1; g < NG - 1; ++g) {
        const df u = two_sum(t.h, -lv[g]);
        lo = __fadd_rn(lo, u.l);
        t.h = u.h;
    }
    lo = __fsub_rn(lo, lv[NG - 1]);
    return quick_two_sum(t.h, lo);
}

// C[m x nn] -= Ap[m x K] * Bp[K x nn]; all double-float complex, column-major.
// tri != 0: only tiles holding an element with row >= column are updated.  The
// team slices the operands together and deals out the tiles in row-band order,
// in contiguous runs.  A wait that ran out sets s.err: the CTA then issues no
// more copies or MMAs but keeps to the barriers, and its items are marked.
template <int NS, class Team>
static __device__ void mixed_gemm_sub(float4* __restrict__ C, int ldc, const float4* Ap, int lda, const float4* Bp, int ldb,
                               int m, int nn, int K, int tri, MixSmem& s, const MixScratch& X, uint32_t tmem, Phases& ph,
                               const Team& tm) {
    constexpr int TN = SliceCfg<NS>::TN, NG = SliceCfg<NS>::NG, AB = a_band<NS>(), BB = b_band<NS>();
    constexpr int CW = TN / 2;  // columns of a tile per thread (two warps per TMEM lane quadrant)
    if (m <= 0 || nn <= 0 || K <= 0) return;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform, so is the branch around the MMAs
    const size_t team = blockIdx.x / tm.size;
    uint8_t* imgA = X.imgA + team * X.a_stride;
    uint8_t* imgB = X.imgB + team * X.b_stride;
    float* gea = X.ea + team * X.e_stride;
    float* geb = X.eb + team * X.e_stride;
    uint8_t* sA = s.u.g.buf;
    uint8_t* sB = s.u.g.buf + AB;
    stat_start(s);
    slice_panel_rows<NS>(Ap, lda, m, K, imgA, gea, tm);
    slice_block_cols<NS>(Bp, ldb, nn, K, imgB, geb, tm);
    fence_proxy_async_all();
    tm.sync();
    if (tm.size > 1) fence_proxy_async_all();
    stat_add(s, PH_SLICE);
    const int nbi = (m + MT_M - 1) / MT_M, nbj = (nn + TN - 1) / TN;
    // tile list in row-band order: band bi holds the tiles of columns [0, width(bi))
    auto width = [&](int bi) { return tri ? min(nbj, (bi * MT_M + MT_M - 1) / TN + 1) : nbj; };
    int todo = 0;
    for (int b = 0; b < nbi; ++b) todo += width(b);
    int bi = 0, bj = 0;
    if (tm.size > 1) {
        const int total = todo;
        bj = (int)((long long)total * tm.rank / tm.size);
        todo = (int)((long long)total * (tm.rank + 1) / tm.size) - bj;
        while (bi < nbi && bj >= width(bi)) bj -= width(bi++);
    }
    // A tile's B operand, and with six slices its column scales (read in the epilogue, beside
    // the next tile's copy, hence two of them): 304 ln det at d = 2, n = 2048 513 -> 491 ms
    // against a global load each, which waits behind the stores to C.  With four slices the
    // second copy cost 3% at n = 1024.
    auto load_b = [&](int col, int p) {
        const uint8_t* src = imgB + (size_t)col * (BB + EB_BYTES);
        mbar_arrive_expect_tx(&s.bar_b, NS == 6 ? BB + EB_BYTES : BB);
        bulk_g2s(sB, src, BB, &s.bar_b);
        if (NS == 6) bulk_g2s(s.eb[p], src + BB, EB_BYTES, &s.bar_b);
    };
    bool pend = todo > 0 && !s.err;  // warp 0: this tile's operand copies were issued
    pend = __shfl_sync(0xffffffffu, pend, 0);
    if (tid == 0 && pend) {
        mbar_arrive_expect_tx(&s.bar_a, AB);
        bulk_g2s(sA, imgA + (size_t)bi * AB, AB / 2, &s.bar_a);
        bulk_g2s(sA + AB / 2, imgA + (size_t)bi * AB + AB / 2, AB / 2, &s.bar_a);
        load_b(bj, 0);
    }
    int par = 0;  // which of s.eb the current tile's scales are in
    // warp 0: have this tile's operands landed?
    auto operands = [&](bool new_band, int limit) {
        bool ok = pend;
        if (pend) {
            if (new_band) {
                ok = mbar_wait(&s.bar_a, ph.a, limit);
                if (!ok) mbar_wait(&s.bar_a, ph.a);  // let the copy in flight land before moving on
                ph.a ^= 1;
            }
            ok = mbar_wait(&s.bar_b, ph.b) && ok;
            ph.b ^= 1;
        }
        return __all_sync(0xffffffffu, ok) != 0;
    };
    // The wait for a tile's operands comes before the barrier that ends the tile before,
    // so that its MMAs are issued at once: behind the barrier the wait queued up with the
    // CTA's loads of C (2.4k of 19.5k cycles a tile at n = 1024, and 3k for the loads).
    bool ready = warp == 0 && todo > 0 && operands(true, X.first_wait);
    // Six slices: the other warps read the first tile's column scales, which came with the copy
    // warp 0 has waited for.  (The later tiles' wait is ahead of the barrier between tiles.)
    if (NS == 6) __syncthreads();
    const int q = warp & 3, hcol = warp >> 2;  // TMEM lane quadrant, column half of this warp
    const int rloc = 32 * q + lane;
    while (todo > 0) {
        int nbi2 = bi, nbj2 = bj + 1;
        if (nbj2 >= width(bi)) { nbj2 = 0; ++nbi2; }
        if (warp == 0) {
            if (ready) {
                tc_fence_after();
                issue_tile_mmas<NS>(smem_u32(sA), smem_u32(sB), &s.bar_mma, tmem, elect_lane());
            } else if (lane == 0) {
                s.err = 1;                // operands missing: no MMA is issued;
                mbar_arrive(&s.bar_mma);  // release this tile's MMA wait at once
            }
            __syncwarp();
        }
        // this thread's row and CW columns of C, and its row scale, on their way while the
        // tensor core works
        const int row = bi * MT_M + rloc;
        const bool row_ok = row < m;
        const float ea_r = row_ok ? gea[row] : 0.0f;
        float4 cpre[CW];
#pragma unroll
        for (int j = 0; j < CW; ++j) {
            const int col = bj * TN + CW * hcol + j;
            cpre[j] = (row_ok && col < nn) ? C[row + (size_t)col * ldc] : make_float4(0, 0, 0, 0);
        }
        const bool mw = mbar_wait(&s.bar_mma, ph.mma);
        if (!mw && lane == 0) {
            s.err = 1;
            s.mma_stuck = 1 + (int)ph.mma;
        }
        ph.mma ^= 1;
        // operands of the next tile: smem is free once the MMAs completed (none after a failed wait)
        if (warp == 0) {
            pend = __shfl_sync(0xffffffffu, todo > 1 && !s.err, 0);
            if (lane == 0 && pend) {
                if (nbi2 != bi) {
                    mbar_arrive_expect_tx(&s.bar_a, AB);
                    bulk_g2s(sA, imgA + (size_t)nbi2 * AB, AB / 2, &s.bar_a);
                    bulk_g2s(sA + AB / 2, imgA + (size_t)nbi2 * AB + AB / 2, AB / 2, &s.bar_a);
                }
                load_b(nbj2, par ^ 1);
            }
        }
        tc_fence_after();
        // epilogue: TMEM lanes 32(w%4).. (rows), columns CW(w/4)..+CW-1
        constexpr int EC = NS == 6 ? 2 : 4;  // columns at a time
#pragma unroll
        for (int cc = 0; cc < CW; cc += EC) {
            float lr[EC][NG], li[EC][NG];
            const uint32_t base = tmem + ((uint32_t)(32 * q) << 16) + CW * hcol + cc;
            if constexpr (NS == 6) {
                float g[4 * NG][2];
#pragma unroll
                for (int a = 0; a < 4 * NG; ++a) tmem_ld2(base + TN * a, g[a][0], g[a][1]);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < EC; ++j)
#pragma unroll
                    for (int gg = 0; gg < NG; ++gg) {
                        // integers below 2^24 in the exact groups: exact sums
                        lr[j][gg] = __fsub_rn(g[4 * gg][j], g[4 * gg + 3][j]);
                        li[j][gg] = __fadd_rn(g[4 * gg + 1][j], g[4 * gg + 2][j]);
                    }
            } else {
                float g[2 * NG][4];
#pragma unroll
                for (int a = 0; a < 2 * NG; ++a) tmem_ld4(base + TN * a, g[a]);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < EC; ++j)
#pragma unroll
                    for (int gg = 0; gg < NG; ++gg) {
                        lr[j][gg] = g[2 * gg][j];
                        li[j][gg] = g[2 * gg + 1][j];
                    }
            }
            if (row_ok) {
#pragma unroll
                for (int j = 0; j < EC; ++j) {
                    const int col = bj * TN + CW * hcol + cc + j;
                    if (col < nn) {
                        // 2^(ea+eb-16), exact
                        const float sc = ea_r * (NS == 6 ? s.eb[par][CW * hcol + cc + j] : geb[col]);
                        const float4 cv = cpre[cc + j];
                        dfc c = dfc{df{cv.x, cv.y}, df{cv.z, cv.w}};
#pragma unroll
                        for (int gg = 0; gg < NG; ++gg) {
                            lr[j][gg] *= sc;
                            li[j][gg] *= sc;
                        }
                        c.re = df_sub_levels<NG>(c.re, lr[j]);
                        c.im = df_sub_levels<NG>(c.im, li[j]);
                        dfc_store(C + row + (size_t)col * ldc, c);
                    }
                }
            }
        }
        if (warp == 0) ready = todo > 1 && operands(nbi2 != bi, WAIT_LIMIT);
        tc_fence_before();
        __syncthreads();
        bi = nbi2;
        bj = nbj2;
        par ^= 1;
        --todo;
    }
    stat_add(s, PH_TILES);
}

// ---------------------------------------------------------------- double-float panel, TRSM, solves
// row of the CTA's largest v >= 0 (smallest row on ties; v = -1: no row), in
// every thread: the FP32 bit patterns order like the values, so the search is
// two warp reductions, and one barrier (candidates double-buffered by `par`)
__device__ __forceinline__ int block_pivotf(float v, int row, int par, MixSmem& s) {
    constexpr int NW = NT / 32;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int k = v < 0.0f ? -1 : __float_as_int(v);
    int m = __reduce_max_sync(FULL, k);
    row = __reduce_min_sync(FULL, k == m ? row : 0x7fffffff);
    if (lane == 0) { s.red_k[par][warp] = m; s.red_p[par][warp] = row; }
    __syncthreads();
    k = s.red_k[par][lane & (NW - 1)];
    row = s.red_p[par][lane & (NW - 1)];
    m = __reduce_max_sync(FULL, k);
    return __reduce_min_sync(FULL, k == m ? row : 0x7fffffff);
}

// 1 / b in double-float, with b scaled by a power of two first so that its
// squared modulus stays inside the FP32 range whatever the pivot's size
__device__ __forceinline__ dfc dfc_recip_pow2(dfc b) {
    int e;
    frexpf(fmaxf(fabsf(b.re.h), fabsf(b.im.h)), &e);
    const float sc = ldexpf(1.0f, -e);
    const dfc r = dfc_recip(dfc{df{b.re.h * sc, b.re.l * sc}, df{b.im.h * sc, b.im.l * sc}});
    return dfc{df{r.re.h * sc, r.re.l * sc}, df{r.im.h * sc, r.im.l * sc}};
}

// Panel factorisation in double-float: LAPACK's getf2 pivoting (|Re|+|Im|,
// first index on ties, full-panel row interchanges), organised in sub-panels
// of SW columns.  Inside a sub-panel the rank-1 updates touch only its own
// columns; the rest of the panel then takes one rank-SW update per sub-panel
// (U rows by unit-lower substitution in shared memory).  The panel of a large
// matrix does not stay in L2 across 304 resident CTAs, so this cuts its
// memory traffic (the full-width rank-1 form re-reads and re-writes the whole
// remaining panel once per column) by about 2.4x at the same arithmetic.
// One warp takes the interchange, the pivot row and the pivot's double-float
// reciprocal (an FP64 division, on a pipe at 1/64 of the FP32 rate, held the
// whole CTA at the next barrier): two barriers a column.  4096 ln det at n = 64:
// 4.95 ms with three barriers, every thread's own reciprocal and a thread per row
// of the rank-4 update, 3.49 now.
// Not inlined: its registers are then allocated apart from the engine's
// tensor-core epilogue, which holds the kernel at the 128-register cap.
constexpr int SW = 4;

static __device__ __noinline__ void df_panel(float4* A, int n, int j0, int jb, int* ipiv, MixSmem& s) {
    const int tid = threadIdx.x;
    const int cend = j0 + jb;
    float bv = -1.0f;
    int bi = n;
    for (int i = j0 + tid; i < n; i += NT) {
        const float v = dfc_abs1(dfc_load(A + i + (size_t)j0 * n));
        if (v > bv) { bv = v; bi = i; }
    }
    for (int c0 = j0; c0 < cend; c0 += SW) {
        const int sw = min(c0 + SW, cend);  // sub-panel columns [c0, sw)
        for (int c = c0; c < sw; ++c) {
            int p = block_pivotf(bv, bi, c & 1, s);
            if (p >= n) p = c;
            if (tid < 32) {
                const size_t col = (size_t)(j0 + tid) * n;
                float4 a = make_float4(0, 0, 0, 0), t = a;
                if (tid < jb) {
                    a = A[c + col];
                    t = p != c ? A[p + col] : a;
                }
                const bool piv0 = t.x == 0.0f && t.z == 0.0f;
                const bool nz = !__shfl_sync(0xffffffffu, (int)piv0, c - j0);
                if (tid < jb) {
                    if (nz && p != c) {
                        A[c + col] = t;
                        A[p + col] = a;
                    }
                    s.u.p.urow[tid] = nz ? t : a;
                }
                if (tid == c - j0) {
                    ipiv[c] = p;
                    if (!nz && s.info == 0) s.info = c + 1;
                    s.nz = nz;
                    if (nz) dfc_store(&s.rpiv, dfc_recip_pow2(dfc{df{t.x, t.y}, df{t.z, t.w}}));
                }
            }
            __syncthreads();
            const bool nz = s.nz != 0;
            const dfc r = dfc_load(&s.rpiv);
            bv = -1.0f;
            bi = n;
            if (nz) {
                for (int i = c + 1 + tid; i < n; i += NT) {
                    float4* pc = A + i + (size_t)c * n;
                    const dfc l = dfc_mul(dfc_load(pc), r);
                    dfc_store(pc, l);
                    if (c + 1 < sw) {
                        float4* q1 = A + i + (size_t)(c + 1) * n;
                        const dfc a = dfc_fms(dfc_load(q1), l, dfc_load(&s.u.p.urow[c + 1 - j0]));
                        dfc_store(q1, a);
                        const float v = dfc_abs1(a);
                        if (v > bv) { bv = v; bi = i; }
                        for (int cc = c + 2; cc < sw; ++cc) {
                            float4* qp = A + i + (size_t)cc * n;
                            dfc_store(qp, dfc_fms(dfc_load(qp), l, dfc_load(&s.u.p.urow[cc - j0])));
                        }
                    }
                }
            } else if (c + 1 < sw) {
                for (int i = c + 1 + tid; i < n; i += NT) {
                    const float v = dfc_abs1(dfc_load(A + i + (size_t)(c + 1) * n));
                    if (v > bv) { bv = v; bi = i; }
                }
            }
        }
        if (sw < cend) {
            const int cw = sw - c0, rem = cend - sw;
            __syncthreads();  // the sub-panel's last column is complete
            // L11 (unit lower, cw x cw) into shared memory
            if (tid < cw * cw) {
                const int r = tid / cw, q = tid % cw;
                if (q < r) s.u.p.T2[r][q] = A[c0 + r + (size_t)(c0 + q) * n];
            }
            __syncthreads();
            // U rows of the sub-panel for columns [sw, cend): u_r = a_r - sum_{q<r} L_rq u_q
            if (tid < rem) {
                const size_t col = (size_t)(sw + tid) * n;
                dfc u[SW];
#pragma unroll
                for (int r = 0; r < SW; ++r) {
                    if (r < cw) {
                        dfc a = dfc_load(A + c0 + r + col);
#pragma unroll
                        for (int q = 0; q < r; ++q) a = dfc_fms(a, dfc_load(&s.u.p.T2[r][q]), u[q]);
                        u[r] = a;
                        dfc_store(A + c0 + r + col, a);
                        dfc_store(&s.u.p.T[r][tid], a);
                    }
                }
            }
            __syncthreads();
            // rank-cw update of rows >= sw; argmax of column sw on the way.  A warp takes 32
            // rows; where the rows do not fill the CTA several warps share them, each with
            // every G-th column.
            bv = -1.0f;
            bi = n;
            const int nrb = (n - sw + 31) / 32, G = max(1, (NT / 32) / nrb);
            const int g = nrb < NT / 32 ? (tid >> 5) / nrb : 0;
            const int i0 = sw + (nrb < NT / 32 ? ((tid >> 5) % nrb) * 32 + (tid & 31) : tid);
            if (g < G)
                for (int i = i0; i < n; i += NT) {
                    dfc l[SW];
#pragma unroll
                    for (int q = 0; q < SW; ++q)
                        if (q < cw) l[q] = dfc_load(A + i + (size_t)(c0 + q) * n);
                    for (int t = g; t < rem; t += G) {
                        float4* qp = A + i + (size_t)(sw + t) * n;
                        dfc a = dfc_load(qp);
#pragma unroll
                        for (int q = 0; q < SW; ++q)
                            if (q < cw) a = dfc_fms(a, l[q], dfc_load(&s.u.p.T[q][t]));
                        dfc_store(qp, a);
                        if (t == 0) {
                            const float v = dfc_abs1(a);
                            if (v > bv) { bv = v; bi = i; }
                        }
                    }
                }
        }
    }
    __syncthreads();
}

// double-float arithmetic of the shared-memory panel (panel.cuh)
struct PanelDf {
    using E = float4;
    static __device__ __forceinline__ dfc v(E a) { return dfc{df{a.x, a.y}, df{a.z, a.w}}; }
    static __device__ __forceinline__ E e(dfc a) { return make_float4(a.re.h, a.re.l, a.im.h, a.im.l); }
    static __device__ __forceinline__ long long key(E a) {
        const float m = dfc_abs1(v(a));
        return m >= 0.0f ? (long long)__float_as_int(m) : -1LL;
    }
    static __device__ __forceinline__ bool zero(E a) { return a.x == 0.0f && a.z == 0.0f; }
    static __device__ __forceinline__ E fms(E a, E l, E u) { return e(dfc_fms(v(a), v(l), v(u))); }
    static __device__ __forceinline__ E prepare(E p, int& mode) {
        mode = 1;
        return e(dfc_recip_pow2(v(p)));
    }
    static __device__ __forceinline__ E scale(E l, E r, int) { return e(dfc_mul(v(l), v(r))); }
};

// As factor_panel of the FP64 engine, but a CTA alone takes shared memory too where
// the panel fits (up to 128 rows): 4096 ln det at n = 64 3.49 -> 2.91 ms.
template <class Team>
__device__ __forceinline__ void df_factor_panel(float4* A, int n, int j0, int jb, int* ipiv, MixSmem& s, const Team& tm) {
    constexpr size_t BYTES = a_band<4>() + b_band<4>();
    const int m = n - j0;
    if (tm.size > 1 && !panel_fits<float4>(m, 1, BYTES) && panel_fits<float4>(m, tm.size, BYTES))
        panel_smem<PanelDf, NT>(A, n, j0, jb, ipiv, s.u.g.buf, s.info, tm);
    else if (tm.rank != 0) return;
    else if (panel_fits<float4>(m, 1, BYTES)) panel_smem<PanelDf, NT>(A, n, j0, jb, ipiv, s.u.g.buf, s.info, Solo{});
    else df_panel(A, n, j0, jb, ipiv, s);
}

__device__ __forceinline__ void dcol_lower_unit(float4* __restrict__ b, int jb, const float4 (*T)[NB + 1]) {
    for (int rb = 0; rb < jb; rb += CH) {
        dfc y[CH];
#pragma unroll
        for (int r = 0; r < CH; ++r) y[r] = (rb + r < jb) ? dfc_load(b + rb + r) : dfc{df{0, 0}, df{0, 0}};
        for (int q = 0; q < rb; ++q) {
            const dfc xq = dfc_load(b + q);
#pragma unroll
            for (int r = 0; r < CH; ++r) y[r] = dfc_fms(y[r], dfc_load(&T[rb + r][q]), xq);
        }
#pragma unroll
        for (int r = 1; r < CH; ++r)
#pragma unroll
            for (int q = 0; q < r; ++q) y[r] = dfc_fms(y[r], dfc_load(&T[rb + r][rb + q]), y[q]);
#pragma unroll
        for (int r = 0; r < CH; ++r)
            if (rb + r < jb) dfc_store(b + rb + r, y[r]);
    }
}

// upper solve; T's diagonal holds the reciprocals of U_rr
__device__ __forceinline__ void dcol_upper(float4* __restrict__ b, int jb, const float4 (*T)[NB + 1]) {
    for (int rb = ((jb - 1) / CH) * CH; rb >= 0; rb -= CH) {
        dfc y[CH];
#pragma unroll
        for (int r = 0; r < CH; ++r) y[r] = (rb + r < jb) ? dfc_load(b + rb + r) : dfc{df{0, 0}, df{0, 0}};
        for (int q = jb - 1; q >= rb + CH; --q) {
            const dfc xq = dfc_load(b + q);
#pragma unroll
            for (int r = 0; r < CH; ++r) y[r] = dfc_fms(y[r], dfc_load(&T[rb + r][q]), xq);
        }
#pragma unroll
        for (int r = CH - 1; r >= 0; --r) {
            if (rb + r < jb) {
                dfc acc = y[r];
#pragma unroll
                for (int q = CH - 1; q > r; --q)
                    if (rb + q < jb) acc = dfc_fms(acc, dfc_load(&T[rb + r][rb + q]), y[q]);
                y[r] = dfc_mul(acc, dfc_load(&T[rb + r][rb + r]));
            }
        }
#pragma unroll
        for (int r = 0; r < CH; ++r)
            if (rb + r < jb) dfc_store(b + rb + r, y[r]);
    }
}

// The same solves with one row a lane, for a warp per column (few columns); every
// element takes its updates in the order of the column solves.
__device__ __forceinline__ dfc dfc_shfl(dfc v, int src) {
    const unsigned FULL = 0xffffffffu;
    return dfc{df{__shfl_sync(FULL, v.re.h, src), __shfl_sync(FULL, v.re.l, src)},
               df{__shfl_sync(FULL, v.im.h, src), __shfl_sync(FULL, v.im.l, src)}};
}
__device__ __forceinline__ dfc drow_lower_unit(dfc x, int jb, const float4 (*T)[NB + 1]) {
    const int lane = threadIdx.x & 31;
    for (int q = 0; q + 1 < jb; ++q) {
        const dfc xq = dfc_shfl(x, q);
        if (lane > q && lane < jb) x = dfc_fms(x, dfc_load(&T[lane][q]), xq);
    }
    return x;
}
__device__ __forceinline__ dfc drow_upper(dfc x, int jb, const float4 (*T)[NB + 1]) {
    const int lane = threadIdx.x & 31;
    for (int q = jb - 1; q >= 0; --q) {
        if (lane == q) x = dfc_mul(x, dfc_load(&T[q][q]));
        const dfc xq = dfc_shfl(x, q);
        if (lane < q) x = dfc_fms(x, dfc_load(&T[lane][q]), xq);
    }
    return x;
}

static __device__ void load_lower_block(const float4* A, int n, int j0, int jb, MixSmem& s) {
    for (int e = threadIdx.x; e < NB * NB; e += NT) {
        int r = e % NB, q = e / NB;
        s.u.p.T[r][q] = (r < jb && q < r) ? A[(j0 + r) + (size_t)(j0 + q) * n] : make_float4(0, 0, 0, 0);
    }
    __syncthreads();
}

static __device__ void load_upper_block(const float4* A, int n, int j0, int jb, MixSmem& s) {
    for (int e = threadIdx.x; e < NB * NB; e += NT) {
        int r = e % NB, q = e / NB;
        float4 v = make_float4(0, 0, 0, 0);
        if (r < jb && q < jb && q > r) v = A[(j0 + r) + (size_t)(j0 + q) * n];
        if (r == q) {
            if (r < jb) {
                const dfc u = dfc_load(A + (j0 + r) + (size_t)(j0 + r) * n);
                const zc ri = 1.0 / mk(df_to_double(u.re), df_to_double(u.im));
                const df a = df_from_double(ri.re), b = df_from_double(ri.im);
                v = make_float4(a.h, a.l, b.h, b.l);
            } else {
                v = make_float4(1, 0, 0, 0);
            }
        }
        s.u.p.T[r][q] = v;
    }
    __syncthreads();
}

// one column through a panel's interchanges (panel_moves), one load and one store a lane
__device__ __forceinline__ void move_rows(float4* a, int j0, int jb, int inner, int orow, int ocur) {
    const int lane = threadIdx.x & 31;
    const float4 z = make_float4(0, 0, 0, 0);
    const float4 v = lane < jb ? a[inner] : z, w = orow >= 0 ? a[ocur] : z;
    __syncwarp();
    if (lane < jb) a[j0 + lane] = v;
    if (orow >= 0) a[orow] = w;
}

// The panel's row interchanges on the columns outside it, then the TRSM
// U12 = L11^-1 A12 of the columns right of it.  keep_l = false leaves the columns
// left of the panel alone: a ln det reads only U's diagonal and the pivots.
template <class Team>
static __device__ void df_swaps_trsm(float4* A, int n, int j0, int jb, const int* ipiv, MixSmem& s, bool keep_l, const Team& tm) {
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    load_lower_block(A, n, j0, jb, s);
    int inner, orow, ocur;
    panel_moves(ipiv, j0, jb, inner, orow, ocur);
    const bool moves = __any_sync(0xffffffffu, inner != j0 + lane);
    const int right = j0 + jb, nr = cta_columns(n - right, tm);
    const int wide = thread_columns(nr, NT);  // the first `wide` a thread each
    if (keep_l && moves) {
        const int nl = cta_columns(j0, tm);
        for (int x = warp; x < nl; x += NW) {
            const int col = cta_column(x, tm);
            if (col < j0) move_rows(A + (size_t)col * n, j0, jb, inner, orow, ocur);
        }
    }
    if (moves)
        for (int x = warp; x < nr; x += NW) {
            const int col = right + cta_column(x, tm);
            if (col < n) move_rows(A + (size_t)col * n, j0, jb, inner, orow, ocur);
        }
    __syncthreads();
    for (int x = wide + warp; x < nr; x += NW) {
        const int col = right + cta_column(x, tm);
        if (col >= n) continue;
        float4* a = A + (size_t)col * n + j0;
        const dfc v = drow_lower_unit(lane < jb ? dfc_load(a + lane) : dfc{df{0, 0}, df{0, 0}}, jb, s.u.p.T);
        if (lane < jb) dfc_store(a + lane, v);
    }
    if (wide > 0) {
        for (int x = tid; x < wide; x += NT) {
            const int col = right + cta_column(x, tm);
            if (col < n) dcol_lower_unit(A + (size_t)col * n + j0, jb, s.u.p.T);
        }
    }
    tm.sync();
}

template <int NS, class Team>
static __device__ void lu_mixed(float4* A, int n, int* ipiv, bool keep_l, MixSmem& s, const MixScratch& X, uint32_t tmem,
                                Phases& ph, const Team& tm) {
    for (int j0 = 0; j0 < n; j0 += NB) {
        const int jb = min(NB, n - j0);
        stat_start(s);
        df_factor_panel(A, n, j0, jb, ipiv, s, tm);
        if (tm.size > 1) tm.sync();
        stat_add(s, PH_PANEL);
        df_swaps_trsm(A, n, j0, jb, ipiv, s, keep_l, tm);
        stat_add(s, PH_TRSM);
        const int r0 = j0 + jb;
        mixed_gemm_sub<NS>(A + r0 + (size_t)r0 * n, n, A + r0 + (size_t)j0 * n, n, A + j0 + (size_t)r0 * n, n, n - r0, n - r0,
                           jb, 0, s, X, tmem, ph, tm);
        if (tm.size > 1) tm.sync();
    }
}

// tr(A^-1 B) from the mixed LU of A; B (double-float, n x n) is destroyed
template <int NS, class Team>
static __device__ zc trace_solve_mixed(const float4* A, float4* B, int n, const int* ipiv, MixSmem& s, const MixScratch& X,
                                  uint32_t tmem, Phases& ph, const Team& tm) {
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int mine = cta_columns(n, tm);
    const dfc zero{df{0, 0}, df{0, 0}};
    for (int j0 = 0; j0 < n; j0 += NB) {
        const int jb = min(NB, n - j0);
        int inner, orow, ocur;
        panel_moves(ipiv, j0, jb, inner, orow, ocur);
        if (!__any_sync(0xffffffffu, inner != j0 + lane)) continue;
        for (int x = warp; x < mine; x += NW) {
            const int col = cta_column(x, tm);
            if (col < n) move_rows(B + (size_t)col * n, j0, jb, inner, orow, ocur);
        }
        __syncwarp();
    }
    __syncthreads();
    for (int j0 = 0; j0 < n; j0 += NB) {
        const int jb = min(NB, n - j0);
        load_lower_block(A, n, j0, jb, s);
        const int wide = thread_columns(mine, NT);
        for (int x = wide + warp; x < mine; x += NW) {
            const int col = cta_column(x, tm);
            if (col >= n) continue;
            float4* b = B + (size_t)col * n + j0;
            const dfc v = drow_lower_unit(lane < jb ? dfc_load(b + lane) : zero, jb, s.u.p.T);
            if (lane < jb) dfc_store(b + lane, v);
        }
        for (int x = tid; x < wide; x += NT) {
            const int col = cta_column(x, tm);
            if (col < n) dcol_lower_unit(B + (size_t)col * n + j0, jb, s.u.p.T);
        }
        tm.sync();
        const int r0 = j0 + jb;
        mixed_gemm_sub<NS>(B + r0, n, A + r0 + (size_t)j0 * n, n, B + j0, n, n - r0, n, jb, 0, s, X, tmem, ph, tm);
        if (tm.size > 1) tm.sync();
    }
    const int nblk = (n + NB - 1) / NB;
    for (int kb = nblk - 1; kb >= 0; --kb) {
        const int j0 = kb * NB, jb = min(NB, n - j0), ncol = j0 + jb;
        load_upper_block(A, n, j0, jb, s);
        const int cols = cta_columns(ncol, tm);
        const int wide = thread_columns(cols, NT);
        for (int x = wide + warp; x < cols; x += NW) {
            const int col = cta_column(x, tm);
            if (col >= ncol) continue;
            float4* b = B + (size_t)col * n + j0;
            const dfc v = drow_upper(lane < jb ? dfc_load(b + lane) : zero, jb, s.u.p.T);
            if (lane < jb) dfc_store(b + lane, v);
        }
        for (int x = tid; x < wide; x += NT) {
            const int col = cta_column(x, tm);
            if (col < ncol) dcol_upper(B + (size_t)col * n + j0, jb, s.u.p.T);
        }
        tm.sync();
        mixed_gemm_sub<NS>(B, n, A + (size_t)j0 * n, n, B + j0, n, j0, ncol, jb, 1, s, X, tmem, ph, tm);
        if (tm.size > 1) tm.sync();
    }
    double tr = 0.0, ti = 0.0, z = 0.0;
    for (int i = tid; i < n; i += NT) {
        dfc v = dfc_load(B + i + (size_t)i * n);
        tr += df_to_double(v.re);
        ti += df_to_double(v.im);
    }
    block_sum3(tr, ti, z, s);
    return mk(tr, ti);
}

// (largest, smallest non-zero) of max(|Re|, |Im|) over the entries seen, with v added
__device__ __forceinline__ float2 entry_range(float2 rg, float4 v) {
    const float a = fmaxf(fabsf(v.x), fabsf(v.z));
    return make_float2(fmaxf(rg.x, a), a > 0.0f ? fminf(rg.y, a) : rg.y);
}

// One 32 x 32 tile of a d != 3 matrix (K_nu elements, FP64, grouped by regime)
// stored as double-floats: the direct triangle here, the mirror by the caller.
// Not inlined, so that d = 3 matrices keep the kernel's registers for themselves.
// rg: the largest and the smallest non-zero max(|Re|, |Im|) of the entries seen.
static __device__ __noinline__ float2 assemble_tile_grouped(float4* __restrict__ A, float4* __restrict__ B, int n,
                                                    int d, const double* __restrict__ pos, zc k, int I, int J,
                                                    zc dg0, zc dg1, MixSmem& s, float2 rg) {
    const int tid = threadIdx.x;
    auto cvt = [](zc v) {
        df a = df_from_double(v.re), b = df_from_double(v.im);
        return make_float4(a.h, a.l, b.h, b.l);
    };
    tile_pairs_grouped<NT>(I, J, n, d, pos, k, B != nullptr, s.u.p.list, s.u.p.cnt, [&](int ii, int jj, zc m, zc dm) {
        const float4 fm = cvt(m);
        rg = entry_range(rg, fm);
        s.u.p.T[jj][ii] = fm;
        if (B) {
            const float4 fd = cvt(dm);
            rg = entry_range(rg, fd);
            s.u.p.T2[jj][ii] = fd;
        }
    });
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ii = tid & 31, jj = (tid >> 5) + 8 * q;
        const int i = I * 32 + ii, j = J * 32 + jj;
        if (i < n && j < n && i <= j) {
            float4 fm = s.u.p.T[jj][ii], fd = make_float4(0, 0, 0, 0);
            if (B) fd = s.u.p.T2[jj][ii];
            if (i == j) {
                fm = cvt(dg0);
                rg = entry_range(rg, fm);
                if (B) {
                    fd = cvt(dg1);
                    rg = entry_range(rg, fd);
                }
            }
            A[i + (size_t)j * n] = fm;
            if (B) B[i + (size_t)j * n] = fd;
        }
    }
    return rg;
}

// One 32 x 32 tile of a d = 2 matrix, every element on the FP32 pipe in
// double-float (green_df2.cuh), the pairs grouped by K_nu regime as in the
// FP64 engine (tile_pairs_grouped): classified into three shared-memory lists,
// then consecutive threads take consecutive list entries, so that a warp runs
// one regime's loop.  Direct triangle here, the mirror by the caller.
static __device__ __noinline__ float2 assemble_tile_grouped_df2(float4* __restrict__ A, float4* __restrict__ B, int n,
                                                        int I, int J, zc dg0, zc dg1, MixSmem& s, float2 rg) {
    const int tid = threadIdx.x;
    const Df2Item& P = s.u.p.d2;
    unsigned short* list = s.u.p.list;
    int* cnt = s.u.p.cnt;
    auto dist = [&](int ii, int jj) {
        const float4 pa = s.u.p.ci[ii], pb = s.u.p.cj[jj];
        const df ex = df_sub(df{pa.x, pa.y}, df{pb.x, pb.y});
        const df ey = df_sub(df{pa.z, pa.w}, df{pb.z, pb.w});
        return df_sqrt(df_add(df_mul(ex, ex), df_mul(ey, ey)));
    };
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int p = tid + NT * q, ii = p & 31, jj = p >> 5;
        const int i = I * 32 + ii, j = J * 32 + jj;
        if (i < n && j < n && i < j) {
            const int reg = k_regime_df(P, dist(ii, jj));
            list[reg * 1024 + atomicAdd(&cnt[reg], 1)] = (unsigned short)p;
        }
    }
    __syncthreads();
    const int c0 = cnt[0], c1 = cnt[1], tot = c0 + c1 + cnt[2];
    for (int w = tid; w < tot; w += NT) {
        const int reg = w < c0 ? 0 : (w < c0 + c1 ? 1 : 2);
        const int p = reg == 0 ? list[w] : (reg == 1 ? list[1024 + w - c0] : list[2048 + w - c0 - c1]);
        const int ii = p & 31, jj = p >> 5;
        dfc m, dm;
        pair_elements_df2(s.u.p.tab, P, dist(ii, jj), reg, B != nullptr, m, dm);
        const float4 fm = make_float4(m.re.h, m.re.l, m.im.h, m.im.l);
        rg = entry_range(rg, fm);
        s.u.p.T[jj][ii] = fm;
        if (B) {
            const float4 fd = make_float4(dm.re.h, dm.re.l, dm.im.h, dm.im.l);
            rg = entry_range(rg, fd);
            s.u.p.T2[jj][ii] = fd;
        }
    }
    __syncthreads();
    if (tid < 3) cnt[tid] = 0;
    auto cvt = [](zc v) {
        df a = df_from_double(v.re), b = df_from_double(v.im);
        return make_float4(a.h, a.l, b.h, b.l);
    };
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ii = tid & 31, jj = (tid >> 5) + 8 * q;
        const int i = I * 32 + ii, j = J * 32 + jj;
        if (i < n && j < n && i <= j) {
            float4 fm = s.u.p.T[jj][ii], fd = make_float4(0, 0, 0, 0);
            if (B) fd = s.u.p.T2[jj][ii];
            if (i == j) {
                fm = cvt(dg0);
                rg = entry_range(rg, fm);
                if (B) {
                    fd = cvt(dg1);
                    rg = entry_range(rg, fd);
                }
            }
            A[i + (size_t)j * n] = fm;
            if (B) B[i + (size_t)j * n] = fd;
        }
    }
    return rg;
}

// Assembly of M(k) (and dM/dk into B) as double-floats; returns the largest
// and the smallest non-zero max(|Re|, |Im|) over the entries this thread stored.
template <bool D3ONLY, class Team>
__device__ float2 assemble_df(float4* __restrict__ A, float4* __restrict__ B, int n, int d,
                             const double* __restrict__ pos, const msgpu_model& mdl, zc k, MixSmem& s, const Team& tm) {
    const int tid = threadIdx.x;
    // F^-1 and the two sides of its central difference (dk_invf), one thread of three warps
    if (tid == 0) s.diag[0] = invf(mdl, d, k);
    if (B && tid == 32) s.diag[1] = invf(mdl, d, k + DK_INVF_STEP);
    if (B && tid == 64) s.diag[2] = invf(mdl, d, k - DK_INVF_STEP);
    __syncthreads();
    const zc dg0 = s.diag[0], dg1 = B ? (s.diag[1] - s.diag[2]) / (2.0 * DK_INVF_STEP) : mk(0.0);
    const bool d3 = D3ONLY || d == 3;
    const df kr = df_from_double(k.re), ki = df_from_double(k.im);
    const bool grow = k.im != 0.0;
    const bool grouped = !D3ONLY && d != 3 && d != 1;
    const bool d2 = !D3ONLY && d == 2;  // d = 2: every element on the FP32 pipe too (green_df2.cuh)
    if (d3 || d2) df3_tables_init(s.u.p.tab);
    if (d2 && tid == 0) s.u.p.d2 = df2_item(k);
    if (grouped && tid < 3) s.u.p.cnt[tid] = 0;
    __syncthreads();
    float2 rg = make_float2(0.0f, INFINITY);
    auto cvt = [](zc v) {
        df a = df_from_double(v.re), b = df_from_double(v.im);
        return make_float4(a.h, a.l, b.h, b.l);
    };
    const int nt = (n + 31) / 32;
    int tile = 0;
    for (int J = 0; J < nt; ++J) {
        for (int I = 0; I <= J; ++I) {
            if (tm.size > 1 && tile++ % tm.size != tm.rank) continue;
            if (d3 || d2) {
                // the tile's atoms as double-floats: rows I*32.., columns J*32..
                if (tid < 64) {
                    const int a = (tid < 32 ? I : J) * 32 + (tid & 31);
                    const int dd = d3 ? 3 : 2;
                    df x{0.0f, 0.0f}, y{0.0f, 0.0f}, z{0.0f, 0.0f};
                    if (a < n) {
                        x = df_from_double(pos[dd * a]);
                        y = df_from_double(pos[dd * a + 1]);
                        if (d3) z = df_from_double(pos[3 * a + 2]);
                    }
                    if (tid < 32) {
                        s.u.p.ci[tid] = make_float4(x.h, x.l, y.h, y.l);
                        s.u.p.ciz[tid] = make_float2(z.h, z.l);
                    } else {
                        s.u.p.cj[tid - 32] = make_float4(x.h, x.l, y.h, y.l);
                        s.u.p.cjz[tid - 32] = make_float2(z.h, z.l);
                    }
                }
                __syncthreads();
            }
            if (grouped) {
                rg = d2 ? assemble_tile_grouped_df2(A, B, n, I, J, dg0, dg1, s, rg)
                        : assemble_tile_grouped(A, B, n, d, pos, k, I, J, dg0, dg1, s, rg);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int ii = tid & 31, jj = (tid >> 5) + 8 * q;
                    const int i = I * 32 + ii, j = J * 32 + jj;
                    if (i < n && j < n && i <= j) {
                        float4 fm, fd = make_float4(0, 0, 0, 0);
                        if (i < j && d3) {
                            // the whole element on the FP32 pipe in double-float (green_df.cuh)
                            const float4 pa = s.u.p.ci[ii], pb = s.u.p.cj[jj];
                            const float2 za = s.u.p.ciz[ii], zb = s.u.p.cjz[jj];
                            const df ex = df_sub(df{pa.x, pa.y}, df{pb.x, pb.y});
                            const df ey = df_sub(df{pa.z, pa.w}, df{pb.z, pb.w});
                            const df ez = df_sub(df{za.x, za.y}, df{zb.x, zb.y});
                            const df r = df_sqrt(df_add(df_add(df_mul(ex, ex), df_mul(ey, ey)), df_mul(ez, ez)));
                            dfc a, b;
                            pair_elements_df3t(s.u.p.tab, kr, ki, grow, r, B != nullptr, a, b);
                            fm = make_float4(a.re.h, a.re.l, a.im.h, a.im.l);
                            if (B) fd = make_float4(b.re.h, b.re.l, b.im.h, b.im.l);
                        } else {
                            zc m, dm = mk(0.0);
                            if (i < j) {
                                pair_elements(d, k, atom_distance(d, pos, i, j), B != nullptr, m, dm);
                            } else {
                                m = dg0;
                                dm = dg1;
                            }
                            fm = cvt(m);
                            if (B) fd = cvt(dm);
                        }
                        rg = entry_range(rg, fm);
                        A[i + (size_t)j * n] = fm;
                        s.u.p.T[jj][ii] = fm;
                        if (B) {
                            rg = entry_range(rg, fd);
                            B[i + (size_t)j * n] = fd;
                            s.u.p.T2[jj][ii] = fd;
                        }
                    }
                }
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int jj = tid & 31, ii = (tid >> 5) + 8 * q;
                const int i = I * 32 + ii, j = J * 32 + jj;
                if (j < n && i < j) {
                    A[j + (size_t)i * n] = s.u.p.T[jj][ii];
                    if (B) B[j + (size_t)i * n] = s.u.p.T2[jj][ii];
                }
            }
            __syncthreads();
        }
    }
    return rg;
}

// The range of an item's entries over its team: FP32 bit patterns of non-negative
// values order like the values, so integer reductions serve.
template <class Team>
__device__ __forceinline__ float2 team_range(float2 rg, MixSmem& s, const Team& tm) {
    const int tid = threadIdx.x;
    if (tid == 0) { s.rng[0] = 0; s.rng[1] = 0x7f800000; }
    __syncthreads();
    const int h = __reduce_max_sync(0xffffffffu, __float_as_int(rg.x)), l = __reduce_min_sync(0xffffffffu, __float_as_int(rg.y));
    if ((tid & 31) == 0) {
        atomicMax(&s.rng[0], h);
        atomicMin(&s.rng[1], l);
    }
    __syncthreads();
    int hi = s.rng[0], lo = s.rng[1];
    if (tm.size > 1) {
        if (tid < tm.size) {
            cluster_store(&s.team_rng[tm.rank][0], tid, hi);
            cluster_store(&s.team_rng[tm.rank][1], tid, lo);
        }
        tm.sync();
        for (int r = 0; r < tm.size; ++r) {
            hi = max(hi, s.team_rng[r][0]);
            lo = min(lo, s.team_rng[r][1]);
        }
    }
    return make_float2(__int_as_float(hi), __int_as_float(lo));
}

// after block_argmax: the CTA-wide maximum (thread 0 folded the warp maxima into red_v)
__device__ __forceinline__ double block_max_value(MixSmem& s) {
    double m = s.red_v[0];
    for (int w = 1; w < NT / 32; ++w) m = fmax(m, s.red_v[w]);
    return m;
}

static __device__ zc tracelog_df(const float4* __restrict__ A, int n, const int* __restrict__ ipiv, MixSmem& s) {
    double lr = 0.0, ar = 0.0, odd = 0.0;
    for (int i = threadIdx.x; i < n; i += NT) {
        const dfc u = dfc_load(A + i + (size_t)i * n);
        const double re = df_to_double(u.re), im = df_to_double(u.im);
        lr += log(hypot(re, im));
        ar += atan2(im, re);
        if (ipiv[i] != i) odd += 1.0;
    }
    block_sum3(lr, ar, odd, s);
    if (fmod(odd, 2.0) == 1.0) ar += PI;
    return mk(lr / n, ar / n);
}

// x <- (LU)^-1 x, one right-hand side, double-float (LAPACK-layout LU): the
// interchanges, then blocked substitution; each block's triangle (the reciprocals
// of U's diagonal with it) in shared memory by the team's first warp, one row per
// lane, the rectangular part by all threads of the team, one row each.
template <class Team>
static __device__ void df_solve_vec(const float4* A, float4* x, int n, const int* ipiv, MixSmem& s, const Team& tm) {
    const int tid = threadIdx.x, lane = tid & 31;
    const dfc zero{df{0, 0}, df{0, 0}};
    if (tm.rank == 0 && tid < 32)
        for (int j0 = 0; j0 < n; j0 += NB) {
            int inner, orow, ocur;
            panel_moves(ipiv, j0, min(NB, n - j0), inner, orow, ocur);
            move_rows(x, j0, min(NB, n - j0), inner, orow, ocur);
            __syncwarp();
        }
    tm.sync();
    auto rows = [&](int j0, int jb, int r0, int r1) {
        tm.sync();  // the block's solution is there
        if (tid < jb) s.u.p.urow[tid] = x[j0 + tid];
        __syncthreads();
        const int mine = cta_columns(r1 - r0, tm);  // rows dealt out in blocks of 32, like columns
        for (int y = tid; y < mine; y += NT) {
            const int i = r0 + cta_column(y, tm);
            if (i >= r1) continue;
            dfc acc = dfc_load(x + i);
            const float4* a = A + i + (size_t)j0 * n;
#pragma unroll 4
            for (int q = 0; q < jb; ++q) acc = dfc_fms(acc, dfc_load(a + (size_t)q * n), dfc_load(&s.u.p.urow[q]));
            dfc_store(x + i, acc);
        }
        tm.sync();
    };
    for (int j0 = 0; j0 < n; j0 += NB) {
        const int jb = min(NB, n - j0);
        if (tm.rank == 0) {
            load_lower_block(A, n, j0, jb, s);
            if (tid < 32) {
                const dfc v = drow_lower_unit(lane < jb ? dfc_load(x + j0 + lane) : zero, jb, s.u.p.T);
                if (lane < jb) dfc_store(x + j0 + lane, v);
            }
        }
        rows(j0, jb, j0 + jb, n);
    }
    for (int j0 = (n - 1) / NB * NB; j0 >= 0; j0 -= NB) {
        const int jb = min(NB, n - j0);
        if (tm.rank == 0) {
            load_upper_block(A, n, j0, jb, s);
            if (tid < 32) {
                const dfc v = drow_upper(lane < jb ? dfc_load(x + j0 + lane) : zero, jb, s.u.p.T);
                if (lane < jb) dfc_store(x + j0 + lane, v);
            }
        }
        rows(j0, jb, 0, j0);
    }
}

// a = M^-1 phi from the mixed LU with iterative refinement: r = phi - M a in
// FP64 against the FP64 copy of M, a += (LU)^-1 r (correction in double-float,
// a kept in FP64), until |r| <= 1e-14 |phi| (max norms), the residual stops
// halving, or 8 corrections.  Returns sigma = -Im(conj(phi).a)/k (the optical
// theorem of total_cross_section, ms_matrix_util.c:361).
// The team shares the residuals (a row a thread) and the solves' rectangular parts.
template <class Team>
static __device__ zc refine_solve(const float4* LU, const zc* M, const zc* phi, zc* x, float4* r, float4* t, const MedDev& md,
                           zc k, const int* ipiv, MixSmem& s, const Team& tm) {
    const int n = md.n, tid = threadIdx.x;
    auto to4 = [](zc v) {
        const df a = df_from_double(v.re), b = df_from_double(v.im);
        return make_float4(a.h, a.l, b.h, b.l);
    };
    if (tm.rank == 0)
        for (int i = tid; i < n; i += NT) t[i] = to4(phi[i]);
    __syncthreads();
    df_solve_vec(LU, t, n, ipiv, s, tm);
    if (tm.rank == 0)
        for (int i = tid; i < n; i += NT) {
            const dfc v = dfc_load(t + i);
            x[i] = mk(df_to_double(v.re), df_to_double(v.im));
        }
    tm.sync();
    double pmax = 0.0;
    for (int i = tid; i < n; i += NT) pmax = fmax(pmax, zabs(phi[i]));
    int dummy;
    block_argmax(pmax, tid, s, dummy);
    pmax = block_max_value(s);
    __syncthreads();
    double prev = INFINITY;
    for (int it = 0; it < 8; ++it) {
        // r = phi - M x in FP64, rows over threads (coalesced columns of M)
        double rmax = 0.0;
        for (int i = tm.rank * NT + tid; i < n; i += NT * tm.size) {
            zc acc = phi[i];
            for (int j = 0; j < n; ++j) {
                const zc mv = M[i + (size_t)j * n], xv = x[j];
                acc.re = fma(-mv.re, xv.re, fma(mv.im, xv.im, acc.re));
                acc.im = fma(-mv.re, xv.im, fma(-mv.im, xv.re, acc.im));
            }
            r[i] = to4(acc);
            rmax = fmax(rmax, fabs(acc.re) + fabs(acc.im));
        }
        block_argmax(rmax, tid, s, dummy);
        rmax = block_max_value(s);
        __syncthreads();
        if (tm.size > 1) {
            if (tid < tm.size) cluster_store(&s.team_max[tm.rank], tid, rmax);
            tm.sync();  // and every part of r is there
            for (int q = 0; q < tm.size; ++q) rmax = fmax(rmax, s.team_max[q]);
        }
        if (!(rmax > 1e-14 * pmax) || !(rmax < 0.5 * prev)) break;
        prev = rmax;
        df_solve_vec(LU, r, n, ipiv, s, tm);
        if (tm.rank == 0)
            for (int i = tid; i < n; i += NT) {
                const dfc v = dfc_load(r + i);
                x[i] = x[i] + mk(df_to_double(v.re), df_to_double(v.im));
            }
        tm.sync();
    }
    double dr = 0.0, di = 0.0, z = 0.0;
    for (int i = tid; i < n; i += NT) {
        const zc tt = conjz(phi[i]) * x[i];
        dr += tt.re;
        di += tt.im;
    }
    block_sum3(dr, di, z, s);
    return mk(-di, 0.0) / k;
}

// One instantiation per job kind (0 ln det, 1 dlogf, 2 amplitudes) and per
// dimension class (D3ONLY: every medium of the job has d = 3): each carries
// only its own reduction, solve and Green function, so a kernel's registers
// are not shaped by code it never runs (a never-taken call to the d != 3 tile
// cost the d = 3 ln det kernel 5 %).
// Each comes for one CTA per matrix (Solo) and for a cluster of them (ClusterTeam),
// which a batch that leaves SMs idle takes: one wavefunction at n = 1024, 512 x 512
// pixels, 74 ms with one CTA, 31 with a cluster of 16.
// host entries of the variants (mixed_k*.cu, mixed_t*.cu): the largest number of
// clusters resident (query), or launch
struct MixLaunch {
    int teams, team;  // matrices at a time, CTAs on each
    size_t smem;
    cudaStream_t st;
    bool query;
};
int mixed_variant_0_d3(const EngineParams&, const MixScratch&, const MixLaunch&);
int mixed_variant_1_d3(const EngineParams&, const MixScratch&, const MixLaunch&);
int mixed_variant_2_d3(const EngineParams&, const MixScratch&, const MixLaunch&);
int mixed_variant_0_any(const EngineParams&, const MixScratch&, const MixLaunch&);
int mixed_variant_1_any(const EngineParams&, const MixScratch&, const MixLaunch&);
int mixed_variant_2_any(const EngineParams&, const MixScratch&, const MixLaunch&);
int mixed_team_0_d3(const EngineParams&, const MixScratch&, const MixLaunch&);
int mixed_team_1_d3(const EngineParams&, const MixScratch&, const MixLaunch&);
int mixed_team_2_d3(const EngineParams&, const MixScratch&, const MixLaunch&);
int mixed_team_0_any(const EngineParams&, const MixScratch&, const MixLaunch&);
int mixed_team_1_any(const EngineParams&, const MixScratch&, const MixLaunch&);
int mixed_team_2_any(const EngineParams&, const MixScratch&, const MixLaunch&);

#ifdef MSG_MIXED_KERNEL_BODY
__device__ __forceinline__ void make_team(Solo&) {}
__device__ __forceinline__ void make_team(ClusterTeam& t) { t = this_team(); }

template <int KIND, bool D3ONLY, class Team>
__global__ void __launch_bounds__(NT, 2) k_engine_mixed(EngineParams P, MixScratch X)
{
    extern __shared__ uint8_t smem_raw[];
    MixSmem& s = *reinterpret_cast<MixSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    const int tid = threadIdx.x, warp = tid >> 5;
    if (warp == 0) {
        tmem_alloc(&s.tmem, TMEM_COLS);
        tmem_relinquish();
    }
    if (tid == 0) {
        mbar_init(&s.bar_a, 1);
        mbar_init(&s.bar_b, 1);
        mbar_init(&s.bar_mma, 1);
        s.err = 0;
        s.mma_stuck = 0;
        for (int i = 0; i < PH_N; ++i) s.stat[i] = 0;
        fence_mbar_init();
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s.tmem;
    Team tm;
    make_team(tm);
    Phases ph{0, 0, 0};
    const size_t vec = (((size_t)P.piv_stride + 15) / 16) * 16, team = blockIdx.x / tm.size;
    const size_t slot_all = KIND == 0 ? P.slot : (KIND == 1 ? 2 * P.slot : 2 * P.slot + 4 * vec);
    float4* A = reinterpret_cast<float4*>(P.ws) + team * slot_all;
    float4* B = (KIND == 1) ? A + P.slot : nullptr;
    // kind 2: copy of M, right-hand side phi, solution, residual, correction
    zc* Mc = reinterpret_cast<zc*>(A + P.slot);  // kind 2: M in FP64 for the refinement
    zc* vphi = reinterpret_cast<zc*>(A + 2 * P.slot);
    zc* vx = vphi + vec;
    float4* vr = reinterpret_cast<float4*>(vx + vec);
    float4* vt = vr + vec;
    int* ipiv = P.piv + team * P.piv_stride;
    if (tm.size > 1) tm.sync();  // every CTA of the cluster is there before its shared memory is written
    bool alive = true;
    while (alive) {
        if (tm.rank == 0 && tid == 0) {
            const unsigned q = atomicAdd(P.counter, 1u);
            const int item = q < P.counter[1] ? (int)q : P.nitem;
            s.item = item;
            for (int r = 1; r < tm.size; ++r) cluster_store(&s.item, r, item);
            s.info = 0;
        }
        tm.sync();
        const int q = s.item;
        if (q >= P.nitem) break;
        const int it = P.order[q];
        const MedDev md = P.media[P.item_med[it]];
        const zc k = mk(P.ks[2 * it], P.ks[2 * it + 1]);
        stat_start(s);
        float2 rg = assemble_df<D3ONLY>(A, B, md.n, md.d, md.pos, md.model, k, s, tm);
        stat_add(s, PH_ASSEMBLE);
        rg = team_range(rg, s, tm);
        const double mxd = rg.x, mnd = rg.y;
        // six slices when the entries span more than SPAN_WIDE (SPAN_WIDE_REFINED for amplitude
        // items) or an entry is zero / non-finite, and for every dlogf item (near a root the condition number of M magnifies the LU's
        // error in tr(M^-1 dM/dk)), if this launch has the shared memory for them; else four,
        // and a status bit says so
        const double thr = KIND == 2 ? (double)SPAN_WIDE_REFINED : (double)SPAN_WIDE;
        const bool span_wide = KIND == 1 || !(mxd <= thr * mnd);
        const bool wide = span_wide && P.wide_ok;
        zc res = mk(0.0);
        int st = 0;
        if (!(mxd < (double)RANGE_LIMIT)) {
            st |= MSGPU_S_RANGE;
            res = mk(nan(""), nan(""));
        } else {
            if (KIND == 2) {
                // M in FP64 for the residual, every element as the FP64 engine assembles it;
                // incident plane wave along +x (incident_wave_util.c:76)
                EntryRange er;
                __syncthreads();
                stat_start(s);
                assemble(Mc, nullptr, md.n, md.d, md.pos, md.model, k, s.u.lu, tm, er);
                if (tm.rank == 0)
                    for (int i = tid; i < md.n; i += NT) vphi[i] = zexp(mk(0.0, 1.0) * k * md.pos[i * md.d]);
                stat_add(s, PH_ASSEMBLE);
            }
            tm.sync();
            if (wide) lu_mixed<6>(A, md.n, ipiv, KIND != 0, s, X, tmem, ph, tm);
            else lu_mixed<4>(A, md.n, ipiv, KIND != 0, s, X, tmem, ph, tm);
            if (KIND == 0) {
                if (tm.rank == 0) res = tracelog_df(A, md.n, ipiv, s);
            } else if (KIND == 1) {
                res = wide ? trace_solve_mixed<6>(A, B, md.n, ipiv, s, X, tmem, ph, tm)
                           : trace_solve_mixed<4>(A, B, md.n, ipiv, s, X, tmem, ph, tm);
            } else {
                stat_start(s);
                res = refine_solve(A, Mc, vphi, vx, vr, vt, md, k, ipiv, s, tm);
                stat_add(s, PH_SOLVE);
                if (P.amps && tm.rank == 0)
                    for (int i = tid; i < md.n; i += NT) {
                        P.amps[2 * (P.amp_off[it] + i)] = vx[i].re;
                        P.amps[2 * (P.amp_off[it] + i) + 1] = vx[i].im;
                    }
            }
        }
        // a wait that ran out in some CTA: the team agrees to stop
        __syncthreads();
        int bad = s.err;
        if (tm.size > 1) {
            if (tid < tm.size) cluster_store(&s.team_bad[tm.rank], tid, bad);
            tm.sync();
            for (int r = 0; r < tm.size; ++r) bad |= s.team_bad[r];
        }
        if (bad) {
            alive = false;
            st |= MSGPU_S_TIMEOUT;
            res = mk(nan(""), nan(""));
        }
        if (KIND == 2 && tm.rank == 0 && (st & (MSGPU_S_TIMEOUT | MSGPU_S_RANGE))) void_amplitudes(P, it, tid, NT);
        if (tm.rank == 0 && tid == 0) {
            s.stat[PH_ITEMS] += 1;
            if (span_wide && !wide) st |= MSGPU_S_SPAN;
            P.out[2 * it] = res.re;
            P.out[2 * it + 1] = res.im;
            if (s.info) st |= MSGPU_S_SINGULAR;
            if (!isfinite(res.re) || !isfinite(res.im)) st |= MSGPU_S_NONFINITE;
            P.status[it] = st;
        }
        tm.sync();
    }
    if (!alive && tm.rank == 0 && tid == 0) {
        atomicExch(X.err, 1);
        // the run is abandoned: every item not yet taken is marked, none keeps a stale result
        for (unsigned q = atomicAdd(P.counter, 1u); q < P.counter[1] && (int)q < P.nitem;
             q = atomicAdd(P.counter, 1u)) {
            const int it = P.order[q];
            P.out[2 * it] = P.out[2 * it + 1] = nan("");
            P.status[it] = MSGPU_S_TIMEOUT;
            void_amplitudes(P, it, 0, 1);
        }
    }
    if (X.stats && tid == 0)
        for (int i = 0; i < PH_N; ++i) atomicAdd(X.stats + i, s.stat[i]);
    // an MMA completion wait that ran out may leave MMAs in flight: give them a bounded chance to land
    if (s.mma_stuck && tid == 0) mbar_wait(&s.bar_mma, (uint32_t)(s.mma_stuck - 1), 1 << 20);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, TMEM_COLS);
}

// launch or query of one variant
template <int KIND, bool D3ONLY, class Team>
static int mixed_variant(const EngineParams& P, const MixScratch& X, const MixLaunch& L) {
    auto* kern = k_engine_mixed<KIND, D3ONLY, Team>;
    static bool done[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return MSGPU_E_CUDA;
    if (dev >= 64 || !done[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MIX_SMEM_WIDE) != cudaSuccess ||
            cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            return MSGPU_E_CUDA;
        if (dev < 64) done[dev] = true;
    }
    if (L.query) return max_teams(kern, L.team, NT, L.smem);
    return launch_teams(kern, L.teams, L.team, NT, L.smem, L.st, P, X);
}
#endif

}  // namespace msg
