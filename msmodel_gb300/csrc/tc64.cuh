// tc64.cuh -- the FP64 engine's trailing update C -= A B on the tcgen05 tensor cores.
//
// GB300's FP64 pipe does 2 FMAs a clock per SM (1.25 TFLOP/s on the chip) and
// 4 n^3 / 3 of them are the whole cost of a large complex LU.  Here every row
// of A and every column of B (K <= 32 entries) is scaled by a power of two to
// 71-bit fixed point and cut into eight balanced digits of 9 bits,
//     V = sum_k d_k 2^(9 (7 - k)),  |d_k| <= 256,
// which bf16 holds exactly.  The digit products (i, j) with l = i + j <= 7 are
// summed by tcgen05.mma kind::f16 in the FP32 accumulator of their level l,
// integers of at most (l + 1) 2^22: below 2^24, hence exact, for levels 0..3, and
// beyond it only if almost every digit is extreme (such elements are redone).  The
// levels are put together in 64-bit integers that keep 60 bits of the sum itself
// and meet C in one FP64 addition.
//
// What that leaves out (digit products of level 8 and up, entries more than 2^18
// below their row's largest cut off) is 2^-69 of row maximum x column maximum (rms;
// 2^-63 at most), whatever the element's own size.  So an element whose old and
// new values are both below 2^-TC_REDO of that product is redone on the FP64 pipe
// with the chain of FMAs it would have had there, as is one with a row or column that
// holds an infinity, a NaN or a subnormal maximum: every element is as good as
// the chain's, whatever the matrix.  Redone elements go on a list that the CTA works off
// while the tensor core has the next tile.
//
// Measured against the FP64 pipe's update in the same kernel: 198 ln det at d = 3,
// n = 1024 126 ms and 627, 152 at n = 512 14.5 and 57.9, 304 at n = 160 3.0 and 5.2, 152 dlogf
// at n = 300 11.7 and 45.8; 152 ln det at d = 2, n = 700, where more is redone, 162 and 258.
// Error of ln det / n against a wider LU of the same matrix (n = 300, rms of 6): d = 3,
// real k 2.0e-16 and 1.9e-16, Im k = -0.05 1.3e-16 and 2.4e-16, -1 4.9e-16 and 4.7e-16; d = 2,
// real k 7.6e-16 and 6.8e-16, Im k = -0.3 1.2e-16 and 4.1e-16, -0.55 (entries span 2^13)
// 1.3e-14 and 1.4e-14.  (Seven digits, levels up to 6 and a unit of 2^-55 of the product of
// maxima without redoing anything took 112 ms at n = 1024, but lost up to 400 times
// the chain's error where rows and columns are uneven.)
//
// One CTA of 512 threads per SM: A band 128 rows x 32 (8 digits x Re/Im, 128 KB),
// one B buffer of 32 columns (48 KB), 8 levels x Re/Im x 32 = 512 TMEM columns, all
// there are.  B's rows are stacked -Im, Re, Im, so that A_re times (Re, Im) and A_im
// times (-Im, Re) are one MMA of N = 64 each, 83 cycles apiece.  A is sliced straight into shared
// memory, B once per update into a global image that bulk copies (TMA engine) bring in,
// the next tile's while this one's epilogue runs.
#pragma once
#include <cuda_bf16.h>
#include "lu64.cuh"
#include "umma.cuh"
#include "engine_internal.h"

namespace msg {

constexpr int TC_NT = 512;
constexpr int TC_M = 128;   // tile rows = TMEM lanes
constexpr int TC_N = 32;    // tile columns
constexpr int TC_NS = 8;    // digits = levels
constexpr int TC_ASUB = TC_M * NB * 2;           // one digit of Re or Im of an A band: 8 KB
constexpr int TC_BROWS = 3 * TC_N;               // a B tile's operand rows: -Im, Re, Im of its columns
constexpr int TC_BSUB = TC_BROWS * NB * 2;       // one digit of them: 6 KB
constexpr int TC_ABAND = 2 * TC_NS * TC_ASUB;    // 128 KB
constexpr int TC_BDIG = TC_NS * TC_BSUB;         // 48 KB
constexpr int TC_BTILE = TC_BDIG + TC_N * 4;     // a tile of the image: digits, then the columns' exponents
constexpr uint32_t TC_TMEM = 512;
// Items whose entries span more than 2^TC_SPAN_LOG2, or lie beyond 2^+-300, stay on the
// FP64 pipe: they would have a large part of their elements redone (of media in a ball, d = 3
// below 1 in 300 at real k = 0.6, n = 1024, the least favourable; d = 2, n = 700 3 in 100).
constexpr int TC_SPAN_LOG2 = 16;
constexpr int TC_EXP_MIN = 1023 - 300, TC_EXP_MAX = 1023 + 300;
// An element is redone below 2^-TC_REDO of row maximum x column maximum: there 2^-69 of
// that product is 2^-56 of the element, an eighth of the rounding of one FMA.
constexpr int TC_REDO = 13;
constexpr int TC_BAD = 1 << 20;     // exponent of a row or column whose largest entry is infinite, NaN or subnormal
constexpr int TC_ZERO = -(1 << 17); // ... and of one of zeros
// sums of two biased exponents between which a product is a normal number to its last bit
constexpr int TC_PLO = 2046 - 900, TC_PHI = 2046 + 900;

// shared memory: what lasts through an item, then the FP64 pipe's tiles (panel,
// TRSM, assembly; names as in LuSmemT) over the tensor core's operand buffers
struct Tc64Smem {
    static constexpr int NTH = TC_NT, TNC = TC_NT / 4, TMR = TM;
    static constexpr size_t PANEL_BYTES = TC_ABAND + TC_BDIG;
    __device__ __forceinline__ void* panel_buf() { return g.a; }  // a panel between updates
    uint64_t bar_b, bar_mma;
    uint32_t tmem;
    int err, mma_stuck;
    int ea[TC_M];             // exponents of the A band's rows
    union {
        int emax[TC_M];       // slicing
        zc dlo[NB];           // solves
    };
    int redo_n[3];            // elements to redo, by tile number mod 3
    unsigned short redo[2][TC_M * TC_N];  // ... (row in the tile) 32 + column, by tile parity
    int rng[2];               // the item's entry range (EntryRange), this CTA's part
    int team_rng[16][2];      // ... and every CTA's of the team
    int team_bad[16];         // every CTA's flag of a wait that ran out
    zc urow[NB];
    zc piv, rpiv;
    zc diag[2];
    long long red_k[2][TC_NT / 32];
    int red_p[2][TC_NT / 32];
    double red_v[TC_NT / 32];
    int red_i[TC_NT / 32];
    double red_s[3][TC_NT / 32];
    int info, bcast_i, item, nz;
    union {
        alignas(128) uint8_t base;
        struct {
            zc As[NB][TM];
            zc Bs[NB][TNC];
            zc T[NB][NB + 1];
        };
        struct {
            uint8_t a[TC_ABAND];
            uint8_t b[TC_BDIG];
        } g;
    };
};

// (with the 1 KB the system takes: beyond 196 KB the L1 cache shrinks from 60 to 28 KB,
// which costs 5% at n = 1024)
static_assert(sizeof(Tc64Smem) + 128 <= 195 * 1024, "shared memory leaves the L1 cache its share");

// 71-bit fixed point of x for a row whose largest entry has biased exponent E,
// round(x 2^(1022 - E + 71)), |.| <= 2^71, as hi 2^27 + lo
__device__ __forceinline__ void tc_fixed(double x, int E, long long& hi, int& lo) {
    const long long b = __double_as_longlong(x);
    const int ex = (int)(b >> 52) & 0x7ff;
    const int sh = E - max(ex, 1);
    const long long m = (b & 0xfffffffffffffLL) | (ex ? 0x10000000000000LL : 0);
    const int mask = (1 << 27) - 1;
    if (sh <= 18) {
        hi = m >> (9 + sh);
        lo = (int)((unsigned long long)m << (18 - sh)) & mask;
    } else {
        const long long v = sh > 72 ? 0 : (m + (1LL << (sh - 19))) >> (sh - 18);
        hi = v >> 27;
        lo = (int)v & mask;
    }
    if (b < 0) {
        hi = -hi;
        lo = -lo;
    }
}

// balanced 9-bit digit of v, which moves to the next
template <class T>
__device__ __forceinline__ int tc_digit(T& v) {
    const int d = (int)(((unsigned)v + 256u) & 511u) - 256;
    v = (v - d) >> 9;
    return d;
}

__device__ __forceinline__ uint32_t tc_pack(int a, int b) {
    // |a|, |b| <= 256: exact in bf16; the integers become floats by the 1.5 x 2^23 offset
    const float fa = __int_as_float(0x4B400000 + a) - 12582912.0f, fb = __int_as_float(0x4B400000 + b) - 12582912.0f;
    __nv_bfloat162 v = __floats2bfloat162_rn(fa, fb);
    return *reinterpret_cast<uint32_t*>(&v);
}

// digits of 8 consecutive k of one row: put(digit, 0 Re / 1 Im, 8 bf16)
template <class Put>
__device__ __forceinline__ void tc_store_digits(const zc* v, int E, Put put) {
    const bool none = E >= TC_BAD || E <= 0;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        long long x[8];
        int y[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            x[k] = 0;
            y[k] = 0;
            if (!none) tc_fixed(c ? v[k].im : v[k].re, E, x[k], y[k]);
        }
#pragma unroll
        for (int s = TC_NS - 1; s >= 0; --s) {
            int d[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (s == TC_NS - 4) x[k] += y[k];  // the low part's carry
                d[k] = s >= TC_NS - 3 ? tc_digit(y[k]) : s > 0 ? tc_digit(x[k]) : (int)x[k];
            }
            put(s, c, make_uint4(tc_pack(d[0], d[1]), tc_pack(d[2], d[3]), tc_pack(d[4], d[5]), tc_pack(d[6], d[7])));
        }
    }
}

// largest of 8 entries' |components|: the high word of the double (0 only for zeros)
__device__ __forceinline__ int tc_emax(const zc* v) {
    int h = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        h = max(h, (__double2hiint(v[k].re) & 0x7fffffff) | (__double2loint(v[k].re) != 0));
        h = max(h, (__double2hiint(v[k].im) & 0x7fffffff) | (__double2loint(v[k].im) != 0));
    }
    return h;
}

// the exponent that goes with a row's digits, from its tc_emax
__device__ __forceinline__ int tc_row_exp(int h) {
    const int e = h >> 20;
    return h == 0 ? TC_ZERO : e == 0 || e == 0x7ff ? TC_BAD : e;
}

// per-kernel state of the tensor-core update
struct TcState {
    uint8_t* img;      // the team's B image: ceil(nmax / 32) tiles of TC_BTILE
    uint32_t tmem;
    uint32_t ph_b, ph_mma;  // phases of bar_b and bar_mma
    int first_wait;    // poll limit of an update's first operand wait
    bool use;          // the item's updates run on the tensor cores
};

// A band: rows [r0, r0 + 128) of the m x K panel, digits into shared memory
static __device__ void tc_slice_a(const zc* Ap, int lda, int r0, int m, int K, Tc64Smem& s) {
    const int tid = threadIdx.x, r = tid & (TC_M - 1), kb = tid / TC_M;
    zc v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int kk = 8 * kb + k;
        v[k] = (r0 + r < m && kk < K) ? Ap[r0 + r + (size_t)kk * lda] : mk(0.0);
    }
    if (tid < TC_M) s.emax[tid] = 0;
    __syncthreads();
    atomicMax(&s.emax[r], tc_emax(v));
    __syncthreads();
    const int E = tc_row_exp(s.emax[r]);
    if (kb == 0) s.ea[r] = E;
    uint8_t* dst = s.g.a + cm_offset(r, 8 * kb, TC_M);
    tc_store_digits(v, E, [&](int d, int c, uint4 w) { *reinterpret_cast<uint4*>(dst + (2 * d + c) * TC_ASUB) = w; });
}

// B image: columns [0, nn) of the K x nn block, four threads a column
template <class Team>
static __device__ void tc_slice_b(const zc* Bp, int ldb, int nn, int K, uint8_t* img, const Team& tm) {
    const int np = (nn + TC_N - 1) / TC_N * TC_N, kb = threadIdx.x & 3;
    for (int j = tm.rank * (TC_NT / 4) + (threadIdx.x >> 2); j < np; j += tm.size * (TC_NT / 4)) {
        uint8_t* tile = img + (size_t)(j / TC_N) * TC_BTILE;
        const int r = j % TC_N;
        zc v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int kk = 8 * kb + k;
            v[k] = (j < nn && kk < K) ? Bp[kk + (size_t)j * ldb] : mk(0.0);
        }
        int e = tc_emax(v);
        const unsigned grp = 0xfu << (threadIdx.x & 28);
        e = max(e, __shfl_xor_sync(grp, e, 1));
        e = max(e, __shfl_xor_sync(grp, e, 2));
        const int E = tc_row_exp(e);
        if (kb == 0) *reinterpret_cast<int*>(tile + TC_BDIG + 4 * r) = E;
        tc_store_digits(v, E, [&](int d, int c, uint4 w) {
            uint8_t* p = tile + d * TC_BSUB;
            *reinterpret_cast<uint4*>(p + cm_offset((c + 1) * TC_N + r, 8 * kb, TC_BROWS)) = w;
            const uint32_t neg = 0x80008000u;
            if (c) *reinterpret_cast<uint4*>(p + cm_offset(r, 8 * kb, TC_BROWS)) = make_uint4(w.x ^ neg, w.y ^ neg, w.z ^ neg, w.w ^ neg);
        });
    }
}

// the products of one tile, issued by warp 0 (lead: its elected lane)
__device__ __forceinline__ void tc_issue_tile(uint32_t a0, uint32_t b0, uint64_t* bar, uint32_t tmem, uint32_t lead) {
    const uint32_t id2 = idesc_bf16(TC_M, 2 * TC_N);
    const uint64_t da0 = sdesc(a0, TC_M * 16, 128), db0 = sdesc(b0, TC_BROWS * 16, 128);
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
        // a descriptor's start address counts 16-byte units, a K step of 16 is two core-matrix columns
        auto dA = [&](int i, int c) { return da0 + (ks * (TC_M * 32) + (2 * i + c) * TC_ASUB) / 16; };
        auto dB = [&](int j, int row) { return db0 + (ks * (TC_BROWS * 32) + j * TC_BSUB + row * 16) / 16; };
#pragma unroll
        for (int l = 0; l < TC_NS; ++l) {
            const uint32_t t = tmem + 2 * TC_N * l;
#pragma unroll
            for (int i = 0; i <= l; ++i) {
                umma_bf16_lead(t, dA(i, 0), dB(l - i, TC_N), id2, (ks == 0 && i == 0) ? 0u : 1u, lead);
                umma_bf16_lead(t, dA(i, 1), dB(l - i, 0), id2, 1, lead);
            }
        }
    }
    umma_commit_lead(bar, lead);
}

// Sum of the levels, level l of weight 2^(-16 - 9 l) of row maximum x column
// maximum, as v 2^xe of that product: at least 60 bits of the sum unless it is exact.
// False if a level of weight may have left the exact integers on the way: its
// partial sums stay within (l + 1) 2^22, so one that passed 2^24 ends above 2^25 - (l + 1) 2^22.
__device__ __forceinline__ bool tc_levels(const float* L, long long& v, int& xe) {
    int i[TC_NS];
#pragma unroll
    for (int l = 0; l < TC_NS; ++l) i[l] = __float2int_rn(L[l]);
    // levels 0..3 in units of 2^-43, levels 4..7 in units of 2^-79
    const long long h = ((long long)i[0] << 27) + ((long long)i[1] << 18) + ((long long)i[2] << 9) + i[3];
    const long long lo = ((long long)i[4] << 27) + ((long long)i[5] << 18) + ((long long)i[6] << 9) + i[7];
    const int s = min(36, __clzll(h ^ (h >> 63)) - 4);  // |h 2^s| < 2^60
    v = (h << s) + ((lo + ((1LL << (36 - s)) >> 1)) >> (36 - s));
    xe = -43 - s;
    return abs(i[4]) < 3 << 22 && abs(i[5]) < 2 << 22;
}

// v 2^xe, rounded to the nearest double (halves away from zero) in integer
// arithmetic: a conversion instruction would take the FP64 pipe as long as the
// one addition the update needs
__device__ __forceinline__ double tc_double(long long v, int xe) {
    unsigned long long u = v < 0 ? -v : v;
    const int lz = __clzll(u);
    u <<= lz & 63;
    const int e = xe + 1023 + 63 - lz;
    long long b = ((long long)(e - 1) << 52) + (long long)((u >> 11) + ((u >> 10) & 1));
    if (e < 1 || v == 0) b = 0;  // nothing to subtract, or nothing beside C
    return __longlong_as_double(b | (v & (long long)0x8000000000000000ULL));
}

// one element's update on the FP64 pipe, the operations of gemm_sub in their order
static __device__ __noinline__ void tc_redo(zc* C, int ldc, const zc* Ap, int lda, const zc* Bp, int ldb, int K, int row,
                                            int col) {
    zc a = C[row + (size_t)col * ldc];
    const zc* l = Ap + row;
    const zc* u = Bp + (size_t)col * ldb;
    int k = 0;
    for (; k + 8 <= K; k += 8) {  // eight operands on their way ahead of the chain
        zc lk[8], uk[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            lk[j] = l[(size_t)(k + j) * lda];
            uk[j] = u[k + j];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) a = zfms(a, lk[j], uk[j]);
    }
    for (; k < K; ++k) a = zfms(a, l[(size_t)k * lda], u[k]);
    C[row + (size_t)col * ldc] = a;
}

// C[m x nn] -= Ap[m x K] Bp[K x nn], all column-major; tri: only tiles holding
// an element with row >= column.  The team deals out the tiles in row-band
// order, in contiguous runs.  A wait that ran out sets s.err: the CTA then
// issues no more MMAs but keeps to the barriers, and its items are marked.
template <class Team>
static __device__ __noinline__ void tc_update(zc* C, int ldc, const zc* Ap, int lda, const zc* Bp,
                                 int ldb, int m, int nn, int K, int tri, Tc64Smem& s, Team tm, TcState& t) {
    if (m <= 0 || nn <= 0 || K <= 0) return;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform, so is the branch around the MMAs
    const uint32_t tmem = __shfl_sync(0xffffffffu, t.tmem, 0);
    if (tid < 3) s.redo_n[tid] = 0;
    tc_slice_b(Bp, ldb, nn, K, t.img, tm);
    fence_proxy_async_all();
    tm.sync();
    fence_proxy_async_all();
    const int nbi = (m + TC_M - 1) / TC_M, nbj = (nn + TC_N - 1) / TC_N;
    // tiles of row band bi: columns [0, width(bi))
    auto width = [&](int bi) { return tri ? min(nbj, (bi * TC_M + TC_M - 1) / TC_N + 1) : nbj; };
    int total = 0;
    for (int b = 0; b < nbi; ++b) total += width(b);
    int todo = (int)((long long)total * (tm.rank + 1) / tm.size), at = (int)((long long)total * tm.rank / tm.size);
    todo -= at;
    int bi = 0, bj = at;
    while (bi < nbi && bj >= width(bi)) bj -= width(bi++);
    auto load_b = [&](int col) {
        mbar_arrive_expect_tx(&s.bar_b, TC_BDIG);
        bulk_g2s(s.g.b, t.img + (size_t)col * TC_BTILE, TC_BDIG, &s.bar_b);
    };
    // the elements on the list of tile number x, tile (i, j): a chain of 64 FMAs, 4 k cycles, that
    // is over before the next tile's MMAs unless warp 0, which issues them, takes part
    // (ln det at n = 1024, one such element a tile: update 80 M cycles, 84 with warp 0)
    auto redo = [&](int x, int i, int j) {
        const int cnt = s.redo_n[x % 3];
        if (warp == 0) return;
        for (int e = tid - 32; e < cnt; e += TC_NT - 32) {
            const int c = s.redo[x & 1][e];
            tc_redo(C, ldc, Ap, lda, Bp, ldb, K, i * TC_M + c / TC_N, j * TC_N + c % TC_N);
        }
    };
    int limit = t.first_wait;
    // warp 0: this tile's B copy is under way (none is issued once a wait has run out)
    bool pend = __shfl_sync(0xffffffffu, todo > 0 && !s.err, 0);
    if (tid == 0 && pend) load_b(bj);
    int band = -1, x = 0, bi0 = 0, bj0 = 0;  // band in shared memory, tile number, the tile before
    const int q = warp & 3, cg = warp >> 2;  // TMEM lane quadrant, group of 8 columns
    const int rloc = 32 * q + lane;
    for (; todo > 0; --todo, ++x) {
        if (bi != band) {  // the previous tile's MMAs are complete: the band's buffer is free
            tc_slice_a(Ap, lda, bi * TC_M, m, K, s);
            fence_proxy_async();
            __syncthreads();
            band = bi;
        }
        if (warp == 0) {
            bool ok = pend;
            if (pend) {
                ok = mbar_wait(&s.bar_b, t.ph_b, limit);
                if (!ok) mbar_wait(&s.bar_b, t.ph_b);  // let the copy in flight land before moving on
                t.ph_b ^= 1;
                limit = WAIT_LIMIT;
            }
            if (__all_sync(0xffffffffu, ok && !s.err)) {
                tc_fence_after();
                tc_issue_tile(smem_u32(s.g.a), smem_u32(s.g.b), &s.bar_mma, tmem, elect_lane());
            } else if (lane == 0) {
                s.err = 1;                // operands missing: no MMA is issued;
                mbar_arrive(&s.bar_mma);  // release this tile's MMA wait at once
            }
            __syncwarp();
        }
        // While the tensor core works: what the tile before left to redo (its list is complete since
        // the barrier, the list after this tile's is empty again), then this thread's row and 8
        // columns of C
        if (x > 0) redo(x - 1, bi0, bj0);
        if (tid == 0) s.redo_n[(x + 1) % 3] = 0;
        const int row = bi * TC_M + rloc, col0 = bj * TC_N + 8 * cg;
        const bool row_ok = row < m;
        zc* cp = C + row + (size_t)col0 * ldc;
        zc cpre[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) cpre[j] = (row_ok && col0 + j < nn) ? cp[(size_t)j * ldc] : mk(0.0);
        const int2* gb = reinterpret_cast<const int2*>(t.img + (size_t)bj * TC_BTILE + TC_BDIG) + 4 * cg;
        int2 eb[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) eb[j] = gb[j];
        const bool mw = mbar_wait(&s.bar_mma, t.ph_mma);
        if (!mw && lane == 0) {
            s.err = 1;
            s.mma_stuck = 1 + (int)t.ph_mma;
        }
        t.ph_mma ^= 1;
        bi0 = bi;
        bj0 = bj;
        if (++bj >= width(bi)) {
            bj = 0;
            ++bi;
        }
        if (warp == 0) {
            // the B buffer is free: the next tile's operand (none after a failed wait)
            pend = __shfl_sync(0xffffffffu, todo > 1 && !s.err, 0);
            if (lane == 0 && pend) load_b(bj);
            __syncwarp();
        }
        tc_fence_after();
        const int ea = s.ea[rloc];
#pragma unroll
        for (int j0 = 0; j0 < 8; j0 += 2) {
            float g[2][2 * TC_NS];
            const uint32_t base = tmem + ((uint32_t)(32 * q) << 16) + 8 * cg + j0;
#pragma unroll
            for (int a = 0; a < 2 * TC_NS; ++a) tmem_ld2(base + TC_N * a, g[0][a], g[1][a]);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (row_ok && col0 + j0 + j < nn) {
                    float lr[TC_NS], li[TC_NS];
#pragma unroll
                    for (int l = 0; l < TC_NS; ++l) {
                        lr[l] = g[j][2 * l];
                        li[l] = g[j][2 * l + 1];
                    }
                    // row maximum x column maximum is below 2^(p - 2044)
                    const int p = ea + (j ? eb[j0 / 2].y : eb[j0 / 2].x);
                    long long vr, vi;
                    int xr, xi;
                    const bool exact = tc_levels(lr, vr, xr) & tc_levels(li, vi, xi);
                    const zc c = cpre[j0 + j];
                    const zc w = mk(c.re - tc_double(vr, p - 2044 + xr), c.im - tc_double(vi, p - 2044 + xi));
                    const int ec = max(max(__double2hiint(c.re) & 0x7fffffff, __double2hiint(c.im) & 0x7fffffff),
                                       max(__double2hiint(w.re) & 0x7fffffff, __double2hiint(w.im) & 0x7fffffff)) >> 20;
                    // (a product below the normal range is no loss beside an element 2^61 times as large)
                    const bool bad = !exact || p > TC_PHI || ec < p - 1021 - TC_REDO || (p < TC_PLO && ec < p - 1021 + 61);
                    if (!bad) cp[(size_t)(j0 + j) * ldc] = w;
                    else s.redo[x & 1][atomicAdd(&s.redo_n[x % 3], 1)] = (unsigned short)(rloc * TC_N + 8 * cg + j0 + j);
                }
            }
        }
        tc_fence_before();
        __syncthreads();
    }
    if (x > 0) redo(x - 1, bi0, bj0);
    __syncthreads();
}

// the FP64 pipe's update, kept out of line beside it
template <class Team>
static __device__ __noinline__ void dfma_update(zc* C, int ldc, const zc* Ab, int lda, const zc* Bb, int ldb, int m, int nn,
                                                int kk, int tri, Tc64Smem& s, Team tm) {
    gemm_sub(C, ldc, Ab, lda, Bb, ldb, m, nn, kk, s, tm, tri);
}

// the engine's update: tensor cores or the FP64 pipe, by item
struct TcUpdate {
    TcState& t;
    // an item whose entries lie too far apart, or too far out, goes to the FP64 pipe
    template <class Team>
    __device__ __forceinline__ void begin(const EntryRange& rg, int n, Tc64Smem& s, const Team& tm) const {
        const int tid = threadIdx.x;
        if (tid == 0) { s.rng[0] = 0; s.rng[1] = 0x7fffffff; }
        __syncthreads();
        const int h = __reduce_max_sync(0xffffffffu, rg.hi), l = __reduce_min_sync(0xffffffffu, rg.lo);
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
        const int eh = hi >> 20, el = lo >> 20;
        t.use = n >= TC_NMIN && eh <= TC_EXP_MAX && el >= TC_EXP_MIN && eh - el <= TC_SPAN_LOG2;
    }
    // a wait of this item ran out in some CTA of the team (the CTAs then agree to stop)
    template <class Team>
    __device__ __forceinline__ bool failed(Tc64Smem& s, const Team& tm) const {
        int bad = s.err;
        if (tm.size > 1) {
            if (threadIdx.x < tm.size) cluster_store(&s.team_bad[tm.rank], threadIdx.x, bad);
            tm.sync();
            for (int r = 0; r < tm.size; ++r) bad |= s.team_bad[r];
        }
        return bad != 0;
    }
    template <class Team>
    __device__ __forceinline__ void operator()(zc* C, int ldc, const zc* Ab, int lda, const zc* Bb, int ldb, int m, int nn,
                                               int kk, int tri, Tc64Smem& s, const Team& tm) const {
        if (t.use) tc_update(C, ldc, Ab, lda, Bb, ldb, m, nn, kk, tri, s, tm, t);
        else dfma_update(C, ldc, Ab, lda, Bb, ldb, m, nn, kk, tri, s, tm);
    }
};

}  // namespace msg
