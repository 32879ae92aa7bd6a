// tc64.cuh -- the FP64 engine's trailing update C -= A B on the tcgen05
// tensor cores, exact to more bits than the FP64 pipe's chain of FMAs keeps.
//
// GB300's FP64 pipe does 2 FMAs a clock per SM (1.25 TFLOP/s on the chip) and
// 4 n^3 / 3 of them are the whole cost of a large complex LU.  Here every row
// of A and every column of B (K <= 32 entries) is scaled by a power of two to
// 62-bit fixed point and cut into seven balanced digits of 9 bits,
//     V = sum_k d_k 2^(9 (6 - k)),  |d_k| <= 256,
// which bf16 holds exactly.  The digit products (i, j) with l = i + j <= 6 are
// summed by tcgen05.mma kind::f16 in the FP32 accumulator of their level l:
// integers, below 2^24 for levels 0..3 whatever the data and beyond it only if
// almost every digit of a row is extreme, where the last bit lost is 2^-52 of
// a product of maxima.  The levels are put together in 64-bit integers
// (resolution 2^-55 of rowmax x colmax, against the up to 64 roundings of
// 2^-53 of the partial sum in a chain of FMAs) and meet C in one FP64 addition.
// The rounding is relative to the row and column maxima, so an item whose
// entries span more than TC_SPAN_LOG2 keeps the FP64 pipe's update.
//
// Measured (d = 3, ln det): 198 items at n = 1024 143 ms against 768 ms with the
// FP64 pipe's update (0.88 of its measured peak), 152 at n = 512 15.9 ms against
// 57, 304 at n = 160 3.7 against 4.9; the FP64 pipe is 54% busy then (panel, TRSM,
// assembly and one addition per update), the tensor pipe 4%.
//
// One CTA of 512 threads per SM: A band 128 rows x 32 (7 digits x Re/Im, 112 KB),
// two B buffers of 32 columns (28 KB each), 7 levels x Re/Im x 32 = 448 TMEM
// columns.  B's rows are stacked Re, Im, so that A_re times (Re, Im) is one MMA of
// N = 64: three MMAs a complex product, 83 cycles for the wide and 57 for each
// narrow one.  (A third block of rows, -Im, makes it two wide MMAs, but the 28 KB
// it takes from the L1 cache cost the panel and the TRSM as much at n = 1024 and
// 5% of the call at n = 100.)  A is sliced straight into shared memory, B once per update into a
// global image that bulk copies (TMA engine) bring in a tile ahead.
#pragma once
#include <cuda_bf16.h>
#include "lu64.cuh"
#include "umma.cuh"
#include "engine_internal.h"

namespace msg {

constexpr int TC_NT = 512;
constexpr int TC_M = 128;   // tile rows = TMEM lanes
constexpr int TC_N = 32;    // tile columns
constexpr int TC_NS = 7;    // digits = levels
constexpr int TC_ASUB = TC_M * NB * 2;           // one digit of Re or Im of an A band: 8 KB
constexpr int TC_BROWS = 2 * TC_N;               // a B tile's operand rows: Re, Im of its columns
constexpr int TC_BSUB = TC_BROWS * NB * 2;       // one digit of them: 4 KB
constexpr int TC_ABAND = 2 * TC_NS * TC_ASUB;    // 112 KB
constexpr int TC_BDIG = TC_NS * TC_BSUB;         // 28 KB
constexpr int TC_BTILE = TC_BDIG + TC_N * 4;     // digits, then the columns' exponents
constexpr uint32_t TC_TMEM = 512;
// Items whose entries span more than 2^TC_SPAN_LOG2 stay on the FP64 pipe.  Up to
// there the errors against 64-bit LAPACK are those of the FP64 pipe: ln det at
// d = 2, n = 1400, Im k = -0.3 (span 2^15.5) 2.0e-13 mean against 1.9e-13, d = 3,
// n = 700, Im k = -1 (2^12.1) 3.5e-14 against 5.3e-14, n = 1024, real k (2^8.4)
// 1.7e-16 against 1.5e-16; amplitudes n = 1024 5.2e-14 against 6.7e-14.
constexpr int TC_SPAN_LOG2 = 16;
// ... as do items with entries so large or small that a product's scale could leave the normal range
constexpr int TC_EXP_MIN = 1023 - 300, TC_EXP_MAX = 1023 + 300;
constexpr int TC_BAD = 1 << 20;  // exponent of a row or column with an infinity or a NaN

// shared memory: what lasts through an item, then the FP64 pipe's tiles (panel,
// TRSM, assembly; names as in LuSmemT) over the tensor core's operand buffers
struct Tc64Smem {
    static constexpr int NTH = TC_NT, TNC = TC_NT / 4, TMR = TM;
    static constexpr size_t PANEL_BYTES = TC_ABAND + 2 * (size_t)((TC_BTILE + 127) / 128 * 128);
    __device__ __forceinline__ void* panel_buf() { return g.a; }  // a panel between updates
    uint64_t bar_b[2], bar_mma;
    uint32_t tmem;
    int err, mma_stuck;
    int ea[TC_M];             // exponents of the A band's rows
    int emax[TC_M];
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
            uint8_t b[2][(TC_BTILE + 127) / 128 * 128];
        } g;
    };
};

// 62-bit fixed point of x for a row whose largest entry has biased exponent E:
// round(x 2^(1022 - E + 62)), |.| <= 2^62
__device__ __forceinline__ long long tc_fixed(double x, int E) {
    const long long b = __double_as_longlong(x);
    const int ex = (int)(b >> 52) & 0x7ff;
    const int sh = E - max(ex, 1);
    long long m = (b & 0xfffffffffffffLL) | (ex ? 0x10000000000000LL : 0);
    m <<= 9;
    m = sh > 62 ? 0 : sh > 0 ? (m + (1LL << (sh - 1))) >> sh : m;
    return b < 0 ? -m : m;
}

// balanced 9-bit digit of v, which moves to the next
__device__ __forceinline__ int tc_digit(long long& v) {
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
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        long long x[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = E >= TC_BAD ? 0 : tc_fixed(c ? v[k].im : v[k].re, E);
#pragma unroll
        for (int s = TC_NS - 1; s > 0; --s) {
            int d[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) d[k] = tc_digit(x[k]);
            put(s, c, make_uint4(tc_pack(d[0], d[1]), tc_pack(d[2], d[3]), tc_pack(d[4], d[5]), tc_pack(d[6], d[7])));
        }
        put(0, c, make_uint4(tc_pack((int)x[0], (int)x[1]), tc_pack((int)x[2], (int)x[3]), tc_pack((int)x[4], (int)x[5]),
                             tc_pack((int)x[6], (int)x[7])));
    }
}

// biased exponent of the largest component of 8 entries
__device__ __forceinline__ int tc_emax(const zc* v) {
    int h = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
        h = max(h, max(__double2hiint(v[k].re) & 0x7fffffff, __double2hiint(v[k].im) & 0x7fffffff));
    return h >> 20;
}

// the exponent that goes with a row's digits
__device__ __forceinline__ int tc_row_exp(int e) { return e == 0x7ff ? TC_BAD : max(e, 1); }

// per-kernel state of the tensor-core update
struct TcState {
    uint8_t* img;      // the team's B image: ceil(nmax / 32) tiles of TC_BTILE
    uint32_t tmem;
    uint32_t ph_b, ph_mma;  // phases of bar_b (a bit each) and bar_mma
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
            *reinterpret_cast<uint4*>(tile + d * TC_BSUB + cm_offset(c * TC_N + r, 8 * kb, TC_BROWS)) = w;
        });
    }
}

// the products of one tile, issued by warp 0 (lead: its elected lane)
__device__ __forceinline__ void tc_issue_tile(uint32_t a0, uint32_t b0, uint64_t* bar, uint32_t tmem, uint32_t lead) {
    const uint32_t id2 = idesc_bf16(TC_M, 2 * TC_N), idp = idesc_bf16(TC_M, TC_N), idn = idesc_bf16(TC_M, TC_N, false, true);
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
                umma_bf16_lead(t, dA(i, 0), dB(l - i, 0), id2, (ks == 0 && i == 0) ? 0u : 1u, lead);
                umma_bf16_lead(t, dA(i, 1), dB(l - i, TC_N), idn, 1, lead);
                umma_bf16_lead(t + TC_N, dA(i, 1), dB(l - i, 0), idp, 1, lead);
            }
        }
    }
    umma_commit_lead(bar, lead);
}

// sum of the levels, weight 2^(39 - 9 l), in units of 2^-55 (rowmax x colmax scale)
__device__ __forceinline__ long long tc_levels(const float* L) {
    int i[TC_NS];
#pragma unroll
    for (int l = 0; l < TC_NS; ++l) i[l] = __float2int_rn(L[l]);
    // levels 5 and 6 lie below the unit: rounded together
    long long v = (long long)(((i[5] << 3) + (i[6] >> 6) + 256) >> 9);
    v += (long long)i[4] * 8;
    v += (long long)i[3] * 4096;
    v += (long long)i[2] * (1 << 21);
    v += (long long)i[1] * (1 << 30);
    v += (long long)i[0] * (1LL << 39);
    return v;
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
    if (e < 1 || v == 0) b = 0;  // nothing to subtract, or below the normal range
    return __longlong_as_double(b | (v & (long long)0x8000000000000000ULL));
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
    uint32_t ph_b = t.ph_b;
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
    auto load_b = [&](int buf, int col) {
        mbar_arrive_expect_tx(&s.bar_b[buf], TC_BTILE);
        bulk_g2s(s.g.b[buf], t.img + (size_t)col * TC_BTILE, TC_BTILE, &s.bar_b[buf]);
    };
    auto next = [&](int& i, int& j) {
        if (++j >= width(i)) { j = 0; ++i; }
    };
    int buf = 0, limit = t.first_wait;
    // warp 0: this tile's B copy is under way (none is issued once a wait has run out)
    bool pend = __shfl_sync(0xffffffffu, todo > 0 && !s.err, 0);
    if (tid == 0 && pend) load_b(0, bj);
    int band = -1;
    const int q = warp & 3, cg = warp >> 2;  // TMEM lane quadrant, group of 8 columns
    const int rloc = 32 * q + lane;
    while (todo > 0) {
        int bi2 = bi, bj2 = bj;
        next(bi2, bj2);
        if (bi != band) {  // the previous tile's MMAs are complete: the band's buffer is free
            tc_slice_a(Ap, lda, bi * TC_M, m, K, s);
            fence_proxy_async();
            __syncthreads();
            band = bi;
        }
        if (warp == 0) {
            bool ok = pend;
            if (pend) {
                ok = mbar_wait(&s.bar_b[buf], (ph_b >> buf) & 1, limit);
                if (!ok) mbar_wait(&s.bar_b[buf], (ph_b >> buf) & 1);  // let the copy in flight land before moving on
                ph_b ^= 1u << buf;
                limit = WAIT_LIMIT;
            }
            pend = false;
            if (__all_sync(0xffffffffu, ok && !s.err)) {
                tc_fence_after();
                tc_issue_tile(smem_u32(s.g.a), smem_u32(s.g.b[buf]), &s.bar_mma, tmem, elect_lane());
                pend = todo > 1;
                if (lane == 0 && pend) load_b(buf ^ 1, bj2);
            } else if (lane == 0) {
                s.err = 1;                // operands missing: no MMA is issued;
                mbar_arrive(&s.bar_mma);  // release this tile's MMA wait at once
            }
            __syncwarp();
        }
        // this thread's row and 8 columns of C, on their way while the tensor core works
        const int row = bi * TC_M + rloc, col0 = bj * TC_N + 8 * cg;
        const bool row_ok = row < m;
        zc* cp = C + row + (size_t)col0 * ldc;
        zc cpre[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) cpre[j] = (row_ok && col0 + j < nn) ? cp[(size_t)j * ldc] : mk(0.0);
        const bool mw = mbar_wait(&s.bar_mma, t.ph_mma);
        if (!mw && lane == 0) {
            s.err = 1;
            s.mma_stuck = 1 + (int)t.ph_mma;
        }
        t.ph_mma ^= 1;
        tc_fence_after();
        const int ea = s.ea[rloc];
        const int* eb = reinterpret_cast<const int*>(s.g.b[buf] + TC_BDIG) + 8 * cg;
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
                    // a product of maxima is 2^(ea + eb - 2044); the unit is 2^-55 of it
                    const int xe = ea + eb[j0 + j] - 2044 - 55;
                    zc c = cpre[j0 + j];
                    if (ea + eb[j0 + j] >= TC_BAD) {
                        c = mk(nan(""), nan(""));
                    } else {
                        c.re -= tc_double(tc_levels(lr), xe);
                        c.im -= tc_double(tc_levels(li), xe);
                    }
                    cp[(size_t)(j0 + j) * ldc] = c;
                }
            }
        }
        tc_fence_before();
        __syncthreads();
        buf ^= 1;
        bi = bi2;
        bj = bj2;
        --todo;
    }
    t.ph_b = ph_b;
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
    // an item whose entries lie too far apart, or too far out, for the fixed point
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
