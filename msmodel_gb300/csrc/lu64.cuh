// lu64.cuh -- CTA-level FP64 complex dense kernels: blocked right-looking
// LU with partial pivoting, the triangular solves of LAPACK zgetrs, and the
// Foldy-Lax matrix assembly.  A matrix lives in global memory (column-major,
// leading dimension n) and belongs to a team: one CTA where there are matrices
// enough to fill the chip, so that thousands of (k, realisation) matrices
// factor concurrently with no inter-CTA traffic, or the CTAs of a cluster.
// Every element takes the same operations in the same order in any team.
//
// GB300's FP64 pipe (about 2 FMA lanes per SM per clock) bounds what is here: panel,
// TRSM, assembly, solves, and the trailing updates of matrices up to 96 rows (larger
// ones': tc64.cuh).  Memory traffic is a few percent of the time.
//
// Pivoting follows LAPACK zgetf2/zgetrf: the pivot of column j is the first
// row of maximum |Re|+|Im| (IZAMAX), ipiv is kept 0-based here, interchanges
// are applied to whole rows (LAPACK layout of L), a zero pivot sets info and
// skips the scaling, the multipliers are scaled by the reciprocal of the
// pivot when |pivot| >= DBL_MIN and divided otherwise.
#pragma once
#include <float.h>
#include "cplx.cuh"
#include "green.cuh"

namespace msg {

constexpr int NT = 256;  // threads per CTA
constexpr int NB = 32;   // panel width
constexpr int TM = 64;   // DFMA trailing-update tile rows

// complex a - l u in two FMAs per component: a product, an FMA and a difference
// (what a - l * u compiles to) would hold the FP64 pipe half as long again
MSG_D zc zfms(zc a, zc l, zc u) {
    a.re = fma(-l.re, u.re, a.re);
    a.re = fma(l.im, u.im, a.re);
    a.im = fma(-l.re, u.im, a.im);
    a.im = fma(-l.im, u.re, a.im);
    return a;
}

// a b with the products' roundings fixed, so that every inlined copy gives the same bits
MSG_D zc zmulf(zc a, zc b) {
    return mk(fma(a.re, b.re, -__dmul_rn(a.im, b.im)), fma(a.re, b.im, __dmul_rn(a.im, b.re)));
}

// The CTAs that factor one matrix together.  Solo: one CTA, the barrier is
// __syncthreads.  ClusterTeam: the CTAs of a thread-block cluster; its barrier
// (release / acquire at cluster scope) orders their global-memory accesses.
struct Solo {
    static constexpr int rank = 0, size = 1;
    __device__ __forceinline__ void sync() const { __syncthreads(); }
};
// A batch that leaves SMs idle gives each matrix several CTAs: the 32 targets of
// one resonance search at n = 100 take 45 ms against 83 ms with one CTA each
// (FP64-pipe updates, panel included), one dlogf at d = 2, n = 50 1.7 against 2.5.
struct ClusterTeam {
    int rank, size;
    __device__ __forceinline__ void sync() const {
        if (size == 1) {
            __syncthreads();
        } else {
            asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        }
    }
};

__device__ __forceinline__ ClusterTeam this_team() {
    uint32_t r, n;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
    return ClusterTeam{(int)r, (int)n};
}
// the same shared-memory variable in CTA `rank` of the cluster := v
__device__ __forceinline__ void cluster_store(int* p, int rank, int v) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

__device__ __forceinline__ void cluster_store(double* p, int rank, double v) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// a 16-byte shared-memory variable of CTA `rank` of the cluster
template <class E>
__device__ __forceinline__ E cluster_load(const E* p, int rank) {
    static_assert(sizeof(E) == 16, "one 128-bit load");
    uint32_t a;
    E v;
    uint32_t* w = reinterpret_cast<uint32_t*>(&v);
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                 : "r"(a)
                 : "memory");
    return v;
}
__device__ __forceinline__ void cluster_store(long long* p, int rank, long long v) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}

// shared memory of a CTA of NTH threads: tiles of TMR rows, NTH / 16 x 4 = TNC columns
template <int NTHREADS, int TILE_ROWS = TM>
struct __align__(16) LuSmemT {
    static constexpr int NTH = NTHREADS, TMR = TILE_ROWS;
    static constexpr int TNC = NTHREADS / 4;  // trailing-update tile columns (64 for 256 threads)
    zc As[NB][TMR];      // L21 tile  (k-major; 32 KB for 64 rows)
    zc Bs[NB][TNC];      // U12 tile  (k-major)
    // the two tiles' space holds a panel between updates
    __device__ __forceinline__ void* panel_buf() { return &As[0][0]; }
    static constexpr size_t PANEL_BYTES = sizeof(zc) * NB * (TMR + TNC);
    zc T[NB][NB + 1];    // 16.5 KB diagonal block / assembly transpose
    zc urow[NB];         // pivot row of the panel
    zc dlo[NB];          // what the reciprocals of U's diagonal in T leave out (DiagQuot)
    zc piv, rpiv;        // the pivot and its reciprocal
    zc diag[2];          // F^-1(k), d F^-1/dk
    long long red_k[2][NTHREADS / 32];
    int red_p[2][NTHREADS / 32];
    double red_v[NTHREADS / 32];
    int red_i[NTHREADS / 32];
    double red_s[3][NTHREADS / 32];
    int info;
    int bcast_i;
    int item;
    int nz;
};
using LuSmem = LuSmemT<NT>;

template <class S>
__device__ __forceinline__ void block_argmax(double v, int i, S& s, int& oi) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        double v2 = __shfl_down_sync(FULL, v, off);
        int i2 = __shfl_down_sync(FULL, i, off);
        if (v2 > v || (v2 == v && i2 < i)) { v = v2; i = i2; }
    }
    if (lane == 0) { s.red_v[warp] = v; s.red_i[warp] = i; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double bv = s.red_v[0];
        int bi = s.red_i[0];
        for (int w = 1; w < S::NTH / 32; w++) {
            double v2 = s.red_v[w];
            int i2 = s.red_i[w];
            if (v2 > bv || (v2 == bv && i2 < bi)) { bv = v2; bi = i2; }
        }
        s.bcast_i = bi;
    }
    __syncthreads();
    oi = s.bcast_i;
}

// sum of three doubles over the CTA; result valid in every thread
template <class S>
__device__ __forceinline__ void block_sum3(double& a, double& b, double& c, S& s) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_down_sync(FULL, a, off);
        b += __shfl_down_sync(FULL, b, off);
        c += __shfl_down_sync(FULL, c, off);
    }
    if (lane == 0) { s.red_s[0][warp] = a; s.red_s[1][warp] = b; s.red_s[2][warp] = c; }
    __syncthreads();
    a = b = c = 0.0;
    for (int w = 0; w < S::NTH / 32; w++) { a += s.red_s[0][w]; b += s.red_s[1][w]; c += s.red_s[2][w]; }
    __syncthreads();
}

// Pivot keys: |Re| + |Im| >= 0 as its bit pattern, which orders like the value,
// so that the search compares integers and leaves the FP64 pipe alone; a NaN
// (never chosen, as in IZAMAX's comparison) and "no row" are -1.
MSG_D long long pivot_key(zc a) {
    const long long b = __double_as_longlong(abs1(a));
    return b > 0x7FF0000000000000LL ? -1LL : b;
}

// row of the warp's largest key, the smallest row on ties: three warp reductions
__device__ __forceinline__ void warp_pivot(long long& key, int& row) {
    const unsigned FULL = 0xffffffffu;
    const int hi = (int)(key >> 32);
    const int mh = __reduce_max_sync(FULL, hi);
    const unsigned lo = hi == mh ? (unsigned)key : 0u;
    const unsigned ml = __reduce_max_sync(FULL, lo);
    row = __reduce_min_sync(FULL, hi == mh && lo == ml ? row : 0x7fffffff);
    key = ((long long)mh << 32) | ml;
}

// row of the CTA's largest key (smallest row on ties), in every thread; one
// barrier: the warps' candidates are double-buffered by `par`
template <class S>
__device__ __forceinline__ int block_pivot(long long key, int row, int par, S& s) {
    constexpr int NW = S::NTH / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    warp_pivot(key, row);
    if (lane == 0) { s.red_k[par][warp] = key; s.red_p[par][warp] = row; }
    __syncthreads();
    key = s.red_k[par][lane & (NW - 1)];
    row = s.red_p[par][lane & (NW - 1)];
    warp_pivot(key, row);
    return row;
}

// 1 / b by one reciprocal of |b|^2 where the squares stay well inside the
// exponent range (one division on the panel's serial chain, zrecip has two)
__device__ __forceinline__ zc pivot_recip(zc b) {
    const int e = max(__double2hiint(b.re) & 0x7fffffff, __double2hiint(b.im) & 0x7fffffff) >> 20;
    if (e < 1023 - 500 || e > 1023 + 500) return zrecip(b);
    const double rd = 1.0 / fma(b.re, b.re, b.im * b.im);
    return mk(b.re * rd, -b.im * rd);
}

// Factor the panel A[j0:n, j0:j0+jb) in place by one CTA; interchanges inside
// the panel only.  Sub-panels of SWP columns: inside one the rank-1 updates
// touch only its own columns, the rest of the panel then takes one rank-SWP
// update (U rows by unit-lower substitution), so the panel is read and written
// once per sub-panel and not once per column; each element still takes its
// updates in the order of the columns.  Per column the pivot's reciprocal is
// one lane's work (256 threads each doing the hypot and the divisions held
// the FP64 pipe, 2 lanes a clock, for ~10k cycles a column) and there are two
// barriers.  4096 ln det at n = 64 (d = 3): 19.6 ms with the full-width rank-1
// form and a reciprocal per thread; 11.6 ms with one reciprocal; 6.8 ms with the
// columns of few rows spread over the warps, warp reductions in the pivot search
// and the small update tiles (11k -> 6k cycles a column at n = 100); 5.7 ms with four
// CTAs of 128 threads per SM.
constexpr int SWP = 4;
template <class S>
static __device__ __noinline__ void panel_factor(zc* A, int n, int j0, int jb, int* ipiv, S& s) {
    constexpr int NTH = S::NTH;
    const int tid = threadIdx.x;
    const int cend = j0 + jb;
    long long bk = -1;
    int bi = n;
    for (int i = j0 + tid; i < n; i += NTH) {
        const long long k = pivot_key(A[i + (size_t)j0 * n]);
        if (k > bk) { bk = k; bi = i; }
    }
    for (int c0 = j0; c0 < cend; c0 += SWP) {
        const int sw = min(c0 + SWP, cend);
        for (int c = c0; c < sw; ++c) {
            int p = block_pivot(bk, bi, c & 1, s);
            if (p >= n) p = c;
            if (tid < 32) {
                // the interchange of rows c and p within the panel, one column a lane
                const size_t col = (size_t)(j0 + tid) * n;
                zc a = mk(0.0), b = mk(0.0);
                if (tid < jb) {
                    a = A[c + col];
                    b = p != c ? A[p + col] : a;
                    s.urow[tid] = b;
                }
                const bool nz = __shfl_sync(0xffffffffu, (int)!is_zero(b), c - j0) != 0;
                if (nz && p != c && tid < jb) {
                    A[c + col] = b;
                    A[p + col] = a;
                }
                if (!nz && tid < jb) s.urow[tid] = a;  // a zero column: no interchange
                if (tid == c - j0) {
                    ipiv[c] = p;
                    if (!nz && s.info == 0) s.info = c + 1;
                    // |b| >= DBL_MIN, by the exponents where they decide it
                    const int hb = max(__double2hiint(b.re) & 0x7fffffff, __double2hiint(b.im) & 0x7fffffff);
                    const bool recip = nz && (hb >= 0x00100000 || zabs(b) >= DBL_MIN);
                    s.nz = nz ? (recip ? 1 : 2) : 0;
                    s.piv = b;
                    s.rpiv = recip ? pivot_recip(b) : mk(0.0);
                }
            }
            __syncthreads();
            const int nz = s.nz;
            const zc r = s.rpiv;
            bk = -1;
            bi = n;
            if (nz) {
                for (int i = c + 1 + tid; i < n; i += NTH) {
                    zc l = A[i + (size_t)c * n];
                    l = nz == 1 ? zmulf(l, r) : l / s.piv;
                    A[i + (size_t)c * n] = l;
                    if (c + 1 < sw) {
                        const zc a = zfms(A[i + (size_t)(c + 1) * n], l, s.urow[c + 1 - j0]);
                        A[i + (size_t)(c + 1) * n] = a;
                        const long long k = pivot_key(a);
                        if (k > bk) { bk = k; bi = i; }
                        for (int cc = c + 2; cc < sw; ++cc) {
                            zc* q = A + i + (size_t)cc * n;
                            *q = zfms(*q, l, s.urow[cc - j0]);
                        }
                    }
                }
            } else if (c + 1 < sw) {
                for (int i = c + 1 + tid; i < n; i += NTH) {
                    const long long k = pivot_key(A[i + (size_t)(c + 1) * n]);
                    if (k > bk) { bk = k; bi = i; }
                }
            }
        }
        if (sw < cend) {
            const int cw = sw - c0, rem = cend - sw;
            __syncthreads();  // the sub-panel's last column is complete
            // U rows of the sub-panel right of it: u_r = a_r - sum_{q<r} L_rq u_q
            if (tid < rem) {
                const size_t col = (size_t)(sw + tid) * n;
                zc u[SWP];
#pragma unroll
                for (int r = 0; r < SWP; ++r) {
                    if (r < cw) {
                        zc a = A[c0 + r + col];
#pragma unroll
                        for (int q = 0; q < r; ++q) a = zfms(a, A[c0 + r + (size_t)(c0 + q) * n], u[q]);
                        u[r] = a;
                        A[c0 + r + col] = a;
                        s.T[r][tid] = a;
                    }
                }
            }
            __syncthreads();
            bk = -1;
            bi = n;
            // a warp takes 32 rows; where the rows do not fill the CTA several warps share
            // them, each with every G-th column (a thread alone on a row would leave the
            // other warps' share of the FP64 pipe idle for 28 columns)
            const int nrb = (n - sw + 31) / 32, G = max(1, (NTH / 32) / max(nrb, 1));
            const int g = nrb < NTH / 32 ? (tid >> 5) / nrb : 0;
            const int i0 = sw + (nrb < NTH / 32 ? ((tid >> 5) % nrb) * 32 + (tid & 31) : tid);
            if (g < G)
                for (int i = i0; i < n; i += NTH) {
                    zc l[SWP];
#pragma unroll
                    for (int q = 0; q < SWP; ++q) l[q] = q < cw ? A[i + (size_t)(c0 + q) * n] : mk(0.0);
                    for (int t = g; t < rem; t += G) {
                        zc* q = A + i + (size_t)(sw + t) * n;
                        zc a = *q;
#pragma unroll
                        for (int e = 0; e < SWP; ++e)
                            if (e < cw) a = zfms(a, l[e], s.T[e][t]);
                        *q = a;
                        if (t == 0) {
                            const long long k = pivot_key(a);
                            if (k > bk) { bk = k; bi = i; }
                        }
                    }
                }
        }
    }
    __syncthreads();
}

// Column solves used by the blocked TRSM steps.  One thread owns one column
// b[0..jb) (global memory); the jb x jb triangle sits in s.T.  Rows are
// processed in chunks of CH so that only CH complex values live in registers;
// solved values of earlier chunks are re-read from memory.
constexpr int CH = 8;

__device__ __forceinline__ void col_solve_lower_unit(zc* __restrict__ b, int jb, const zc (*T)[NB + 1]) {
    for (int rb = 0; rb < jb; rb += CH) {
        zc y[CH];
#pragma unroll
        for (int r = 0; r < CH; ++r) y[r] = (rb + r < jb) ? b[rb + r] : mk(0.0);
        for (int q = 0; q < rb; ++q) {
            const zc xq = b[q];
#pragma unroll
            for (int r = 0; r < CH; ++r) y[r] = zfms(y[r], T[rb + r][q], xq);
        }
#pragma unroll
        for (int r = 1; r < CH; ++r)
#pragma unroll
            for (int q = 0; q < r; ++q) y[r] = zfms(y[r], T[rb + r][rb + q], y[q]);
#pragma unroll
        for (int r = 0; r < CH; ++r)
            if (rb + r < jb) b[rb + r] = y[r];
    }
}

// Division by a diagonal element U_rr, prepared once for the block's columns: hi the
// rounded reciprocal, lo = hi (1 - U_rr hi), so that a hi + a lo loses nothing to the
// reciprocal's rounding (|error| <= 2 2^-53 of the quotient; Smith's quotient reaches 2.2,
// a product with the rounded reciprocal alone 2.7).  Far from 1 in the exponent range,
// where a reciprocal may overflow, hi is U_rr itself, lo marked by an infinity, and the
// solve divides.
struct DiagQuot {
    zc hi, lo;
    static __device__ __forceinline__ DiagQuot prepare(zc u) {
        const int e = max(__double2hiint(u.re) & 0x7fffffff, __double2hiint(u.im) & 0x7fffffff) >> 20;
        if (e < 1023 - 500 || e > 1023 + 500) return {u, mk(__longlong_as_double(0x7ff0000000000000LL))};
        const zc h = pivot_recip(u);
        // 1 - u h, every difference exact: the two products of the real part add up to 1
        // within rounding, those of the imaginary part to 0
        const double p = __dmul_rn(u.re, h.re), q = -__dmul_rn(u.im, h.im);
        const double pe = fma(u.re, h.re, -p), qe = fma(-u.im, h.im, -q);
        const double r = __dmul_rn(u.re, h.im), t = __dmul_rn(u.im, h.re);
        const double re = fma(u.re, h.im, -r), te = fma(u.im, h.re, -t);
        const zc d = mk(((1.0 - fmax(p, q)) - fmin(p, q)) - (pe + qe), -((r + t) + (re + te)));
        return {h, zmulf(h, d)};
    }
    // a / U_rr; far: some element of the block is one to divide by (load_upper)
    static __device__ __forceinline__ zc of(zc a, zc hi, zc lo, bool far) {
        if (far && __double2hiint(lo.re) == 0x7ff00000) return a / hi;
        const zc t = zmulf(a, lo);
        return mk(fma(a.re, hi.re, fma(-a.im, hi.im, t.re)), fma(a.re, hi.im, fma(a.im, hi.re, t.im)));
    }
};

// the upper solve; T's diagonal and dlo hold the prepared divisions by U_rr
__device__ __forceinline__ void col_solve_upper(zc* __restrict__ b, int jb, const zc (*T)[NB + 1], const zc* dlo,
                                                bool far) {
    for (int rb = ((jb - 1) / CH) * CH; rb >= 0; rb -= CH) {
        zc y[CH];
#pragma unroll
        for (int r = 0; r < CH; ++r) y[r] = (rb + r < jb) ? b[rb + r] : mk(0.0);
        for (int q = jb - 1; q >= rb + CH; --q) {
            const zc xq = b[q];
#pragma unroll
            for (int r = 0; r < CH; ++r) y[r] = zfms(y[r], T[rb + r][q], xq);
        }
#pragma unroll
        for (int r = CH - 1; r >= 0; --r) {
            if (rb + r < jb) {
                zc acc = y[r];
#pragma unroll
                for (int q = CH - 1; q > r; --q)
                    if (rb + q < jb) acc = zfms(acc, T[rb + r][rb + q], y[q]);
                y[r] = DiagQuot::of(acc, T[rb + r][rb + r], dlo[rb + r], far);
            }
        }
#pragma unroll
        for (int r = 0; r < CH; ++r)
            if (rb + r < jb) b[rb + r] = y[r];
    }
}

// The same solves with one row a lane, for a warp per column: where a CTA has few
// columns, one thread per column would put them on a warp or two, a quarter of
// the FP64 pipe each, for jb^2/2 steps.  Every element takes its updates in the
// order of the column solves, so the results are the same bits.
__device__ __forceinline__ zc row_solve_lower_unit(zc x, int jb, const zc (*T)[NB + 1]) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    for (int q = 0; q + 1 < jb; ++q) {
        const zc xq = mk(__shfl_sync(FULL, x.re, q), __shfl_sync(FULL, x.im, q));
        if (lane > q && lane < jb) x = zfms(x, T[lane][q], xq);
    }
    return x;
}
// (The division of row q is one lane's, but its instructions take the pipe for the whole
// warp: the halves of the warp do its real and its imaginary part, 4 instructions in
// place of 8: 32 dlogf at n = 100 1.26 -> 1.19 ms.)
__device__ __forceinline__ zc row_solve_upper(zc x, int jb, const zc (*T)[NB + 1], const zc* dlo, bool far) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, part = lane >> 4;
    for (int q = jb - 1; q >= 0; --q) {
        const double ar = __shfl_sync(FULL, x.re, q), ai = __shfl_sync(FULL, x.im, q);
        zc xq;
        if (far && __double2hiint(dlo[q].re) == 0x7ff00000) {
            xq = mk(ar, ai) / T[q][q];
        } else {
            // DiagQuot::of, component `part`
            const double* h = &T[q][q].re;
            const double* l = &dlo[q].re;
            const double b = part ? ai : -ai;
            const double v = fma(ar, h[part], fma(b, h[1 - part], fma(ar, l[part], __dmul_rn(b, l[1 - part]))));
            xq = mk(__shfl_sync(FULL, v, 0), __shfl_sync(FULL, v, 16));
        }
        if (lane == q) x = xq;
        if (lane < q) x = zfms(x, T[lane][q], xq);
    }
    return x;
}

// Columns go to the team in blocks of 32, block b to CTA b % size: the columns
// of this CTA below ncol
template <class Team>
__device__ __forceinline__ int cta_columns(int ncol, const Team& tm) {
    const int nb = (ncol + 31) / 32, mine = (nb - tm.rank + tm.size - 1) / tm.size;
    return mine * 32;
}
// ... and the x-th of them (may be >= ncol in the last block)
template <class Team>
__device__ __forceinline__ int cta_column(int x, const Team& tm) { return ((x >> 5) * tm.size + tm.rank) * 32 + (x & 31); }
// few columns: a warp for each column and a lane for each row is the faster solve
// (~2k cycles a column on the whole SM, against ~127k for up to 128 columns with
// a thread each: 166k -> 59k cycles a panel at n = 100)
__device__ __forceinline__ bool few_columns(int cols) { return cols <= 64; }
// ... so of a CTA's columns as many go a thread each as fill its nth threads, and
// the rest too unless they are few
__device__ __forceinline__ int thread_columns(int cols, int nth) {
    const int full = cols / nth * nth;
    return few_columns(cols - full) ? full : cols;
}

// The net effect of a panel's interchanges, worked out by every warp for
// itself: row j0 + lane receives row `inner`, and row `orow` (-1: none), one of
// the rows below the panel that took part, receives row `ocur`.  One load and
// one store per moved row then replace the chain of up to 32 exchanges.
__device__ __forceinline__ void panel_moves(const int* ipiv, int j0, int jb, int& inner, int& orow, int& ocur) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int pv = lane < jb ? ipiv[j0 + lane] : j0 + lane;
    inner = j0 + lane;
    orow = -1;
    ocur = -1;
    int used = 0;
    for (int c = 0; c < jb; ++c) {
        const int p = __shfl_sync(FULL, pv, c);
        if (p == j0 + c) continue;
        const int ic = __shfl_sync(FULL, inner, c);
        if (p < j0 + jb) {
            const int ip = __shfl_sync(FULL, inner, p - j0);
            if (lane == c) inner = ip;
            if (lane == p - j0) inner = ic;
        } else {
            const unsigned hit = __ballot_sync(FULL, orow == p);
            const int u = hit ? __ffs(hit) - 1 : used++;
            const int cur = hit ? __shfl_sync(FULL, ocur, u) : p;
            if (lane == u) { orow = p; ocur = ic; }
            if (lane == c) inner = cur;
        }
    }
}

template <class S>
static __device__ void load_lower(const zc* A, int n, int j0, int jb, S& s) {
    for (int e = threadIdx.x; e < NB * NB; e += S::NTH) {
        int r = e % NB, q = e / NB;
        s.T[r][q] = (r < jb && q < r) ? A[(j0 + r) + (size_t)(j0 + q) * n] : mk(0.0);
    }
    __syncthreads();
}

// the upper triangle, its diagonal as prepared divisions; true if one of them divides
template <class S>
static __device__ bool load_upper(const zc* A, int n, int j0, int jb, S& s) {
    bool far = false;
    for (int e = threadIdx.x; e < NB * NB; e += S::NTH) {
        int r = e % NB, q = e / NB;
        zc v = mk(0.0);
        if (r < jb && q < jb && q >= r) v = A[(j0 + r) + (size_t)(j0 + q) * n];
        if (q == r && r < jb) {
            const DiagQuot d = DiagQuot::prepare(v);
            v = d.hi;
            s.dlo[r] = d.lo;
            far |= __double2hiint(d.lo.re) == 0x7ff00000;
        }
        s.T[r][q] = v;
    }
    return __syncthreads_or(far) != 0;
}

// Apply the panel's interchanges to every other column and compute
// U12 = L11^-1 A12 (columns right of the panel).  keep_l = false leaves the
// columns left of the panel alone: a ln det reads only U's diagonal and the
// pivots afterwards.
template <class S, class Team>
static __device__ void panel_swaps_trsm(zc* A, int n, int j0, int jb, const int* ipiv, bool keep_l, S& s, const Team& tm) {
    constexpr int NW = S::NTH / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    load_lower(A, n, j0, jb, s);
    int inner, orow, ocur;
    panel_moves(ipiv, j0, jb, inner, orow, ocur);
    const bool moves = __any_sync(0xffffffffu, inner != j0 + lane);
    const int right = j0 + jb, nr = cta_columns(n - right, tm);
    const int wide = thread_columns(nr, S::NTH);  // the first `wide` a thread each
    if (keep_l && moves) {
        const int nl = cta_columns(j0, tm);
        for (int x = warp; x < nl; x += NW) {
            const int col = cta_column(x, tm);
            if (col >= j0) continue;
            zc* a = A + (size_t)col * n;
            const zc v = lane < jb ? a[inner] : mk(0.0), w = orow >= 0 ? a[ocur] : mk(0.0);
            __syncwarp();
            if (lane < jb) a[j0 + lane] = v;
            if (orow >= 0) a[orow] = w;
        }
    }
    if (wide < nr || moves)
        for (int x = (moves ? 0 : wide) + warp; x < nr; x += NW) {
            const int col = right + cta_column(x, tm);
            if (col >= n) continue;
            zc* a = A + (size_t)col * n;
            zc v = lane < jb ? a[inner] : mk(0.0);
            const zc w = orow >= 0 ? a[ocur] : mk(0.0);
            __syncwarp();
            if (x >= wide) v = row_solve_lower_unit(v, jb, s.T);
            if (lane < jb) a[j0 + lane] = v;
            if (orow >= 0) a[orow] = w;
        }
    if (wide > 0) {
        __syncthreads();
        for (int x = tid; x < wide; x += S::NTH) {
            const int col = right + cta_column(x, tm);
            if (col < n) col_solve_lower_unit(A + (size_t)col * n + j0, jb, s.T);
        }
    }
    tm.sync();
}

// C[m x nn] -= Ablk[m x kk] * Bblk[kk x nn] (all column-major); kk <= NB.
// tri != 0: only tiles that hold some element with row >= col are updated.
// The team deals the tiles round robin; the caller's barrier ends the update.
// A thread holds R x R elements: R = 4 (64 x 64 tiles for 256 threads), or R = 2
// for blocks of at most 32 rows or columns, most of whose larger tile would be
// work on padding.
template <int R, class S, class Team>
static __device__ void gemm_sub_r(zc* C, int ldc, const zc* Ab, int lda, const zc* Bb,
                           int ldb, int m, int nn, int kk, S& s, const Team& tm, int tri) {
    constexpr int NTH = S::NTH, TM = 16 * R, TNC = NTH / 16 * R, CST = NTH / 16;
    if (m <= 0 || nn <= 0 || kk <= 0) return;
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    int t = 0;
    for (int ti = 0; ti < m; ti += TM) {
        bool have_a = false;
        for (int tj = 0; tj < nn; tj += TNC) {
            if (tri && ti + TM - 1 < tj) break;
            if (tm.size > 1 && t++ % tm.size != tm.rank) continue;
            if (!have_a) {
                have_a = true;
                for (int e = tid; e < NB * TM; e += NTH) {
                    int r = e % TM, k = e / TM;
                    zc v = mk(0.0);
                    if (k < kk && ti + r < m) v = Ab[(ti + r) + (size_t)k * lda];
                    s.As[k][r] = v;
                }
            }
            for (int e = tid; e < NB * TNC; e += NTH) {
                int k = e % NB, c = e / NB;
                zc v = mk(0.0);
                if (k < kk && tj + c < nn) v = Bb[k + (size_t)(tj + c) * ldb];
                s.Bs[k][c] = v;
            }
            __syncthreads();
            zc acc[R][R];
#pragma unroll
            for (int a = 0; a < R; ++a)
#pragma unroll
                for (int b = 0; b < R; ++b) {
                    int r = ti + tx + 16 * a, c = tj + ty + CST * b;
                    acc[a][b] = (r < m && c < nn) ? C[r + (size_t)c * ldc] : mk(0.0);
                }
#pragma unroll 2
            for (int k = 0; k < kk; ++k) {
                zc av[R], bw[R];
#pragma unroll
                for (int a = 0; a < R; ++a) av[a] = s.As[k][tx + 16 * a];
#pragma unroll
                for (int b = 0; b < R; ++b) bw[b] = s.Bs[k][ty + CST * b];
#pragma unroll
                for (int a = 0; a < R; ++a)
#pragma unroll
                    for (int b = 0; b < R; ++b) acc[a][b] = zfms(acc[a][b], av[a], bw[b]);
            }
#pragma unroll
            for (int a = 0; a < R; ++a)
#pragma unroll
                for (int b = 0; b < R; ++b) {
                    int r = ti + tx + 16 * a, c = tj + ty + CST * b;
                    if (r < m && c < nn) C[r + (size_t)c * ldc] = acc[a][b];
                }
            __syncthreads();
        }
    }
}

template <class S, class Team>
static __device__ void gemm_sub(zc* C, int ldc, const zc* Ab, int lda, const zc* Bb, int ldb, int m, int nn, int kk, S& s,
                         const Team& tm, int tri = 0) {
    if (S::TMR < TM || m <= 32 || nn <= 32) gemm_sub_r<2>(C, ldc, Ab, lda, Bb, ldb, m, nn, kk, s, tm, tri);
    else if constexpr (S::TMR >= TM) gemm_sub_r<4>(C, ldc, Ab, lda, Bb, ldb, m, nn, kk, s, tm, tri);
}

// the trailing update on the FP64 pipe (DFMA); another kernel may pass its own
struct EntryRange;
struct DfmaUpdate {
    template <class S, class Team>
    __device__ __forceinline__ void begin(const EntryRange&, int, S&, const Team&) const {}
    template <class S, class Team>
    __device__ __forceinline__ bool failed(S&, const Team&) const { return false; }
    template <class S, class Team>
    __device__ __forceinline__ void operator()(zc* C, int ldc, const zc* Ab, int lda, const zc* Bb, int ldb, int m, int nn,
                                               int kk, int tri, S& s, const Team& tm) const {
        gemm_sub(C, ldc, Ab, lda, Bb, ldb, m, nn, kk, s, tm, tri);
    }
};

// A team's panels short enough are factored in shared memory (panel.cuh), by all
// of it above PANEL_SOLO rows (below, a barrier a column costs more than the rows
// it takes off the first CTA): one ln det at n = 1024 16.6 -> 8.7 ms, n = 300
// 2.28 -> 1.69.  Longer ones, and those of a CTA alone, whose columns the FP64 pipe
// bounds either way (n = 100: 708k cycles out of global memory, 742k in shared),
// take panel_factor.
constexpr int PANEL_SOLO = 64;
struct PanelFp64;
template <class E>
__device__ __forceinline__ bool panel_fits(int m, int size, size_t bytes);
template <class Ar, int NTH, class Team>
static __device__ __noinline__ void panel_smem(typename Ar::E* A, int n, int j0, int jb, int* ipiv, void* buf, int& info,
                                               Team tm);
template <class S, class Team>
__device__ __forceinline__ void factor_panel(zc* A, int n, int j0, int jb, int* ipiv, S& s, const Team& tm) {
    const int m = n - j0;
    if (tm.size > 1 && m > PANEL_SOLO && panel_fits<zc>(m, tm.size, S::PANEL_BYTES))
        panel_smem<PanelFp64, S::NTH>(A, n, j0, jb, ipiv, s.panel_buf(), s.info, tm);
    else if (tm.rank != 0) return;
    else if (tm.size > 1 && panel_fits<zc>(m, 1, S::PANEL_BYTES))
        panel_smem<PanelFp64, S::NTH>(A, n, j0, jb, ipiv, s.panel_buf(), s.info, Solo{});
    else panel_factor(A, n, j0, jb, ipiv, s);
}

// In-place LU of A (n x n, ld n).  ipiv 0-based.  Sets s.info of the team's
// first CTA (1-based first zero pivot).
template <class S, class Team, class Update>
static __device__ void lu_factor(zc* A, int n, int* ipiv, bool keep_l, S& s, const Team& tm,
                                 const Update& update) {
    for (int j0 = 0; j0 < n; j0 += NB) {
        const int jb = min(NB, n - j0);
        factor_panel(A, n, j0, jb, ipiv, s, tm);
        if (tm.size > 1) tm.sync();
        panel_swaps_trsm(A, n, j0, jb, ipiv, keep_l, s, tm);
        const int r0 = j0 + jb;
        update(A + r0 + (size_t)r0 * n, n, A + r0 + (size_t)j0 * n, n, A + j0 + (size_t)r0 * n, n, n - r0, n - r0, jb, 0, s,
               tm);
        if (tm.size > 1) tm.sync();
    }
}

// ln det(A)/n with the reference's branch: sum log|U_ii| + i (sum Arg U_ii + pi [odd interchanges]).
template <class S>
static __device__ zc lu_tracelog(const zc* A, int n, const int* ipiv, S& s) {
    double lr = 0.0, ar = 0.0, odd = 0.0;
    for (int i = threadIdx.x; i < n; i += S::NTH) {
        zc u = A[i + (size_t)i * n];
        lr += log(hypot(u.re, u.im));
        ar += atan2(u.im, u.re);
        if (ipiv[i] != i) odd += 1.0;
    }
    block_sum3(lr, ar, odd, s);
    if (fmod(odd, 2.0) == 1.0) ar += PI;
    return mk(lr / n, ar / n);
}

// tr(A^-1 B) given the LU of A (LAPACK layout) and B (n x n, ld n), B destroyed:
// B <- P B, forward solve with unit-lower L, backward solve with U restricted
// to the rows each diagonal element needs (X_jj depends on rows >= j only).
template <class S, class Team, class Update>
static __device__ zc lu_trace_solve(const zc* A, zc* B, int n, const int* ipiv,
                             S& s, const Team& tm, const Update& update) {
    constexpr int NTH = S::NTH, NW = NTH / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int mine = cta_columns(n, tm);
    // P B: each warp takes its columns through every panel's interchanges
    for (int j0 = 0; j0 < n; j0 += NB) {
        const int jb = min(NB, n - j0);
        int inner, orow, ocur;
        panel_moves(ipiv, j0, jb, inner, orow, ocur);
        if (!__any_sync(0xffffffffu, inner != j0 + lane)) continue;
        for (int x = warp; x < mine; x += NW) {
            const int col = cta_column(x, tm);
            if (col >= n) continue;
            zc* b = B + (size_t)col * n;
            const zc v = lane < jb ? b[inner] : mk(0.0), w = orow >= 0 ? b[ocur] : mk(0.0);
            __syncwarp();
            if (lane < jb) b[j0 + lane] = v;
            if (orow >= 0) b[orow] = w;
            __syncwarp();
        }
    }
    __syncthreads();
    // forward: L X = P B
    for (int j0 = 0; j0 < n; j0 += NB) {
        const int jb = min(NB, n - j0);
        load_lower(A, n, j0, jb, s);
        const int wide = thread_columns(mine, NTH);
        for (int x = wide + warp; x < mine; x += NW) {
            const int col = cta_column(x, tm);
            if (col >= n) continue;
            zc* b = B + (size_t)col * n + j0;
            const zc v = row_solve_lower_unit(lane < jb ? b[lane] : mk(0.0), jb, s.T);
            if (lane < jb) b[lane] = v;
        }
        for (int x = tid; x < wide; x += NTH) {
            const int col = cta_column(x, tm);
            if (col < n) col_solve_lower_unit(B + (size_t)col * n + j0, jb, s.T);
        }
        tm.sync();
        const int r0 = j0 + jb;
        update(B + r0, n, A + r0 + (size_t)j0 * n, n, B + j0, n, n - r0, n, jb, 0, s, tm);
        if (tm.size > 1) tm.sync();
    }
    // backward: U X = Y, columns [0, j0+jb) of block row j0 only
    const int nblk = (n + NB - 1) / NB;
    for (int kb = nblk - 1; kb >= 0; --kb) {
        const int j0 = kb * NB, jb = min(NB, n - j0), ncol = j0 + jb;
        const bool far = load_upper(A, n, j0, jb, s);
        const int cols = cta_columns(ncol, tm);
        const int wide = thread_columns(cols, NTH);
        for (int x = wide + warp; x < cols; x += NW) {
            const int col = cta_column(x, tm);
            if (col >= ncol) continue;
            zc* b = B + (size_t)col * n + j0;
            const zc v = row_solve_upper(lane < jb ? b[lane] : mk(0.0), jb, s.T, s.dlo, far);
            if (lane < jb) b[lane] = v;
        }
        for (int x = tid; x < wide; x += NTH) {
            const int col = cta_column(x, tm);
            if (col < ncol) col_solve_upper(B + (size_t)col * n + j0, jb, s.T, s.dlo, far);
        }
        tm.sync();
        // Y[0:j0, 0:ncol] -= U[0:j0, j0:j0+jb] X[j0:j0+jb, 0:ncol]   (rows >= cols only)
        update(B, n, A + (size_t)j0 * n, n, B + j0, n, j0, ncol, jb, 1, s, tm);
        if (tm.size > 1) tm.sync();
    }
    double tr = 0.0, ti = 0.0, z = 0.0;
    for (int i = tid; i < n; i += NTH) {
        zc v = B[i + (size_t)i * n];
        tr += v.re;
        ti += v.im;
    }
    block_sum3(tr, ti, z, s);
    return mk(tr, ti);
}

// x <- A^-1 x for one right-hand side x[n] (global), LAPACK-layout LU: the
// interchanges, then blocked forward and backward substitution; each block's
// triangle comes into shared memory, with the divisions by U's diagonal prepared (a
// whole division a step by one lane held up the chain), and is solved by warp 0 (one row
// per lane), the rectangular remainder by all threads (one row per thread,
// coalesced column reads).
template <class S>
static __device__ void lu_solve_vec(const zc* A, zc* x, int n, const int* ipiv, S& s) {
    constexpr int NTH = S::NTH;
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid < 32)
        for (int j0 = 0; j0 < n; j0 += NB) {
            const int jb = min(NB, n - j0);
            int inner, orow, ocur;
            panel_moves(ipiv, j0, jb, inner, orow, ocur);
            const zc v = lane < jb ? x[inner] : mk(0.0), w = orow >= 0 ? x[ocur] : mk(0.0);
            __syncwarp();
            if (lane < jb) x[j0 + lane] = v;
            if (orow >= 0) x[orow] = w;
            __syncwarp();
        }
    __syncthreads();
    auto rows = [&](int j0, int jb, int r0, int r1) {
        for (int i = r0 + tid; i < r1; i += NTH) {
            zc acc = x[i];
            const zc* a = A + i + (size_t)j0 * n;
#pragma unroll 8
            for (int q = 0; q < jb; ++q) acc = zfms(acc, a[(size_t)q * n], s.urow[q]);
            x[i] = acc;
        }
        __syncthreads();
    };
    for (int j0 = 0; j0 < n; j0 += NB) {
        const int jb = min(NB, n - j0);
        load_lower(A, n, j0, jb, s);
        if (tid < 32) {
            const zc v = row_solve_lower_unit(lane < jb ? x[j0 + lane] : mk(0.0), jb, s.T);
            if (lane < jb) x[j0 + lane] = s.urow[lane] = v;
        }
        __syncthreads();
        rows(j0, jb, j0 + jb, n);
    }
    for (int j0 = (n - 1) / NB * NB; j0 >= 0; j0 -= NB) {
        const int jb = min(NB, n - j0);
        const bool far = load_upper(A, n, j0, jb, s);
        if (tid < 32) {
            const zc v = row_solve_upper(lane < jb ? x[j0 + lane] : mk(0.0), jb, s.T, s.dlo, far);
            if (lane < jb) x[j0 + lane] = s.urow[lane] = v;
        }
        __syncthreads();
        rows(j0, jb, 0, j0);
    }
}

// Off-diagonal matrix elements -G (and -dG/dk) for one pair distance.
__device__ __forceinline__ void pair_elements(int d, zc k, double r, bool want_deriv, zc& m, zc& dm) {
    if (d == 3) {
        pair_elements_d3(k, r, want_deriv, m, dm);
        return;
    }
    if (d == 2 && want_deriv) {
        // M = K_0(z) / (2 pi), dM/dk = -(k / 2 pi) G_0 = i r K_1(z) / (2 pi), z = -i k r (the general
        // G_0 = -(-ik / (2 pi r))^-1 K_-1 / (2 pi) raises a complex power for every pair)
        zc k0, k1;
        bessel_k01(-(mk(-k.im, k.re) * r), k0, k1);
        m = k0 / TWOPI;
        dm = (r / TWOPI) * mk(-k1.im, k1.re);
        return;
    }
    m = -free_green(d, k, r);
    if (want_deriv) dm = -dk_free_green(d, k, r);
}

// K_nu regime of the pair's argument z = -i k r (the reference's switch,
// green_bessel.c:208-218): 0 asymptotic, 1 ascending series, 2 Miller.
__device__ __forceinline__ int k_regime(zc k, double r) {
    const double x = k.im * r, y = -k.re * r;
    if (x * x + y * y > 256.0) return 0;
    if (x < 3.0 - y * y / 12.0) return 1;
    return 2;
}

// Pairs i < j of the 32 x 32 tile (I, J) for d != 3, evaluated grouped by K_nu
// regime: the three loops differ several-fold in length, and a warp that
// mixes them runs all of them.  Every pair goes to one of three lists in
// shared memory (list: 3 x 1024 entries, cnt: 3 counters, both zero on entry
// and on return), then consecutive threads take consecutive list entries;
// put(ii, jj, m, dm) receives each element.  Entries of a list are in no
// fixed order, but every element is a function of (k, r) alone.
template <int NTH, class Put>
__device__ __forceinline__ void tile_pairs_grouped(int I, int J, int n, int d, const double* __restrict__ pos, zc k,
                                                   bool want_deriv, unsigned short* list, int* cnt, Put put, int q0 = 0,
                                                   int q1 = 1024 / NTH) {
    const int tid = threadIdx.x;
    for (int q = q0; q < q1; ++q) {
        const int p = tid + NTH * q, ii = p & 31, jj = p >> 5;
        const int i = I * 32 + ii, j = J * 32 + jj;
        if (i < n && j < n && i < j) {
            const int reg = k_regime(k, atom_distance(d, pos, i, j));
            list[reg * 1024 + atomicAdd(&cnt[reg], 1)] = (unsigned short)p;
        }
    }
    __syncthreads();
    const int c0 = cnt[0], c1 = cnt[1], tot = c0 + c1 + cnt[2];
    for (int w = tid; w < tot; w += NTH) {
        const int p = w < c0 ? list[w] : (w < c0 + c1 ? list[1024 + w - c0] : list[2048 + w - c0 - c1]);
        const int ii = p & 31, jj = p >> 5;
        zc m, dm = mk(0.0);
        pair_elements(d, k, atom_distance(d, pos, I * 32 + ii, J * 32 + jj), want_deriv, m, dm);
        put(ii, jj, m, dm);
    }
    __syncthreads();
    if (tid < 3) cnt[tid] = 0;
}

// The largest and the smallest non-zero max(|Re|, |Im|) of the entries a thread
// has seen, as the high words of the doubles (which order like the values).
struct EntryRange {
    int hi = 0, lo = 0x7fffffff;
    __device__ __forceinline__ void add(zc v) {
        const int a = max(__double2hiint(v.re) & 0x7fffffff, __double2hiint(v.im) & 0x7fffffff);
        hi = max(hi, a);
        if (a > 0) lo = min(lo, a);
    }
};

// Assemble M(k) into A and, if B != nullptr, dM/dk into B (ld n, column-major).
// Tiles of 32 x 32 pairs above the diagonal are evaluated once and written to
// both triangles, the mirrored tile through shared memory to keep stores
// coalesced.  A team deals out strips of a tile (NTH / 32 of its columns), round
// robin: one dlogf at d = 2, n = 50 has three tiles, of which K_nu is the most work.
template <class S, class Team>
static __device__ void assemble(zc* __restrict__ A, zc* __restrict__ B, int n, int d, const double* __restrict__ pos,
                         const msgpu_model& mdl, zc k, S& s, const Team& tm, EntryRange& rg) {
    constexpr int NTH = S::NTH, RQ = NTH / 32, NQ = 32 / RQ;  // tile rows per pass, passes
    const int tid = threadIdx.x;
    // F^-1 and the two sides of its central difference (dk_invf), a long scalar
    // FP64 chain each, by one thread of three warps
    const double h = DK_INVF_STEP;
    if (tid == 0) s.diag[0] = invf(mdl, d, k);
    if (B && tid == 32) s.urow[0] = invf(mdl, d, k + h);
    if (B && tid == 64) s.urow[1] = invf(mdl, d, k - h);
    __syncthreads();
    const zc dg0 = s.diag[0], dg1 = B ? (s.urow[0] - s.urow[1]) / (2.0 * h) : mk(0.0);
    rg.add(dg0);
    if (B) rg.add(dg1);
    zc (*T2)[NB + 1] = reinterpret_cast<zc(*)[NB + 1]>(&s.As[0][0]);
    // d != 3: pair lists of the regime grouping behind it, in the (idle) tile buffers
    constexpr size_t T2_BYTES = sizeof(zc) * NB * (NB + 1), AS_BYTES = sizeof(zc) * NB * S::TMR;
    unsigned short* list = reinterpret_cast<unsigned short*>(reinterpret_cast<char*>(&s.As[0][0]) +
                                                             (AS_BYTES > T2_BYTES ? AS_BYTES : T2_BYTES));
    int* cnt = reinterpret_cast<int*>(list + 3 * 1024);
    const bool grouped = d != 3 && d != 1;
    if (grouped && tid < 3) cnt[tid] = 0;
    __syncthreads();
    const int nt = (n + 31) / 32;
    const int strips = tm.size > 1 ? NQ : 1, units = nt * (nt + 1) / 2 * strips;
    int I = 0, J = 0, at = 0;  // tile of unit `at`
    for (int u = tm.rank; u < units; u += tm.size) {
        for (; at < u / strips; ++at)
            if (++I > J) { I = 0; ++J; }
        const int q0 = tm.size > 1 ? u % strips : 0, q1 = tm.size > 1 ? q0 + 1 : NQ;
        {
            if (grouped) {
                tile_pairs_grouped<NTH>(I, J, n, d, pos, k, B != nullptr, list, cnt, [&](int ii, int jj, zc m, zc dm) {
                    s.T[jj][ii] = m;
                    rg.add(m);
                    if (B) {
                        T2[jj][ii] = dm;
                        rg.add(dm);
                    }
                }, q0, q1);
                for (int q = q0; q < q1; ++q) {
                    const int ii = tid & 31, jj = (tid >> 5) + RQ * q;
                    const int i = I * 32 + ii, j = J * 32 + jj;
                    if (i < n && j < n && i <= j) {
                        A[i + (size_t)j * n] = i < j ? s.T[jj][ii] : dg0;
                        if (B) B[i + (size_t)j * n] = i < j ? T2[jj][ii] : dg1;
                    }
                }
            } else {
            for (int q = q0; q < q1; ++q) {
                const int ii = tid & 31, jj = (tid >> 5) + RQ * q;
                const int i = I * 32 + ii, j = J * 32 + jj;
                if (i < n && j < n && i <= j) {
                    zc m, dm = mk(0.0);
                    if (i < j) {
                        pair_elements(d, k, atom_distance(d, pos, i, j), B != nullptr, m, dm);
                    } else {
                        m = dg0;
                        dm = dg1;
                    }
                    A[i + (size_t)j * n] = m;
                    s.T[jj][ii] = m;
                    rg.add(m);
                    if (B) {
                        rg.add(dm);
                        B[i + (size_t)j * n] = dm;
                        T2[jj][ii] = dm;
                    }
                }
            }
            }
            __syncthreads();
            // the mirrored elements: a lane takes a column j, of this unit's strip
            const int jj = tid & 31, j = J * 32 + jj;
            if (j < n && jj >= RQ * q0 && jj < RQ * q1)
                for (int ii = tid >> 5; ii < 32; ii += RQ) {
                    const int i = I * 32 + ii;
                    if (i < j) {
                        A[j + (size_t)i * n] = s.T[jj][ii];
                        if (B) B[j + (size_t)i * n] = T2[jj][ii];
                    }
                }
            __syncthreads();
        }
    }
    if (tm.size > 1) tm.sync();
}

}  // namespace msg

#include "panel.cuh"
