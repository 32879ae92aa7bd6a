// eigvals.cu -- the eigenvalues mu of M(k), the input of the reference's
// mu-plane histograms (eigvals, src/core/ms_matrix_util.c:147, zgeev_ without
// eigenvectors; run_chistogram_omp and run_imag_mu_histogram_omp,
// src/core/ms_core.c:173-282).
//
// One persistent CTA per matrix slot, FP64 throughout (the reference's
// arithmetic), items dealt to CTAs in order:
//   1. M(k) assembled by the FP64 engine's assembly (lu64.cuh), or the
//      normalized N(k) = i - G(k)/I(k,0) of the mu-plane task's mtype=normalized
//      (build_normalized_matrix, ms_matrix_util.c:50) made from it in place;
//   2. reduction to upper Hessenberg form by Householder reflectors, as
//      LAPACK's unblocked zgehd2 (reflector of zlarfg; H applied from the
//      right to rows 0..n-1, H^H from the left to the trailing rows), the
//      reflector in shared memory, the right update one thread per row and the
//      left update one warp per column (coalesced both ways);
//   3. eigenvalues of the Hessenberg matrix by the single-shift complex QR
//      algorithm of LAPACK's zlahqr with wantt = wantz = false (real
//      subdiagonals, the Ahues-Kressner deflation test, Wilkinson shifts with
//      exceptional shifts every 10 iterations without deflation, the search
//      for two consecutive small subdiagonals, 2 x 2 reflectors chasing the
//      bulge through the active block): warp 0 chases the bulge through a window
//      of up to 30 steps on its diagonal block, the CTA takes the columns and
//      rows outside it through the window's reflectors.
// zgeev also balances the matrix first (zgebal); this path does not: M(k)'s
// entries do not span the magnitudes balancing is for, and the eigenvalues
// agree with the reference's to ~1e-13 of the largest.  Eigenvalues come out
// in deflation order, as zgeev's.
#include <cuda_runtime.h>
#include <float.h>
#include <algorithm>
#include <mutex>
#include <vector>
#include "msgpu.h"
#include "lu64.cuh"
#include "engine_internal.h"

namespace msg {

// shared memory: the assembly's and the reductions' LuSmem; the Householder
// vector overlays its two tile buffers (4096 complex values: n <= 4097)
constexpr int EIG_NMAX = NB * (TM + LuSmem::TNC) + 1;

struct EigParams {
    int nitem;
    const int* item_n;       // order per item
    const int* item_d;
    const size_t* item_pos;  // offset of the item's positions in pos
    const msgpu_model* item_model;
    const double* pos;
    const double* ks;        // 2 per item
    const size_t* item_out;  // offset of the item's eigenvalues in mu
    zc* mu;
    int* status;
    zc* work;                // one nmax x nmax slot per CTA
    size_t slot;
    int normalized;          // N(k) = i - G(k)/I(k,0) in place of M(k)
    double* trg2;            // per item Tr[G^+ G]/N of the matrix (tracegtwo), or nullptr
};

__device__ __forceinline__ double dlapy3(double x, double y, double z) {
    const double w = fmax(fabs(x), fmax(fabs(y), fabs(z)));
    if (w == 0.0) return fabs(x) + fabs(y) + fabs(z);
    const double a = x / w, b = y / w, c = z / w;
    return w * sqrt(a * a + b * b + c * c);
}

// 2^-e of a modulus m = f 2^e; 1 where there is nothing to scale by (0, infinite, NaN)
__device__ __forceinline__ double unit_scale(double m) {
    if (!(m > 0.0) || !(m < INFINITY)) return 1.0;
    return scalbn(1.0, max(-1000, min(1000, -ilogb(m))));
}
// do squares that add up to s lose nothing to the exponent range?
__device__ __forceinline__ bool squares_safe(double s) { return s > 1e-280 && s < 1e280; }

// Householder reduction to upper Hessenberg form (zgehd2, ilo = 1, ihi = n)
static __device__ void hessenberg(zc* __restrict__ A, int n, LuSmem& s) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    zc* v = &s.As[0][0];
    for (int j = 0; j + 2 < n; ++j) {
        const int m = n - j - 1;  // length of the reflector
        zc* col = A + (size_t)j * n + j + 1;
        double ss = 0.0, z1 = 0.0, z2 = 0.0;
        for (int i = 1 + tid; i < m; i += NT) ss += zabs2(col[i]);
        block_sum3(ss, z1, z2, s);
        double xnorm = sqrt(ss);
        if (!squares_safe(ss)) {
            // squares out of range, or zeros: the norm of the column scaled by its largest entry
            double mx = 0.0;
            int im = m, at;
            for (int i = 1 + tid; i < m; i += NT) {
                const double v = fmax(fabs(col[i].re), fabs(col[i].im));
                if (v > mx) { mx = v; im = i; }
            }
            block_argmax(mx, im, s, at);
            const double sc = at < m ? unit_scale(fmax(fabs(col[at].re), fabs(col[at].im))) : 1.0;
            ss = 0.0;
            for (int i = 1 + tid; i < m; i += NT) ss += zabs2(sc * col[i]);
            block_sum3(ss, z1, z2, s);
            xnorm = sqrt(ss) / sc;
        }
        const zc alpha = col[0];
        __syncthreads();  // every thread has read alpha before column j changes
        if (xnorm == 0.0 && alpha.im == 0.0) continue;  // H = I (tau = 0)
        // zlarfg: beta = -sign(Re alpha) |(alpha, x)|, tau = (beta - alpha) / beta,
        // v = (1, x / (alpha - beta))
        const double beta = -copysign(dlapy3(alpha.re, alpha.im, xnorm), alpha.re);
        const zc tau = mk((beta - alpha.re) / beta, -alpha.im / beta);
        const zc scal = 1.0 / (alpha - beta);
        for (int i = tid; i < m; i += NT) {
            v[i] = i == 0 ? mk(1.0) : col[i] * scal;
            col[i] = i == 0 ? mk(beta) : mk(0.0);
        }
        __syncthreads();
        // from the right: A[0:n, j+1:n] -= tau (A v) v^H
        for (int r = tid; r < n; r += NT) {
            zc* row = A + r + (size_t)(j + 1) * n;
            zc w = mk(0.0);
            for (int c = 0; c < m; ++c) w += row[(size_t)c * n] * v[c];
            w = tau * w;
            for (int c = 0; c < m; ++c) row[(size_t)c * n] -= w * conjz(v[c]);
        }
        __syncthreads();
        // from the left with conj(tau): A[j+1:n, j+1:n] -= conj(tau) v (v^H A)
        const zc ctau = conjz(tau);
        for (int c = j + 1 + warp; c < n; c += NT / 32) {
            zc* cc = A + (size_t)c * n + j + 1;
            zc w = mk(0.0);
            for (int i = lane; i < m; i += 32) w += conjz(v[i]) * cc[i];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                w.re += __shfl_xor_sync(0xffffffffu, w.re, off);
                w.im += __shfl_xor_sync(0xffffffffu, w.im, off);
            }
            w = ctau * w;
            for (int i = lane; i < m; i += 32) cc[i] -= v[i] * w;
        }
        __syncthreads();
    }
}

// zlarfg for n = 2 and real x: on return a = beta (real), v2 the reflector's second
// entry, the reflector I - t1 (1, v2)(1, v2)^H, and t2 = t1 v2, which is real.  (The
// bulge's lower entry is a product of t2 and a subdiagonal entry, both real.)  The
// warp that chases the bulge is bound by how many FP64 instructions it issues, 64
// clocks each: one reciprocal square root gives beta and 1 / beta, one division the
// rest, 32 of them in all where a square root, two divisions and complex products
// took 47.  Where |a|^2 + x^2 leaves the exponent range (entries below 1e-140 or above
// 1e140) both are scaled to 1 first, as zlarfg does; only beta depends on the scale.
__device__ __forceinline__ void larfg2(zc& a, double x, zc& t1, zc& v2, double& t2) {
    double b2 = fma(x, x, fma(a.re, a.re, a.im * a.im)), back = 1.0;
    if (x == 0.0 && a.im == 0.0) {
        t1 = v2 = mk(0.0);
        t2 = 0.0;
        return;
    }
    if (!squares_safe(b2)) {
        const double sc = unit_scale(fmax(fabs(x), fmax(fabs(a.re), fabs(a.im))));
        a = sc * a;
        x *= sc;
        b2 = fma(x, x, fma(a.re, a.re, a.im * a.im));
        back = 1.0 / sc;  // a power of two
    }
    const double rs = rsqrt(b2);
    double beta = b2 * rs;
    beta = -copysign(fma(0.5 * rs, fma(-beta, beta, b2), beta), a.re);
    const double rb = copysign(rs, beta);
    const zc d = mk(a.re - beta, a.im);
    t1 = mk(-d.re * rb, -d.im * rb);
    t2 = -x * rb;
    const double y = x / fma(d.re, d.re, d.im * d.im);
    v2 = mk(d.re * y, -d.im * y);
    a = mk(beta * back);
}

// reflectors a bulge-chase window makes, and its rows and columns
constexpr int HQR_W = 30, HQR_D = HQR_W + 2;

// what the CTA shares in the QR iteration
struct HqrShared {
    zc temp;
    zc t1[2][HQR_W], v2[2][HQR_W];  // reflectors of the last two windows
    double t2[2][HQR_W];
    zc win[HQR_D][HQR_D + 1];       // the diagonal block of the window being chased
    int l, m, flag;
};

// One reflector (t1, v2, t2) on the pair (a, b) of a column, from the left
__device__ __forceinline__ void hqr_left(zc t1, zc v2, double t2, zc& a, zc& b) {
    const zc sum = conjz(t1) * a + t2 * b;
    a -= sum;
    b -= sum * v2;
}
// ... and on the pair (a, b) of a row, from the right
__device__ __forceinline__ void hqr_right(zc t1, zc v2, double t2, zc& a, zc& b) {
    const zc sum = t1 * a + t2 * b;
    a -= sum;
    b -= sum * conjz(v2);
}

// A window's ns reflectors (rows and columns lo..lo+ns) on columns [c0, c1] from the
// left and on rows [r0, r1] from the right, a lane a column or row, 32 of them at a
// time for warp w of nw.
static __device__ void hqr_far(zc* __restrict__ H, int n, const HqrShared& q, int par, int lo, int ns, int c0, int c1, int r0,
                               int r1, int w, int nw) {
    const int lane = threadIdx.x & 31;
    const int bc = c1 >= c0 ? (c1 - c0 + 32) / 32 : 0, br = r1 >= r0 ? (r1 - r0 + 32) / 32 : 0;
    for (int b = w; b < bc + br; b += nw) {
        const bool left = b < bc;
        const int x = left ? c0 + 32 * b + lane : r0 + 32 * (b - bc) + lane;
        if (x > (left ? c1 : r1)) continue;
        zc* p = left ? H + lo + (size_t)x * n : H + x + (size_t)lo * n;
        const size_t st = left ? 1 : n;
        zc a = p[0];
        for (int s = 0; s < ns; ++s) {
            zc v = p[(s + 1) * st];
            if (left) hqr_left(q.t1[par][s], q.v2[par][s], q.t2[par][s], a, v);
            else hqr_right(q.t1[par][s], q.v2[par][s], q.t2[par][s], a, v);
            p[s * st] = a;
            a = v;
        }
        p[ns * st] = a;
    }
}

// Eigenvalues of the upper Hessenberg H (n x n, ld n) into w by zlahqr's
// single-shift QR (wantt = wantz = false).  A sweep is chased in windows of up to
// HQR_W steps: warp 0 makes the reflectors on the window's diagonal block in
// shared memory, every lane with the scalar chain to itself, a column or row of
// the block each; then the CTA takes each column right of the block and each row
// above it through all of the window's reflectors, a thread a column or row, the
// next window's columns first and the rest beside the next window's chase.  (A
// step at a time across the CTA, three barriers and three global round trips each,
// took 8k cycles a step at n = 256: 415 ms for 64 matrices on as many SMs.)  The
// deflation test and the search for the sweep's start look at 32 rows at once.
// Returns 0, or i + 1 if eigenvalue i and above did not converge within
// 30 max(10, n) iterations (zlahqr's info).
static __device__ int hqr_cta(zc* __restrict__ H, int n, zc* __restrict__ w, HqrShared& q) {
    const int tid = threadIdx.x;
    auto h = [&](int r, int c) -> zc& { return H[r + (size_t)c * n]; };
    if (n == 1) {
        if (tid == 0) w[0] = h(0, 0);
        return 0;
    }
    const int ilo = 0, ihi = n - 1;
    // subdiagonal entries made real by diagonal unitary similarity
    for (int i = ilo + 1; i <= ihi; ++i) {
        if (tid == 0) {
            const zc hs = h(i, i - 1);
            q.flag = hs.im != 0.0;
            if (q.flag) {
                const zc sc = hs / abs1(hs);
                q.temp = conjz(sc) / zabs(sc);
                h(i, i - 1) = mk(zabs(hs));
            }
        }
        __syncthreads();
        if (q.flag) {
            const zc sc = q.temp;
            for (int j = i + tid; j <= ihi; j += NT) h(i, j) = h(i, j) * sc;
            __syncthreads();
            const int top = min(ihi, i + 1);
            for (int j = ilo + tid; j <= top; j += NT) h(j, i) = h(j, i) * conjz(sc);
        }
        __syncthreads();
    }
    const double safmin = DBL_MIN, ulp = DBL_EPSILON;
    const double smlnum = safmin * ((double)(ihi - ilo + 1) / ulp);
    const int itmax = 30 * max(10, ihi - ilo + 1);
    constexpr int KEXSH = 10;
    int kdefl = 0;
    int i = ihi;
    zc v0 = mk(0.0), v1 = mk(0.0);  // warp 0's reflector vector
    while (i >= ilo) {
        int l = ilo;
        bool done = false;
        for (int its = 0; its <= itmax; ++its) {
            if (tid < 32) {
                // a single small subdiagonal element: the largest k in (l, i] that has one, else l
                auto small = [&](int k) {
                    const zc hkk1 = h(k, k - 1);
                    if (abs1(hkk1) <= smlnum) return true;
                    double tst = abs1(h(k - 1, k - 1)) + abs1(h(k, k));
                    if (tst == 0.0) {
                        if (k - 2 >= ilo) tst += fabs(h(k - 1, k - 2).re);
                        if (k + 1 <= ihi) tst += fabs(h(k + 1, k).re);
                    }
                    if (fabs(hkk1.re) > ulp * tst) return false;
                    const double a1 = abs1(hkk1), a2 = abs1(h(k - 1, k));
                    const double ab = fmax(a1, a2), ba = fmin(a1, a2);
                    const double b1 = abs1(h(k, k)), b2 = abs1(h(k - 1, k - 1) - h(k, k));
                    const double aa = fmax(b1, b2), bb = fmin(b1, b2);
                    const double sab = aa + ab;
                    return ba * (ab / sab) <= fmax(smlnum, ulp * (bb * (aa / sab)));
                };
                int k = l;
                for (int top = i; top > l; top -= 32) {
                    const unsigned hit = __ballot_sync(0xffffffffu, top - tid > l && small(top - tid));
                    if (hit) {
                        k = top - (__ffs(hit) - 1);
                        break;
                    }
                }
                __syncwarp();
                if (tid == 0) {
                    if (k > ilo) h(k, k - 1) = mk(0.0);
                    q.l = k;
                }
                if (k < i) {
                    const int kd = kdefl + 1;
                    zc t;
                    if (kd % (2 * KEXSH) == 0) {
                        t = h(i, i) + 0.75 * fabs(h(i, i - 1).re);
                    } else if (kd % KEXSH == 0) {
                        t = h(k, k) + 0.75 * fabs(h(k + 1, k).re);
                    } else {  // Wilkinson's shift
                        t = h(i, i);
                        const zc u = zsqrt(h(i - 1, i)) * zsqrt(h(i, i - 1));
                        double s = abs1(u);
                        if (s != 0.0) {
                            const zc x = 0.5 * (h(i - 1, i - 1) - t);
                            const double sx = abs1(x);
                            s = fmax(s, sx);
                            const zc xs = x / s, us = u / s;
                            zc y = s * zsqrt(xs * xs + us * us);
                            if (sx > 0.0) {
                                const zc xn = x / sx;
                                if (xn.re * y.re + xn.im * y.im < 0.0) y = -y;
                            }
                            t = t - u * (u / (x + y));
                        }
                    }
                    // two consecutive small subdiagonal elements: start the sweep at row m,
                    // the largest in (k, i-1] that has them, else k; the bulge's first vector
                    auto start = [&](int m) {
                        zc h11s = h(m, m) - t;
                        double h21 = h(m + 1, m).re;
                        const double s = abs1(h11s) + fabs(h21);
                        v0 = h11s / s;
                        v1 = mk(h21 / s);
                    };
                    int m = k;
                    for (int top = i - 1; top > k; top -= 32) {
                        bool ok = false;
                        const int mm = top - tid;
                        if (mm > k) {
                            start(mm);
                            const double h10 = h(mm, mm - 1).re;
                            ok = fabs(h10) * fabs(v1.re) <= ulp * (abs1(v0) * (abs1(h(mm, mm)) + abs1(h(mm + 1, mm + 1))));
                        }
                        const unsigned hit = __ballot_sync(0xffffffffu, ok);
                        if (hit) {
                            m = top - (__ffs(hit) - 1);
                            break;
                        }
                    }
                    start(m);
                    if (tid == 0) q.m = m;
                }
            }
            __syncthreads();
            l = q.l;
            if (l >= i) {
                done = true;
                break;
            }
            ++kdefl;
            const int i1 = l, i2 = i, m = q.m;
            // the single-shift QR sweep
            int prev_lo = 0, prev_hi = -1, prev_ns = 0, par = 0;  // the window whose far part is still to do
            for (int lo = m; lo < i;) {
                // a sweep that starts below l rescales the block after its first step: that one alone
                const int ns = min(lo == m && m > l ? 1 : HQR_W, i - lo), hi = min(lo + ns + 1, i), dim = hi - lo + 1;
                if (tid < 32) {
                    for (int e = tid; e < dim * dim; e += 32) q.win[e % dim][e / dim] = h(lo + e % dim, lo + e / dim);
                    if (lo > m) {
                        v0 = h(lo, lo - 1);
                        v1 = h(lo + 1, lo - 1);
                    }
                    __syncwarp();
                    for (int s = 0; s < ns; ++s) {
                        if (s > 0) {
                            v0 = q.win[s][s - 1];
                            v1 = q.win[s + 1][s - 1];
                        }
                        zc t1, v2;
                        double t2;
                        larfg2(v0, v1.re, t1, v2, t2);
                        __syncwarp();
                        if (tid == 0) {
                            q.t1[par][s] = t1;
                            q.v2[par][s] = v2;
                            q.t2[par][s] = t2;
                            if (s > 0) {
                                q.win[s][s - 1] = v0;
                                q.win[s + 1][s - 1] = mk(0.0);
                            } else if (lo > m) {
                                h(lo, lo - 1) = v0;
                                h(lo + 1, lo - 1) = mk(0.0);
                            }
                        }
                        if (tid >= s && tid < dim) hqr_left(t1, v2, t2, q.win[s][tid], q.win[s + 1][tid]);
                        __syncwarp();
                        if (tid <= min(s + 2, dim - 1)) hqr_right(t1, v2, t2, q.win[tid][s], q.win[tid][s + 1]);
                        __syncwarp();
                    }
                    for (int e = tid; e < dim * dim; e += 32) h(lo + e % dim, lo + e / dim) = q.win[e % dim][e / dim];
                } else if (prev_ns > 0 && (tid >> 5) % 4 != 0) {
                    // the far part of the window before, by the warps that do not share warp 0's FP64 pipe
                    hqr_far(H, n, q, par ^ 1, prev_lo, prev_ns, min(prev_hi + HQR_D, i2) + 1, i2, i1, prev_lo - 1,
                            (tid >> 5) / 4 * 3 + (tid >> 5) % 4 - 1, NT / 128 * 3);
                }
                __syncthreads();
                // the columns of the next window first
                hqr_far(H, n, q, par, lo, ns, hi + 1, min(hi + HQR_D, i2), 0, -1, tid >> 5, NT / 32);
                __syncthreads();
                prev_lo = lo;
                prev_hi = hi;
                prev_ns = ns;
                if (lo == m && m > l) {
                    // far part at once, then keep H(m, m-1) real.  Row j in S =
                    // [m, i] \ {m+1} takes temp right of the diagonal, column j in S takes
                    // conj(temp) above it (zlahqr, one row and column at a time); an
                    // entry in both keeps its value
                    hqr_far(H, n, q, par, lo, ns, min(hi + HQR_D, i2) + 1, i2, i1, lo - 1, tid >> 5, NT / 32);
                    prev_ns = 0;
                    zc temp = 1.0 - q.t1[par][0];
                    temp = temp / zabs(temp);
                    __syncthreads();
                    if (tid == 0) {
                        h(m + 1, m) = h(m + 1, m) * conjz(temp);
                        if (m + 2 <= i) h(m + 2, m + 1) = h(m + 2, m + 1) * temp;
                    }
                    auto in_s = [&](int x) { return x >= m && x <= i && x != m + 1; };
                    const int na = i - i1 + 1;
                    for (int e = tid; e < na * na; e += NT) {
                        const int r = i1 + e % na, c = i1 + e / na;
                        if (r >= c) continue;
                        const bool a = in_s(r), b = in_s(c);
                        if (a && !b) h(r, c) = h(r, c) * temp;
                        else if (b && !a) h(r, c) = h(r, c) * conjz(temp);
                    }
                    __syncthreads();
                }
                lo += ns;
                par ^= 1;
            }
            if (prev_ns > 0) {
                hqr_far(H, n, q, par ^ 1, prev_lo, prev_ns, min(prev_hi + HQR_D, i2) + 1, i2, i1, prev_lo - 1, tid >> 5, NT / 32);
                __syncthreads();
            }
            // H(i, i-1) made real
            if (tid == 0) {
                const zc temp = h(i, i - 1);
                q.flag = temp.im != 0.0;
                if (q.flag) {
                    const double rt = zabs(temp);
                    q.temp = temp / rt;
                    h(i, i - 1) = mk(rt);
                }
            }
            __syncthreads();
            if (q.flag) {
                const zc u = q.temp;
                for (int c = i + 1 + tid; c <= i2; c += NT) h(i, c) = h(i, c) * conjz(u);
                for (int r = i1 + tid; r < i; r += NT) h(r, i) = h(r, i) * u;
            }
            __syncthreads();
        }
        if (!done) return i + 1;
        if (tid == 0) w[i] = h(i, i);
        kdefl = 0;
        i = l - 1;
    }
    return 0;
}

__global__ void __launch_bounds__(NT, 2) k_eigvals(EigParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    LuSmem& s = *reinterpret_cast<LuSmem*>(smem_raw);
    __shared__ HqrShared q;
    zc* A = P.work + (size_t)blockIdx.x * P.slot;
    for (int it = blockIdx.x; it < P.nitem; it += gridDim.x) {
        const int n = P.item_n[it];
        const zc k = mk(P.ks[2 * it], P.ks[2 * it + 1]);
        EntryRange rg;
        assemble(A, nullptr, n, P.item_d[it], P.pos + P.item_pos[it], P.item_model[it], k, s, Solo{}, rg);
        __syncthreads();
        if (P.normalized) {
            // build_normalized_matrix (ms_matrix_util.c:50): off the diagonal -G(k, r_ij) / I(k, 0),
            // that is M_ij / I(k, 0); i on the diagonal
            if (threadIdx.x == 0) s.diag[0] = free_green_imag(P.item_d[it], k, 0.0);
            __syncthreads();
            const zc iz = s.diag[0];
            for (size_t e = threadIdx.x; e < (size_t)n * n; e += NT) {
                const size_t r = e % n, c = e / n;
                A[e] = r == c ? mk(0.0, 1.0) : A[e] / iz;
            }
            __syncthreads();
        }
        if (P.trg2) {
            // tracegtwo (ms_matrix_util.c:167): 2 sum_{i<j} |A_ij|^2 / n, the matrix symmetric
            double t = 0.0, z1 = 0.0, z2 = 0.0;
            for (size_t e = threadIdx.x; e < (size_t)n * n; e += NT)
                if (e % n < e / n) t += zabs2(A[e]);
            block_sum3(t, z1, z2, s);
            if (threadIdx.x == 0) P.trg2[it] = 2.0 * t / n;
        }
        hessenberg(A, n, s);
        const int info = hqr_cta(A, n, P.mu + P.item_out[it], q);
        if (threadIdx.x == 0) P.status[it] = info > 0 ? MSGPU_S_NOCONV : 0;
        __syncthreads();
    }
}

}  // namespace msg

namespace {
std::mutex g_eig_mu;
}

extern "C" int msgpu_eigvals_batch_mtype(int mtype, int nmed, const msgpu_medium* media, int nitem,
                                         const int* item_med, const double* ks, double* mu, int* status,
                                         double* trg2) {
    using namespace msg;
    if ((mtype != MSGPU_MTYPE_MSMATRIX && mtype != MSGPU_MTYPE_NORMALIZED) || nmed < 1 || !media || nitem < 1 || !ks ||
        !mu)
        return record_error(MSGPU_E_ARG, "eigvals: bad argument (mtype 0 or 1, nmed >= 1, nitem >= 1, non-null pointers)");
    int nmax = 0;
    size_t npos = 0;
    std::vector<size_t> med_pos(nmed);
    for (int m = 0; m < nmed; ++m) {
        if (media[m].n < 1 || media[m].d < 1 || !media[m].pos)
            return record_error(MSGPU_E_ARG, "eigvals: a medium has n < 1, d < 1 or no positions");
        nmax = std::max(nmax, media[m].n);
        med_pos[m] = npos;
        npos += (size_t)media[m].n * media[m].d;
    }
    if (nmax > EIG_NMAX) return record_error(MSGPU_E_SIZE, "eigvals: n > 4097 (the reflector lives in shared memory)");
    for (int i = 0; i < nitem; ++i)
        if (item_med && (item_med[i] < 0 || item_med[i] >= nmed))
            return record_error(MSGPU_E_ARG, "eigvals: item_med out of range");
    const int sms = msgpu_sm_count();  // initialises the device and the kernels' attributes
    if (sms < 1) return record_error(MSGPU_E_NODEV, "eigvals: no CUDA device");
    std::lock_guard<std::mutex> lk(g_eig_mu);
    // on every call: the attribute belongs to the current device
    if (cudaFuncSetAttribute(k_eigvals, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LuSmem)) !=
        cudaSuccess)
        return record_error(MSGPU_E_CUDA, "eigvals: cudaFuncSetAttribute (shared memory) failed");
    std::vector<int> hn(nitem), hd(nitem);
    std::vector<size_t> hpos(nitem), hout(nitem);
    std::vector<msgpu_model> hmodel(nitem);
    size_t nout = 0;
    for (int i = 0; i < nitem; ++i) {
        const int mi = item_med ? item_med[i] : 0;
        hn[i] = media[mi].n;
        hd[i] = media[mi].d;
        hpos[i] = med_pos[mi];
        hmodel[i] = media[mi].model;
        hout[i] = nout;
        nout += (size_t)media[mi].n;
    }
    const size_t slot = (size_t)nmax * nmax;
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return record_error(MSGPU_E_CUDA, "eigvals: cudaMemGetInfo failed");
    const size_t budget = free_b > ((size_t)4 << 30) ? free_b - ((size_t)4 << 30) : free_b / 2;
    const int grid = (int)std::min<size_t>({(size_t)nitem, (size_t)2 * sms, std::max<size_t>(1, budget / (slot * 16))});
    double *dpos = nullptr, *dks = nullptr;
    zc *dmu = nullptr, *dwork = nullptr;
    int *dn = nullptr, *dd = nullptr, *dst = nullptr;
    double* dtrg = nullptr;
    size_t *dposo = nullptr, *douto = nullptr;
    msgpu_model* dmodel = nullptr;
    auto cleanup = [&]() {
        cudaFree(dpos); cudaFree(dks); cudaFree(dmu); cudaFree(dwork); cudaFree(dn); cudaFree(dd);
        cudaFree(dst); cudaFree(dposo); cudaFree(douto); cudaFree(dmodel); cudaFree(dtrg);
    };
    if (cudaMalloc(&dpos, sizeof(double) * npos) || cudaMalloc(&dks, sizeof(double) * 2 * nitem) ||
        cudaMalloc(&dmu, sizeof(zc) * nout) || cudaMalloc(&dwork, sizeof(zc) * slot * grid) ||
        cudaMalloc(&dn, sizeof(int) * nitem) || cudaMalloc(&dd, sizeof(int) * nitem) ||
        cudaMalloc(&dst, sizeof(int) * nitem) || cudaMalloc(&dposo, sizeof(size_t) * nitem) ||
        cudaMalloc(&douto, sizeof(size_t) * nitem) || cudaMalloc(&dmodel, sizeof(msgpu_model) * nitem) ||
        (trg2 && cudaMalloc(&dtrg, sizeof(double) * nitem))) {
        cleanup();
        return record_error(MSGPU_E_CUDA, "eigvals: device allocation failed");
    }
    bool ok = true;
    for (int m = 0; m < nmed && ok; ++m)
        ok = cudaMemcpy(dpos + med_pos[m], media[m].pos, sizeof(double) * (size_t)media[m].n * media[m].d,
                        cudaMemcpyHostToDevice) == cudaSuccess;
    ok = ok && cudaMemcpy(dks, ks, sizeof(double) * 2 * nitem, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(dn, hn.data(), sizeof(int) * nitem, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(dd, hd.data(), sizeof(int) * nitem, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(dposo, hpos.data(), sizeof(size_t) * nitem, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(douto, hout.data(), sizeof(size_t) * nitem, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(dmodel, hmodel.data(), sizeof(msgpu_model) * nitem, cudaMemcpyHostToDevice) == cudaSuccess;
    ok = ok && cudaMemset(dmu, 0, sizeof(zc) * nout) == cudaSuccess;  // unconverged values read 0
    if (!ok) {
        cleanup();
        return record_error(MSGPU_E_CUDA, "eigvals: host-to-device copy failed");
    }
    EigParams P{nitem, dn, dd, dposo, dmodel, dpos, dks, douto, dmu, dst, dwork, slot,
                mtype == MSGPU_MTYPE_NORMALIZED, dtrg};
    k_eigvals<<<grid, NT, sizeof(LuSmem)>>>(P);
    count_launches(1);
    std::vector<int> hst(nitem);
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(mu, dmu, sizeof(zc) * nout, cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(hst.data(), dst, sizeof(int) * nitem, cudaMemcpyDeviceToHost) != cudaSuccess ||
        (trg2 && cudaMemcpy(trg2, dtrg, sizeof(double) * nitem, cudaMemcpyDeviceToHost) != cudaSuccess)) {
        cleanup();
        return record_error(MSGPU_E_CUDA, "eigvals: kernel launch, execution or device-to-host copy failed");
    }
    if (status)
        for (int i = 0; i < nitem; ++i) status[i] = hst[i];
    cleanup();
    return 0;
}

extern "C" int msgpu_eigvals_batch(int nmed, const msgpu_medium* media, int nitem, const int* item_med,
                                   const double* ks, double* mu, int* status) {
    return msgpu_eigvals_batch_mtype(MSGPU_MTYPE_MSMATRIX, nmed, media, nitem, item_med, ks, mu, status, nullptr);
}
