// fp64_engine.cuh -- the FP64 engine's work loop, shared by its two kernels:
// k_engine_fp64 (engine.cu; every update on the FP64 pipe) and k_engine_tc64
// (tc64.cu; trailing updates on the tensor cores).
#pragma once
#include "lu64.cuh"
#include "engine_internal.h"

namespace msg {

// complex elements of one CTA slot: the matrix, plus dM/dk (kind 1) or the
// right-hand side (kind 2)
__host__ __device__ inline size_t slot_elems(int kind, size_t slot, int nmax) {
    if (kind == 1) return 2 * slot;
    // kind 2: the matrix, its copy for the refinement residual (mixed engine), four vectors;
    // kinds 1, 3: the matrix and a right-hand-side matrix; kind 4: the matrix and two vectors
    const size_t vec = (((size_t)nmax + 15) / 16) * 16;
    if (kind == 2) return 2 * slot + 4 * vec;
    if (kind == 1 || kind == 3) return 2 * slot;
    if (kind == 4) return slot + 2 * vec;
    return slot;
}

// cnormalize (complex_vector_util.c:47): x /= fac, fac = |x| x_i0/|x_i0| with
// x_i0 the first nonzero entry (locks the phase); returns fac
template <class S>
static __device__ zc cnormalize_block(zc* __restrict__ x, int n, S& s) {
    double nr = 0.0, z0 = 0.0, z1 = 0.0;
    for (int i = threadIdx.x; i < n; i += S::NTH) nr += zabs2(x[i]);
    block_sum3(nr, z0, z1, s);
    double nzv = -1.0;
    int nzi = n;
    for (int i = threadIdx.x; i < n; i += S::NTH)
        if (x[i].re != 0.0 || x[i].im != 0.0) {
            nzv = 1.0;
            nzi = min(nzi, i);
        }
    int i0;
    block_argmax(nzv, nzi, s, i0);
    if (i0 >= n) return mk(1.0);
    const zc xi = x[i0];
    const zc fac = (sqrt(nr) / zabs(xi)) * xi;
    __syncthreads();  // every thread read x[i0] before it is rescaled
    const zc rf = 1.0 / fac;
    for (int i = threadIdx.x; i < n; i += S::NTH) x[i] = x[i] * rf;
    __syncthreads();
    return fac;
}

// inverse_iteration (ms_matrix_util.c:279) on the LU already in A: from
// `start` (n complex values, the caller's previous eigenvector) or else the
// constant unit vector, x <- normalize(A^-1 x) until |x - x_old| < 1e-10 or 50
// steps (the reference's ivit_maxit / ivit_toler); returns lambda = 1 / fac,
// the eigenvalue of smallest modulus, x the eigenvector; conv = 0 if not reached.
template <class S>
static __device__ zc inverse_iteration(const zc* __restrict__ A, zc* __restrict__ x, zc* __restrict__ xold, int n,
                                       const int* __restrict__ ipiv, S& s, int& conv,
                                       const double* __restrict__ start) {
    for (int i = threadIdx.x; i < n; i += S::NTH) x[i] = start ? mk(start[2 * i], start[2 * i + 1]) : mk(1.0);
    __syncthreads();
    zc fac = cnormalize_block(x, n, s);
    conv = 0;
    for (int it = 0; it < 50; ++it) {
        for (int i = threadIdx.x; i < n; i += S::NTH) xold[i] = x[i];
        __syncthreads();
        lu_solve_vec(A, x, n, ipiv, s);
        fac = cnormalize_block(x, n, s);
        double d2 = 0.0, z0 = 0.0, z1 = 0.0;
        for (int i = threadIdx.x; i < n; i += S::NTH) d2 += zabs2(x[i] - xold[i]);
        block_sum3(d2, z0, z1, s);
        if (sqrt(d2) < 1e-10) {
            conv = 1;
            break;
        }
    }
    return 1.0 / fac;
}

// A team (the CTAs of a cluster, one or more) takes the next item from the
// queue, assembles M(k) (and dM/dk) into its slot, factors it together and
// reduces it by its first CTA, then takes the next item.
template <class S, class Update>
static __device__ void run_items_fp64(const EngineParams& P, S& s, const ClusterTeam& tm, const Update& up) {
    const int tid = threadIdx.x, team = blockIdx.x / tm.size;
    zc* A = P.ws + (size_t)team * slot_elems(P.kind, P.slot, P.piv_stride);
    zc* B = (P.kind >= 1) ? A + P.slot : nullptr;
    int* ipiv = P.piv + (size_t)team * P.piv_stride;
    if (tm.size > 1) tm.sync();  // every CTA of the cluster is there before its shared memory is written
    for (;;) {
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
        int it = 0;
        MedDev md{0, P.given_n, nullptr, {}};
        zc k = mk(0.0);
        EntryRange rg;
        if (P.given_n > 0) {
            const size_t nn = (size_t)md.n * md.n;
            for (size_t e = (size_t)tm.rank * S::NTH + tid; e < nn; e += (size_t)tm.size * S::NTH) rg.add(A[e]);
        } else {
            it = P.order[q];
            md = P.media[P.item_med[it]];
            k = mk(P.ks[2 * it], P.ks[2 * it + 1]);
            assemble(A, P.kind == 1 ? B : nullptr, md.n, md.d, md.pos, md.model, k, s, tm, rg);
        }
        up.begin(rg, md.n, s, tm);
        zc res = mk(0.0);
        int conv = 1;
        if (P.kind == 3) {
            // traceinv (ms_matrix_util.c:319): tr(M^-1 I) by the n-right-hand-side solve
            for (size_t e = (size_t)tm.rank * S::NTH + tid; e < (size_t)md.n * md.n; e += (size_t)tm.size * S::NTH)
                B[e] = (e % (md.n + 1) == 0) ? mk(1.0) : mk(0.0);
            tm.sync();
        }
        if (P.kind == 2 && tm.rank == 0) {
            // incident plane wave along +x (reference incident_wave_util.c:76, ms_core.c:616-618)
            for (int i = tid; i < md.n; i += S::NTH) B[i] = zexp(mk(0.0, 1.0) * k * md.pos[i * md.d]);
            __syncthreads();
        }
        lu_factor(A, md.n, ipiv, P.kind != 0, s, tm, up);
        if (P.kind == 1 || P.kind == 3) {
            res = lu_trace_solve(A, B, md.n, ipiv, s, tm, up);
        } else if (tm.rank != 0) {
            // the reductions and the solves of one vector are the first CTA's
        } else if (P.kind == 0) {
            res = lu_tracelog(A, md.n, ipiv, s);
        } else if (P.kind == 4) {
            const size_t vec = (((size_t)P.piv_stride + 15) / 16) * 16;
            res = inverse_iteration(A, B, B + vec, md.n, ipiv, s, conv,
                                    P.warm && P.amps ? P.amps + 2 * P.amp_off[it] : nullptr);
            if (P.amps)
                for (int i = tid; i < md.n; i += S::NTH) {
                    P.amps[2 * (P.amp_off[it] + i)] = B[i].re;
                    P.amps[2 * (P.amp_off[it] + i) + 1] = B[i].im;
                }
        } else {
            lu_solve_vec(A, B, md.n, ipiv, s);
            // optical theorem sigma = -Im(conj(phi).a)/k (reference ms_matrix_util.c:361)
            double dr = 0.0, di = 0.0, z = 0.0;
            for (int i = tid; i < md.n; i += S::NTH) {
                zc ph = zexp(mk(0.0, 1.0) * k * md.pos[i * md.d]);
                zc t = conjz(ph) * B[i];
                dr += t.re;
                di += t.im;
                if (P.amps) {
                    P.amps[2 * (P.amp_off[it] + i)] = B[i].re;
                    P.amps[2 * (P.amp_off[it] + i) + 1] = B[i].im;
                }
            }
            block_sum3(dr, di, z, s);
            res = mk(-di, 0.0) / k;
        }
        const bool bad = up.failed(s, tm);
        if (bad) {
            res = mk(nan(""), nan(""));
            if (tm.rank == 0 && P.given_n <= 0) void_amplitudes(P, it, tid, S::NTH);
        }
        if (tm.rank == 0 && tid == 0) {
            P.out[2 * it] = res.re;
            P.out[2 * it + 1] = res.im;
            int st = bad ? MSGPU_S_TIMEOUT : 0;
            if (s.info) st |= MSGPU_S_SINGULAR;
            if (!isfinite(res.re) || !isfinite(res.im)) st |= MSGPU_S_NONFINITE;
            if (!conv) st |= MSGPU_S_NOCONV;
            P.status[it] = st;
            if (P.given_n > 0) *P.info = s.info;
            // a run given up: every item not yet taken is marked, none keeps a stale result
            if (bad && P.given_n <= 0)
                for (unsigned u = atomicAdd(P.counter, 1u); u < P.counter[1] && (int)u < P.nitem;
                     u = atomicAdd(P.counter, 1u)) {
                    P.out[2 * P.order[u]] = P.out[2 * P.order[u] + 1] = nan("");
                    P.status[P.order[u]] = MSGPU_S_TIMEOUT;
                    void_amplitudes(P, P.order[u], 0, 1);
                }
        }
        tm.sync();
        if (bad) break;
    }
}

}  // namespace msg
