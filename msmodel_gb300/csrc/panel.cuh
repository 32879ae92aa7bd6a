// panel.cuh -- panel factorisation in shared memory, by one CTA or shared by the
// CTAs of a cluster; for both engines (FP64 and double-float entries).
//
// A panel of 32 columns is a serial chain: per column a pivot search, a row
// interchange, a reciprocal and a rank-1 update.  Out of global memory each of
// those steps waits for L2 (the last update's stores have left the L1 cache),
// and one CTA alone has only its own SM's share of the FP64 pipe, 2 FMAs a clock.
// Here each CTA of the team holds R rows of the panel in shared memory (512 bytes
// a row; rank 0 the diagonal block), and one cluster barrier a column carries
// the candidates: every CTA publishes its best row's key and keeps a copy of that
// row and rank 0 of row c, the winner's copy is read through distributed shared
// memory.  Every element takes its updates in the order of the columns, as in the
// global-memory panel, so the bits are the same.
#pragma once

namespace msg {

// arithmetic of FP64 entries (zc); the double-float one is in mixed_engine.cuh
struct PanelFp64 {
    using E = zc;
    static __device__ __forceinline__ long long key(E a) { return pivot_key(a); }
    static __device__ __forceinline__ bool zero(E a) { return is_zero(a); }
    static __device__ __forceinline__ E fms(E a, E l, E u) { return zfms(a, l, u); }
    // 1 / p, or (mode 2) p itself where the multipliers are to be divided by it
    static __device__ __forceinline__ E prepare(E p, int& mode) {
        const int hb = max(__double2hiint(p.re) & 0x7fffffff, __double2hiint(p.im) & 0x7fffffff);
        mode = hb >= 0x00100000 || zabs(p) >= DBL_MIN ? 1 : 2;
        return mode == 1 ? pivot_recip(p) : p;
    }
    static __device__ __forceinline__ E scale(E l, E r, int mode) { return mode == 1 ? zmulf(l, r) : l / r; }
};

template <class E>
struct PanelShared {
    E row_p[2][NB], row_c[2][NB];  // copies of the CTA's candidate row and (rank 0) of row c, by column parity
    E urow[NB];
    E rpiv;
    long long key[2][16];          // every CTA's candidate
    int row[2][16];
    long long red_k[2][16];
    int red_p[2][16];
    int mode;                      // 0 zero pivot, 1 multiply by rpiv, 2 divide by it
};

// rows of a panel of m rows on each CTA of a team: whole warps, the diagonal block on rank 0
__device__ __forceinline__ int panel_rows(int m, int size) {
    return max(NB, ((m + size - 1) / size + 31) / 32 * 32);
}
// does a panel of m rows fit `bytes` of shared memory on each CTA?
template <class E>
__device__ __forceinline__ bool panel_fits(int m, int size, size_t bytes) {
    return sizeof(PanelShared<E>) + (size_t)panel_rows(m, size) * NB * sizeof(E) <= bytes;
}

// Factor the panel A[j0:n, j0:j0+jb) (LAPACK getf2 pivoting, first row of the
// largest |Re| + |Im|), interchanges inside the panel; buf: the same offset of
// shared memory in every CTA of the team.  info: rank 0's zero-pivot index.
// The caller's team barrier follows.
template <class Ar, int NTH, class Team>
static __device__ __noinline__ void panel_smem(typename Ar::E* A, int n, int j0, int jb, int* ipiv, void* buf, int& info,
                                               Team tm) {
    using E = typename Ar::E;
    constexpr int NW = NTH / 32;
    const unsigned FULL = 0xffffffffu;
    PanelShared<E>& ps = *reinterpret_cast<PanelShared<E>*>(buf);
    E* P = reinterpret_cast<E*>(reinterpret_cast<char*>(buf) + sizeof(PanelShared<E>));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m = n - j0, R = panel_rows(m, tm.size), r0 = tm.rank * R, rows = max(0, min(R, m - r0));
    // a warp takes 32 rows; where the rows do not fill the CTA several warps share
    // them, each with every G-th column
    const int nrb = (rows + 31) / 32, G = nrb > 0 ? max(1, NW / nrb) : 1;
    const int g = nrb > 0 && nrb < NW ? warp / nrb : 0, rb0 = nrb > 0 && nrb < NW ? warp % nrb : warp;
    for (int e = tid; e < R * jb; e += NTH) {
        const int i = e % R, t = e / R;
        if (i < rows) P[t * R + i] = A[j0 + r0 + i + (size_t)(j0 + t) * n];
    }
    __syncthreads();
    long long bk = -1;
    int bi = 0x7fffffff;  // panel row
    for (int i = tid; i < rows; i += NTH) {
        const long long k = Ar::key(P[i]);
        if (k > bk) { bk = k; bi = r0 + i; }
    }
    for (int c = 0; c < jb; ++c) {
        const int par = c & 1;
        // this CTA's candidate
        warp_pivot(bk, bi);
        if (lane == 0) { ps.red_k[par][warp] = bk; ps.red_p[par][warp] = bi; }
        __syncthreads();
        bk = ps.red_k[par][lane & (NW - 1)];
        bi = ps.red_p[par][lane & (NW - 1)];
        warp_pivot(bk, bi);
        int p = bk >= 0 ? bi : c;  // no candidate (every entry a NaN): row c
        if (tm.size > 1) {
            if (warp == 0) {
                if (bk >= 0 && lane < jb) ps.row_p[par][lane] = P[lane * R + bi - r0];
                if (tm.rank == 0 && lane < jb) ps.row_c[par][lane] = P[lane * R + c];
                if (lane < tm.size) {
                    cluster_store(&ps.key[par][tm.rank], lane, bk);
                    cluster_store(&ps.row[par][tm.rank], lane, bi);
                }
            }
            tm.sync();
            bk = lane < tm.size ? ps.key[par][lane] : -1;
            bi = lane < tm.size ? ps.row[par][lane] : 0x7fffffff;
            warp_pivot(bk, bi);
            p = bk >= 0 ? bi : c;
        }
        if (warp == 0) {
            const int po = p / R;  // the pivot row's CTA
            E u{};
            if (lane < jb) {
                if (tm.size == 1) {
                    u = P[lane * R + p];
                    ps.row_c[par][lane] = P[lane * R + c];
                } else {
                    u = bk >= 0 ? cluster_load(&ps.row_p[par][lane], po) : cluster_load(&ps.row_c[par][lane], 0);
                }
            }
            const bool nz = !__shfl_sync(FULL, (int)Ar::zero(u), c);
            if (lane < jb && nz && p != c) {
                // rows c and p exchanged; a zero column keeps its order
                if (po == tm.rank) P[lane * R + p - r0] = tm.size == 1 ? ps.row_c[par][lane] : cluster_load(&ps.row_c[par][lane], 0);
                if (tm.rank == 0) P[lane * R + c] = u;
            }
            if (lane < jb) ps.urow[lane] = u;
            if (lane == c) {
                int mode = 0;
                if (nz) ps.rpiv = Ar::prepare(u, mode);
                ps.mode = mode;
                if (tm.rank == 0) {
                    ipiv[j0 + c] = j0 + p;
                    if (!nz && info == 0) info = j0 + c + 1;
                }
            }
        }
        __syncthreads();
        const int mode = ps.mode;
        bk = -1;
        bi = 0x7fffffff;
        if (mode) {
            const E r = ps.rpiv;
            for (int i = tid; i < rows; i += NTH)
                if (r0 + i > c) P[c * R + i] = Ar::scale(P[c * R + i], r, mode);
            __syncthreads();
            if (g < G)
                for (int rb = rb0; rb < nrb; rb += NW) {
                    const int i = rb * 32 + lane;
                    if (i < rows && r0 + i > c) {
                        const E l = P[c * R + i];
                        for (int t = c + 1 + g; t < jb; t += G) {
                            const E a = Ar::fms(P[t * R + i], l, ps.urow[t]);
                            P[t * R + i] = a;
                            if (t == c + 1) {
                                const long long k = Ar::key(a);
                                if (k > bk) { bk = k; bi = r0 + i; }
                            }
                        }
                    }
                }
        } else if (c + 1 < jb) {
            for (int i = tid; i < rows; i += NTH)
                if (r0 + i > c) {
                    const long long k = Ar::key(P[(c + 1) * R + i]);
                    if (k > bk) { bk = k; bi = r0 + i; }
                }
        }
    }
    __syncthreads();
    for (int e = tid; e < R * jb; e += NTH) {
        const int i = e % R, t = e / R;
        if (i < rows) A[j0 + r0 + i + (size_t)(j0 + t) * n] = P[t * R + i];
    }
    __syncthreads();
}

}  // namespace msg
