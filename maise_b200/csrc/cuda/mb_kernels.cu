/*
 * mb_kernels.cu -- sm_100a kernels of libmaise_b200 (FP64 one-structure path).
 *
 *   k_wrap          wrap positions into the cell (JAR, src/cell.c:445-508)
 *   k_nlist_brute   all (atom, image) pairs within Rc (LIST, src/cell.c:82-185)
 *   k_cell_*        integer cell-list build (one CTA, or bin, scan, fill and
 *                   sort kernels for more than 4096 atoms) and
 *   k_nlist_cell    the same neighbour set from the 27 adjacent cells
 *   k_efs_tri       the descriptor pass of the reference bases: per atom the
 *                   triplet list, descriptors, MLP and reverse pass below with
 *                   every factor of a triplet evaluated in registers
 *   k_efs           one CTA per central atom, any basis: G2/G4 descriptors
 *                   (src/nprs.c:500-566), MLP forward and dE/dG
 *                   (src/nmlp.c:367-431), then the reverse pass that turns
 *                   dE_i/dG_i into forces on i and its neighbours and the
 *                   virial (src/nprs.c:567-770 contracted as in
 *                   src/nmlp.c:433-479) without materialising dG/dx
 *   k_finalize      energy and virial reductions in fixed order, noise
 *                   zeroing and enthalpy (src/cmod.c:153-191)
 *   k_nvt_*         NVT thermostat and integrator (src/cmod.c:403-453)
 *
 * The wrap and the neighbour test use explicitly rounded operations
 * (__dadd_rn/__dmul_rn, never contracted into FMAs) in the reference's
 * operation order, so the selected neighbour set is the reference's.
 */
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include "../mb_internal.h"

#define FULL 0xffffffffu

namespace {

__device__ __forceinline__ double xadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double xsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double xmul(double a, double b) { return __dmul_rn(a, b); }

/* ------------------------------------------------------------------ */
/* wrap                                                                */
/* ------------------------------------------------------------------ */

/* JAR on atom i's position: Cartesian -> fractional, into [0, 1), back */
__device__ __forceinline__ void wrap_atom(int i, double *__restrict__ X, const mb_cell &c, int *status) {
    double x[3];
    for (int q = 0; q < 3; q++) {
        double s = 0.0;
        for (int j = 0; j < 3; j++) s = xadd(s, xmul(X[3 * i + j], c.R[3 * q + j]));
        x[q] = s;
    }
    for (int q = 0; q < 3; q++) {
        int it = 0;
        while (x[q] < 0.0 && it < 4096) { x[q] = xadd(x[q], 1.0); it++; }
        while (x[q] >= 1.0 && it < 4096) { x[q] = xsub(x[q], 1.0); it++; }
        if (!(x[q] >= 0.0 && x[q] < 1.0)) atomicOr(status, MB_ST_WRAP);
    }
    for (int q = 0; q < 3; q++) {
        double s = 0.0;
        for (int j = 0; j < 3; j++) s = xadd(s, xmul(x[j], c.L[3 * j + q]));
        X[3 * i + q] = s;
    }
}

/* JAR on every atom; F (if set) is cleared for the pass that follows */
__global__ void k_wrap(int N, double *__restrict__ X, mb_cell c, int *status, double *__restrict__ F) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    wrap_atom(i, X, c, status);
    if (F) F[3 * i] = F[3 * i + 1] = F[3 * i + 2] = 0.0;
}

/* Start of a pass on host arrays: positions and species read from pinned host
 * memory, JAR (periodic cells), forces cleared.  One launch in the place of two
 * copies, a clear and k_wrap, which for a small structure each cost more than
 * they move (with the results stored by k_finalize, and the list kernel below,
 * a 32-atom E/F/S call went from 120 to 77 us). */
__global__ void k_intake(int N, const double *__restrict__ hx, mb_cell c, const int *__restrict__ hspc,
                         double *__restrict__ X, int *__restrict__ spc, int *status, double *__restrict__ F) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    X[3 * i] = hx[3 * i];
    X[3 * i + 1] = hx[3 * i + 1];
    X[3 * i + 2] = hx[3 * i + 2];
    spc[i] = hspc[i];
    if (c.ND > 0) wrap_atom(i, X, c, status);
    if (F) F[3 * i] = F[3 * i + 1] = F[3 * i + 2] = 0.0;
}

/* ------------------------------------------------------------------ */
/* neighbour list                                                      */
/* ------------------------------------------------------------------ */

/* displacement of atom j's image (i0,i1,i2) from atom i and its squared
 * length, formed exactly as src/cell.c:115-121 */
__device__ __forceinline__ double image_disp(const mb_cell &c, const double *xi, const double *xj, int i0, int i1,
                                             int i2, double *d) {
    double r = 0.0;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        double x = 0.0;
        x = xadd(x, xmul((double)i0, c.L[q]));
        x = xadd(x, xmul((double)i1, c.L[3 + q]));
        x = xadd(x, xmul((double)i2, c.L[6 + q]));
        x = xadd(x, xsub(xj[q], xi[q]));
        d[q] = x;
        r = xadd(r, xmul(x, x));
    }
    return r;
}

/* append the accepted candidates of a round to atom i's list, in lane order */
__device__ __forceinline__ void list_append(bool ok, int j, const double *d, double r2, size_t row, int cap, int lane,
                                            int &count, int *__restrict__ nj, double4 *__restrict__ nd) {
    const unsigned m = __ballot_sync(FULL, ok);
    const int pos = count + __popc(m & ((1u << lane) - 1u));
    if (ok && pos < cap) {
        nj[row + pos] = j;
        nd[row + pos] = make_double4(d[0], d[1], d[2], sqrt(r2));
    }
    count += __popc(m);
}

/* One warp per atom; candidates in the reference's order (j, then images).
 * Cells with 16 to 128 images: the lanes hold the images' shifts (formed in
 * image_disp's order, so the sums round as there) and walk the atoms j
 * together.  Otherwise (clusters above all) the lanes walk the flat candidate
 * index; with that for every cell, its two divisions a candidate took 16 us
 * for 32 atoms of 27 images and 22 us for 47 of 125 (now 8 and 11). */
#define BRUTE_IMG 4
__global__ void k_nlist_brute(int N, int NM, int cap, const double *__restrict__ X, mb_cell c, double rc2,
                              int *__restrict__ nn, int *__restrict__ nj, double4 *__restrict__ nd, int *status) {
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= N) return;
    int i = warp;
    const size_t row = (size_t)i * cap;
    int w0 = 2 * c.Nq[0] + 1, w1 = 2 * c.Nq[1] + 1, w2 = 2 * c.Nq[2] + 1;
    int nimg = w0 * w1 * w2;
    double xi[3] = {X[3 * i], X[3 * i + 1], X[3 * i + 2]};
    int count = 0;
    if (nimg >= 16 && nimg <= 32 * BRUTE_IMG) {
        double sh[BRUTE_IMG][3];
        const int zero = (c.Nq[0] * w1 + c.Nq[1]) * w2 + c.Nq[2]; /* the unshifted image */
#pragma unroll
        for (int t = 0; t < BRUTE_IMG; t++) {
            const int im = 32 * t + lane, i2 = im % w2 - c.Nq[2], u = im / w2, i1 = u % w1 - c.Nq[1], i0 = u / w1 - c.Nq[0];
#pragma unroll
            for (int q = 0; q < 3; q++) {
                double x = 0.0;
                x = xadd(x, xmul((double)i0, c.L[q]));
                x = xadd(x, xmul((double)i1, c.L[3 + q]));
                sh[t][q] = xadd(x, xmul((double)i2, c.L[6 + q]));
            }
        }
        /* four rounds' distances side by side (their FP64 chains overlap), then
         * four appends: images 0-31 of atoms j..j+3, or all images of atom j */
        const int T = nimg > 32 ? BRUTE_IMG : 1;
        for (int j0 = 0; j0 < N; j0 += BRUTE_IMG / T) {
            double d[BRUTE_IMG][3], r2[BRUTE_IMG];
            bool ok[BRUTE_IMG];
            int jj[BRUTE_IMG];
#pragma unroll
            for (int u = 0; u < BRUTE_IMG; u++) {
                const int j = T == 1 ? min(j0 + u, N - 1) : j0, im = (T == 1 ? 0 : 32 * u) + lane;
                jj[u] = j;
                r2[u] = 0.0;
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    d[u][q] = xadd(T == 1 ? sh[0][q] : sh[u][q], xsub(X[3 * j + q], xi[q]));
                    r2[u] = xadd(r2[u], xmul(d[u][q], d[u][q]));
                }
                ok[u] = im < nimg && r2[u] < rc2 && !(j == i && im == zero) && (T > 1 || j0 + u < N);
            }
#pragma unroll
            for (int u = 0; u < BRUTE_IMG; u++) list_append(ok[u], jj[u], d[u], r2[u], row, cap, lane, count, nj, nd);
        }
    } else {
        long long total = (long long)N * nimg;
        for (long long base = 0; base < total; base += 32) {
            long long cidx = base + lane;
            bool ok = false;
            int j = 0, i0 = 0, i1 = 0, i2 = 0;
            double d[3] = {0, 0, 0}, r2 = 0.0;
            if (cidx < total) {
                if (nimg == 1) {
                    j = (int)cidx;
                } else {
                    j = (int)(cidx / nimg);
                    int im = (int)(cidx % nimg);
                    i2 = im % w2 - c.Nq[2];
                    int t = im / w2;
                    i1 = t % w1 - c.Nq[1];
                    i0 = t / w1 - c.Nq[0];
                }
                if (!(j == i && i0 == 0 && i1 == 0 && i2 == 0)) {
                    double xj[3] = {X[3 * j], X[3 * j + 1], X[3 * j + 2]};
                    r2 = image_disp(c, xi, xj, i0, i1, i2, d);
                    ok = r2 < rc2;
                }
            }
            list_append(ok, j, d, r2, row, cap, lane, count, nj, nd);
        }
    }
    if (lane == 0) {
        nn[i] = count < cap ? count : cap;
        if (count >= NM) atomicOr(status, MB_ST_NBR_OVERFLOW);
        if (count > cap) atomicOr(status, MB_ST_CAP_OVERFLOW);
        atomicMax(&status[1], count);
    }
}

__device__ __forceinline__ int cell_index(const mb_cell &c, const double *x, int *cq) {
    for (int q = 0; q < 3; q++) {
        double f = x[0] * c.R[3 * q] + x[1] * c.R[3 * q + 1] + x[2] * c.R[3 * q + 2];
        int k = (int)floor(f * c.M[q]);
        k = k < 0 ? 0 : (k >= c.M[q] ? c.M[q] - 1 : k);
        cq[q] = k;
    }
    return (cq[0] * c.M[1] + cq[1]) * c.M[2] + cq[2];
}

__global__ void k_cell_bin(int N, const double *__restrict__ X, mb_cell c, int *cell_of, int *cnt) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    int cq[3];
    int k = cell_index(c, X + 3 * i, cq);
    cell_of[i] = k;
    atomicAdd(&cnt[k], 1);
}

/* exclusive scan of the cell counts by one CTA of 1024 threads; start[ncell] = N */
__global__ void k_cell_scan(int ncell, const int *cnt, int *start) {
    __shared__ int wsum[32];
    const int t = threadIdx.x, nt = blockDim.x, lane = t & 31, w = t >> 5;
    const int per = (ncell + nt - 1) / nt, lo = t * per, hi = min(lo + per, ncell);
    int s = 0;
    for (int k = lo; k < hi; k++) s += cnt[k];
    int x = s; /* inclusive scan over the warp */
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
        int v = lane < (nt >> 5) ? wsum[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, v, o);
            if (lane >= o) v += y;
        }
        wsum[lane] = v;
    }
    __syncthreads();
    int e = x - s + (w > 0 ? wsum[w - 1] : 0);
    for (int k = lo; k < hi; k++) {
        start[k] = e;
        e += cnt[k];
    }
    if (t == nt - 1) start[ncell] = e;
}

__global__ void k_cell_fill(int N, const int *cell_of, const int *start, int *cursor, int *atoms) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    int k = cell_of[i];
    int pos = atomicAdd(&cursor[k], 1);
    atoms[start[k] + pos] = i;
}

/* order each cell's atoms by index so the neighbour order is deterministic:
 * one warp per cell, each atom placed at its rank (the number of smaller
 * indices in the cell; indices are distinct); cells of more than
 * 32 * CELL_SORT_PER_LANE atoms are sorted by one lane */
#define CELL_SORT_PER_LANE 8
__global__ void k_cell_sort(int ncell, const int *start, int *atoms) {
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (k >= ncell) return;
    const int lo = start[k], n = start[k + 1] - lo;
    if (n <= 32 * CELL_SORT_PER_LANE) {
        int v[CELL_SORT_PER_LANE], r[CELL_SORT_PER_LANE];
#pragma unroll
        for (int q = 0; q < CELL_SORT_PER_LANE; q++) {
            const int e = q * 32 + lane;
            v[q] = e < n ? atoms[lo + e] : 0x7fffffff;
            r[q] = 0;
        }
        const int rounds = (n + 31) >> 5;
        for (int f = 0; f < n; f++) {
            const int w = atoms[lo + f];
#pragma unroll
            for (int q = 0; q < CELL_SORT_PER_LANE; q++)
                if (q < rounds) r[q] += w < v[q];
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < CELL_SORT_PER_LANE; q++)
            if (q * 32 + lane < n) atoms[lo + r[q]] = v[q];
    } else if (lane == 0) {
        for (int a = lo + 1; a < lo + n; a++) {
            int v = atoms[a], b = a - 1;
            while (b >= lo && atoms[b] > v) {
                atoms[b + 1] = atoms[b];
                b--;
            }
            atoms[b + 1] = v;
        }
    }
}

/* The whole build in one CTA: bins and counts (shared atomics), their scan, the
 * atoms by cell, and each atom to its rank in its cell (the number of smaller
 * indices, so the order does not depend on the atomics).  Up to
 * CELL_BUILD_MAX atoms and cells the four kernels and two clears above are
 * launches and gaps, not work: 19 us for 487 atoms and 21 for 4000, against 3.4
 * and 8.6 here (an E/F/S call of 487 atoms 130 -> 121 us).  The time grows with
 * the atoms a thread holds, and beyond 4096 those and their cells no longer fit
 * 4 registers and the 48 KB of shared memory. */
#define CELL_BUILD_MAX 4096
__global__ void __launch_bounds__(1024) k_cell_build(int N, const double *__restrict__ X, mb_cell c, int ncell,
                                                     int *__restrict__ cell_of, int *__restrict__ start,
                                                     int *__restrict__ atoms) {
    extern __shared__ int cell_sm[];
    __shared__ int wsum[32];
    int *cnt = cell_sm, *lst = cell_sm + ncell; /* [ncell], [N] */
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    constexpr int PER = CELL_BUILD_MAX / 1024;
    int mine[PER];
    for (int k = t; k < ncell; k += 1024) cnt[k] = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < PER; q++) {
        const int i = q * 1024 + t;
        if (i < N) {
            int cq[3];
            mine[q] = cell_index(c, X + 3 * i, cq);
            cell_of[i] = mine[q];
            atomicAdd(&cnt[mine[q]], 1);
        }
    }
    __syncthreads();
    /* exclusive scan, a run of cells a thread; cnt[k] becomes cell k's cursor */
    const int per = (ncell + 1023) >> 10, lo = min(t * per, ncell), hi = min(lo + per, ncell);
    int s = 0;
    for (int k = lo; k < hi; k++) s += cnt[k];
    int x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
        int v = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, v, o);
            if (lane >= o) v += y;
        }
        wsum[lane] = v;
    }
    __syncthreads();
    int e = x - s + (w > 0 ? wsum[w - 1] : 0);
    for (int k = lo; k < hi; k++) {
        const int n = cnt[k];
        start[k] = cnt[k] = e;
        e += n;
    }
    if (t == 0) start[ncell] = N;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < PER; q++)
        if (q * 1024 + t < N) lst[atomicAdd(&cnt[mine[q]], 1)] = q * 1024 + t;
    __syncthreads();
    /* cnt[k] is now the end of cell k */
#pragma unroll
    for (int q = 0; q < PER; q++) {
        const int i = q * 1024 + t;
        if (i < N) {
            const int from = mine[q] ? cnt[mine[q] - 1] : 0, to = cnt[mine[q]];
            int r = from;
#pragma unroll 4
            for (int p = from; p < to; p++) r += lst[p] < i;
            atoms[r] = i;
        }
    }
}

/* One warp per atom over the 27 adjacent cells.  Periodic directions have
 * at least 3 bins no thinner than Rc, so every image within Rc lies in an
 * adjacent bin and each (atom, image) pair is visited once; the exact test
 * then selects the reference's set.  The 27 cells' atom ranges are laid end
 * to end (cell order a, b, e; atoms in index order within a cell) and
 * walked 32 candidates per round, every lane busy. */
__global__ void k_nlist_cell(int N, int NM, int cap, const double *__restrict__ X, mb_cell c, double rc2,
                             const int *__restrict__ cell_of, const int *__restrict__ start,
                             const int *__restrict__ atoms, int *__restrict__ nn, int *__restrict__ nj,
                             double4 *__restrict__ nd, int *status) {
    __shared__ int s_off[4][32], s_lo[4][32], s_img[4][32];
    const int w = (threadIdx.x >> 5) & 3;
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= N) return;
    int i = warp;
    double xi[3] = {X[3 * i], X[3 * i + 1], X[3 * i + 2]};
    int ci = cell_of[i];
    int cq[3] = {ci / (c.M[1] * c.M[2]), (ci / c.M[2]) % c.M[1], ci % c.M[2]};
    /* lane k < 27 describes adjacent cell k = 9 (a+1) + 3 (b+1) + (e+1) */
    int lo = 0, cnt = 0, pimg = 0;
    if (lane < 27) {
        const int dd[3] = {lane / 9 - 1, (lane / 3) % 3 - 1, lane % 3 - 1};
        int cc[3], img[3];
        bool skip = false;
        for (int q = 0; q < 3; q++) {
            int k = cq[q] + dd[q];
            img[q] = 0;
            if (q < c.ND) {
                if (k < 0) { k += c.M[q]; img[q] = -1; }
                else if (k >= c.M[q]) { k -= c.M[q]; img[q] = 1; }
            } else if (k < 0 || k >= c.M[q]) {
                skip = true;
            }
            cc[q] = k;
        }
        if (!skip) {
            const int cell = (cc[0] * c.M[1] + cc[1]) * c.M[2] + cc[2];
            lo = start[cell];
            cnt = start[cell + 1] - lo;
        }
        pimg = (img[0] + 1) * 9 + (img[1] + 1) * 3 + (img[2] + 1);
    }
    int off = cnt; /* inclusive scan of the cell sizes */
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, off, o);
        if (lane >= o) off += y;
    }
    const int total = __shfl_sync(FULL, off, 31);
    s_off[w][lane] = off - cnt; /* exclusive */
    s_lo[w][lane] = lo;
    s_img[w][lane] = pimg;
    __syncwarp();
    int count = 0;
    for (int base = 0; base < total; base += 32) {
        const int t = base + lane;
        bool ok = false;
        int j = 0, img[3] = {0, 0, 0};
        double d[3] = {0, 0, 0}, r2 = 0.0;
        if (t < total) {
            /* the last of the 27 cells whose range starts at or before t */
            int k = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1)
                if (k + step < 27 && s_off[w][k + step] <= t) k += step;
            j = atoms[s_lo[w][k] + (t - s_off[w][k])];
            const int pi = s_img[w][k];
            img[0] = pi / 9 - 1;
            img[1] = (pi / 3) % 3 - 1;
            img[2] = pi % 3 - 1;
            if (!(j == i && img[0] == 0 && img[1] == 0 && img[2] == 0)) {
                double xj[3] = {X[3 * j], X[3 * j + 1], X[3 * j + 2]};
                r2 = image_disp(c, xi, xj, img[0], img[1], img[2], d);
                ok = r2 < rc2;
            }
        }
        unsigned m = __ballot_sync(FULL, ok);
        int pos = count + __popc(m & ((1u << lane) - 1u));
        if (ok && pos < cap) {
            nj[(size_t)i * cap + pos] = j;
            nd[(size_t)i * cap + pos] = make_double4(d[0], d[1], d[2], sqrt(r2));
        }
        count += __popc(m);
    }
    if (lane == 0) {
        nn[i] = count < cap ? count : cap;
        if (count >= NM) atomicOr(status, MB_ST_NBR_OVERFLOW);
        if (count > cap) atomicOr(status, MB_ST_CAP_OVERFLOW);
        atomicMax(&status[1], count);
    }
}

/* ------------------------------------------------------------------ */
/* descriptor / MLP / force kernel                                     */
/* ------------------------------------------------------------------ */

__device__ __forceinline__ double fcut(double rc, double r) { return r > rc ? 0.0 : 0.5 * (cospi(r / rc) + 1.0); }

__device__ __forceinline__ void fcut_d(double rc, double r, double &f, double &df) {
    if (r > rc) {
        f = 0.0;
        df = 0.0;
        return;
    }
    double s, co;
    sincospi(r / rc, &s, &co);
    f = 0.5 * (co + 1.0);
    df = -0.5 * CUDART_PI / rc * s;
}

/* (1 + lambda c)^zeta * 2^(1-zeta) for every (zeta, lambda), and optionally
 * the derivative in c; integer zeta by repeated squaring.  NZ and NLAM are
 * upper bounds (exact for the specialised kernels); zl = z*NLAM + l. */
/* PZ = false leaves out the normalisation powz[z] = 2^(1 - zeta) (the
 * caller folds it into the per-block grid instead: for the reference
 * bases it is a power of two, so the results are unchanged bit for bit) */
template <int NZ, int NLAM, bool PZ = true>
__device__ __forceinline__ void angular(const mb_params &P, double c, double *lz, double *lzp) {
    auto pz = [&](int z) { return PZ ? P.powz[z] : 1.0; };
    if (NZ == 4 && P.zeta_std) {
        /* zeta = 1, 2, 4, 16 (the reference bases): powers by squaring */
#pragma unroll
        for (int l = 0; l < NLAM; l++) {
            if (l >= P.nlam) break;
            const double lam = P.lam[l], b1 = 1.0 + lam * c, b2 = b1 * b1, b4 = b2 * b2, b8 = b4 * b4;
            if constexpr (PZ) {
                lz[0 * NLAM + l] = P.powz[0] * b1;
                lz[1 * NLAM + l] = P.powz[1] * b2;
                lz[2 * NLAM + l] = P.powz[2] * b4;
                lz[3 * NLAM + l] = P.powz[3] * (b8 * b8);
            } else {
                lz[0 * NLAM + l] = b1;
                lz[1 * NLAM + l] = b2;
                lz[2 * NLAM + l] = b4;
                lz[3 * NLAM + l] = b8 * b8;
            }
            if (lzp) {
                if constexpr (PZ) {
                    lzp[0 * NLAM + l] = P.powz[0] * lam;
                    lzp[1 * NLAM + l] = P.powz[1] * 2.0 * lam * b1;
                    lzp[2 * NLAM + l] = P.powz[2] * 4.0 * lam * (b2 * b1);
                    lzp[3 * NLAM + l] = P.powz[3] * 16.0 * lam * (b8 * b4 * b2 * b1);
                } else {
                    lzp[0 * NLAM + l] = lam;
                    lzp[1 * NLAM + l] = 2.0 * lam * b1;
                    lzp[2 * NLAM + l] = 4.0 * lam * (b2 * b1);
                    lzp[3 * NLAM + l] = 16.0 * lam * (b8 * b4 * b2 * b1);
                }
            }
        }
        return;
    }
#pragma unroll
    for (int l = 0; l < NLAM; l++) {
        if (l >= P.nlam) break;
        double lam = P.lam[l];
        double base = 1.0 + lam * c;
        if (P.zeta_int) {
            double sq[7];
            sq[0] = base;
#pragma unroll
            for (int k = 1; k < 7; k++) sq[k] = sq[k - 1] * sq[k - 1];
#pragma unroll
            for (int z = 0; z < NZ; z++) {
                if (z >= P.nz) break;
                int zb = P.zbits[z], mb = P.zm1bits[z];
                double pw = 1.0, pm = 1.0;
#pragma unroll
                for (int k = 0; k < 7; k++) {
                    if (zb & (1 << k)) pw *= sq[k];
                    if (mb & (1 << k)) pm *= sq[k];
                }
                lz[z * NLAM + l] = pz(z) * pw;
                if (lzp) lzp[z * NLAM + l] = pz(z) * P.zeta[z] * lam * pm;
            }
        } else {
#pragma unroll
            for (int z = 0; z < NZ; z++) {
                if (z >= P.nz) break;
                lz[z * NLAM + l] = pz(z) * pow(base, P.zeta[z]);
                if (lzp) lzp[z * NLAM + l] = pz(z) * P.zeta[z] * lam * pow(base, P.zeta[z] - 1.0);
            }
        }
    }
}

struct EfsArgs {
    int N, cap, mode;
    double urep;
    const int *nn, *nj;
    const double4 *nd;
    const int *spc;
    const mb_params *params;
    const double *weights;
    double *EA, *EU, *G, *F, *vir;
    unsigned long long *counters; /* [0] pairs, [1] accepted forward triplets */
    size_t smem_group;            /* shared-memory bytes of one atom group */
    int tl_cap;                   /* triplet-list entries of one atom group */
};

/* shared-memory carve-up of one atom group of k_efs */
struct EfsSmem {
    int *j, *sp;
    double4 *d;
    double *ir, *fa, *fb, *P, *Fnb, *G, *grid, *red, *tmp, *h;
    double *stage; /* per warp: 32 triplets x EFS_STG doubles (tensor-core forward) */
    unsigned *tl;  /* accepted (j,k) pairs: per-warp regions of tlw entries */
    int *blk;      /* [block][warp][2] ranges of each warp's region per species block */
    int *seg;      /* [0..3] counts, [4..7] offsets */
};

#define MB_MAX_BLOCKS 6 /* species blocks (a<=b) for 3 species */

__host__ __device__ inline size_t align8(size_t x) { return (x + 7) & ~(size_t)7; }
__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }
/* row stride of the per-neighbour exponential factors: even, so that rows
 * start on 16 bytes (the neighbour capacity is a multiple of 8) */
__host__ __device__ constexpr int nep(int ne) { return (ne + 1) & ~1; }

#define EFS_STG 16 /* staging row: 8 exponential + 8 angular values */

/* Staging slot of value q (0-7 exponential, 8-15 angular) of a warp's
 * triplet t (0-31): rows of 16 doubles whose columns are rotated by
 * 4 (t & 3) + ((t >> 2) & 3).  An 8-byte shared access is served a
 * half-warp at a time; the writes (one q, 16 consecutive t) and the
 * mma operand reads (4 consecutive t x 4 consecutive q) then both touch
 * 16 distinct banks.  (A padded row of 17 left the operand reads 4-way
 * conflicted.) */
__device__ __forceinline__ int stg_slot(int t, int q) { return t * EFS_STG + ((q + 4 * (t & 3) + ((t >> 2) & 3)) & 15); }

/* Sizes of the regions that share one block of memory: the forward
 * staging rows (tensor-core forward, live only while the forward triplets
 * run) and Fnb + grid + red + h (block reductions, MLP and reverse pass,
 * all after it). */
__host__ __device__ inline size_t efs_union_bytes(int cap, int nzl_cells, int warps, int stage) {
    const size_t st = stage ? sizeof(double) * warps * 32 * EFS_STG : 0;
    const size_t rest = sizeof(double) * (cap * 3 + nzl_cells + warps * 64 + 4 * MB_MAXH);
    return align16(st > rest ? st : rest);
}

__host__ __device__ inline size_t efs_smem_bytes(int cap, int D, int ne, int ng2, int nzl_cells, int warps, int tl,
                                                 int stage) {
    size_t b = 0;
    b += efs_union_bytes(cap, nzl_cells, warps, stage); /* stage | Fnb, grid, red, h */
    b += align8(sizeof(int) * cap) * 2;           /* j, sp */
    b += sizeof(double4) * cap;                   /* d */
    b += sizeof(double) * cap * 3;                /* ir, fa, fb */
    b += sizeof(double) * cap * nep(ne);          /* P */
    b += align16(sizeof(double) * D);             /* G */
    /* tmp (G2 terms) and tl (triplet list) share one region: tmp is dead
     * before the first list entry is written */
    const size_t tmp_b = sizeof(double) * cap * (ng2 > 1 ? ng2 : 1), tl_b = align8(sizeof(unsigned) * tl);
    b += tmp_b > tl_b ? tmp_b : tl_b; /* tmp | tl */
    b += align8(sizeof(int) * MB_MAX_BLOCKS * warps * 2);
    b += sizeof(int) * 8;
    return b;
}

__device__ inline EfsSmem efs_carve(char *base, int cap, int D, int ne, int ng2, int nzl_cells, int warps, int tl,
                                   int stage) {
    /* one atom group's region; `warps` = warps per atom */
    EfsSmem s;
    char *p = base;
    s.stage = (double *)p;
    s.Fnb = (double *)p;
    s.grid = s.Fnb + cap * 3;
    s.red = s.grid + nzl_cells;
    s.h = s.red + warps * 64;
    p += efs_union_bytes(cap, nzl_cells, warps, stage);
    s.d = (double4 *)p; p += sizeof(double4) * cap;
    s.ir = (double *)p; p += sizeof(double) * cap;
    s.fa = (double *)p; p += sizeof(double) * cap;
    s.fb = (double *)p; p += sizeof(double) * cap;
    s.P = (double *)p; p += sizeof(double) * cap * nep(ne);
    s.G = (double *)p; p += align16(sizeof(double) * D);
    {
        const size_t tmp_b = sizeof(double) * cap * (ng2 > 1 ? ng2 : 1), tl_b = align8(sizeof(unsigned) * tl);
        s.tmp = (double *)p;
        s.tl = (unsigned *)p;
        p += tmp_b > tl_b ? tmp_b : tl_b;
    }
    s.j = (int *)p; p += align8(sizeof(int) * cap);
    s.sp = (int *)p; p += align8(sizeof(int) * cap);
    s.blk = (int *)p; p += align8(sizeof(int) * MB_MAX_BLOCKS * warps * 2);
    s.seg = (int *)p;
    return s;
}

/* Sum of 64 per-lane values across a warp: afterwards lane l holds the
 * sums of values 2l and 2l+1 (recursive halving). */
__device__ __forceinline__ void warp_reduce64(double *v, int lane) {
#pragma unroll
    for (int step = 0; step < 5; step++) {
        const int off = 16 >> step, half = 32 >> step;
        const bool upper = (lane & off) != 0;
#pragma unroll
        for (int k = 0; k < half; k++) {
            double send = upper ? v[k] : v[k + half];
            double keep = upper ? v[k + half] : v[k];
            v[k] = keep + __shfl_xor_sync(FULL, send, off);
        }
    }
}

/* Sum of 16 per-lane values across a warp: lanes l and l ^ 1 end with the
 * total of value l >> 1 (four halving steps and one exchange). */
__device__ __forceinline__ double warp_reduce16(double *v, int lane) {
#pragma unroll
    for (int step = 0; step < 4; step++) {
        const int off = 16 >> step, half = 8 >> step;
        const bool upper = (lane & off) != 0;
#pragma unroll
        for (int k = 0; k < half; k++) {
            const double send = upper ? v[k] : v[k + half];
            const double keep = upper ? v[k + half] : v[k];
            v[k] = keep + __shfl_xor_sync(FULL, send, off);
        }
    }
    return v[0] + __shfl_xor_sync(FULL, v[0], 1);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

template <int WPA>
__device__ __forceinline__ void group_sync() {
    if (WPA == 1)
        __syncwarp();
    else
        __syncthreads();
}

/* Reduction of a 64-cell accumulator grid over the atom's group into
 * s.red[0..63] (warp 0 adds the warps' partial sums in a fixed order). */
template <int WPA, class Smem>
__device__ __forceinline__ void group_reduce64(double *v, Smem &s, int gwarp, int lane) {
    warp_reduce64(v, lane);
    if (WPA == 1) {
        s.red[2 * lane] = v[0];
        s.red[2 * lane + 1] = v[1];
        __syncwarp();
        return;
    }
    s.red[gwarp * 64 + 2 * lane] = v[0];
    s.red[gwarp * 64 + 2 * lane + 1] = v[1];
    __syncthreads();
    if (gwarp == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < WPA; w++) {
            a += s.red[w * 64 + 2 * lane];
            b += s.red[w * 64 + 2 * lane + 1];
        }
        __syncwarp();
        s.red[2 * lane] = a;
        s.red[2 * lane + 1] = b;
    }
    __syncthreads();
}

/* As group_reduce64 for values already summed over the warp (lane l holds
 * cells 2l and 2l+1, the layout of a tensor-core accumulator fragment). */
template <int WPA, class Smem>
__device__ __forceinline__ void group_store64(double v0, double v1, Smem &s, int gwarp, int lane) {
    if (WPA == 1) {
        s.red[2 * lane] = v0;
        s.red[2 * lane + 1] = v1;
        __syncwarp();
        return;
    }
    s.red[gwarp * 64 + 2 * lane] = v0;
    s.red[gwarp * 64 + 2 * lane + 1] = v1;
    __syncthreads();
    if (gwarp == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < WPA; w++) {
            a += s.red[w * 64 + 2 * lane];
            b += s.red[w * 64 + 2 * lane + 1];
        }
        __syncwarp();
        s.red[2 * lane] = a;
        s.red[2 * lane + 1] = b;
    }
    __syncthreads();
}

/* D(8x8) += A(8x4) B(4x8) in FP64 on the tensor cores (mma.sync m8n8k4):
 * lane l holds A[l/4][l%4], B[l%4][l/4] and D[l/4][2(l%4) + {0, 1}]. */
__device__ __forceinline__ void dmma884(double &c0, double &c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

/* Candidates of block (a, b): the na x nb square for a != b; for a == b
 * only the strict upper triangle (col > row), enumerated directly up to 256
 * neighbours of the species (the square with the lower half skipped above) */
__device__ __forceinline__ bool block_tri(const EfsSmem &s, int a, int b) { return a == b && s.seg[a] <= 256; }
__device__ __forceinline__ int block_candidates(const EfsSmem &s, int a, int b) {
    const int na = s.seg[a], nb = s.seg[b];
    return block_tri(s, a, b) ? na * (na - 1) / 2 : na * nb;
}

/* Append the accepted candidates (j, k) of block (a, b) to this warp's
 * list region in row-major order, 32 candidates per round with every lane
 * busy, the warps of an atom taking every WPA-th round.  Square: row =
 * (c + 0.5) / nb in FP32 is exact (the fraction stays >= 0.5 / nb away from
 * an integer).  Triangle: row r starts at r (2 na - r - 1) / 2, inverted
 * with one FP32 square root and corrected by one row either way (exact for
 * na <= 256 under +-2 ulp of sqrt error).  Returns the next candidate
 * index; stops early when the region is full. */
template <int WPA, class Accept>
__device__ __forceinline__ int fill_chunks(const EfsSmem &s, int a, int b, int c, int &pos, int hi, int lane,
                                           Accept accept) {
    const int na = s.seg[a], nb = s.seg[b], oa = s.seg[4 + a], ob = s.seg[4 + b];
    const bool tri = block_tri(s, a, b);
    const int C = block_candidates(s, a, b);
    const float inv_nb = nb > 0 ? 1.0f / (float)nb : 0.0f, tb = (float)(2 * na - 1);
    for (; c < C && pos + 32 <= hi; c += 32 * WPA) {
        const int cc = c + lane;
        bool ok = false;
        int jj = 0, kk = 0;
        if (cc < C) {
            int r, col;
            if (tri) {
                r = __float2int_rz(0.5f * (tb - sqrtf(tb * tb - 8.0f * (float)cc)));
                if ((r + 1) * (2 * na - r - 2) / 2 <= cc) r++;
                else if (r * (2 * na - r - 1) / 2 > cc) r--;
                r = min(max(r, 0), na - 2);
                col = min(max(cc - r * (2 * na - r - 1) / 2 + r + 1, r + 1), na - 1);
            } else {
                r = __float2int_rz(((float)cc + 0.5f) * inv_nb);
                col = cc - r * nb;
            }
            jj = oa + r;
            kk = ob + col;
            ok = (a != b || col > r) && accept(jj, kk);
        }
        const unsigned m = __ballot_sync(FULL, ok);
        if (ok) s.tl[pos + __popc(m & ((1u << lane) - 1u))] = (unsigned)jj | ((unsigned)kk << 16);
        pos += __popc(m);
    }
    __syncwarp();
    return c;
}

/* body(jj, kk) over list entries [from, to), one entry per lane */
template <class Body>
__device__ __forceinline__ void run_list(const EfsSmem &s, int from, int to, int lane, Body body) {
    for (int t = from + lane; t < to; t += 32) {
        const unsigned pk = s.tl[t];
        body((int)(pk & 0xffffu), (int)(pk >> 16));
    }
}

/* body(jj, kk) -> the entry's force on neighbour j, over list entries
 * [from, to): each lane takes a contiguous run of K entries (K odd, so that
 * the lanes' reads of the list fall in distinct banks).  The list runs row
 * by row, so a lane's entries mostly share j: their j-side forces are summed
 * in registers and added to Fnb once per change of j.  The body must not
 * exchange values across lanes (lanes leave the loop at different times). */
template <class Body>
__device__ __forceinline__ void run_list_runs(const EfsSmem &s, int from, int to, int lane, Body body) {
    int K = (to - from + 31) >> 5;
    if (K > 0) K |= 1;
    const int t0 = from + lane * K;
    int cj = -1;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    for (int step = 0; step < K; step++) {
        const int t = t0 + step;
        if (t >= to) break;
        const unsigned pk = s.tl[t];
        const int jj = (int)(pk & 0xffffu), kk = (int)(pk >> 16);
        if (jj != cj) {
            if (cj >= 0) {
                atomicAdd(&s.Fnb[3 * cj], -sx);
                atomicAdd(&s.Fnb[3 * cj + 1], -sy);
                atomicAdd(&s.Fnb[3 * cj + 2], -sz);
            }
            cj = jj;
            sx = sy = sz = 0.0;
        }
        const double3 g = body(jj, kk);
        sx += g.x;
        sy += g.y;
        sz += g.z;
    }
    if (cj >= 0) {
        atomicAdd(&s.Fnb[3 * cj], -sx);
        atomicAdd(&s.Fnb[3 * cj + 1], -sy);
        atomicAdd(&s.Fnb[3 * cj + 2], -sz);
    }
}

/* body(jj, kk, valid) with the whole warp converged on every round (for
 * bodies that exchange values across lanes or issue warp-wide tensor-core
 * instructions, which need all 32 lanes at one call site); lanes past the
 * end get valid = false and jj = -1 - lane, so equal jj values stay
 * adjacent */
template <class Body>
__device__ __forceinline__ void run_list_all(const EfsSmem &s, int from, int to, int lane, Body body) {
    for (int base = from; base < to; base += 32) {
        const int t = base + lane;
        const bool valid = t < to;
        const unsigned pk = valid ? s.tl[t] : 0u;
        body(valid ? (int)(pk & 0xffffu) : -1 - lane, (int)(pk >> 16), valid);
    }
}

/* Enumerate block (a,b) for this warp and process it, reusing the list
 * entries [blk[0], blk[1]) when `reuse` and filling (in rounds when the
 * region overflows) otherwise.  Records the range for later reuse and
 * returns 0 if the region overflowed (then the range is not reusable). */
/* how for_block runs a body over list entries */
enum { RUN_LANES = 0, RUN_CONVERGED = 1, RUN_RUNS = 2 };

template <int RUN, class Body>
__device__ __forceinline__ void run_entries(const EfsSmem &s, int from, int to, int lane, Body body) {
    if constexpr (RUN == RUN_CONVERGED)
        run_list_all(s, from, to, lane, body);
    else if constexpr (RUN == RUN_RUNS)
        run_list_runs(s, from, to, lane, body);
    else
        run_list(s, from, to, lane, body);
}

template <int WPA, int RUN = RUN_LANES, class Accept, class Body>
__device__ __forceinline__ int for_block(const EfsSmem &s, int a, int b, int *blk, int reuse, int &pos, int lo,
                                         int hi, int warp, int lane, Accept accept, Body body) {
    if (reuse) {
        run_entries<RUN>(s, blk[0], blk[1], lane, body);
        return 1;
    }
    int start = pos, c = warp * 32, whole = 1;
    const int C = block_candidates(s, a, b);
    for (;;) {
        const int from = pos;
        c = fill_chunks<WPA>(s, a, b, c, pos, hi, lane, accept);
        run_entries<RUN>(s, from, pos, lane, body);
        __syncwarp();
        if (c >= C) break;
        whole = 0; /* region full: restart it for the next round */
        start = pos = lo;
    }
    blk[0] = start;
    blk[1] = pos;
    return whole;
}

/* The 4-atoms-per-CTA shape holds two CTAs per SM (its shared memory per
 * atom decides that), so it may use up to 256 registers a thread: asking for
 * two blocks per SM lets it run without spills instead of the register
 * budget of three. */
template <int NE, int NZ, int NLAM, int WPA, int APB>
__global__ void __launch_bounds__(WPA * 32 * APB, APB >= 4 ? 2 : 1) k_efs(EfsArgs A) {
    constexpr int NZL = NZ * NLAM;
    constexpr int WARPS = WPA;
    constexpr int NEP = nep(NE);
    /* the reference bases (<= 8 exponents x 8 angular terms): the forward
     * grid is accumulated on the FP64 tensor cores */
    constexpr bool TC_FWD = NE <= 8 && NZL == 8;
    extern __shared__ __align__(16) char smem_raw[];
    __shared__ mb_params Ps;
    {
        const int *src = reinterpret_cast<const int *>(A.params);
        int *dst = reinterpret_cast<int *>(&Ps);
        for (int k = threadIdx.x; k < (int)(sizeof(mb_params) / sizeof(int)); k += blockDim.x) dst[k] = src[k];
        __syncthreads();
    }
    const mb_params &P = Ps;
    const int NT = WPA * 32, group = threadIdx.x / NT;
    const int tid = threadIdx.x % NT, lane = threadIdx.x & 31, warp = tid >> 5;
    const int i = blockIdx.x * APB + group;
    if (i >= A.N) return; /* whole atom groups only: no barrier spans two groups */
    const int D = P.D, ns = P.nspc, ng2 = P.ng2, ne = P.ne;
    EfsSmem s = efs_carve(smem_raw + (size_t)group * A.smem_group, A.cap, D, NE, ng2, NE * NZL, WARPS, A.tl_cap,
                          TC_FWD);
    const int tlw = A.tl_cap / WPA, tl_lo = warp * tlw, tl_hi = tl_lo + tlw;
    int tl_pos = tl_lo, tl_whole = 1;
    const int n = A.nn[i];
    const int s0 = A.spc[i];
    const double *net = A.weights + P.w_off[s0];

    /* ---- stage neighbours, stably sorted by species relative to s0 ---- */
    for (int t = tid; t < D; t += NT) s.G[t] = 0.0;
    if (warp == 0) {
        /* counts and stable ranks per relative species from warp ballots */
        const int *nj_i = A.nj + (size_t)i * A.cap;
        const unsigned below = (1u << lane) - 1u;
        int cnt[4] = {0, 0, 0, 0};
        for (int base = 0; base < n; base += 32) {
            const int t = base + lane;
            const int ds = t < n ? (A.spc[nj_i[t]] - s0 + ns) % ns : -1;
#pragma unroll
            for (int v = 0; v < 4; v++) cnt[v] += __popc(__ballot_sync(FULL, ds == v));
        }
        int off[4];
        off[0] = 0;
#pragma unroll
        for (int v = 1; v < 4; v++) off[v] = off[v - 1] + cnt[v - 1];
        if (lane < 4) {
            s.seg[lane] = cnt[lane];
            s.seg[4 + lane] = off[lane];
        }
        int run[4] = {0, 0, 0, 0};
        for (int base = 0; base < n; base += 32) {
            const int t = base + lane;
            const int j = t < n ? nj_i[t] : 0;
            const int sp = t < n ? A.spc[j] : 0;
            const int ds = t < n ? (sp - s0 + ns) % ns : -1;
            int dst = 0;
#pragma unroll
            for (int v = 0; v < 4; v++) {
                const unsigned m = __ballot_sync(FULL, ds == v);
                if (ds == v) dst = off[v] + run[v] + __popc(m & below);
                run[v] += __popc(m);
            }
            if (t < n) {
                s.j[dst] = j;
                s.sp[dst] = sp;
                const double4 dv = A.nd[(size_t)i * A.cap + t];
                s.d[dst] = dv;
                s.ir[dst] = 1.0 / dv.w;
            }
        }
    }
    group_sync<WPA>();
    if (tid == 0 && A.counters) atomicAdd(&A.counters[0], (unsigned long long)n);

    constexpr int CELLS = ((NE * NZL + 63) / 64) * 64;
    /* list gate: the union of the forward and derivative triplet gates
     * (they coincide unless species blocks carry different cutoffs) */
    auto accept_union = [&](int jj, int kk) -> bool {
        double4 d1 = s.d[jj], d2 = s.d[kk];
        int sj = s.sp[jj], sk = s.sp[kk];
        int p01 = s0 * s0 + sj * sj, p02 = s0 * s0 + sk * sk, p12 = sj * sj + sk * sk;
        double dx = d1.x - d2.x, dy = d1.y - d2.y, dz = d1.z - d2.z;
        double r3s = dx * dx + dy * dy + dz * dz;
        bool fwd = d1.w < P.f_rc2[p01] && d1.w < P.f_rc4[p01] && d2.w < P.f_rc4[p02] && r3s < P.f_rc4sq[p12];
        bool rev = d1.w < P.d_rc4 && d2.w < P.d_rc4 && r3s < P.d_rc4sq;
        return fwd || rev;
    };
    if (A.mode != MB_MODE_VJP) {
    /* ---- forward pair terms: fc, exponential factors, G2, repulsion ---- */
    for (int t = tid; t < n; t += NT) {
        double r = s.d[t].w;
        int sj = s.sp[t], p = s0 * s0 + sj * sj;
        double fa = fcut(P.f_rc2[p], r);
        s.fa[t] = fa;
        s.fb[t] = fcut(P.f_rc4[p], r);
#pragma unroll
        for (int e = 0; e < NEP; e++)
            s.P[t * NEP + e] = e < ne ? exp(-P.f_eta4[p][e] * r * r) : 0.0;
        bool gate = r < P.f_rc2[p];
        for (int f = 0; f < ng2; f++) {
            double x = r - P.f_rs[p][f];
            s.tmp[t * ng2 + f] = gate ? fa * exp(-P.f_eta2[p][f] * (x * x)) : 0.0;
        }
    }
    group_sync<WPA>();
    /* G2 sums per relative species in neighbour order (deterministic) */
    for (int w = tid; w < ns * ng2; w += NT) {
        int v = w / ng2, f = w % ng2;
        double acc = 0.0;
        for (int t = s.seg[4 + v]; t < s.seg[4 + v] + s.seg[v]; t++) acc += s.tmp[t * ng2 + f];
        s.G[P.ind2[v] + f] = acc;
    }
    if (A.urep > 0.0 && tid == 0) {
        double eu = 0.0;
        for (int t = 0; t < n; t++) {
            double r = s.d[t].w, R = P.rm[s0] + P.rm[s.sp[t]];
            if (r < R) eu += A.urep * fcut(R, r) * R / r;
        }
        A.EU[i] = eu;
    }
    group_sync<WPA>(); /* the G2 terms in tmp are read; the triplet list reuses their space */

    /* ---- forward triplet terms, block by block of (species j, species k) ---- */
    {
        int blkid = 0;
        unsigned long long nacc = 0;
        for (int a = 0; a < ns; a++)
            for (int b = a; b < ns; b++, blkid++) {
                /* the species of j and k are fixed within the block (neighbours are
                 * sorted by species relative to s0): hoist their parameters */
                const int sja = (a + s0) % ns, skb = (b + s0) % ns;
                const int p01 = s0 * s0 + sja * sja, p02 = s0 * s0 + skb * skb, p12 = sja * sja + skb * skb;
                const double rc2_01 = P.f_rc2[p01], rc4_01 = P.f_rc4[p01], rc4_02 = P.f_rc4[p02];
                const double rc4sq_12 = P.f_rc4sq[p12], rc4_12 = P.f_rc4[p12];
                const double drc4 = P.d_rc4, drc4sq = P.d_rc4sq;
                auto accept_blk = [&](int jj, int kk) -> bool {
                    const double4 d1 = s.d[jj], d2 = s.d[kk];
                    const double dx = d1.x - d2.x, dy = d1.y - d2.y, dz = d1.z - d2.z;
                    const double r3s = dx * dx + dy * dy + dz * dz;
                    return (d1.w < rc2_01 && d1.w < rc4_01 && d2.w < rc4_02 && r3s < rc4sq_12) ||
                           (d1.w < drc4 && d2.w < drc4 && r3s < drc4sq);
                };
                const double *eta12 = P.f_eta4[p12];
                if constexpr (TC_FWD) {
                    /* Each lane takes one listed triplet and forms its 8 exponential
                     * factors ex[e] and 8 angular terms lz[zl]; the grid
                     * G[e][zl] += sum_t ex_t[e] lz_t[zl] is then an outer-product
                     * sum, done 4 triplets at a time by mma.sync m8n8k4 in FP64
                     * with the values staged through shared memory.  The
                     * accumulator fragment leaves lane l with cells 2l, 2l+1. */
                    double c0 = 0.0, c1 = 0.0;
                    double *stw = s.stage + warp * 32 * EFS_STG;
                    auto body = [&](int jj, int kk, bool valid) {
                        double ex[8], lz[NZL];
#pragma unroll
                        for (int q = 0; q < 8; q++) ex[q] = 0.0;
#pragma unroll
                        for (int q = 0; q < NZL; q++) lz[q] = 0.0;
                        if (valid) {
                            const double4 d1 = s.d[jj], d2 = s.d[kk];
                            const double dx = d1.x - d2.x, dy = d1.y - d2.y, dz = d1.z - d2.z;
                            const double r3s = dx * dx + dy * dy + dz * dz;
                            if (d1.w < rc2_01 && d1.w < rc4_01 && d2.w < rc4_02 && r3s < rc4sq_12) {
                                nacc++;
                                const double r3 = sqrt(r3s);
                                const double c = (d1.x * d2.x + d1.y * d2.y + d1.z * d2.z) * (s.ir[jj] * s.ir[kk]);
                                const double A3 = 2.0 * s.fa[jj] * s.fb[kk] * fcut(rc4_12, r3);
                                angular<NZ, NLAM>(P, c, lz, nullptr);
                                const double2 *pj = reinterpret_cast<const double2 *>(s.P + jj * NEP);
                                const double2 *pk = reinterpret_cast<const double2 *>(s.P + kk * NEP);
#pragma unroll
                                for (int h = 0; h < NEP / 2; h++) {
                                    const double2 x = pj[h], y = pk[h];
#pragma unroll
                                    for (int q = 0; q < 2; q++) {
                                        const int e = 2 * h + q;
                                        if (e < NE && e < ne)
                                            ex[e] = A3 * (q ? x.y * y.y : x.x * y.x) * exp(-eta12[e] * r3s);
                                    }
                                }
                            }
                        }
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            stw[stg_slot(lane, q)] = ex[q];
                            stw[stg_slot(lane, 8 + q)] = lz[q];
                        }
                        __syncwarp();
#pragma unroll
                        for (int st = 0; st < 8; st++) {
                            const int t = 4 * st + (lane & 3);
                            dmma884(c0, c1, stw[stg_slot(t, lane >> 2)], stw[stg_slot(t, 8 + (lane >> 2))]);
                        }
                        __syncwarp();
                    };
                    int *blk = s.blk + (blkid * WPA + warp) * 2;
                    tl_whole &= for_block<WPA, RUN_CONVERGED>(s, a, b, blk, 0, tl_pos, tl_lo, tl_hi, warp, lane, accept_blk, body);
                    group_sync<WPA>();
                    group_store64<WPA>(c0, c1, s, warp, lane);
                    {
                        /* every feature is its own descriptor entry: one per thread */
                        const int base = P.ind4[a * a + b * b];
                        for (int f = tid; f < P.ng4; f += NT)
                            s.G[base + f] += s.red[P.g4_e[f] * NZL + (P.g4_zl[f] / P.nlam) * NLAM + P.g4_zl[f] % P.nlam];
                    }
                    group_sync<WPA>();
                } else {
                double acc[CELLS];
#pragma unroll
                for (int k = 0; k < CELLS; k++) acc[k] = 0.0;
                auto body = [&](int jj, int kk) {
                    double4 d1 = s.d[jj], d2 = s.d[kk];
                    double dx = d1.x - d2.x, dy = d1.y - d2.y, dz = d1.z - d2.z;
                    double r3s = dx * dx + dy * dy + dz * dz;
                    if (!(d1.w < rc2_01 && d1.w < rc4_01 && d2.w < rc4_02 && r3s < rc4sq_12)) return;
                    nacc++;
                    double r3 = sqrt(r3s);
                    double c = (d1.x * d2.x + d1.y * d2.y + d1.z * d2.z) * (s.ir[jj] * s.ir[kk]);
                    double A3 = 2.0 * s.fa[jj] * s.fb[kk] * fcut(rc4_12, r3);
                    double lz[NZL];
#pragma unroll
                    for (int k = 0; k < NZL; k++) lz[k] = 0.0;
                    angular<NZ, NLAM>(P, c, lz, nullptr);
                    const double2 *pj = reinterpret_cast<const double2 *>(s.P + jj * NEP);
                    const double2 *pk = reinterpret_cast<const double2 *>(s.P + kk * NEP);
#pragma unroll
                    for (int h = 0; h < NEP / 2; h++) {
                        const double2 x = pj[h], y = pk[h];
#pragma unroll
                        for (int q = 0; q < 2; q++) {
                            const int e = 2 * h + q;
                            if (e >= NE || e >= ne) break;
                            const double ex = A3 * (q ? x.y * y.y : x.x * y.x) * exp(-eta12[e] * r3s);
#pragma unroll
                            for (int zl = 0; zl < NZL; zl++) acc[e * NZL + zl] += ex * lz[zl];
                        }
                    }
                };
                int *blk = s.blk + (blkid * WPA + warp) * 2;
                tl_whole &= for_block<WPA>(s, a, b, blk, 0, tl_pos, tl_lo, tl_hi, warp, lane, accept_blk, body);
                group_sync<WPA>();
#pragma unroll
                for (int ch = 0; ch < CELLS / 64; ch++) {
                    group_reduce64<WPA>(acc + 64 * ch, s, warp, lane);
                    {
                        int ds = a * a + b * b, base = P.ind4[ds];
                        for (int f = tid; f < P.ng4; f += NT) {
                            int cell = P.g4_e[f] * NZL + (P.g4_zl[f] / P.nlam) * NLAM + P.g4_zl[f] % P.nlam;
                            if (cell / 64 == ch) s.G[base + f] += s.red[cell % 64];
                        }
                    }
                    group_sync<WPA>();
                }
                }
            }
        if (A.counters) {
            for (int o = 16; o > 0; o >>= 1) nacc += __shfl_xor_sync(FULL, nacc, o);
            if (lane == 0) atomicAdd(&A.counters[1], nacc);
        }
    }

    if (A.mode == MB_MODE_DESCRIPTORS) {
        for (int t = tid; t < D; t += NT) A.G[(size_t)i * D + t] = s.G[t];
        return;
    }
    } /* end of the forward part (skipped for MB_MODE_VJP) */

    /* ---- MLP: forward (src/nmlp.c:367-431) and dE/dG ---- */
    const int h1 = P.h1, h2 = P.h2;
    const double *off = net, *W0 = off + D, *b0 = W0 + h1 * D, *W1 = b0 + h1, *b1 = W1 + h2 * h1, *W2 = b1 + h2,
                 *b2 = W2 + h2;
    double *H1 = s.h, *H2 = s.h + MB_MAXH, *Dl1 = s.h + 2 * MB_MAXH, *Dl2 = s.h + 3 * MB_MAXH;
    if (A.mode != MB_MODE_VJP) {
        for (int m = warp; m < h1; m += WARPS) {
            double acc = 0.0;
            for (int l = lane; l < D; l += 32) acc += (s.G[l] - off[l]) * W0[m * D + l];
            acc = warp_sum(acc);
            if (lane == 0) H1[m] = tanh(b0[m] + acc);
        }
        group_sync<WPA>();
        if (warp == 0) {
            double v = 0.0;
            if (lane < h2) {
                v = b1[lane];
                for (int k = 0; k < h1; k++) v += H1[k] * W1[lane * h1 + k];
                v = tanh(v);
                H2[lane] = v;
            }
            double e = lane < h2 ? v * W2[lane] : 0.0;
            e = warp_sum(e);
            if (lane == 0) A.EA[i] = b2[0] + e;
            __syncwarp();
            if (lane < h2) Dl2[lane] = W2[lane] * (1.0 - v * v);
            __syncwarp();
            if (lane < h1) {
                double g = 0.0;
                for (int m = 0; m < h2; m++) g += Dl2[m] * W1[m * h1 + lane];
                Dl1[lane] = g * (1.0 - H1[lane] * H1[lane]);
            }
        }
        group_sync<WPA>();
        if (A.mode == MB_MODE_ENERGY) return;
        /* s.G <- dE_i/dG_i */
        for (int l = tid; l < D; l += NT) {
            double g = 0.0;
            for (int k = 0; k < h1; k++) g += Dl1[k] * W0[k * D + l];
            s.G[l] = g;
        }
    } else {
        for (int l = tid; l < D; l += NT) s.G[l] = A.G[(size_t)i * D + l];
    }
    group_sync<WPA>();

    /* ---- reverse pair terms with the species-0 parameters ---- */
    double fi[3] = {0.0, 0.0, 0.0}, vr[6] = {0, 0, 0, 0, 0, 0};
    for (int t = tid; t < n; t += NT) {
        double4 d = s.d[t];
        double r = d.w, ir = 1.0 / r;
        double f4, df4, f2, df2;
        fcut_d(P.d_rc4, r, f4, df4);
        fcut_d(P.d_rc2, r, f2, df2);
        s.fa[t] = f4;
        s.fb[t] = df4;
#pragma unroll
        for (int e = 0; e < NEP; e++)
            s.P[t * NEP + e] = e < ne ? exp(-P.d_eta4[e] * r * r) : 0.0;
        int ds1 = (s.sp[t] - s0 + ns) % ns;
        const double *g = s.G + P.ind2[ds1];
        double cpair = 0.0;
        for (int f = 0; f < ng2; f++) {
            double x = r - P.d_rs[f], eta = P.d_eta2[f];
            cpair += g[f] * exp(-eta * x * x) * (-2.0 * eta * x * f2 + df2);
        }
        /* dE/dd = cpair d / r : force +on i, -on j; virial -= (dE/dd) (x) d */
        double cr = cpair * ir;
        double v0 = cr * d.x, v1 = cr * d.y, v2 = cr * d.z;
        fi[0] += v0; fi[1] += v1; fi[2] += v2;
        s.Fnb[3 * t] = -v0; s.Fnb[3 * t + 1] = -v1; s.Fnb[3 * t + 2] = -v2;
        if (A.urep > 0.0) {
            double R = P.rm[s0] + P.rm[s.sp[t]];
            if (r < R) {
                /* CELL_UREP on the ordered pair (i, j): force on i only (src/cmod.c:100-112) */
                double fu, dfu;
                fcut_d(R, r, fu, dfu);
                double tu = -2.0 * A.urep * R / (r * r) * (-fu / r + dfu);
                fi[0] -= tu * d.x; fi[1] -= tu * d.y; fi[2] -= tu * d.z;
                vr[0] += 0.5 * tu * d.x * d.x; vr[1] += 0.5 * tu * d.y * d.y; vr[2] += 0.5 * tu * d.z * d.z;
                vr[3] += 0.5 * tu * d.x * d.y; vr[4] += 0.5 * tu * d.y * d.z; vr[5] += 0.5 * tu * d.z * d.x;
            }
        }
    }
    group_sync<WPA>();

    /* ---- reverse triplet terms (list of the forward pass reused) ---- */
    {
        const int reuse = (A.mode != MB_MODE_VJP) && tl_whole;
        int blkid = 0;
        tl_pos = tl_lo;
        for (int a = 0; a < ns; a++)
            for (int b = a; b < ns; b++, blkid++) {
                const int ds = a * a + b * b, base = P.ind4[ds];
                for (int t = tid; t < NE * NZL; t += NT) s.grid[t] = 0.0;
                group_sync<WPA>();
                for (int f = tid; f < P.ng4; f += NT)
                    atomicAdd(&s.grid[P.g4_e[f] * NZL + (P.g4_zl[f] / P.nlam) * NLAM + P.g4_zl[f] % P.nlam], s.G[base + f]);
                group_sync<WPA>();
                /* returns the entry's force on neighbour j; run_list_runs sums
                 * those per lane and adds them once per change of j */
                auto body = [&](int jj, int kk) -> double3 {
                    const double4 d1 = s.d[jj], d2 = s.d[kk];
                    const double wx = d2.x - d1.x, wy = d2.y - d1.y, wz = d2.z - d1.z;
                    const double r3s = wx * wx + wy * wy + wz * wz;
                    if (!(d1.w < P.d_rc4 && d2.w < P.d_rc4 && r3s < P.d_rc4sq)) return make_double3(0.0, 0.0, 0.0);
                    double r3 = sqrt(r3s);
                    double r1 = d1.w, r2 = d2.w, ir1 = s.ir[jj], ir2 = s.ir[kk], ir3 = 1.0 / r3;
                    double c = (d1.x * d2.x + d1.y * d2.y + d1.z * d2.z) * (ir1 * ir2);
                    double f3, df3;
                    fcut_d(P.d_rc4, r3, f3, df3);
                    double f1 = s.fa[jj], df1 = s.fb[jj], f2 = s.fa[kk], df2 = s.fb[kk];
                    double lz[NZL], lzp[NZL];
#pragma unroll
                    for (int k = 0; k < NZL; k++) { lz[k] = 0.0; lzp[k] = 0.0; }
                    angular<NZ, NLAM>(P, c, lz, lzp);
                    const double2 *pj = reinterpret_cast<const double2 *>(s.P + jj * NEP);
                    const double2 *pk = reinterpret_cast<const double2 *>(s.P + kk * NEP);
                    double Q = 0.0, Qe = 0.0, Qc = 0.0;
#pragma unroll
                    for (int h = 0; h < NEP / 2; h++) {
                        const double2 x = pj[h], y = pk[h];
#pragma unroll
                        for (int q = 0; q < 2; q++) {
                            const int e = 2 * h + q;
                            if (e >= NE || e >= ne) break;
                            const double ex = (q ? x.y * y.y : x.x * y.x) * exp(-P.d_eta4[e] * r3s);
                            double u = 0.0, v = 0.0;
#pragma unroll
                            for (int zl = 0; zl < NZL; zl += 2) {
                                const double2 cg = *reinterpret_cast<const double2 *>(s.grid + e * NZL + zl);
                                u += cg.x * lz[zl] + cg.y * lz[zl + 1];
                                v += cg.x * lzp[zl] + cg.y * lzp[zl + 1];
                            }
                            Q += ex * u;
                            Qe += P.d_eta4[e] * ex * u;
                            Qc += ex * v;
                        }
                    }
                    double Af = 2.0 * f1 * f2 * f3;
                    double T1 = 2.0 * df1 * f2 * f3 * Q - 2.0 * r1 * Af * Qe;
                    double T2 = 2.0 * f1 * df2 * f3 * Q - 2.0 * r2 * Af * Qe;
                    double T3 = 2.0 * f1 * f2 * df3 * Q - 2.0 * r3 * Af * Qe;
                    double Tc = Af * Qc;
                    double a11 = T1 * ir1 - Tc * c * ir1 * ir1, a22 = T2 * ir2 - Tc * c * ir2 * ir2;
                    double a12 = Tc * ir1 * ir2, a3 = T3 * ir3;
                    const double g1x = a11 * d1.x + a12 * d2.x - a3 * wx;
                    const double g1y = a11 * d1.y + a12 * d2.y - a3 * wy;
                    const double g1z = a11 * d1.z + a12 * d2.z - a3 * wz;
                    const double g2x = a22 * d2.x + a12 * d1.x + a3 * wx;
                    const double g2y = a22 * d2.y + a12 * d1.y + a3 * wy;
                    const double g2z = a22 * d2.z + a12 * d1.z + a3 * wz;
                    fi[0] += g1x + g2x; fi[1] += g1y + g2y; fi[2] += g1z + g2z;
                    atomicAdd(&s.Fnb[3 * kk], -g2x);
                    atomicAdd(&s.Fnb[3 * kk + 1], -g2y);
                    atomicAdd(&s.Fnb[3 * kk + 2], -g2z);
                    return make_double3(g1x, g1y, g1z);
                };
                int *blk = s.blk + (blkid * WPA + warp) * 2;
                for_block<WPA, RUN_RUNS>(s, a, b, blk, reuse, tl_pos, tl_lo, tl_hi, warp, lane, accept_union, body);
                group_sync<WPA>();
            }
    }

    /* virial of atom i's energy: every neighbour force (pairs and triplets)
     * times its displacement -- the sum -(dE/dd) (x) d taken per neighbour */
    for (int t = tid; t < n; t += NT) {
        const double4 d = s.d[t];
        const double fx = s.Fnb[3 * t], fy = s.Fnb[3 * t + 1], fz = s.Fnb[3 * t + 2];
        vr[0] += fx * d.x; vr[1] += fy * d.y; vr[2] += fz * d.z;
        vr[3] += fx * d.y; vr[4] += fy * d.z; vr[5] += fz * d.x;
    }

    /* ---- write forces and the virial of atom i ---- */
    {
        double v[64];
#pragma unroll
        for (int k = 0; k < 64; k++) v[k] = 0.0;
        v[0] = fi[0]; v[1] = fi[1]; v[2] = fi[2];
#pragma unroll
        for (int k = 0; k < 6; k++) v[3 + k] = vr[k];
        group_reduce64<WPA>(v, s, warp, lane);
        if (tid == 0) {
            atomicAdd(&A.F[3 * i], s.red[0]);
            atomicAdd(&A.F[3 * i + 1], s.red[1]);
            atomicAdd(&A.F[3 * i + 2], s.red[2]);
            for (int k = 0; k < 6; k++) A.vir[(size_t)i * 6 + k] = s.red[3 + k];
        }
        for (int t = tid; t < n; t += NT) {
            int j = s.j[t];
            atomicAdd(&A.F[3 * j], s.Fnb[3 * t]);
            atomicAdd(&A.F[3 * j + 1], s.Fnb[3 * t + 1]);
            atomicAdd(&A.F[3 * j + 2], s.Fnb[3 * t + 2]);
        }
    }
}

/* ------------------------------------------------------------------ */
/* fused triplet kernel (reference bases)                               */
/* ------------------------------------------------------------------ */

/* k_efs_tri: the whole descriptor pass of an atom -- neighbour sort, G2,
 * triplet list, forward grid, MLP, reverse pass -- with every factor of a
 * triplet evaluated in registers.  It applies to bases whose forward and
 * derivative functions share one cutoff and whose pair-mixed G4 exponents
 * equal the species-0 ones (every reference model; src/nprs.c:222-252 mixes
 * identical blocks), see mb_tri.
 *
 * What bounds it: instruction issue and the latency of dependent FP64
 * operations at the 14 warps per SM that shared memory and 128 registers a
 * thread allow (the 4000-atom ternary alloy, 2 warps per atom: issue slots 46%
 * busy, FP64 pipe 33%, 1450 instructions per 32 triplets, of them 470 FP64).
 * The j-k leg of a triplet is an entry of j's own list, and an earlier form of
 * this pass looked its factors up there (leg tables and triplet lists in
 * global memory, found through hashes, in three kernels): nine 16-byte loads a
 * triplet from scattered 80-byte rows kept the L1 pipe 67% busy, and listing
 * the triplets took a kernel of its own.  Here exp(-eta_e rho) and the cutoff
 * are polynomials of the squared distances (mb_tri), about 100 FMAs in 7
 * independent chains: no table, no square root, no trigonometry and no memory
 * traffic per triplet.  The pass over that alloy went from 520 to 375 us, over
 * the 20000-atom particle from 1.20 to 0.87 ms, over a 487-atom alloy from 140
 * to 75 us. */

#define TRI_ROW 10                        /* doubles of a neighbour's row; 80 bytes: 16-byte loads of
                                           * consecutive rows fall in distinct banks */
#define TRI_PER_LANE (MB_TRI_MAX_CAP / 32)
#define TRI_NONE 0xffffu                  /* padding entry of a triplet list */

struct TriArgs {
    int N, cap, mode, tlw; /* tlw: list entries of one warp */
    double urep;
    const int *nn, *nj;
    const double4 *nd;
    const int *spc;
    const double *weights, *w0; /* w0: first-layer weights by input (mb_tri) */
    double *EA, *EU, *G, *F, *vir;
    unsigned long long *counters;
    size_t smem_group;
    mb_params P; /* by value: read from the kernel-parameter space through the constant cache */
    mb_tri T;
};

#define TRI_STG 36 /* staging: [16 values][TRI_STG triplets]; both the lane-wise writes and the
                    * mma operand reads touch 16 distinct banks a half-warp */
#define TRI_TS 20  /* row stride of the reverse pass's 8 x 16 tiles (4 mod 16: operand reads of the
                    * tile and of its transpose are conflict-free) */

/* shared-memory carve-up of one atom group of k_efs_tri; regions whose
 * lifetimes do not overlap share storage */
struct TriSmem {
    double *row;        /* [cap][TRI_ROW]: x, y, z, 1/r, r^2, f, h, r */
    double *stage;      /* per warp TRI_STG x 16 (forward) | */
    double *G, *h, *hp; /* descriptors or dE/dG, hidden layers and their partial sums | */
    double *tile;       /* per warp 3 x 8 x TRI_TS (reverse) */
    double *red;        /* [warp][block][64] forward sums | */
    double *Fnb, *grid; /* neighbour forces per warp [cap][4], dE/dG by (eta, zeta, lambda) cell per block */
    double *g2;         /* [warp][species][ng2] | */
    double *fin;        /* [warp][9] */
    unsigned short *tl; /* [warp][tlw] triplets a | b << 8 */
    int *j;
    int *bnd;           /* [warp][8] starts of the species blocks in the warp's list, and the end */
    int *seg;           /* [0..3] counts, [4..7] offsets by relative species */
};

__host__ __device__ inline int tri_nblk(int ns) { return ns * (ns + 1) / 2; }

/* list entries of one warp: it takes every warps-th group of 4 columns, and
 * column b of the upper triangle holds b pairs; up to 3 padding entries per
 * species block */
__host__ __device__ inline int tri_list(int cap, int warps) {
    int most = 0;
    for (int w = 0; w < warps; w++) {
        int sum = 0;
        for (int b = 4 * w; b < cap; b += 4 * warps) sum += 4 * b + 6;
        most = sum > most ? sum : most;
    }
    return (most + 4 * MB_MAX_BLOCKS + 7) & ~7;
}

__host__ __device__ inline size_t tri_r1_bytes(int D, int warps) {
    const size_t st = sizeof(double) * warps * 16 * TRI_STG;
    const size_t mid = sizeof(double) * (D + (D & 1) + 4 * MB_MAXH + 16 * warps);
    const size_t ti = sizeof(double) * warps * 24 * TRI_TS;
    return align16(st > mid ? (st > ti ? st : ti) : (mid > ti ? mid : ti));
}

__host__ __device__ inline size_t tri_r2_bytes(int cap, int ns, int warps) {
    const size_t red = sizeof(double) * warps * tri_nblk(ns) * 64;
    const size_t rev = sizeof(double) * (64 * tri_nblk(ns) + 4 * cap * warps);
    return align16(red > rev ? red : rev);
}

__host__ __device__ inline size_t tri_small(int ns, int ng2, int warps) {
    const int g2 = ns * ng2 > 9 ? ns * ng2 : 9;
    return align16(sizeof(double) * warps * g2);
}

__host__ __device__ inline size_t tri_smem_bytes(int cap, int D, int ns, int ng2, int warps) {
    return align16(sizeof(double) * cap * TRI_ROW + tri_r1_bytes(D, warps) + tri_r2_bytes(cap, ns, warps) +
                   tri_small(ns, ng2, warps) + align16(sizeof(short) * tri_list(cap, warps) * warps) +
                   align16(sizeof(int) * cap) + sizeof(int) * (8 * warps + 8));
}

__device__ inline TriSmem tri_carve(char *p, int cap, int D, int ns, int ng2, int warps, int tlw) {
    TriSmem s;
    s.row = (double *)p; p += sizeof(double) * cap * TRI_ROW;
    s.stage = (double *)p;
    s.tile = (double *)p;
    s.G = (double *)p;
    s.h = s.G + D + (D & 1);
    s.hp = s.h + 4 * MB_MAXH;
    p += tri_r1_bytes(D, warps);
    s.red = (double *)p;
    s.grid = (double *)p;
    s.Fnb = s.grid + 64 * tri_nblk(ns);
    p += tri_r2_bytes(cap, ns, warps);
    s.g2 = (double *)p;
    s.fin = (double *)p;
    p += tri_small(ns, ng2, warps);
    s.tl = (unsigned short *)p; p += align16(sizeof(short) * tlw * warps);
    s.j = (int *)p; p += align16(sizeof(int) * cap);
    s.bnd = (int *)p; p += sizeof(int) * 8 * warps;
    s.seg = (int *)p;
    return s;
}

/* exp(-eta_e rho) for e < NE: the polynomial and its two squarings, the chains
 * side by side over one coefficient at a time (two per 16-byte shared load), or
 * exp() for the ne exponents there are (EXP, steep bases). */
template <int NE, bool EXP>
__device__ __forceinline__ void tri_exp(const mb_tri_tab &tab, int ne, double rho, double *E) {
    if constexpr (EXP) {
#pragma unroll
        for (int e = 0; e < NE; e++) E[e] = e < ne ? exp(-tab.eta[e] * rho) : 0.0;
        return;
    }
    const double2 *c = reinterpret_cast<const double2 *>(tab.ex), *kw = reinterpret_cast<const double2 *>(tab.kw);
    double w[NE];
#pragma unroll
    for (int e = 0; e < NE; e += 2) {
        const double2 k = kw[e / 2];
        w[e] = fma(k.x, rho, -1.0);
        if (e + 1 < NE) w[e + 1] = fma(k.y, rho, -1.0);
    }
#pragma unroll
    for (int k = 0; k <= MB_TRI_DEG; k += 2) {
        const double2 ck = c[k / 2];
#pragma unroll
        for (int e = 0; e < NE; e++) E[e] = k ? fma(E[e], w[e], ck.x) : ck.x;
#pragma unroll
        for (int e = 0; e < NE; e++) E[e] = fma(E[e], w[e], ck.y);
    }
#pragma unroll
    for (int q = 0; q < MB_TRI_SQ; q++)
#pragma unroll
        for (int e = 0; e < NE; e++) E[e] *= E[e];
}

__device__ __forceinline__ double tri_f(const mb_tri_tab &tab, double v) {
    const double2 *c = reinterpret_cast<const double2 *>(tab.f);
    double p = fma(c[0].x, v, c[0].y);
#pragma unroll
    for (int k = 1; k <= MB_TRI_FDEG / 2; k++) p = fma(fma(p, v, c[k].x), v, c[k].y);
    return p;
}

__device__ __forceinline__ double2 tri_fh(const mb_tri_tab &tab, double v) {
    const double2 *c = reinterpret_cast<const double2 *>(tab.fh);
    double2 p = c[0];
#pragma unroll
    for (int k = 1; k <= MB_TRI_FDEG; k++) {
        const double2 ck = c[k];
        p.x = fma(p.x, v, ck.x);
        p.y = fma(p.y, v, ck.y);
    }
    return p;
}

/* (1 + lambda c)^zeta without its normalisation, and the derivative in c.
 * STD: zeta = 1, 2, 4, 16 and lambda = -1, +1 (the reference bases), straight
 * multiplications; otherwise any integer zeta. */
template <bool STD>
__device__ __forceinline__ void tri_angular(const mb_params &P, double c, double *lz, double *lzp) {
    if constexpr (STD) {
#pragma unroll
        for (int l = 0; l < 2; l++) {
            const double lam = l ? 1.0 : -1.0, b1 = 1.0 + lam * c, b2 = b1 * b1, b4 = b2 * b2, b8 = b4 * b4;
            lz[l] = b1;
            lz[2 + l] = b2;
            lz[4 + l] = b4;
            lz[6 + l] = b8 * b8;
            if (lzp) {
                const double b3 = b1 * b2;
                lzp[l] = lam;
                lzp[2 + l] = 2.0 * lam * b1;
                lzp[4 + l] = 4.0 * lam * b3;
                lzp[6 + l] = 16.0 * lam * (b4 * b8) * b3;
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < 8; k++) {
            lz[k] = 0.0;
            if (lzp) lzp[k] = 0.0;
        }
        angular<4, 2, false>(P, c, lz, lzp);
    }
}

/* absolute species of relative species v of an atom of species s0 */
__device__ __forceinline__ int abs_species(int s0, int v, int ns) {
    const int x = s0 + v;
    return x >= ns ? x - ns : x;
}

/* NE: exponents evaluated (ne <= NE); WPA: warps per atom; APB: atoms per
 * CTA; STD: the reference's function table (mb_tri), whose powers are
 * straight-line code (the general form is 20% slower: the branches keep the
 * compiler from interleaving the chains); EXP: exponents too steep for the
 * polynomial, exp() in its place (E/F/S calls of 32, 500 and 4000 atoms with
 * exponents up to 1 / A^2: 120, 245 and 967 us on k_efs, 79, 129 and 574 here;
 * up to 8 exponents and all function cells 364, 940 and 6727 against 89, 143 and
 * 676).  All shapes are compiled for 16 resident warps per SM (128 registers a
 * thread). */
template <int NE, int WPA, int APB, bool STD, bool EXP>
__global__ void __launch_bounds__(WPA * 32 * APB, 512 / (WPA * 32 * APB)) k_efs_tri(const __grid_constant__ TriArgs A) {
    constexpr int NZL = 8;
    extern __shared__ __align__(16) char smem_raw[];
    __shared__ __align__(16) mb_tri_tab tab; /* polynomial coefficients: 16-byte broadcast loads */
    const mb_params &P = A.P;
    const mb_tri &T = A.T;
    for (int k = threadIdx.x; k < (int)(sizeof(mb_tri_tab) / sizeof(double)); k += blockDim.x)
        reinterpret_cast<double *>(&tab)[k] = reinterpret_cast<const double *>(&T.tab)[k];
    __syncthreads();
    const int NT = WPA * 32, group = threadIdx.x / NT;
    const int tid = threadIdx.x % NT, lane = threadIdx.x & 31, warp = tid >> 5;
    const int i = blockIdx.x * APB + group;
    if (i >= A.N) return; /* whole atom groups only: no barrier spans two groups */
    const int D = P.D, ns = P.nspc, ng2 = P.ng2, ne = P.ne, cap = A.cap, nblk = tri_nblk(ns);
    TriSmem s = tri_carve(smem_raw + (size_t)group * A.smem_group, cap, D, ns, ng2, WPA, A.tlw);
    const int n = A.nn[i], s0 = A.spc[i];
    const double *net = A.weights + P.w_off[s0];

    /* ---- stage the neighbours, stably sorted by species relative to s0:
     * every warp finds all the ranks (ballots) and writes its share of the rows ---- */
    {
        const size_t row = (size_t)i * cap;
        int jv[TRI_PER_LANE], rv[TRI_PER_LANE], cnt[MB_MAXSPC] = {0, 0, 0};
        constexpr int MINE = (TRI_PER_LANE + WPA - 1) / WPA; /* rows this warp writes, per lane */
        double4 dv[MINE];
#pragma unroll
        for (int q = 0; q < TRI_PER_LANE; q++) {
            const int t = q * 32 + lane;
            jv[q] = t < n ? A.nj[row + t] : -1;
        }
#pragma unroll
        for (int k = 0; k < MINE; k++) {
            const int t = (k * WPA + warp) * 32 + lane;
            if (t < n) dv[k] = A.nd[row + t];
        }
#pragma unroll
        for (int q = 0; q < TRI_PER_LANE; q++) {
            rv[q] = -1;
            if (jv[q] >= 0) {
                const int d = A.spc[jv[q]] - s0;
                rv[q] = d < 0 ? d + ns : d;
            }
        }
        unsigned bal[TRI_PER_LANE][MB_MAXSPC];
#pragma unroll
        for (int q = 0; q < TRI_PER_LANE; q++)
#pragma unroll
            for (int v = 0; v < MB_MAXSPC; v++) {
                bal[q][v] = v < ns && 32 * q < n ? __ballot_sync(FULL, rv[q] == v) : 0u;
                cnt[v] += __popc(bal[q][v]);
            }
        if (warp == 0 && lane < 4) {
            s.seg[lane] = lane == 0 ? cnt[0] : lane == 1 ? cnt[1] : lane == 2 ? cnt[2] : 0;
            s.seg[4 + lane] = lane == 0 ? 0 : lane == 1 ? cnt[0] : lane == 2 ? cnt[0] + cnt[1] : n;
        }
        const unsigned below = (1u << lane) - 1u;
        int run[MB_MAXSPC] = {0, cnt[0], cnt[0] + cnt[1]};
#pragma unroll
        for (int q = 0; q < TRI_PER_LANE; q++) {
            if (q % WPA == warp && rv[q] >= 0) {
                const int v = rv[q];
                const int dst = (v == 0 ? run[0] + __popc(bal[q][0] & below)
                                        : v == 1 ? run[1] + __popc(bal[q][1] & below) : run[2] + __popc(bal[q][2] & below));
                const double4 d = dv[q / WPA];
                const double r2 = d.x * d.x + d.y * d.y + d.z * d.z;
                const double2 fh = tri_fh(tab, fma(r2, T.sv, -1.0));
                double2 *o = reinterpret_cast<double2 *>(s.row + TRI_ROW * dst);
                o[0] = make_double2(d.x, d.y);
                o[1] = make_double2(d.z, 1.0 / d.w);
                o[2] = make_double2(r2, fh.x);
                o[3] = make_double2(fh.y, d.w);
                s.j[dst] = jv[q];
            }
#pragma unroll
            for (int v = 0; v < MB_MAXSPC; v++) run[v] += __popc(bal[q][v]);
        }
    }
    group_sync<WPA>();
    if (tid == 0 && A.counters) atomicAdd(&A.counters[0], (unsigned long long)n);
    const int o1 = s.seg[5], o2 = s.seg[6]; /* where relative species 1 and 2 begin */

    if (A.mode != MB_MODE_VJP) {
        /* ---- G2 (src/nprs.c:518-526): lane = (neighbour mod 4, function mod 8),
         * fixed-order partial sums per warp ---- */
        for (int f0 = 0; f0 < ng2; f0 += 8)
            for (int v = 0; v < ns; v++) {
                const int f = f0 + (lane & 7), sj = abs_species(s0, v, ns), p = s0 * s0 + sj * sj;
                double acc = 0.0;
                if (f < ng2) {
                    const double rs = P.f_rs[p][f], eta = P.f_eta2[p][f];
                    const int end = s.seg[4 + v] + s.seg[v];
                    for (int t = s.seg[4 + v] + warp * 4 + (lane >> 3); t < end; t += 4 * WPA) {
                        const double x = s.row[TRI_ROW * t + 7] - rs;
                        acc += s.row[TRI_ROW * t + 5] * exp(-eta * (x * x));
                    }
                }
                acc += __shfl_xor_sync(FULL, acc, 8);
                acc += __shfl_xor_sync(FULL, acc, 16);
                if (lane < 8 && f < ng2) s.g2[(warp * ns + v) * ng2 + f] = acc;
            }
        if (A.urep > 0.0 && warp == 0) {
            double eu = 0.0;
            for (int t = lane; t < n; t += 32) {
                const int v = (t >= o1) + (t >= o2);
                const double r = s.row[TRI_ROW * t + 7], R = P.rm[s0] + P.rm[abs_species(s0, v, ns)];
                if (r < R) eu += A.urep * fcut(R, r) * R / r;
            }
            eu = warp_sum(eu);
            if (lane == 0) A.EU[i] = eu;
        } else if (tid == 0) {
            A.EU[i] = 0.0;
        }
    }

    /* ---- triplet list: per species block (al <= be) the pairs a < b of the
     * atom's entries whose j-k distance is below the cutoff.  PRS_BP takes the
     * triplet when |DX_j - DX_k| < Rc (src/nprs.c:528-537, src/cell.c:175-181):
     * the squared distance summed without contraction as the reference forms
     * it, against the threshold for which sqrt(s) < Rc holds exactly.  The
     * block is walked in stripes of 8 rows (a >> 3) and groups of 4 columns
     * (b >> 2), a candidate per lane, the atom's warps taking every WPA-th
     * group; accepted pairs are appended column by column, so that a run of a
     * list shares one stripe and few columns (the reverse pass sums such runs
     * as 8 x 8 tiles).  A block's part is padded to a multiple of 4 entries, so
     * that the tensor-core steps of the forward pass hold one block each. ---- */
    unsigned short *tl = s.tl + warp * A.tlw;
    int *bnd = s.bnd + 8 * warp;
    int pos = 0;
    {
        int blkid = 0, pad = 0;
        const unsigned below = (1u << lane) - 1u;
        for (int al = 0; al < ns; al++)
            for (int be = al; be < ns; be++, blkid++) {
                if (lane == 0) bnd[blkid] = pos;
                const int sj = abs_species(s0, al, ns), sk = abs_species(s0, be, ns);
                const double thr = P.f_rc4thr[sj * sj + sk * sk];
                const int oa = s.seg[4 + al], ea = oa + s.seg[al], ob = s.seg[4 + be], eb = ob + s.seg[be];
                for (int st = oa >> 3; 8 * st < ea && ea > oa; st++) {
                    const int a = 8 * st + (lane & 7);
                    const double *pa = s.row + TRI_ROW * a;
                    const double ax = pa[0], ay = pa[1], az = pa[2];
                    /* the lane's columns: lo <= b < eb (none for rows outside the
                     * block; what is read past the rows is discarded) */
                    const int lo = a >= oa && a < ea ? max(ob, a + 1) : 0x7fffffff;
                    /* groups g = warp (mod WPA) from the stripe's first column on */
                    int g = max(ob, max(oa, 8 * st) + 1) >> 2;
                    g += (warp - g) & (WPA - 1);
                    const double *pb = s.row + TRI_ROW * (4 * g + (lane >> 3));
                    unsigned ent = (unsigned)a | (unsigned)(4 * g + (lane >> 3)) << 8;
#pragma unroll 1
                    for (int b = 4 * g + (lane >> 3); b - (lane >> 3) < eb; b += 4 * WPA) {
                        const double2 b01 = *reinterpret_cast<const double2 *>(pb);
                        const double dx = xsub(ax, b01.x), dy = xsub(ay, b01.y), dz = xsub(az, pb[2]);
                        const bool ok = xadd(xadd(xmul(dx, dx), xmul(dy, dy)), xmul(dz, dz)) < thr && b >= lo && b < eb;
                        const unsigned m = __ballot_sync(FULL, ok);
                        if (ok) tl[pos + __popc(m & below)] = (unsigned short)ent;
                        pos += __popc(m);
                        pb += 4 * WPA * TRI_ROW;
                        ent += 4u * WPA << 8;
                    }
                }
                if (lane < (-pos & 3)) tl[pos + lane] = (unsigned short)TRI_NONE;
                pad += -pos & 3;
                pos = (pos + 3) & ~3;
            }
        if (lane == 0) bnd[blkid] = pos;
        if (A.counters && lane == 0) atomicAdd(&A.counters[1], (unsigned long long)(pos - pad));
    }
    __syncwarp();

    if (A.mode != MB_MODE_VJP) {
        /* ---- forward: each lane forms a triplet's 8 exponential and 8 angular
         * factors, staged through shared memory; the grid sum_t ex_t[e] lz_t[zl]
         * of a block is an outer-product sum on the FP64 tensor cores, 4
         * triplets a step, left in lane l as cells 2l, 2l+1 ---- */
        double c0 = 0.0, c1 = 0.0;
        double *stw = s.stage + warp * 16 * TRI_STG + lane;
        const double *str = s.stage + warp * 16 * TRI_STG + (lane >> 2) * TRI_STG + (lane & 3);
        double2 *red = reinterpret_cast<double2 *>(s.red + (size_t)warp * nblk * 64) + lane;
        int blk = 0, nb = bnd[1];
        for (int base = 0; base < pos; base += 32) {
            const unsigned ent = base + lane < pos ? tl[base + lane] : TRI_NONE;
            const bool valid = ent != TRI_NONE;
            /* padding lanes evaluate entry (0, 0) with weight 0 */
            const unsigned ab = valid ? ent : 0u;
            const double2 *pa = reinterpret_cast<const double2 *>(s.row + TRI_ROW * (ab & 0xffu));
            const double2 *pb = reinterpret_cast<const double2 *>(s.row + TRI_ROW * (ab >> 8));
            const double2 a0 = pa[0], a1 = pa[1], a2 = pa[2], b0 = pb[0], b1 = pb[1], b2 = pb[2];
            const double wx = b0.x - a0.x, wy = b0.y - a0.y, wz = b1.x - a1.x;
            const double s3 = wx * wx + wy * wy + wz * wz;
            const double c = (a0.x * b0.x + a0.y * b0.y + a1.x * b1.x) * (a1.y * b1.y);
            double A3 = 2.0 * a2.y * b2.y * tri_f(tab, fma(s3, T.sv, -1.0));
            if (!valid) A3 = 0.0;
            double ex[8], lz[NZL];
            ex[7] = 0.0;
            tri_exp<NE, EXP>(tab, ne, a2.x + b2.x + s3, ex);
            tri_angular<STD>(P, c, lz, nullptr);
#pragma unroll
            for (int q = 0; q < 8; q++) {
                stw[q * TRI_STG] = q < NE ? A3 * ex[q] : 0.0;
                stw[(8 + q) * TRI_STG] = lz[q];
            }
            __syncwarp();
#pragma unroll
            for (int st = 0; st < 8; st++) {
                if (base + 4 * st >= nb && blk + 1 < nblk) {
                    /* the next block begins (past the last one the values are zeros) */
                    do {
                        red[32 * blk] = make_double2(c0, c1);
                        c0 = c1 = 0.0;
                        blk++;
                        nb = bnd[blk + 1];
                    } while (base + 4 * st >= nb && blk + 1 < nblk);
                }
                dmma884(c0, c1, str[4 * st], str[4 * st + 8 * TRI_STG]);
            }
            __syncwarp();
        }
        for (; blk < nblk; blk++) {
            red[32 * blk] = make_double2(c0, c1);
            c0 = c1 = 0.0;
        }
        group_sync<WPA>();
        /* descriptors: the warps' sums in warp order; the cells carry the zeta
         * normalisation left out of the angular terms (a power of two) */
        for (int w = tid; w < ns * ng2; w += NT) {
            const int v = w / ng2, f = w - v * ng2;
            double g = 0.0;
            for (int k = 0; k < WPA; k++) g += s.g2[(k * ns + v) * ng2 + f];
            s.G[P.ind2[v] + f] = g;
        }
        for (int f = tid; f < P.ng4; f += NT) {
            const int cell = T.fn_cell[f];
            const double pz = P.powz[(cell & 7) >> 1];
            int b = 0;
            for (int al = 0; al < ns; al++)
                for (int be = al; be < ns; be++, b++) {
                    double g = 0.0;
                    for (int k = 0; k < WPA; k++) g += s.red[(size_t)(k * nblk + b) * 64 + cell];
                    s.G[P.ind4[al * al + be * be] + f] = g * pz;
                }
        }
        group_sync<WPA>();
        if (A.mode == MB_MODE_DESCRIPTORS) {
            for (int t = tid; t < D; t += NT) A.G[(size_t)i * D + t] = s.G[t];
            return;
        }
    }

    /* ---- MLP: forward (src/nmlp.c:367-431) and dE/dG ---- */
    const int h1 = P.h1, h2 = P.h2;
    const double *w0 = A.w0 + (size_t)s0 * D * T.wrow;
    const double *b0 = net + D + h1 * D, *W1 = b0 + h1, *b1 = W1 + h2 * h1, *W2 = b1 + h2,
                 *b2 = W2 + h2;
    double *H1 = s.h, *Dl1 = s.h + 2 * MB_MAXH, *Dl2 = s.h + 3 * MB_MAXH;
    if (A.mode != MB_MODE_VJP) {
        if (h1 <= 16) {
            /* an input a lane: its row of first-layer weights in 16-byte loads,
             * every unit's partial sum in each lane, one halving reduction per
             * warp, then the warps in order */
            double acc[16];
#pragma unroll
            for (int m = 0; m < 16; m++) acc[m] = 0.0;
#pragma unroll 2
            for (int l = tid; l < D; l += NT) {
                const double2 *w = reinterpret_cast<const double2 *>(w0 + (size_t)l * T.wrow);
                double2 r[8];
#pragma unroll
                for (int m = 0; m < 8; m++)
                    if (2 * m < h1) r[m] = w[m];
                const double x = s.G[l] - w0[(size_t)l * T.wrow + h1];
#pragma unroll
                for (int m = 0; m < 8; m++)
                    if (2 * m < h1) {
                        acc[2 * m] = fma(x, r[m].x, acc[2 * m]);
                        acc[2 * m + 1] = fma(x, r[m].y, acc[2 * m + 1]);
                    }
            }
            const double tot = warp_reduce16(acc, lane);
            if (!(lane & 1)) s.hp[16 * warp + (lane >> 1)] = tot;
            group_sync<WPA>();
            if (tid < h1) {
                double v = b0[tid];
                for (int w = 0; w < WPA; w++) v += s.hp[16 * w + tid];
                H1[tid] = tanh(v);
            }
        } else {
            for (int m = warp; m < h1; m += WPA) {
                double acc = 0.0;
                for (int l = lane; l < D; l += 32)
                    acc += (s.G[l] - w0[(size_t)l * T.wrow + h1]) * w0[(size_t)l * T.wrow + m];
                acc = warp_sum(acc);
                if (lane == 0) H1[m] = tanh(b0[m] + acc);
            }
        }
        group_sync<WPA>();
        if (warp == 0) {
            double v = 0.0, w2 = 0.0;
            if (lane < h2) {
                v = b1[lane];
                w2 = W2[lane];
#pragma unroll 8
                for (int k = 0; k < h1; k++) v = fma(H1[k], W1[lane * h1 + k], v);
                v = tanh(v);
            }
            const double e = warp_sum(w2 * v);
            if (lane == 0) A.EA[i] = b2[0] + e;
            if (lane < h2) Dl2[lane] = w2 * (1.0 - v * v);
            __syncwarp();
            if (lane < h1) {
                double g = 0.0;
#pragma unroll 8
                for (int m = 0; m < h2; m++) g = fma(Dl2[m], W1[m * h1 + lane], g);
                Dl1[lane] = g * (1.0 - H1[lane] * H1[lane]);
            } else if (lane == h1) {
                Dl1[lane] = 0.0;
            }
        }
        group_sync<WPA>();
        if (A.mode == MB_MODE_ENERGY) return;
        for (int l = tid; l < D; l += NT) {
            const double2 *w = reinterpret_cast<const double2 *>(w0 + (size_t)l * T.wrow);
            double g = 0.0;
            if (h1 <= 16) {
                double2 r[8];
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (2 * k < h1) r[k] = w[k];
                /* an odd h1's last pair holds off[l], against Dl1[h1] = 0 */
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (2 * k < h1) {
                        const double2 d = reinterpret_cast<const double2 *>(Dl1)[k];
                        g = fma(d.y, r[k].y, fma(d.x, r[k].x, g));
                    }
            } else {
                for (int k = 0; k < h1; k++) g = fma(Dl1[k], w0[(size_t)l * T.wrow + k], g);
            }
            s.G[l] = g;
        }
    } else {
        for (int l = tid; l < D; l += NT) s.G[l] = A.G[(size_t)i * D + l];
    }
    group_sync<WPA>();

    /* ---- dE/dG by grid cell, and the reverse pair terms with the species-0 parameters ---- */
    for (int cell = tid; cell < 64; cell += NT) {
        const int f0 = T.cell_fn[cell];
        const int f1 = f0 >= 0 ? T.fn_next[f0] : -1;
        const double pz = P.powz[(cell & 7) >> 1];
        int b = 0;
        for (int al = 0; al < ns; al++)
            for (int be = al; be < ns; be++, b++) {
                const double *g = s.G + P.ind4[al * al + be * be];
                double v = f0 >= 0 ? g[f0] : 0.0;
                for (int f = f1; f >= 0; f = T.fn_next[f]) v += g[f];
                s.grid[64 * b + cell] = v * pz;
            }
    }
    double fi[3] = {0.0, 0.0, 0.0}, vr[6] = {0, 0, 0, 0, 0, 0};
    /* lane = (neighbour mod 4, function mod 8) as in the forward sums */
    for (int t0 = 4 * warp; t0 < n; t0 += 4 * WPA) {
        const int t = min(t0 + (lane >> 3), n - 1);
        const double *d = s.row + TRI_ROW * t;
        const double r = d[7], f2 = d[5], df2 = d[6] * r;
        const int v = (t >= o1) + (t >= o2);
        const double *g = s.G + (v == 0 ? P.ind2[0] : v == 1 ? P.ind2[1] : P.ind2[2]);
        double cpair = 0.0;
        for (int f = lane & 7; f < ng2; f += 8) {
            const double x = r - P.d_rs[f], eta = P.d_eta2[f];
            cpair += g[f] * exp(-eta * x * x) * (-2.0 * eta * x * f2 + df2);
        }
        cpair += __shfl_xor_sync(FULL, cpair, 1);
        cpair += __shfl_xor_sync(FULL, cpair, 2);
        cpair += __shfl_xor_sync(FULL, cpair, 4);
        const int q = lane & 7;
        if (t0 + (lane >> 3) < n && q < 4) {
            s.Fnb[4 * t + q] = q < 3 ? -cpair * d[3] * d[q] : 0.0;
            for (int w = 1; w < WPA; w++) s.Fnb[4 * (cap * w + t) + q] = 0.0;
        }
    }
    if (A.urep > 0.0)
        for (int t = tid; t < n; t += NT) {
            const double *d = s.row + TRI_ROW * t;
            const int v = (t >= o1) + (t >= o2);
            const double r = d[7], R = P.rm[s0] + P.rm[abs_species(s0, v, ns)];
            if (r < R) {
                /* CELL_UREP on the ordered pair (i, j): force on i only (src/cmod.c:100-112) */
                double fu, dfu;
                fcut_d(R, r, fu, dfu);
                const double tu = -2.0 * A.urep * R / (r * r) * (-fu / r + dfu);
                fi[0] -= tu * d[0]; fi[1] -= tu * d[1]; fi[2] -= tu * d[2];
                vr[0] += 0.5 * tu * d[0] * d[0]; vr[1] += 0.5 * tu * d[1] * d[1]; vr[2] += 0.5 * tu * d[2] * d[2];
                vr[3] += 0.5 * tu * d[0] * d[1]; vr[4] += 0.5 * tu * d[1] * d[2]; vr[5] += 0.5 * tu * d[2] * d[0];
            }
        }
    group_sync<WPA>();

    /* ---- reverse triplet terms: 32 list entries a round, an entry a lane.
     * The force on j is -(p1 d_j + sc d_k), on k -(p2 d_k + sc d_j), so a run
     * of entries with one stripe of rows and 16 columns is three 8 x 16 tiles:
     * sum_b sc_ab d_b, sum_a sc_ab d_a and the row and column sums of p1 and p2
     * are products of the tiles with the displacements, done on the FP64 tensor
     * cores and added to the warp's own Fnb with plain
     * loads and stores.  (Shared FP64 atomics are compare-and-swap loops: six
     * of them and a segmented warp sum per triplet were a third of the reverse
     * pass.)  The force on i is minus the sum of its neighbours'. ---- */
    {
        double2 *Fw = reinterpret_cast<double2 *>(s.Fnb + 4 * cap * warp) + (lane & 1);
        double *tile = s.tile + warp * 24 * TRI_TS;
        double2 *ztile = reinterpret_cast<double2 *>(tile) + lane;
        const double *tr = tile + TRI_TS * (lane >> 2) + (lane & 3), *tc = tile + TRI_TS * (lane & 3) + (lane >> 2);
        const int m4 = lane >> 2, k4 = lane & 3;
        const bool xyz = m4 < 3;                    /* mma columns 0-2: displacements */
        const double one = m4 == 3 ? 1.0 : 0.0;     /* column 3: sums of p1 and p2 */
        const double *rx = s.row + (xyz ? m4 : 0);
        const double2 *rq = reinterpret_cast<const double2 *>(s.row) + (lane & 1);
#pragma unroll
        for (int q = 0; q < 8; q++)
            if (q < 7 || lane < 16) ztile[q * 32] = make_double2(0.0, 0.0);
        __syncwarp();
        int eb[MB_MAX_BLOCKS - 1];
#pragma unroll
        for (int k = 0; k < MB_MAX_BLOCKS - 1; k++) eb[k] = k + 1 < nblk ? bnd[k + 1] : 0x7fffffff;
        for (int base = 0; base < pos; base += 32) {
            const int t = base + lane;
            const unsigned ent = t < pos ? tl[t] : TRI_NONE;
            const bool valid = ent != TRI_NONE;
            const unsigned ab = valid ? ent : 0u; /* padding lanes evaluate entry (0, 0) and add nothing */
            const int a = (int)(ab & 0xffu), b = (int)(ab >> 8);
            int blk = 0;
#pragma unroll
            for (int k = 0; k < MB_MAX_BLOCKS - 1; k++) blk += t >= eb[k];
            const double *grid = s.grid + 64 * min(blk, nblk - 1);
            const double2 *pa = reinterpret_cast<const double2 *>(s.row + TRI_ROW * a);
            const double2 *pb = reinterpret_cast<const double2 *>(s.row + TRI_ROW * b);
            const double2 a0 = pa[0], a1 = pa[1], a2 = pa[2], q0 = pb[0], q1 = pb[1], q2 = pb[2];
            const double ha = pa[3].x, hb = pb[3].x;
            const double wx = q0.x - a0.x, wy = q0.y - a0.y, wz = q1.x - a1.x;
            const double s3 = wx * wx + wy * wy + wz * wz;
            const double ir12 = a1.y * q1.y;
            const double c = (a0.x * q0.x + a0.y * q0.y + a1.x * q1.x) * ir12;
            double E[8], lz[NZL], lzp[NZL];
            tri_exp<NE, EXP>(tab, ne, a2.x + q2.x + s3, E);
            tri_angular<STD>(P, c, lz, lzp);
            double Q = 0.0, Qe = 0.0, Qc = 0.0, eta[8];
#pragma unroll
            for (int e = 0; e < NE; e += 2) {
                const double2 x = reinterpret_cast<const double2 *>(tab.eta)[e / 2];
                eta[e] = x.x;
                eta[e + 1] = x.y;
            }
#pragma unroll
            for (int e = 0; e < NE; e++) {
                double u = 0.0, v = 0.0;
#pragma unroll
                for (int zl = 0; zl < NZL; zl += 2) {
                    if (STD && e < MB_TRI_LOW && zl >= 4) break;
                    const double2 cg = *reinterpret_cast<const double2 *>(grid + e * NZL + zl);
                    u = fma(cg.y, lz[zl + 1], fma(cg.x, lz[zl], u));
                    v = fma(cg.y, lzp[zl + 1], fma(cg.x, lzp[zl], v));
                }
                const double Eu = E[e] * u;
                Q += Eu;
                Qe = fma(eta[e], Eu, Qe);
                Qc = fma(E[e], v, Qc);
            }
            /* legs: f = fc(r), h = fc'(r)/r (i-j: a, i-k: b, j-k: 3); with
             * T = 2 f_a f_b f_3 sum: dT/dr / r of each leg, and dT/dcos */
            const double2 fh = tri_fh(tab, fma(s3, T.sv, -1.0));
            const double fab = 2.0 * a2.y * q2.y, Af = fab * fh.x, Y = 2.0 * Af * Qe, f3Q = 2.0 * fh.x * Q;
            const double Tc = Af * Qc, tcc = Tc * c;
            const double a3 = fab * fh.y * Q - Y;
            const double p1 = ha * q2.y * f3Q - Y - tcc * a1.y * a1.y + a3;
            const double p2 = a2.y * hb * f3Q - Y - tcc * q1.y * q1.y + a3;
            const double sc = Tc * ir12 - a3;

            /* column number among the warp's own columns */
            const int col = (((b >> 2) / WPA) << 2) | (b & 3);
            unsigned rem = __ballot_sync(FULL, valid);
            while (rem) {
                const int first = __shfl_sync(FULL, (a & ~7) | (col << 8), __ffs(rem) - 1);
                const int a0r = first & 0xff, c0 = first >> 8;
                const unsigned ra = (unsigned)(a - a0r), cc = (unsigned)(col - c0);
                const bool mine = ((rem >> lane) & 1u) && ra < 8u && cc < 16u;
                double *o = tile + TRI_TS * ra + cc;
                if (mine) {
                    o[0] = sc;
                    o[8 * TRI_TS] = p1;
                    o[16 * TRI_TS] = p2;
                }
                rem &= ~__ballot_sync(FULL, mine);
                const bool wide = __any_sync(FULL, mine && cc >= 8u);
                __syncwarp();
                /* operands: the rows (a) and columns (b) of the tile; past the end
                 * of the list the tile holds zeros and any row of the atom will do */
                double da[2], ea0 = 0.0, ea1 = 0.0;
#pragma unroll
                for (int h = 0; h < 2; h++)
                    da[h] = xyz ? rx[TRI_ROW * min(a0r + 4 * h + k4, n - 1)] : 0.0;
#pragma unroll
                for (int ct = 0; ct < 2; ct++) {
                    if (ct == 1 && !wide) break;
                    double eb0 = 0.0, eb1 = 0.0;
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int c = c0 + 8 * ct + 4 * h + k4, kb = (((c >> 2) * WPA + warp) << 2) | (c & 3);
                        const double db = xyz ? rx[TRI_ROW * min(kb, n - 1)] : 0.0;
                        dmma884(ea0, ea1, tr[8 * ct + 4 * h], db);
                        dmma884(ea0, ea1, tr[8 * ct + 4 * h + 8 * TRI_TS], one);
                        dmma884(eb0, eb1, tc[8 * ct + 4 * h * TRI_TS], da[h]);
                        dmma884(eb0, eb1, tc[8 * ct + (4 * h + 16) * TRI_TS], one);
                    }
                    /* lane 4 m holds x, y of column m, lane 4 m + 1 z and the sum of p2
                     * (its second value goes to the row's unused fourth word) */
                    const double pb = __shfl_sync(FULL, eb1, lane | 1);
                    const int c = c0 + 8 * ct + m4, br = (((c >> 2) * WPA + warp) << 2) | (c & 3);
                    if (k4 < 2 && br < n) {
                        const double2 d = rq[(TRI_ROW / 2) * br], f = Fw[2 * br];
                        Fw[2 * br] = make_double2(f.x - fma(pb, d.x, eb0), f.y - fma(pb, d.y, eb1));
                    }
                    __syncwarp();
                }
                {
                    const double pa = __shfl_sync(FULL, ea1, lane | 1);
                    const int ar = a0r + m4;
                    if (k4 < 2 && ar < n) {
                        const double2 d = rq[(TRI_ROW / 2) * ar], f = Fw[2 * ar];
                        Fw[2 * ar] = make_double2(f.x - fma(pa, d.x, ea0), f.y - fma(pa, d.y, ea1));
                    }
                    /* the tile is left as zeros */
                    if (mine) o[0] = o[8 * TRI_TS] = o[16 * TRI_TS] = 0.0;
                    __syncwarp();
                }
            }
        }
    }
    group_sync<WPA>();

    /* neighbour forces out; the virial of atom i's energy is every neighbour
     * force times its displacement */
    const double2 *F4 = reinterpret_cast<const double2 *>(s.Fnb);
    for (int t = tid; t < n; t += NT) {
        const double *d = s.row + TRI_ROW * t;
        double2 f0 = F4[2 * t], f1 = F4[2 * t + 1];
        for (int w = 1; w < WPA; w++) {
            const double2 g0 = F4[2 * (cap * w + t)], g1 = F4[2 * (cap * w + t) + 1];
            f0.x += g0.x;
            f0.y += g0.y;
            f1.x += g1.x;
        }
        const double fx = f0.x, fy = f0.y, fz = f1.x;
        const int j = s.j[t];
        atomicAdd(&A.F[3 * j], fx);
        atomicAdd(&A.F[3 * j + 1], fy);
        atomicAdd(&A.F[3 * j + 2], fz);
        fi[0] -= fx; fi[1] -= fy; fi[2] -= fz;
        vr[0] += fx * d[0]; vr[1] += fy * d[1]; vr[2] += fz * d[2];
        vr[3] += fx * d[1]; vr[4] += fy * d[2]; vr[5] += fz * d[0];
    }
    {
        /* the atom's force and virial: warp sums, then the warps in a fixed order */
        double v[9] = {fi[0], fi[1], fi[2], vr[0], vr[1], vr[2], vr[3], vr[4], vr[5]};
#pragma unroll
        for (int k = 0; k < 9; k++) v[k] = warp_sum(v[k]);
        if (WPA > 1) {
            if (lane == 0)
                for (int k = 0; k < 9; k++) s.fin[warp * 9 + k] = v[k];
            group_sync<WPA>();
            if (tid == 0)
                for (int k = 0; k < 9; k++) {
                    double t = 0.0;
                    for (int w = 0; w < WPA; w++) t += s.fin[w * 9 + k];
                    v[k] = t;
                }
        }
        if (tid == 0) {
            atomicAdd(&A.F[3 * i], v[0]);
            atomicAdd(&A.F[3 * i + 1], v[1]);
            atomicAdd(&A.F[3 * i + 2], v[2]);
            for (int k = 0; k < 6; k++) A.vir[(size_t)i * 6 + k] = v[3 + k];
        }
    }
}

/* ------------------------------------------------------------------ */
/* forward-mode derivative of the descriptors                           */
/* ------------------------------------------------------------------ */

/* dG = (dG/dx) . dx for a displacement field dx[3N] of the atoms and a
 * homogeneous deformation eps[3][3] of every neighbour displacement
 * (d -> d + eps d): the tangent of the descriptor map that the reference
 * materialises as the derivative blocks Fn (dG_j/dx_i) and Sn (dG/dstrain)
 * of PRS_BP (src/nprs.c:567-770), with the same species-0 derivative
 * parameters.  A unit dx on atom m and axis q gives column q of every
 * Fn block of m; eps = e_a e_b^T gives the (a, b) strain column.
 * One warp per atom (one per CTA); every term is added to the atom's
 * descriptor row in shared memory. */
struct JvpArgs {
    int N, cap;
    const int *nn, *nj;
    const double4 *nd;
    const int *spc;
    const mb_params *params;
    const double *dx;
    double eps[9];
    double *dG;
};

__global__ void __launch_bounds__(32) k_jvp(JvpArgs A) {
    extern __shared__ __align__(16) char jsm[];
    const int i = blockIdx.x, lane = threadIdx.x;
    if (i >= A.N) return;
    const mb_params &P = *A.params;
    const int D = P.D, ns = P.nspc, ng2 = P.ng2, cap = A.cap;
    double4 *d = reinterpret_cast<double4 *>(jsm);
    double *dd = reinterpret_cast<double *>(d + cap); /* [cap][3] tangent of each displacement */
    double *g = dd + 3 * cap;                         /* [D] */
    int *rel = reinterpret_cast<int *>(g + D);        /* [cap] relative species */
    const int n = A.nn[i], s0 = A.spc[i];
    for (int t = lane; t < D; t += 32) g[t] = 0.0;
    for (int t = lane; t < n; t += 32) {
        const size_t o = (size_t)i * cap + t;
        const int j = A.nj[o];
        const double4 v = A.nd[o];
        d[t] = v;
        rel[t] = (A.spc[j] - s0 + ns) % ns;
        const double e[3] = {A.eps[0] * v.x + A.eps[1] * v.y + A.eps[2] * v.z,
                             A.eps[3] * v.x + A.eps[4] * v.y + A.eps[5] * v.z,
                             A.eps[6] * v.x + A.eps[7] * v.y + A.eps[8] * v.z};
        for (int q = 0; q < 3; q++) dd[3 * t + q] = A.dx[3 * j + q] - A.dx[3 * i + q] + e[q];
    }
    __syncwarp();
    /* G2: d/dr [fc(r) exp(-eta (r - rs)^2)] dr, dr = d . dd / r */
    for (int t = lane; t < n; t += 32) {
        const double4 v = d[t];
        const double r = v.w, dr = (v.x * dd[3 * t] + v.y * dd[3 * t + 1] + v.z * dd[3 * t + 2]) / r;
        double f2, df2;
        fcut_d(P.d_rc2, r, f2, df2);
        double *gg = g + P.ind2[rel[t]];
        for (int f = 0; f < ng2; f++) {
            const double x = r - P.d_rs[f], eta = P.d_eta2[f];
            atomicAdd(gg + f, exp(-eta * x * x) * (-2.0 * eta * x * f2 + df2) * dr);
        }
    }
    /* G4 over the pairs a < b of the list (the reference's triplets) */
    const int ne = P.ne, nzl = P.nzl;
    for (int a = 0; a + 1 < n; a++) {
        const double4 d1 = d[a];
        const double r1 = d1.w;
        if (!(r1 < P.d_rc4)) continue;
        const double e1x = dd[3 * a], e1y = dd[3 * a + 1], e1z = dd[3 * a + 2];
        const double dr1 = (d1.x * e1x + d1.y * e1y + d1.z * e1z) / r1;
        double f1, df1;
        fcut_d(P.d_rc4, r1, f1, df1);
        for (int b = a + 1 + lane; b < n; b += 32) {
            const double4 d2 = d[b];
            const double r2 = d2.w;
            const double wx = d2.x - d1.x, wy = d2.y - d1.y, wz = d2.z - d1.z;
            const double r3s = wx * wx + wy * wy + wz * wz;
            if (!(r2 < P.d_rc4 && r3s < P.d_rc4sq)) continue;
            const double r3 = sqrt(r3s);
            const double e2x = dd[3 * b], e2y = dd[3 * b + 1], e2z = dd[3 * b + 2];
            const double dr2 = (d2.x * e2x + d2.y * e2y + d2.z * e2z) / r2;
            const double dr3 = (wx * (e2x - e1x) + wy * (e2y - e1y) + wz * (e2z - e1z)) / r3;
            const double c = (d1.x * d2.x + d1.y * d2.y + d1.z * d2.z) / (r1 * r2);
            const double dc = (e1x * d2.x + e1y * d2.y + e1z * d2.z + d1.x * e2x + d1.y * e2y + d1.z * e2z) / (r1 * r2) -
                              c * (dr1 / r1 + dr2 / r2);
            double f2, df2, f3, df3;
            fcut_d(P.d_rc4, r2, f2, df2);
            fcut_d(P.d_rc4, r3, f3, df3);
            const double Af = 2.0 * f1 * f2 * f3;
            const double dA = 2.0 * (df1 * dr1 * f2 * f3 + f1 * df2 * dr2 * f3 + f1 * f2 * df3 * dr3);
            const double rr = r1 * r1 + r2 * r2 + r3s, drr = r1 * dr1 + r2 * dr2 + r3 * dr3;
            double sv[MB_MAXE], tv[MB_MAXE];
            for (int e = 0; e < ne; e++) {
                const double eta = P.d_eta4[e], E = exp(-eta * rr);
                sv[e] = dA * E + Af * E * (-2.0 * eta * drr);
                tv[e] = Af * E * dc;
            }
            double lz[MB_MAXZL], lzp[MB_MAXZL];
            for (int k = 0; k < MB_MAXZL; k++) lz[k] = lzp[k] = 0.0;
            angular<8, 4>(P, c, lz, lzp);
            /* angular<8, 4> lays (zeta, lambda) out as z * 4 + l */
            const int va = rel[a], vb = rel[b];
            const int lo = va < vb ? va : vb, hi = va < vb ? vb : va;
            double *gg = g + P.ind4[lo * lo + hi * hi];
            for (int f = 0; f < P.ng4; f++) {
                const int e = P.g4_e[f], zl = (P.g4_zl[f] / P.nlam) * 4 + P.g4_zl[f] % P.nlam;
                atomicAdd(gg + f, sv[e] * lz[zl] + tv[e] * lzp[zl]);
            }
        }
    }
    (void)nzl;
    __syncwarp();
    for (int t = lane; t < D; t += 32) A.dG[(size_t)i * D + t] = g[t];
}

/* ------------------------------------------------------------------ */
/* reductions                                                          */
/* ------------------------------------------------------------------ */

/* Atoms per CTA of the multi-CTA reductions: chunks of at least 512 atoms,
 * at most MB_RED_MAXB CTAs; nparts = 0 runs one CTA over all atoms. */
__host__ __device__ inline int red_chunk(int N, int nparts) {
    if (nparts <= 0) return N > 0 ? N : 1;
    const int c = (N + MB_RED_MAXB - 1) / MB_RED_MAXB;
    return c > 512 ? c : 512;
}

/* Sum of acc[0..K-1] over the CTA's 256 threads into red[k][0] (warp trees,
 * then the 8 warps in order). */
template <int K>
__device__ __forceinline__ void block_tree(double (*red)[8], const double *acc, int t) {
    const int lane = t & 31, warp = t >> 5;
#pragma unroll
    for (int k = 0; k < K; k++) {
        const double v = warp_sum(acc[k]);
        if (lane == 0) red[k][warp] = v;
    }
    __syncthreads();
    if (t < K) {
        double s = 0.0;
        for (int w = 0; w < 8; w++) s += red[t][w];
        red[t][0] = s;
    }
    __syncthreads();
}

/* After block_tree: CTA partials go to part[cta][0..K-1]; returns true in
 * the threads of warp 0 of the CTA that finished last, all of which then hold
 * the sums of the partials in tot[] (lanes over CTAs, then a tree: a fixed
 * order), and the ticket is reset. */
template <int K>
__device__ __forceinline__ bool last_cta(double (*red)[8], double *part, unsigned *ticket, double *tot, int t) {
    __shared__ bool is_last;
    const int nb = gridDim.x;
    if (nb == 1) {
        for (int k = 0; k < K; k++) tot[k] = red[k][0];
        return t < 32;
    }
    if (t < K) part[blockIdx.x * 8 + t] = red[t][0];
    __syncwarp();
    if (t == 0) {
        __threadfence();
        is_last = atomicAdd(ticket, 1u) == (unsigned)(nb - 1);
    }
    __syncthreads();
    if (!is_last || t >= 32) return false;
    __threadfence();
    const volatile double *vp = part;
    for (int k = 0; k < K; k++) {
        double s = 0.0;
        for (int c = t; c < nb; c += 32) s += vp[c * 8 + k];
        tot[k] = warp_sum(s);
    }
    if (t == 0) *ticket = 0u;
    return true;
}

/* where a pass's results go on the host (pinned memory; any may be NULL) */
struct HostOut {
    double *out;       /* [16], as the device's */
    int *status;       /* [4] */
    double *F, *X, *EA;
};

/* out[0]=E, out[1]=H, out[2..7]=U: every CTA reduces a fixed chunk of atoms
 * (threads strided, then a tree) and zeroes the chunk's force components
 * below 1e-8 (src/cmod.c:177-184); the last CTA adds the partials.  For a pass
 * on host arrays it also stores the results into pinned host memory (forces,
 * wrapped positions, atom energies, totals, status): one launch in the place
 * of five copies.  Every sum has a fixed order, so results are reproducible. */
__global__ void __launch_bounds__(256) k_finalize(int N, int mode, double pV, const double *EA, const double *EU,
                                                  const double *vir, double *F, double *out, double *part,
                                                  unsigned *ticket, const double *X, const int *status, HostOut ho) {
    __shared__ double red[7][8];
    const int t = threadIdx.x, chunk = red_chunk(N, part ? 1 : 0);
    const int lo = blockIdx.x * chunk, hi = min(N, lo + chunk);
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    for (int i = lo + t; i < hi; i += 256) {
        const double ea = EA[i];
        acc[0] += ea + EU[i];
        if (ho.EA) ho.EA[i] = ea;
        if (mode != MB_MODE_ENERGY)
            for (int k = 0; k < 6; k++) acc[1 + k] += vir[(size_t)i * 6 + k];
    }
    if (mode == MB_MODE_EFS || (mode == MB_MODE_VJP && ho.F))
        for (int i = 3 * lo + t; i < 3 * hi; i += 256) {
            double f = F[i];
            if (mode == MB_MODE_EFS && fabs(f) < 1e-8) F[i] = f = 0.0;
            if (ho.F) ho.F[i] = f;
        }
    if (ho.X)
        for (int i = 3 * lo + t; i < 3 * hi; i += 256) ho.X[i] = X[i];
    block_tree<7>(red, acc, t);
    double tot[7];
    if (last_cta<7>(red, part, ticket, tot, t) && t < 8) {
        /* E, H = E + pV, U (lane 0, 1, 2..7) */
        double v = tot[0];
        for (int k = 1; k < 7; k++)
            if (t == k + 1) v = tot[k];
        if (t == 1) v = tot[0] + pV;
        if (t >= 2 && mode == MB_MODE_EFS && fabs(v) < 1e-8) v = 0.0;
        out[t] = v;
        if (ho.out) {
            ho.out[t] = v;
            ho.out[8 + t] = out[8 + t];
        }
        if (ho.status && t < 4) ho.status[t] = status[t];
    }
}

/* ------------------------------------------------------------------ */
/* NVT step (src/cmod.c:403-407, 440-453)                              */
/* ------------------------------------------------------------------ */

/* K = 1/2 sum m v^2 (CTA chunks, then the partials in CTA order), then
 * xi += dt/tau^2 (2K/(3NT) - 1).  out[8] = K, out[9] = xi;
 * trace[2*step] = H, trace[2*step+1] = K with the step index kept in
 * out[10] and advanced here, so that a captured chunk of steps can be
 * replayed unchanged. */
__global__ void __launch_bounds__(256) k_nvt_thermostat(int N, const double *V, const int *spc, const double *mass,
                                                        double dt, double tau, double T, double *out, double *trace,
                                                        int capTrace, double *part, unsigned *ticket) {
    __shared__ double red[1][8];
    const int t = threadIdx.x, chunk = red_chunk(N, part ? 1 : 0);
    const int lo = blockIdx.x * chunk, hi = min(N, lo + chunk);
    double k[1] = {0.0};
    for (int i = lo + t; i < hi; i += 256) {
        double m = mass[spc[i]];
        k[0] += m * V[3 * i] * V[3 * i] + m * V[3 * i + 1] * V[3 * i + 1] + m * V[3 * i + 2] * V[3 * i + 2];
    }
    block_tree<1>(red, k, t);
    double tot[1];
    if (last_cta<1>(red, part, ticket, tot, t) && t == 0) {
        double K = 0.5 * tot[0];
        double fs = 1.0 / (tau * tau) * (2.0 * K / ((3.0 * (double)N) * T) - 1.0);
        const int step = (int)out[10];
        out[8] = K;
        out[9] += dt * fs;
        out[10] = (double)(step + 1);
        if (step >= 0 && step < capTrace) {
            trace[2 * step] = out[1];
            trace[2 * step + 1] = K;
        }
    }
}

/* the integrator, then (wrap != 0) the step's closing JAR on the moved
 * atom, the same operations as k_wrap in one launch */
__global__ void k_nvt_integrate(int N, double *X, double *V, const double *F, const int *spc, const double *mass,
                                double dt, const double *out, mb_cell c, int wrap, int *status) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    double xi = out[9], m = mass[spc[i]];
    for (int q = 0; q < 3; q++) {
        double v = V[3 * i + q];
        double f = F[3 * i + q] / m - xi * v;
        X[3 * i + q] += v * dt + 0.5 * f * dt * dt;
        V[3 * i + q] = v + f * dt;
    }
    if (wrap) wrap_atom(i, X, c, status);
}

__global__ void k_set_out(double *out, int idx, double v) { out[idx] = v; }

} /* namespace */

/* ------------------------------------------------------------------ */
/* launchers                                                           */
/* ------------------------------------------------------------------ */

/* Shapes of the fused kernel: warps per atom x atoms per block.  One warp
 * per atom keeps many atoms resident per SM (large structures); several
 * warps per atom shorten the latency of small structures. */
struct EfsShape {
    int wpa, apb;
};
static const EfsShape kShapes[] = {{1, 4}, {4, 1}, {8, 1}};
#define EFS_STATIC_SMEM (sizeof(mb_params) + 16) /* k_efs's __shared__ Ps, with alignment slack */
#define TRI_STATIC_SMEM sizeof(mb_tri_tab)        /* k_efs_tri's __shared__ tab */
#define MB_NSHAPES 3
#define MB_MAX_DEVICES_K 64

/* specialised kernel for the reference bases: 7 G4 exponents, 4 zeta, 2 lambda */
static bool efs_fast(const mb_model *m) { return m->P.ne <= 7 && m->P.nz <= 4 && m->P.nlam <= 2; }

/* triplet-list entries per atom group: all candidate pairs when they fit,
 * otherwise at least one row (the capacity) per warp plus slack */
static int tl_entries(int capNB, int wpa) {
    int all = capNB * (capNB - 1) / 2 + 32 * wpa;
    int lim = wpa == 1 ? 2048 : 8192;
    int floor_ = wpa * (capNB + 64);
    int v = all < lim ? all : lim;
    return v > floor_ ? v : floor_;
}

static size_t group_bytes(const mb_model *m, int capNB, int wpa) {
    bool fast = efs_fast(m);
    int ne = fast ? 7 : MB_MAXE;
    int cells = fast ? 7 * 8 : MB_MAXE * 8 * 4;
    return (efs_smem_bytes(capNB, m->P.D, ne, m->P.ng2, cells, wpa, tl_entries(capNB, wpa), fast ? 1 : 0) + 15) &
           ~(size_t)15;
}

extern "C" size_t mbk_efs_smem(const mb_model *m, int capNB, int shape) {
    return group_bytes(m, capNB, kShapes[shape].wpa) * kShapes[shape].apb;
}

extern "C" int mbk_wrap(mb_dev *d, int N, const mb_cell *c, void *stream, long *launches) {
    d->f_clear = 0;
    if (c->ND <= 0 || N <= 0) return 0;
    k_wrap<<<(N + 127) / 128, 128, 0, (cudaStream_t)stream>>>(N, d->X, *c, d->status, d->F);
    d->f_clear = 1;
    (*launches)++;
    return (int)cudaGetLastError();
}

extern "C" int mbk_intake(mb_dev *d, int N, const mb_cell *c, const double *hx, const int *hspc, void *stream,
                          long *launches) {
    k_intake<<<(N + 127) / 128, 128, 0, (cudaStream_t)stream>>>(N, hx, *c, hspc, d->X, d->spc, d->status, d->F);
    d->f_clear = 1;
    (*launches)++;
    return (int)cudaGetLastError();
}

extern "C" int mbk_nlist(mb_dev *d, int N, int NM, const mb_cell *c, double rc, void *stream, long *launches) {
    cudaStream_t st = (cudaStream_t)stream;
    double rc2 = rc * rc;
    int warps_per_block = 4;
    int blocks = (N + warps_per_block - 1) / warps_per_block;
    if (c->M[0] > 0) {
        int ncell = c->M[0] * c->M[1] * c->M[2];
        if (N <= CELL_BUILD_MAX && ncell <= CELL_BUILD_MAX) {
            k_cell_build<<<1, 1024, sizeof(int) * (ncell + N), st>>>(N, d->X, *c, ncell, d->cell_of, d->cell_start,
                                                                     d->cell_atoms);
            *launches += 1;
        } else {
            cudaMemsetAsync(d->cell_cnt, 0, sizeof(int) * ncell, st);
            k_cell_bin<<<(N + 127) / 128, 128, 0, st>>>(N, d->X, *c, d->cell_of, d->cell_cnt);
            k_cell_scan<<<1, 1024, 0, st>>>(ncell, d->cell_cnt, d->cell_start);
            cudaMemsetAsync(d->cell_cnt, 0, sizeof(int) * ncell, st);
            k_cell_fill<<<(N + 127) / 128, 128, 0, st>>>(N, d->cell_of, d->cell_start, d->cell_cnt, d->cell_atoms);
            k_cell_sort<<<(ncell + 3) / 4, 128, 0, st>>>(ncell, d->cell_start, d->cell_atoms); /* a warp per cell */
            *launches += 4;
        }
        k_nlist_cell<<<blocks, warps_per_block * 32, 0, st>>>(N, NM, d->capNB, d->X, *c, rc2, d->cell_of,
                                                              d->cell_start, d->cell_atoms, d->nn, d->nj,
                                                              (double4 *)d->nd, d->status);
        *launches += 1;
    } else {
        /* a warp a CTA: few atoms, as many SMs as there are */
        k_nlist_brute<<<N, 32, 0, st>>>(N, NM, d->capNB, d->X, *c, rc2, d->nn, d->nj,
                                                               (double4 *)d->nd, d->status);
        *launches += 1;
    }
    return (int)cudaGetLastError();
}

template <int NE, int NZ, int NLAM, int WPA, int APB>
static int launch_shape(const EfsArgs &a, cudaStream_t st, cudaEvent_t e0, cudaEvent_t e1) {
    auto kern = k_efs<NE, NZ, NLAM, WPA, APB>;
    size_t smem = a.smem_group * APB;
    /* the shared-memory opt-in is a per-device attribute of the function: set
     * once per device, to the most there is, since a limit of one handle's own
     * size could fall between another thread's limit and its launch */
    static bool configured[MB_MAX_DEVICES_K] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MB_MAX_DEVICES_K) return (int)cudaErrorInvalidDevice;
    /* the 48 KB default and the 227 KB opt-in limit both count the kernel's
     * static shared block (the staged mb_params) as well as the dynamic part */
    if (smem + EFS_STATIC_SMEM > 227 * 1024) return (int)cudaErrorInvalidConfiguration;
    if (smem + EFS_STATIC_SMEM > 48 * 1024 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             227 * 1024 - (int)EFS_STATIC_SMEM);
        if (e != cudaSuccess) return (int)e;
        configured[dev] = true;
    }
    if (e0) mbk_record(e0, st);
    kern<<<(a.N + APB - 1) / APB, WPA * 32 * APB, smem, st>>>(a);
    if (e1) mbk_record(e1, st);
    return (int)cudaGetLastError();
}

static int launch_any(const mb_model *m, int shape, EfsArgs a, cudaStream_t st, cudaEvent_t e0, cudaEvent_t e1) {
    a.smem_group = group_bytes(m, a.cap, kShapes[shape].wpa);
    a.tl_cap = tl_entries(a.cap, kShapes[shape].wpa);
    if (efs_fast(m)) {
        switch (shape) {
            case 0: return launch_shape<7, 4, 2, 1, 4>(a, st, e0, e1);
            case 1: return launch_shape<7, 4, 2, 4, 1>(a, st, e0, e1);
            default: return launch_shape<7, 4, 2, 8, 1>(a, st, e0, e1);
        }
    }
    if (m->P.nz > 8 || m->P.nlam > 4) return (int)cudaErrorInvalidValue;
    switch (shape) {
        case 0: return launch_shape<MB_MAXE, 8, 4, 1, 4>(a, st, e0, e1);
        case 1: return launch_shape<MB_MAXE, 8, 4, 4, 1>(a, st, e0, e1);
        default: return launch_shape<MB_MAXE, 8, 4, 8, 1>(a, st, e0, e1);
    }
}

/* ---- fused triplet kernel ---- */

/* 1 when a pass can run on k_efs_tri: the basis qualifies (mb_tri) and the
 * neighbour capacity is within what its lists and sort hold */
extern "C" int mbk_tri_usable(const mb_dev *d, const mb_model *m) {
    return m->T.ok && d->tri_w && d->capNB <= MB_TRI_MAX_CAP ? 1 : 0;
}

/* One warp per atom for large structures, several where the atoms alone do
 * not fill the SMs; the autotuner times them. */
static const EfsShape kTriShapes[] = {{1, 4}, {1, 2}, {2, 1}, {4, 1}, {8, 1}};
#define MB_NTRISHAPES 5

/* list entries of a warp and shared memory of an atom, for capacity cap */
extern "C" int mbk_tri_list(int cap, int warps) { return tri_list(cap, warps); }
extern "C" size_t mbk_tri_smem(int cap, int D, int ns, int ng2, int warps) {
    return tri_smem_bytes(cap, D, ns, ng2, warps);
}

static size_t tri_group_bytes(const mb_model *m, int capNB, int wpa) {
    return tri_smem_bytes(capNB, m->P.D, m->P.nspc, m->P.ng2, wpa);
}

template <int NE, int WPA, int APB, bool STD, bool EXP>
static int launch_tri(const TriArgs &a, cudaStream_t st) {
    auto kern = k_efs_tri<NE, WPA, APB, STD, EXP>;
    const size_t smem = a.smem_group * APB;
    static bool configured[MB_MAX_DEVICES_K] = {false}; /* as in launch_shape */
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MB_MAX_DEVICES_K) return (int)cudaErrorInvalidDevice;
    if (smem + TRI_STATIC_SMEM > 227 * 1024) return (int)cudaErrorInvalidConfiguration;
    if (smem + TRI_STATIC_SMEM > 48 * 1024 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             227 * 1024 - (int)TRI_STATIC_SMEM);
        if (e != cudaSuccess) return (int)e;
        configured[dev] = true;
    }
    kern<<<(a.N + APB - 1) / APB, WPA * 32 * APB, smem, st>>>(a);
    return (int)cudaGetLastError();
}

template <int NE, bool STD, bool EXP>
static int launch_tri_shape(int shape, const TriArgs &a, cudaStream_t st) {
    switch (shape) {
        case 0: return launch_tri<NE, 1, 4, STD, EXP>(a, st);
        case 1: return launch_tri<NE, 1, 2, STD, EXP>(a, st);
        case 2: return launch_tri<NE, 2, 1, STD, EXP>(a, st);
        case 3: return launch_tri<NE, 4, 1, STD, EXP>(a, st);
        default: return launch_tri<NE, 8, 1, STD, EXP>(a, st);
    }
}

/* k_efs_tri in shape `shape`; the events (if any) bracket it */
static int launch_tri_pass(const mb_model *m, int shape, TriArgs &a, cudaStream_t st, cudaEvent_t e0, cudaEvent_t e1) {
    a.smem_group = tri_group_bytes(m, a.cap, kTriShapes[shape].wpa);
    a.tlw = tri_list(a.cap, kTriShapes[shape].wpa);
    if (e0) mbk_record(e0, st);
    int rc;
    if (m->T.steep)
        rc = m->T.std ? launch_tri_shape<8, true, true>(shape, a, st) : launch_tri_shape<8, false, true>(shape, a, st);
    else if (m->T.std)
        rc = m->P.ne <= 7 ? launch_tri_shape<7, true, false>(shape, a, st) : launch_tri_shape<8, true, false>(shape, a, st);
    else
        rc = launch_tri_shape<8, false, false>(shape, a, st);
    if (e1) mbk_record(e1, st);
    return rc;
}

/* warps per atom and atoms per CTA of shape `shape` of k_efs_tri (tri != 0)
 * or of k_efs */
extern "C" int mbk_shape_dims(int tri, int shape, int *wpa, int *apb) {
    if (shape < 0 || shape >= (tri ? MB_NTRISHAPES : MB_NSHAPES)) return 1;
    const EfsShape &e = tri ? kTriShapes[shape] : kShapes[shape];
    *wpa = e.wpa;
    *apb = e.apb;
    return 0;
}

/* Autotuner: on the first pass of a (mode, size bucket, capacity) the shapes of
 * the kernel it runs on, k_efs_tri's five or k_efs's three, are each timed once
 * (after an untimed launch) and the fastest is kept for later passes of that
 * key. */
static int tune_key(const mb_dev *d, int N, int mode) {
    int bucket = 0;
    while ((1 << bucket) < N) bucket++;
    return (mode << 28) | ((d->tri_on ? 1 : 0) << 26) | (bucket << 20) | (d->capNB & 0xfffff);
}

/* Record a decision; a full table gives up its oldest one, so that a key is
 * not timed again on every call.  The capacity of a handle only grows, and at
 * one capacity there are 4 modes of at most 31 size buckets: the keys in use
 * always fit. */
static void tune_store(mb_dev *d, int key, int val) {
    if (d->tune_n == MB_TUNE_SLOTS) {
        memmove(d->tune_key, d->tune_key + 1, sizeof(int) * (MB_TUNE_SLOTS - 1));
        memmove(d->tune_val, d->tune_val + 1, sizeof(int) * (MB_TUNE_SLOTS - 1));
        d->tune_n--;
    }
    d->tune_key[d->tune_n] = key;
    d->tune_val[d->tune_n++] = val;
}

/* The shape of k_efs_tri for a pass: each is timed once (after an untimed
 * launch) and the fastest kept, recorded as 16 + shape (k_efs, slower at every
 * size measured -- 32 atoms: 73 us against 40; 487: 199 against 64; 4000: 890
 * against 375 -- is not among them; a shape that does not fit is passed over,
 * and up to MB_TRI_MAX_CAP neighbours one warp an atom always does). */
static int tune_tri(mb_dev *d, const mb_model *m, int N, int mode, const TriArgs &a, cudaStream_t st) {
    const int key = tune_key(d, N, mode);
    for (int k = 0; k < d->tune_n; k++)
        if (d->tune_key[k] == key) return d->tune_val[k] - 16;
    int best = 0;
    if (d->tune_fixed >= 0) {
        /* a forced shape is recorded as the decision for this key */
        best = d->tune_fixed < MB_NTRISHAPES ? d->tune_fixed : 0;
    } else {
        TriArgs t = a;
        t.counters = nullptr;
        cudaEvent_t e0, e1;
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        float best_ms = 1e30f;
        for (int sh = 0; sh < MB_NTRISHAPES; sh++) {
            if (tri_group_bytes(m, a.cap, kTriShapes[sh].wpa) * kTriShapes[sh].apb + TRI_STATIC_SMEM > 227 * 1024) continue;
            float ms = 1e30f;
            int bad = 0;
            for (int rep = 0; rep < 2 && !bad; rep++) {
                if (mode == MB_MODE_EFS || mode == MB_MODE_VJP) cudaMemsetAsync(d->F, 0, sizeof(double) * 3 * N, st);
                bad = launch_tri_pass(m, sh, t, st, rep ? e0 : nullptr, rep ? e1 : nullptr);
            }
            if (!bad && cudaEventSynchronize(e1) == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
            if (ms < best_ms) {
                best_ms = ms;
                best = sh;
            }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        cudaGetLastError();
        d->f_clear = 0; /* the trials added to F */
    }
    tune_store(d, key, 16 + best);
    return best;
}

static int tune_shape(mb_dev *d, const mb_model *m, int N, int mode, const EfsArgs &a, cudaStream_t st) {
    int k;
    const int key = tune_key(d, N, mode);
    for (k = 0; k < d->tune_n; k++)
        if (d->tune_key[k] == key) return d->tune_val[k];
    if (d->tune_fixed >= 0) {
        const int v = d->tune_fixed < MB_NSHAPES ? d->tune_fixed : 0;
        tune_store(d, key, v);
        return v;
    }
    EfsArgs t = a;
    t.counters = nullptr;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int best = 0;
    float best_ms = 1e30f;
    for (int sh = 0; sh < MB_NSHAPES; sh++) {
        if (group_bytes(m, a.cap, kShapes[sh].wpa) * kShapes[sh].apb + EFS_STATIC_SMEM > 227 * 1024) continue;
        float ms = 1e30f;
        for (int rep = 0; rep < 2; rep++) {
            if (mode == MB_MODE_EFS || mode == MB_MODE_VJP) cudaMemsetAsync(d->F, 0, sizeof(double) * 3 * N, st);
            if (launch_any(m, sh, t, st, rep ? e0 : nullptr, rep ? e1 : nullptr)) break;
        }
        if (cudaEventSynchronize(e1) == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
        if (ms < best_ms) {
            best_ms = ms;
            best = sh;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaGetLastError();
    tune_store(d, key, best);
    return best;
}

extern "C" int mbk_descriptor_pass(mb_dev *d, const mb_model *m, int N, int mode, double urep, int need_nb_max,
                                   int nb_max, void *stream, long *launches) {
    (void)need_nb_max;
    (void)nb_max;
    cudaStream_t st = (cudaStream_t)stream;
    EfsArgs a;
    a.N = N;
    a.cap = d->capNB;
    a.mode = mode;
    a.urep = urep;
    a.nn = d->nn;
    a.nj = d->nj;
    a.nd = (const double4 *)d->nd;
    a.spc = d->spc;
    a.params = d->params;
    a.weights = d->weights;
    a.EA = d->EA;
    a.EU = d->EU;
    a.G = d->G;
    a.F = d->F;
    a.vir = d->vir;
    a.counters = d->counters;
    a.smem_group = 0;
    if (d->tri_on) {
        TriArgs la;
        la.N = N;
        la.cap = d->capNB;
        la.mode = mode;
        la.tlw = 0;
        la.urep = urep;
        la.nn = d->nn;
        la.nj = d->nj;
        la.nd = (const double4 *)d->nd;
        la.spc = d->spc;
        la.weights = d->weights;
        la.w0 = d->tri_w;
        la.EA = d->EA;
        la.EU = d->EU;
        la.G = d->G;
        la.F = d->F;
        la.vir = d->vir;
        la.counters = d->counters;
        la.smem_group = 0;
        la.P = m->P;
        la.T = m->T;
        const int sh = tune_tri(d, m, N, mode, la, st);
        d->last_shape = 16 + sh;
        cudaEvent_t e0 = 0, e1 = 0;
        if (d->ev_on && d->ev_n < d->ev_cap) {
            e0 = ((cudaEvent_t *)d->ev_pool)[2 * d->ev_n];
            e1 = ((cudaEvent_t *)d->ev_pool)[2 * d->ev_n + 1];
            d->ev_n++;
        }
        if ((mode == MB_MODE_EFS || mode == MB_MODE_VJP) && !d->f_clear)
            cudaMemsetAsync(d->F, 0, sizeof(double) * 3 * N, st);
        d->f_clear = 0;
        const int rc = launch_tri_pass(m, sh, la, st, e0, e1);
        (*launches)++;
        return rc;
    }
    d->f_clear = 0;
    cudaMemsetAsync(d->EU, 0, sizeof(double) * N, st);
    int shape = tune_shape(d, m, N, mode, a, st);
    d->last_shape = shape;
    cudaEvent_t e0 = 0, e1 = 0;
    if (d->ev_on && d->ev_n < d->ev_cap) {
        e0 = ((cudaEvent_t *)d->ev_pool)[2 * d->ev_n];
        e1 = ((cudaEvent_t *)d->ev_pool)[2 * d->ev_n + 1];
        d->ev_n++;
    }
    if (mode == MB_MODE_EFS || mode == MB_MODE_VJP) cudaMemsetAsync(d->F, 0, sizeof(double) * 3 * N, st);
    int rc = launch_any(m, shape, a, st, e0, e1);
    (*launches)++;
    return rc;
}

/* the descriptor tangent for displacements dx[3N] (device) and the
 * deformation eps[9] (host), into dG[N*D] (device) */
extern "C" int mbk_jvp(mb_dev *d, const mb_model *m, int N, const double *dx, const double *eps, double *dG,
                       void *stream, long *launches) {
    if (m->P.nz > 8 || m->P.nlam > 4) return (int)cudaErrorInvalidValue;
    JvpArgs a;
    a.N = N;
    a.cap = d->capNB;
    a.nn = d->nn;
    a.nj = d->nj;
    a.nd = (const double4 *)d->nd;
    a.spc = d->spc;
    a.params = d->params;
    a.dx = dx;
    for (int k = 0; k < 9; k++) a.eps[k] = eps ? eps[k] : 0.0;
    a.dG = dG;
    const size_t smem = sizeof(double4) * d->capNB + sizeof(double) * (3 * (size_t)d->capNB + m->P.D) +
                        sizeof(int) * d->capNB;
    if (smem > 227 * 1024) return (int)cudaErrorInvalidConfiguration;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_jvp, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return (int)e;
    }
    k_jvp<<<N, 32, smem, (cudaStream_t)stream>>>(a);
    (*launches)++;
    return (int)cudaGetLastError();
}

extern "C" int mbk_finalize(mb_dev *d, int N, int mode, double pV, const mb_host_out *host, void *stream,
                            long *launches) {
    const int chunk = red_chunk(N, d->part ? 1 : 0), nb = (N + chunk - 1) / chunk;
    HostOut ho = {nullptr, nullptr, nullptr, nullptr, nullptr};
    if (host) ho = {host->out, host->status, mode == MB_MODE_ENERGY ? nullptr : host->F, host->X, host->EA};
    k_finalize<<<nb > 0 ? nb : 1, 256, 0, (cudaStream_t)stream>>>(N, mode, pV, d->EA, d->EU, d->vir, d->F, d->out,
                                                                   d->part, d->ticket, d->X, d->status, ho);
    (*launches)++;
    return (int)cudaGetLastError();
}

extern "C" int mbk_nvt_update(mb_dev *d, const mb_model *m, int N, double dt, double tau, double T,
                              const mb_cell *c, void *stream, long *launches) {
    cudaStream_t st = (cudaStream_t)stream;
    (void)m;
    /* masses by species live after the weights in the parameter upload (see mb_core.c) */
    const double *mass = d->weights + m->weights_len;
    const int chunk = red_chunk(N, d->part ? 1 : 0), nb = (N + chunk - 1) / chunk;
    k_nvt_thermostat<<<nb > 0 ? nb : 1, 256, 0, st>>>(N, d->V, d->spc, mass, dt, tau, T, d->out, d->trace,
                                                      d->capTrace, d->part ? d->part + MB_RED_MAXB * 8 : nullptr,
                                                      d->ticket ? d->ticket + 1 : nullptr);
    k_nvt_integrate<<<(N + 127) / 128, 128, 0, st>>>(N, d->X, d->V, d->F, d->spc, mass, dt, d->out, *c,
                                                     c->ND > 0 ? 1 : 0, d->status);
    *launches += 2;
    return (int)cudaGetLastError();
}

extern "C" int mbk_set_out(mb_dev *d, int idx, double v, void *stream) {
    k_set_out<<<1, 1, 0, (cudaStream_t)stream>>>(d->out, idx, v);
    return (int)cudaGetLastError();
}

/* events recorded while the stream is being captured become event-record
 * nodes of the graph, so that they time every replay */
extern "C" void mbk_record(void *event, void *stream) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing((cudaStream_t)stream, &cs);
    if (cs == cudaStreamCaptureStatusActive)
        cudaEventRecordWithFlags((cudaEvent_t)event, (cudaStream_t)stream, cudaEventRecordExternal);
    else
        cudaEventRecord((cudaEvent_t)event, (cudaStream_t)stream);
}

/* 1 when the descriptor pass of (N, mode) at the current capacity has its
 * kernel shape already: only then may it be captured (tuning synchronises) */
extern "C" int mbk_shape_ready(const mb_dev *d, int N, int mode) {
    int k;
    if (d->tune_fixed >= 0) return 1;
    const int key = tune_key(d, N, mode);
    for (k = 0; k < d->tune_n; k++)
        if (d->tune_key[k] == key) return 1;
    return 0;
}

/* ------------------------------------------------------------------ */
/* Replayed single-structure passes: the kernel nodes of a captured     */
/* pass that take the cell (or pV) by value, and their update          */
/* ------------------------------------------------------------------ */

template <typename... A>
constexpr int karity(void (*)(A...)) {
    return (int)sizeof...(A);
}

struct CellArg {
    const void *func;
    int arity, index; /* index of the mb_cell argument; -1: the pV argument of k_finalize */
};

static const CellArg kCellArgs[] = {
    {(const void *)k_wrap, karity(k_wrap), 2},
    {(const void *)k_intake, karity(k_intake), 2},
    {(const void *)k_cell_bin, karity(k_cell_bin), 2},
    {(const void *)k_cell_build, karity(k_cell_build), 2},
    {(const void *)k_nlist_cell, karity(k_nlist_cell), 4},
    {(const void *)k_nlist_brute, karity(k_nlist_brute), 4},
    {(const void *)k_finalize, karity(k_finalize), -1},
};

/* Find in `graph` the kernel nodes whose arguments depend on the cell or
 * pV; stores up to `cap` of them (node, table row) and returns how many
 * there are, or -1 on an error. */
extern "C" int mbk_graph_cell_nodes(void *graph, void **nodes, int *rows, int cap) {
    size_t n = 0;
    if (cudaGraphGetNodes((cudaGraph_t)graph, nullptr, &n) != cudaSuccess) return -1;
    cudaGraphNode_t *all = (cudaGraphNode_t *)malloc(sizeof(cudaGraphNode_t) * (n ? n : 1));
    if (cudaGraphGetNodes((cudaGraph_t)graph, all, &n) != cudaSuccess) {
        free(all);
        return -1;
    }
    int found = 0;
    for (size_t k = 0; k < n; k++) {
        cudaGraphNodeType t;
        if (cudaGraphNodeGetType(all[k], &t) != cudaSuccess || t != cudaGraphNodeTypeKernel) continue;
        cudaKernelNodeParams kp;
        if (cudaGraphKernelNodeGetParams(all[k], &kp) != cudaSuccess) continue;
        for (int r = 0; r < (int)(sizeof(kCellArgs) / sizeof(kCellArgs[0])); r++)
            if (kp.func == kCellArgs[r].func) {
                if (found < cap) {
                    nodes[found] = (void *)all[k];
                    rows[found] = r;
                }
                found++;
            }
    }
    free(all);
    return found;
}

/* Point the recorded nodes of the instantiated graph at a new cell and pV. */
extern "C" int mbk_graph_set_cell(void *exec, void *const *nodes, const int *rows, int count, const mb_cell *c,
                                  double pV) {
    for (int k = 0; k < count; k++) {
        cudaKernelNodeParams kp;
        cudaError_t e = cudaGraphKernelNodeGetParams((cudaGraphNode_t)nodes[k], &kp);
        if (e != cudaSuccess) return (int)e;
        const CellArg &a = kCellArgs[rows[k]];
        void *args[16];
        if (a.arity > 16) return (int)cudaErrorInvalidValue;
        for (int q = 0; q < a.arity; q++) args[q] = kp.kernelParams[q];
        mb_cell cell = *c;
        double pv = pV;
        if (a.index >= 0)
            args[a.index] = &cell;
        else
            args[2] = &pv;
        kp.kernelParams = args;
        kp.extra = nullptr;
        e = cudaGraphExecKernelNodeSetParams((cudaGraphExec_t)exec, (cudaGraphNode_t)nodes[k], &kp);
        if (e != cudaSuccess) return (int)e;
    }
    return 0;
}
