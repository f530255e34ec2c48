/*
 * mb_rdf.cu -- duplicate detection of the evolutionary search on the GPU:
 * the per-species-pair radial distribution of every member (RDF,
 * src/cell.c:369-417) and the overlaps of all pairs of members (CxC,
 * src/cell.c:419-430) that COMP_CL (src/eutl.c:394-413) combines and
 * RANK_TR (src/emod.c:351-368) compares against its cutoff.
 *
 *   k_rdf_ref   one CTA per structure, a warp per (i, j) pair of atoms with
 *               its lanes over the periodic images: every image within Rmax of
 *               a pair with species(j) >= species(i) spreads a Gaussian of
 *               width sigma over the bins within 3 sigma of r, a bin a lane,
 *               tapered by cos(pi/2 (x - Rmin)/(Rmax - Rmin)) above Rmin;
 *               same-species blocks halved; optionally scaled to unit length.
 *               The histogram lives in shared memory (FP64) and is written once.
 *   k_gram      the overlap matrix C = R R^T of the S histograms (a dense
 *               FP64 product of S x S outputs over nbins x npair terms) on the
 *               FP64 tensor cores, the terms split over enough CTAs to fill the
 *               GPU; k_gram_sum adds the splits in order.
 */
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdio.h>
#include <stdlib.h>

#include "../../../include/maise_b200.h"

namespace {

constexpr int RDF_THREADS = 512;
constexpr int RDF_MAX_HIST = 200 * 1024; /* bytes of a structure's histograms */
constexpr int RDF_SHIFTS = 128; /* image shifts kept in shared memory (more are formed again per pair) */

/* squared distance of j's image from i in LIST's operation order
 * (src/cell.c:115-121): the image's shift is the same sum of i0 L0, i1 L1,
 * i2 L2 for every pair and is formed once per structure */
__device__ __forceinline__ double rdf_disp2(const double *sh, const double *dij) {
    double r = 0.0;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const double x = __dadd_rn(sh[q], dij[q]);
        r = __dadd_rn(r, __dmul_rn(x, x));
    }
    return r;
}

__device__ __forceinline__ void rdf_shift(const double *L, int i0, int i1, int i2, double *sh) {
#pragma unroll
    for (int q = 0; q < 3; q++) {
        double x = 0.0;
        x = __dadd_rn(x, __dmul_rn((double)i0, L[q]));
        x = __dadd_rn(x, __dmul_rn((double)i1, L[3 + q]));
        sh[q] = __dadd_rn(x, __dmul_rn((double)i2, L[6 + q]));
    }
}

struct RdfArgs {
    int S, nspc, nbins, ND, normalise;
    const int *off, *spc;
    const double *lat, *x;
    double rmin, rmax, sigma;
    double *out; /* [S][npair][nbins] */
};

/* Bound by the Gaussians: a pair within Rmax spreads over 25 of 3000 bins,
 * one exponential and one shared FP64 addition each.  With a thread per
 * (i, j, image) candidate the few accepted lanes of a warp walked their 25
 * bins alone (and every bin its cosine); with the warp on one pair at a time,
 * a bin a lane, 150 structures of 8 to 64 atoms take 202 us instead of
 * 5826. */
__global__ void __launch_bounds__(RDF_THREADS) k_rdf_ref(RdfArgs A) {
    extern __shared__ __align__(16) double hist[]; /* [npair][nbins] */
    __shared__ double L[9], R[9], red[RDF_THREADS / 32], sh[RDF_SHIFTS][3];
    __shared__ int nq[3];
    const int s = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int o = A.off[s], N = A.off[s + 1] - o, ns = A.nspc, nb = A.nbins;
    const int npair = ns * (ns + 1) / 2;
    for (int k = tid; k < npair * nb; k += blockDim.x) hist[k] = 0.0;
    if (tid == 0) {
        for (int k = 0; k < 9; k++) L[k] = A.lat[9 * (size_t)s + k];
        R[6] = L[1] * L[5] - L[2] * L[4];
        R[7] = L[2] * L[3] - L[0] * L[5];
        R[8] = L[0] * L[4] - L[1] * L[3];
        R[0] = L[4] * L[8] - L[5] * L[7];
        R[1] = L[5] * L[6] - L[3] * L[8];
        R[2] = L[3] * L[7] - L[4] * L[6];
        R[3] = L[7] * L[2] - L[8] * L[1];
        R[4] = L[8] * L[0] - L[6] * L[2];
        R[5] = L[6] * L[1] - L[7] * L[0];
        const double t = 1.0 / (L[0] * L[4] * L[8] + L[1] * L[5] * L[6] + L[2] * L[3] * L[7] - L[0] * L[5] * L[7] -
                                L[1] * L[3] * L[8] - L[2] * L[4] * L[6]);
        for (int k = 0; k < 9; k++) R[k] *= t;
        for (int q = 0; q < 3; q++) {
            const double len = sqrt(R[3 * q] * R[3 * q] + R[3 * q + 1] * R[3 * q + 1] + R[3 * q + 2] * R[3 * q + 2]);
            nq[q] = q < A.ND ? (int)ceil(A.rmax * len) : 0;
        }
    }
    __syncthreads();
    const double dr = A.rmax / (double)nb, rc2 = A.rmax * A.rmax;
    const int Do = (int)(3.0 * A.sigma / dr);
    const double DRi = 0.5 / (A.sigma * A.sigma);
    const int w0 = 2 * nq[0] + 1, w1 = 2 * nq[1] + 1, w2 = 2 * nq[2] + 1, nimg = w0 * w1 * w2;
    const int zero = (nq[0] * w1 + nq[1]) * w2 + nq[2]; /* the unshifted image */
    for (int im = tid; im < nimg && im < RDF_SHIFTS; im += blockDim.x) {
        const int t = im / w2;
        rdf_shift(L, t / w1 - nq[0], t % w1 - nq[1], im % w2 - nq[2], sh[im]);
    }
    __syncthreads();
    for (long long ij = warp; ij < (long long)N * N; ij += RDF_THREADS / 32) {
        const int i = (int)(ij / N), j = (int)(ij - (long long)i * N);
        const int si = A.spc[o + i], sj = A.spc[o + j];
        if (sj < si) continue;
        const double *xi = A.x + 3 * (size_t)(o + i), *xj = A.x + 3 * (size_t)(o + j);
        const double dij[3] = {__dsub_rn(xj[0], xi[0]), __dsub_rn(xj[1], xi[1]), __dsub_rn(xj[2], xi[2])};
        const int pair = si * ns - si * (si - 1) / 2 + (sj - si); /* (si, sj), si <= sj, row-major */
        double *h = hist + (size_t)pair * nb;
        for (int base = 0; base < nimg; base += 32) {
            const int im = base + lane;
            double r2 = rc2;
            if (im < nimg && !(i == j && im == zero)) {
                if (im < RDF_SHIFTS) {
                    r2 = rdf_disp2(sh[im], dij);
                } else {
                    double t3[3];
                    const int t = im / w2;
                    rdf_shift(L, t / w1 - nq[0], t % w1 - nq[1], im % w2 - nq[2], t3);
                    r2 = rdf_disp2(t3, dij);
                }
            }
            const double rl = sqrt(r2);
            for (unsigned m = __ballot_sync(0xffffffffu, r2 < rc2); m; m &= m - 1) {
                const double r = __shfl_sync(0xffffffffu, rl, __ffs(m) - 1);
                const int ob = (int)(r / dr);
                for (int k = ob - Do + lane; k <= ob + Do; k += 32) {
                    if (k < 0 || k >= nb) continue;
                    const double xk = (double)k * dr;
                    double f = exp(-(r - xk) * (r - xk) * DRi);
                    if (xk >= A.rmin) f *= cos(0.5 * CUDART_PI * (xk - A.rmin) / (A.rmax - A.rmin));
                    atomicAdd(h + k, f);
                }
            }
        }
    }
    __syncthreads();
    /* same-species blocks hold each pair twice (i-j and j-i): halved */
    for (int m = 0; m < ns; m++) {
        const int pair = m * ns - m * (m - 1) / 2;
        for (int k = tid; k < nb; k += blockDim.x) hist[(size_t)pair * nb + k] *= 0.5;
    }
    __syncthreads();
    double scale = 1.0;
    if (A.normalise) {
        double ss = 0.0;
        for (int k = tid; k < npair * nb; k += blockDim.x) ss += hist[k] * hist[k];
        for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
        if ((tid & 31) == 0) red[tid >> 5] = ss;
        __syncthreads();
        double tot = 0.0;
        for (int w = 0; w < (int)(blockDim.x / 32); w++) tot += red[w];
        scale = tot > 0.0 ? 1.0 / sqrt(tot) : 0.0;
    }
    double *out = A.out + (size_t)s * npair * nb;
    for (int k = tid; k < npair * nb; k += blockDim.x) out[k] = hist[k] * scale;
}

/* Partial sums of C[p][q] = sum_t A[p][t] A[q][t] over the terms of split
 * blockIdx.y, for the 64 x 64 tile blockIdx.x of the upper triangle of tiles
 * (C is symmetric): 4 warps of 32 x 32, operands staged 32 terms at a time in
 * rows of 36 (the mma operand reads, 4 rows x 4 terms a half-warp, touch 16
 * distinct banks).  With one CTA per tile and no split, 150 histograms of
 * 9000 terms ran on 9 SMs for 2707 us; split over 47 CTAs a tile they take
 * 73 us with the final sum. */
#define GRAM_T 64
#define GRAM_K 32
#define GRAM_LD 36
__device__ __forceinline__ void gram_tile(int tile, int nt, int &ti, int &tj) {
    ti = 0;
    while (tile >= nt - ti) {
        tile -= nt - ti;
        ti++;
    }
    tj = ti + tile;
}

__global__ void __launch_bounds__(128) k_gram(int S, int T, int nt, int per, const double *__restrict__ A,
                                              double *__restrict__ part, double *__restrict__ C) {
    __shared__ double a[GRAM_T * GRAM_LD], b[GRAM_T * GRAM_LD];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int ti, tj;
    gram_tile(blockIdx.x, nt, ti, tj);
    const int p0 = ti * GRAM_T, q0 = tj * GRAM_T;
    const int t_lo = blockIdx.y * per, t_hi = min(T, t_lo + per);
    const int wr = (warp >> 1) * 32, wc = (warp & 1) * 32, fr = (lane >> 2) * GRAM_LD + (lane & 3);
    double c[4][4][2] = {};
    for (int t0 = t_lo; t0 < t_hi; t0 += GRAM_K) {
#pragma unroll 4
        for (int e = tid; e < GRAM_T * GRAM_K; e += 128) {
            const int r = e / GRAM_K, k = e % GRAM_K, t = t0 + k;
            a[r * GRAM_LD + k] = (p0 + r < S && t < t_hi) ? A[(size_t)(p0 + r) * T + t] : 0.0;
            b[r * GRAM_LD + k] = (q0 + r < S && t < t_hi) ? A[(size_t)(q0 + r) * T + t] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < GRAM_K; k += 4) {
            double av[4], bv[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                av[u] = a[(wr + 8 * u) * GRAM_LD + fr + k];
                bv[u] = b[(wc + 8 * u) * GRAM_LD + fr + k];
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int v = 0; v < 4; v++)
                    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                                 : "+d"(c[u][v][0]), "+d"(c[u][v][1])
                                 : "d"(av[u]), "d"(bv[v]));
        }
        __syncthreads();
    }
    if (C) { /* no split: straight to both triangles */
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
            for (int v = 0; v < 4; v++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int p = p0 + wr + 8 * u + (lane >> 2), q = q0 + wc + 8 * v + 2 * (lane & 3) + h;
                    if (p < S && q < S) {
                        C[(size_t)p * S + q] = c[u][v][h];
                        if (ti != tj) C[(size_t)q * S + p] = c[u][v][h];
                    }
                }
        return;
    }
    double *o = part + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * GRAM_T * GRAM_T;
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++)
            *reinterpret_cast<double2 *>(o + (wr + 8 * u + (lane >> 2)) * GRAM_T + wc + 8 * v + 2 * (lane & 3)) =
                make_double2(c[u][v][0], c[u][v][1]);
}

/* one thread per output of a tile: its splits in order, to both triangles */
__global__ void __launch_bounds__(256) k_gram_sum(int S, int nt, int nsplit, const double *__restrict__ part,
                                                  double *__restrict__ C) {
    int ti, tj;
    gram_tile(blockIdx.x, nt, ti, tj);
    const int e = blockIdx.y * 256 + threadIdx.x, p = ti * GRAM_T + e / GRAM_T, q = tj * GRAM_T + e % GRAM_T;
    if (p >= S || q >= S) return;
    double acc = 0.0;
#pragma unroll 4
    for (int k = 0; k < nsplit; k++) acc += part[((size_t)k * gridDim.x + blockIdx.x) * GRAM_T * GRAM_T + e];
    C[(size_t)p * S + q] = acc;
    if (ti != tj) C[(size_t)q * S + p] = acc;
}

}  // namespace

extern "C" int mb_handle_fail(int code, const char *msg);

static int rdf_cuda(cudaError_t e, const char *what) {
    if (e == cudaSuccess) return MB_OK;
    static __thread char msg[200];
    snprintf(msg, sizeof(msg), "%s: %s", what, cudaGetErrorString(e));
    return mb_handle_fail(MB_ERR_CUDA, msg);
}

extern "C" int mb_rdf(int device, int S, const int *nat, const int *atmn, const double *lat, const double *x, int ND,
                      int nspc, int nbins, double rmin, double rmax, double sigma, int normalise, double *rdf) {
    if (S < 1 || !nat || !atmn || !lat || !x || !rdf || nspc < 1 || nspc > 3 || nbins < 1 || !(rmax > 0.0) ||
        !(rmin <= rmax) || !(sigma > 0.0) || ND < 0 || ND > 3)
        return mb_handle_fail(MB_ERR_ARG, "bad arguments");
    const int npair = nspc * (nspc + 1) / 2;
    const size_t smem = sizeof(double) * (size_t)npair * nbins;
    if (smem > RDF_MAX_HIST) return mb_handle_fail(MB_ERR_ARG, "nbins x species pairs exceed the shared histogram");
    int *off = (int *)malloc(sizeof(int) * (S + 1));
    off[0] = 0;
    for (int s = 0; s < S; s++) {
        if (nat[s] < 1) {
            free(off);
            return mb_handle_fail(MB_ERR_ARG, "empty structure");
        }
        off[s + 1] = off[s] + nat[s];
    }
    for (int k = 0; k < off[S]; k++)
        if (atmn[k] < 0 || atmn[k] >= nspc) {
            free(off);
            return mb_handle_fail(MB_ERR_ARG, "species index out of range");
        }
    int rc = rdf_cuda(cudaSetDevice(device), "cudaSetDevice");
    /* one allocation: offsets, species, lattices, positions, results */
    const size_t nout = (size_t)S * npair * nbins;
    const size_t b_spc = (sizeof(int) * (S + 1) + 15) & ~(size_t)15;
    const size_t b_lat = b_spc + ((sizeof(int) * (size_t)off[S] + 15) & ~(size_t)15);
    const size_t b_x = b_lat + ((sizeof(double) * 9 * S + 15) & ~(size_t)15), b_out = b_x + ((sizeof(double) * 3 * (size_t)off[S] + 15) & ~(size_t)15);
    char *d = nullptr;
    if (!rc) rc = rdf_cuda(cudaMalloc(&d, b_out + sizeof(double) * nout), "cudaMalloc");
    int *d_off = (int *)d, *d_spc = (int *)(d + b_spc);
    double *d_lat = (double *)(d + b_lat), *d_x = (double *)(d + b_x), *d_out = (double *)(d + b_out);
    if (!rc) rc = rdf_cuda(cudaMemcpy(d_off, off, sizeof(int) * (S + 1), cudaMemcpyHostToDevice), "H2D");
    if (!rc) rc = rdf_cuda(cudaMemcpy(d_spc, atmn, sizeof(int) * off[S], cudaMemcpyHostToDevice), "H2D");
    if (!rc) rc = rdf_cuda(cudaMemcpy(d_lat, lat, sizeof(double) * 9 * S, cudaMemcpyHostToDevice), "H2D");
    if (!rc) rc = rdf_cuda(cudaMemcpy(d_x, x, sizeof(double) * 3 * off[S], cudaMemcpyHostToDevice), "H2D");
    if (!rc && smem + 4096 > 48 * 1024) /* (k_rdf_ref's static arrays count too) */
        rc = rdf_cuda(cudaFuncSetAttribute(k_rdf_ref, cudaFuncAttributeMaxDynamicSharedMemorySize, RDF_MAX_HIST),
                      "shared-memory opt-in"); /* one limit for every call: other threads may be launching */
    if (!rc) {
        RdfArgs a;
        a.S = S; a.nspc = nspc; a.nbins = nbins; a.ND = ND; a.normalise = normalise ? 1 : 0;
        a.off = d_off; a.spc = d_spc; a.lat = d_lat; a.x = d_x;
        a.rmin = rmin; a.rmax = rmax; a.sigma = sigma; a.out = d_out;
        k_rdf_ref<<<S, RDF_THREADS, smem>>>(a);
        rc = rdf_cuda(cudaGetLastError(), "k_rdf_ref");
    }
    if (!rc) rc = rdf_cuda(cudaMemcpy(rdf, d_out, sizeof(double) * nout, cudaMemcpyDeviceToHost), "D2H");
    cudaFree(d);
    free(off);
    return rc;
}

extern "C" int mb_rdf_overlap(int device, int S, int len, const double *rdf, double *cxc) {
    if (S < 1 || len < 1 || !rdf || !cxc) return mb_handle_fail(MB_ERR_ARG, "bad arguments");
    int rc = rdf_cuda(cudaSetDevice(device), "cudaSetDevice");
    /* tiles of the upper triangle, and as many splits of the terms as give
     * about two CTAs an SM without going below two stages of GRAM_K terms */
    const int nt = (S + GRAM_T - 1) / GRAM_T;
    const long long tiles = (long long)nt * (nt + 1) / 2;
    int sms = 148, nsplit, per;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    nsplit = (int)((2LL * sms + tiles - 1) / tiles);
    if (nsplit > len / (2 * GRAM_K)) nsplit = len / (2 * GRAM_K);
    if (nsplit < 1) nsplit = 1;
    per = ((len + nsplit - 1) / nsplit + GRAM_K - 1) / GRAM_K * GRAM_K;
    nsplit = (len + per - 1) / per;
    /* one allocation (each costs 0.3 ms with its release): RDFs, overlaps, the splits' sums */
    const size_t na = (size_t)S * len, nc = (size_t)S * S, part0 = (na + nc + 1) & ~(size_t)1;
    const size_t npart = nsplit > 1 ? (size_t)nsplit * tiles * GRAM_T * GRAM_T : 0;
    double *d_a = nullptr;
    if (!rc) rc = rdf_cuda(cudaMalloc(&d_a, sizeof(double) * (part0 + npart)), "cudaMalloc");
    double *d_c = d_a + na, *d_part = d_a + part0;
    if (!rc) rc = rdf_cuda(cudaMemcpy(d_a, rdf, sizeof(double) * (size_t)S * len, cudaMemcpyHostToDevice), "H2D");
    if (!rc) {
        k_gram<<<dim3((unsigned)tiles, nsplit), 128>>>(S, len, nt, per, d_a, d_part, nsplit > 1 ? nullptr : d_c);
        if (nsplit > 1) k_gram_sum<<<dim3((unsigned)tiles, GRAM_T * GRAM_T / 256), 256>>>(S, nt, nsplit, d_part, d_c);
        rc = rdf_cuda(cudaGetLastError(), "k_gram");
    }
    if (!rc) rc = rdf_cuda(cudaMemcpy(cxc, d_c, sizeof(double) * (size_t)S * S, cudaMemcpyDeviceToHost), "D2H");
    cudaFree(d_a);
    return rc;
}
