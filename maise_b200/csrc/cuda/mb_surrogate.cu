/*
 * mb_surrogate.cu -- kernels of the surrogate screen for EA offspring.
 *
 * The screen ranks unrelaxed offspring by a predicted relaxed enthalpy per
 * atom so that only the best fraction goes on to a full relaxation.  Its
 * input is a per-species-pair radial histogram (the analogue of RDF,
 * src/cell.c:369-417, at 128 bins); its model is a small FP32 MLP
 * (nin -> 128 -> 64 -> 64 -> 1, SiLU) trained with Adam on
 * unrelaxed -> relaxed pairs.  Nothing here exists in the reference, which
 * relaxes every offspring.
 *
 * Kernels:
 *   k_rdf       one CTA per structure, a warp over (i, j) pairs of atoms with its
 *               lanes over the images that can lie within rmax; distances
 *               within rmax are queued per warp and spread as tapered Gaussians
 *               8 bins at a time into a shared histogram (FP64 distances and
 *               weights, FP32 shared atomics); writes the histogram / N.
 *   k_gemm      register-tiled FP32 GEMM (tiles of 64x64 or 32x32), C = op(A) op(B), with
 *               fused epilogues: bias + SiLU (keeping the pre-activation),
 *               bias only, plain store, and product with SiLU'(Z) for the
 *               backward pass.  The layers are at most 4096 x 768 x 128,
 *               FP32 by specification, so SIMT FMA tiles are used.
 *   k_colsum    bias gradients (column sums of dZ).
 *   k_mse       squared-error loss and its gradient for one batch.
 *   k_adam      Adam update of the flat parameter vector.
 *   k_gather    minibatch rows by index, standardised on the fly.
 *   k_colstats  per-feature mean and 1/std of the training features.
 */
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../host/mb_surrogate_k.h"

/* ------------------------------------------------------------ histogram */

/* Images kept per structure: those whose shift can bring a minimum-image
 * displacement (at most the cell's half diagonal long) within rmax.  The
 * (2 n + 1)^3 images of the plane spacings hold 5 to 10 times as many. */
#define RDF_IMGS 512
#define RDF_QUEUE 64 /* distances a warp holds before spreading them */

/* Spread the queued distances: 8 lanes an entry, 4 entries a step. */
__device__ __forceinline__ void rdf_spread(const double *qr, const int *qp, int n, int lane, int nbins, int Do,
                                           double dr, double DR, const double *taper, float *hist) {
    for (int e = lane >> 3; e < n; e += 4) {
        const double r = qr[e];
        const int o = (int)(r / dr);
        float *h = hist + qp[e] * nbins;
        for (int k = o - Do + (lane & 7); k <= o + Do; k += 8) {
            if (k < 0 || k >= nbins) continue;
            const double xk = k * dr;
            atomicAdd(h + k, (float)(taper[k] * exp(-(r - xk) * (r - xk) * DR)));
        }
    }
}

/* Bound by the candidate distances and the Gaussians (7 bins a pair at the
 * default width).  A thread per (i, j) pair walking all images alone, a cosine
 * and an exponential per bin, took 3689 us for 2048 structures of 16 to 48
 * atoms; with the images pruned once per structure and the bins spread over
 * lanes it takes 500 us. */
__global__ void __launch_bounds__(256) k_rdf(int S, const int *__restrict__ off, const int *__restrict__ spc,
                                            const double *__restrict__ lat, const double *__restrict__ x, int nspc,
                                            int nbins, double rmax, double sigma, float *__restrict__ feat,
                                            int *__restrict__ status) {
    extern __shared__ __align__(16) double taper[]; /* [nbins], then the histogram */
    float *hist = reinterpret_cast<float *>(taper + nbins);
    __shared__ double L[9], Li[9], half2;
    __shared__ double fr[3 * SUR_MAX_ATOMS], sh[3 * RDF_IMGS], qr[8][RDF_QUEUE];
    __shared__ int sp[SUR_MAX_ATOMS], qp[8][RDF_QUEUE];
    __shared__ int nimg[3], nsh;
    __shared__ int bad;
    const int s = blockIdx.x, tid = threadIdx.x, bd = blockDim.x, lane = tid & 31, warp = tid >> 5;
    if (s >= S) return;
    const int a0 = off[s], N = off[s + 1] - a0;
    const int P = nspc * (nspc + 1) / 2;
    for (int k = tid; k < P * nbins; k += bd) hist[k] = 0.0f;
    if (tid < 9) L[tid] = lat[9 * s + tid];
    __syncthreads();
    if (tid == 0) {
        /* inverse of the row-vector lattice by cofactors */
        const double c00 = L[4] * L[8] - L[5] * L[7], c01 = L[5] * L[6] - L[3] * L[8], c02 = L[3] * L[7] - L[4] * L[6];
        const double det = L[0] * c00 + L[1] * c01 + L[2] * c02;
        const double id = 1.0 / det;
        Li[0] = c00 * id;
        Li[3] = c01 * id;
        Li[6] = c02 * id;
        Li[1] = (L[2] * L[7] - L[1] * L[8]) * id;
        Li[4] = (L[0] * L[8] - L[2] * L[6]) * id;
        Li[7] = (L[1] * L[6] - L[0] * L[7]) * id;
        Li[2] = (L[1] * L[5] - L[2] * L[4]) * id;
        Li[5] = (L[2] * L[3] - L[0] * L[5]) * id;
        Li[8] = (L[0] * L[4] - L[1] * L[3]) * id;
        /* images needed along each lattice vector: rmax over the plane
         * spacing, plus half a cell for the minimum-image fractional shift */
        const double V = fabs(det);
        bad = (N < 1 || N > SUR_MAX_ATOMS || !(V > 0.0));
        for (int a = 0; a < 3; a++) {
            const double *b = L + 3 * ((a + 1) % 3), *c = L + 3 * ((a + 2) % 3);
            const double cx = b[1] * c[2] - b[2] * c[1], cy = b[2] * c[0] - b[0] * c[2], cz = b[0] * c[1] - b[1] * c[0];
            const double h = V / sqrt(cx * cx + cy * cy + cz * cz);
            const double n = ceil(rmax / h + 0.5);
            if (!(n <= SUR_MAX_IMG)) bad = 1;
            nimg[a] = bad ? 0 : (int)n;
        }
        /* the longest half diagonal bounds a minimum-image displacement */
        half2 = 0.0;
        for (int q = 0; q < 4; q++) {
            double d2 = 0.0;
            for (int c = 0; c < 3; c++) {
                const double v = 0.5 * (L[c] + ((q & 1) ? -L[3 + c] : L[3 + c]) + ((q & 2) ? -L[6 + c] : L[6 + c]));
                d2 += v * v;
            }
            half2 = fmax(half2, d2);
        }
        nsh = 0;
    }
    __syncthreads();
    if (bad) {
        if (tid == 0) atomicOr(status, 1);
        for (int k = tid; k < P * nbins; k += bd) feat[(size_t)s * P * nbins + k] = 0.0f;
        return;
    }
    for (int i = tid; i < N; i += bd) {
        const double *xi = x + 3 * (size_t)(a0 + i);
        for (int c = 0; c < 3; c++) fr[3 * i + c] = xi[0] * Li[c] + xi[1] * Li[3 + c] + xi[2] * Li[6 + c];
        sp[i] = spc[a0 + i];
    }
    for (int k = tid; k < nbins; k += bd) taper[k] = cos(0.5 * M_PI * (k * (rmax / nbins)) / rmax);
    const int n0 = nimg[0], n1 = nimg[1], n2 = nimg[2], w1 = 2 * n1 + 1, w2 = 2 * n2 + 1;
    const double reach = (rmax + sqrt(half2)) * (1.0 + 1e-9), rc2 = rmax * rmax;
    for (int im = tid; im < (2 * n0 + 1) * w1 * w2; im += bd) {
        const double ta = im / (w1 * w2) - n0, tb = (im / w2) % w1 - n1, tc = im % w2 - n2;
        const double vx = ta * L[0] + tb * L[3] + tc * L[6], vy = ta * L[1] + tb * L[4] + tc * L[7],
                     vz = ta * L[2] + tb * L[5] + tc * L[8];
        if (vx * vx + vy * vy + vz * vz <= reach * reach) {
            const int e = atomicAdd(&nsh, 1);
            if (e < RDF_IMGS) {
                sh[3 * e] = ta;
                sh[3 * e + 1] = tb;
                sh[3 * e + 2] = tc;
            }
        }
    }
    __syncthreads();
    /* (a cell so skewed that the list overflows walks every image) */
    const int every = nsh > RDF_IMGS, count = every ? (2 * n0 + 1) * w1 * w2 : nsh;
    const double dr = rmax / nbins;
    const int Do = (int)(3.0 * sigma / dr);
    const double DR = 0.5 / (sigma * sigma);
    int nq = 0;
    /* lanes a pair of atoms takes: as many as there are images to look at.  A
     * warp a pair, whatever the count, looked at 7 images with 32 lanes in
     * cells longer than 2 rmax: screens of 64 structures of 128, 200 and 256
     * atoms took 0.97, 2.00 and 3.10 ms (0.48, 0.80 and 1.18 now).  The loop is
     * inlined twice, for whole warps with the constants folded. */
    auto walk = [&](const int group, const int sub) {
        for (int w0 = warp * (32 / group); w0 < N * N; w0 += 8 * (32 / group)) {
            const int w = w0 + sub;
            const int i = w / N, j = w - i * N;
            const bool pair = w < N * N && sp[j] >= sp[i];
            if (group == 32 ? !pair : !__any_sync(0xffffffffu, pair)) continue;
            int p = 0;
            double d[3] = {0.0, 0.0, 0.0};
            if (group == 32 || pair) {
                const int si = sp[i];
                p = si * nspc - si * (si - 1) / 2 + (sp[j] - si);
                for (int c = 0; c < 3; c++) {
                    const double t = fr[3 * j + c] - fr[3 * i + c];
                    d[c] = t - rint(t);
                }
            }
            for (int base = 0; base < count; base += 32) {
                const int im = base + (lane & (group - 1));
                double r2 = rc2;
                if ((group == 32 || pair) && im < count) {
                    const double u0 = d[0] + (every ? (double)(im / (w1 * w2) - n0) : sh[3 * im]);
                    const double u1 = d[1] + (every ? (double)((im / w2) % w1 - n1) : sh[3 * im + 1]);
                    const double u2 = d[2] + (every ? (double)(im % w2 - n2) : sh[3 * im + 2]);
                    const double vx = u0 * L[0] + u1 * L[3] + u2 * L[6];
                    const double vy = u0 * L[1] + u1 * L[4] + u2 * L[7];
                    const double vz = u0 * L[2] + u1 * L[5] + u2 * L[8];
                    r2 = vx * vx + vy * vy + vz * vz;
                }
                const bool in = r2 < rc2 && r2 != 0.0;
                const unsigned m = __ballot_sync(0xffffffffu, in);
                if (in) {
                    const int e = nq + __popc(m & ((1u << lane) - 1u));
                    qr[warp][e] = sqrt(r2);
                    qp[warp][e] = p;
                }
                nq += __popc(m);
                if (nq > RDF_QUEUE - 32) {
                    __syncwarp();
                    rdf_spread(qr[warp], qp[warp], nq, lane, nbins, Do, dr, DR, taper, hist);
                    __syncwarp();
                    nq = 0;
                }
            }
        }
    };
    const int group = count > 8 ? 16 : count > 4 ? 8 : count > 2 ? 4 : count > 1 ? 2 : 1;
    if (count > 16) walk(32, 0);
    else walk(group, lane / group);
    __syncwarp();
    rdf_spread(qr[warp], qp[warp], nq, lane, nbins, Do, dr, DR, taper, hist);
    __syncthreads();
    const float invN = 1.0f / (float)N;
    for (int k = tid; k < P * nbins; k += bd) {
        const int p = k / nbins;
        int diag = 0;
        for (int m = 0; m < nspc; m++) diag |= (p == m * nspc - m * (m - 1) / 2);
        feat[(size_t)s * P * nbins + k] = hist[k] * (diag ? 0.5f : 1.0f) * invN;
    }
}

/* ----------------------------------------------------------------- GEMM */

#define GB_K 16

__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float dsilu_f(float z) {
    const float s = 1.0f / (1.0f + expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

/* C[m, n] = sum_k A(m, k) B(k, n), A(m, k) = TA ? A[k lda + m] : A[m lda + k],
 * B(k, n) = TB ? B[n ldb + k] : B[k ldb + n]; row-major C with leading
 * dimension ldc; EP selects the epilogue (SUR_EP_*). */
/* Tiles of GB x GB outputs, 256 threads of R x R each (R = GB / 16); the next
 * GB_K terms are loaded into registers while the current ones are multiplied.
 * GB is 64 where such tiles give at least one CTA an SM, 32 below: the first
 * layer of 2048 rows (128 outputs, 768 terms) is 64 tiles of 64, each a chain
 * of 48 load-multiply stages (86 us), and 256 tiles of 32 (35 us).  Every output
 * sums its terms in ascending order in either. */
template <bool TA, bool TB, int EP, int GB>
__global__ void __launch_bounds__(256) k_gemm(int M, int N, int K, const float *__restrict__ A, int lda,
                                             const float *__restrict__ B, int ldb, float *__restrict__ C, int ldc,
                                             const float *__restrict__ bias, float *__restrict__ Z,
                                             const float *__restrict__ Zp) {
    constexpr int R = GB / 16, LOADS = GB * GB_K / 256;
    __shared__ __align__(16) float As[GB_K][GB + 4];
    __shared__ __align__(16) float Bs[GB_K][GB + 4];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * GB, n0 = blockIdx.x * GB;
    float acc[R][R];
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
        for (int j = 0; j < R; j++) acc[i][j] = 0.0f;
    float ra[LOADS], rb[LOADS];
    auto load = [&](int k0) {
#pragma unroll
        for (int r = 0; r < LOADS; r++) {
            const int e = tid + 256 * r;
            const int m = TA ? e % GB : e / GB_K, ka = TA ? e / GB : e % GB_K;
            const int n = TB ? e / GB_K : e % GB, kb = TB ? e % GB_K : e / GB;
            const int gm = m0 + m, gn = n0 + n;
            ra[r] = gm < M && k0 + ka < K ? (TA ? A[(size_t)(k0 + ka) * lda + gm] : A[(size_t)gm * lda + k0 + ka]) : 0.0f;
            rb[r] = gn < N && k0 + kb < K ? (TB ? B[(size_t)gn * ldb + k0 + kb] : B[(size_t)(k0 + kb) * ldb + gn]) : 0.0f;
        }
    };
    load(0);
    for (int k0 = 0; k0 < K; k0 += GB_K) {
#pragma unroll
        for (int r = 0; r < LOADS; r++) {
            const int e = tid + 256 * r;
            As[TA ? e / GB : e % GB_K][TA ? e % GB : e / GB_K] = ra[r];
            Bs[TB ? e % GB_K : e / GB][TB ? e / GB_K : e % GB] = rb[r];
        }
        __syncthreads();
        if (k0 + GB_K < K) load(k0 + GB_K);
#pragma unroll
        for (int kk = 0; kk < GB_K; kk++) {
            float a[R], b[R];
#pragma unroll
            for (int i = 0; i < R; i++) a[i] = As[kk][ty * R + i];
#pragma unroll
            for (int j = 0; j < R; j++) b[j] = Bs[kk][tx * R + j];
#pragma unroll
            for (int i = 0; i < R; i++)
#pragma unroll
                for (int j = 0; j < R; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int gm = m0 + ty * R + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < R; j++) {
            const int gn = n0 + tx * R + j;
            if (gn >= N) continue;
            const size_t o = (size_t)gm * ldc + gn;
            float v = acc[i][j];
            if (EP == SUR_EP_BIAS_SILU) {
                v += bias[gn];
                Z[o] = v;
                C[o] = silu_f(v);
            } else if (EP == SUR_EP_BIAS) {
                C[o] = v + bias[gn];
            } else if (EP == SUR_EP_DSILU) {
                C[o] = v * dsilu_f(Zp[o]);
            } else {
                C[o] = v;
            }
        }
    }
}

extern "C" int surk_gemm(int ta, int tb, int ep, int M, int N, int K, const float *A, int lda, const float *B, int ldb,
                         float *C, int ldc, const float *bias, float *Z, const float *Zp, void *stream) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const bool small = (long)((N + 63) / 64) * ((M + 63) / 64) < sms;
    const int gb = small ? 32 : 64;
    dim3 grid((N + gb - 1) / gb, (M + gb - 1) / gb);
    cudaStream_t st = (cudaStream_t)stream;
#define SUR_GEMM(TA_, TB_, EP_)                                                                             \
    do {                                                                                                    \
        if (small)                                                                                          \
            k_gemm<TA_, TB_, EP_, 32><<<grid, 256, 0, st>>>(M, N, K, A, lda, B, ldb, C, ldc, bias, Z, Zp);  \
        else                                                                                                \
            k_gemm<TA_, TB_, EP_, 64><<<grid, 256, 0, st>>>(M, N, K, A, lda, B, ldb, C, ldc, bias, Z, Zp);  \
    } while (0)
    if (!ta && tb && ep == SUR_EP_BIAS_SILU) SUR_GEMM(false, true, SUR_EP_BIAS_SILU);
    else if (!ta && tb && ep == SUR_EP_BIAS) SUR_GEMM(false, true, SUR_EP_BIAS);
    else if (!ta && !tb && ep == SUR_EP_DSILU) SUR_GEMM(false, false, SUR_EP_DSILU);
    else if (ta && !tb && ep == SUR_EP_STORE) SUR_GEMM(true, false, SUR_EP_STORE);
    else return (int)cudaErrorInvalidValue;
#undef SUR_GEMM
    return (int)cudaGetLastError();
}

/* ------------------------------------------------------- small kernels */

__global__ void k_colsum(int B, int O, const float *__restrict__ dZ, float *__restrict__ out) {
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= O) return;
    float s = 0.0f;
    for (int b = 0; b < B; b++) s += dZ[(size_t)b * O + o];
    out[o] = s;
}

__global__ void __launch_bounds__(256) k_mse(int B, const float *__restrict__ y, const float *__restrict__ t,
                                            float *__restrict__ dy, double *__restrict__ loss) {
    __shared__ double red[256];
    double s = 0.0;
    for (int b = threadIdx.x; b < B; b += blockDim.x) {
        const float e = y[b] - t[b];
        dy[b] = 2.0f * e / (float)B;
        s += (double)e * e;
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *loss = red[0] / B;
}

__global__ void k_adam(long n, float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
    for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) {
        const float gk = g[k];
        const float mk = b1 * m[k] + (1.0f - b1) * gk;
        const float vk = b2 * v[k] + (1.0f - b2) * gk * gk;
        m[k] = mk;
        v[k] = vk;
        p[k] -= lr * (mk * c1) / (sqrtf(vk * c2) + eps);
    }
}

__global__ void k_gather(int B, int F, const int *__restrict__ idx, const float *__restrict__ X,
                         const float *__restrict__ mean, const float *__restrict__ istd, float *__restrict__ out,
                         const float *__restrict__ T, float tmean, float tistd, float *__restrict__ tout) {
    const int b = blockIdx.x;
    if (b >= B) return;
    const long r = idx ? idx[b] : b;
    const float *src = X + (size_t)r * F;
    float *dst = out + (size_t)b * F;
    for (int f = threadIdx.x; f < F; f += blockDim.x) dst[f] = (src[f] - mean[f]) * istd[f];
    if (T && threadIdx.x == 0) tout[b] = (T[r] - tmean) * tistd;
}

__global__ void k_colstats(int S, int F, const float *__restrict__ X, float *__restrict__ mean,
                           float *__restrict__ istd) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= F) return;
    double s = 0.0;
    for (int r = 0; r < S; r++) s += X[(size_t)r * F + f];
    const double mu = s / S;
    double q = 0.0;
    for (int r = 0; r < S; r++) {
        const double e = X[(size_t)r * F + f] - mu;
        q += e * e;
    }
    mean[f] = (float)mu;
    istd[f] = (float)(1.0 / sqrt(q / S + SUR_VAR_FLOOR));
}

/* ------------------------------------------------------------ launchers */

extern "C" int surk_rdf(int S, const int *off, const int *spc, const double *lat, const double *x, int nspc, int nbins,
                        double rmax, double sigma, float *feat, int *status, void *stream) {
    const int P = nspc * (nspc + 1) / 2;
    const size_t hist = sizeof(float) * P * nbins, smem = hist + sizeof(double) * nbins;
    if (nspc < 1 || nspc > SUR_MAX_SPC || nbins < 1 || hist > 48 * 1024) return (int)cudaErrorInvalidValue;
    if (smem > 16 * 1024) { /* with the static arrays (26 KB) past the default limit */
        /* the largest size any call has (one species): a limit of a call's own
         * size could fall between another thread's limit and its launch */
        const cudaError_t e = cudaFuncSetAttribute(k_rdf, cudaFuncAttributeMaxDynamicSharedMemorySize, 3 * 48 * 1024);
        if (e != cudaSuccess) return (int)e;
    }
    k_rdf<<<S, 256, smem, (cudaStream_t)stream>>>(S, off, spc, lat, x, nspc, nbins, rmax, sigma, feat, status);
    return (int)cudaGetLastError();
}

extern "C" int surk_colsum(int B, int O, const float *dZ, float *out, void *stream) {
    k_colsum<<<(O + 127) / 128, 128, 0, (cudaStream_t)stream>>>(B, O, dZ, out);
    return (int)cudaGetLastError();
}

extern "C" int surk_mse(int B, const float *y, const float *t, float *dy, double *loss, void *stream) {
    k_mse<<<1, 256, 0, (cudaStream_t)stream>>>(B, y, t, dy, loss);
    return (int)cudaGetLastError();
}

extern "C" int surk_adam(long n, float *p, const float *g, float *m, float *v, float lr, float b1, float b2, float eps,
                         float c1, float c2, void *stream) {
    long blocks = (n + 255) / 256;
    if (blocks > 1184) blocks = 1184; /* 148 SMs x 8 */
    k_adam<<<(int)blocks, 256, 0, (cudaStream_t)stream>>>(n, p, g, m, v, lr, b1, b2, eps, c1, c2);
    return (int)cudaGetLastError();
}

extern "C" int surk_gather(int B, int F, const int *idx, const float *X, const float *mean, const float *istd,
                           float *out, const float *T, float tmean, float tistd, float *tout, void *stream) {
    if (B < 1) return 0;
    k_gather<<<B, 256, 0, (cudaStream_t)stream>>>(B, F, idx, X, mean, istd, out, T, tmean, tistd, tout);
    return (int)cudaGetLastError();
}

extern "C" int surk_colstats(int S, int F, const float *X, float *mean, float *istd, void *stream) {
    k_colstats<<<(F + 127) / 128, 128, 0, (cudaStream_t)stream>>>(S, F, X, mean, istd);
    return (int)cudaGetLastError();
}
