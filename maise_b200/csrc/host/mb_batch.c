/*
 * mb_batch.c -- host side of the population relax: packs the structures,
 * launches the persistent kernel (mb_batch.cu) and returns the results.
 */
#include <cuda_runtime_api.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "../../../include/maise_b200.h"
#include "mb_batch.h"

#define MB_EV2GPA 160.2176565 /* src/util.c:8 */

/* the handle layout is private to mb_core.c; these accessors are defined there */
const mb_model *mb_handle_model(const mb_potential *p);
void *mb_handle_stream(mb_potential *p);
int mb_handle_device(const mb_potential *p);
int mb_handle_fail(int code, const char *msg);
mb_batch_ws *mb_handle_batch(mb_potential *p);
void mb_handle_set_batch_stats(mb_potential *p, const long long *evals, float ms);

/* The population relax and the batched E/F/S share this: with frc/str set
 * the kernel also returns each structure's forces and virial at its final
 * state, and with keep_xyz = 0 the positions and lattices are not copied back. */
static int batch_run(mb_potential *pot, int S, const int *nat, const int *atmn, double *lat, double *x, double p_gpa,
                     double urep, int rlxt, int mitr, double fmax, double *H, int *iters, int *status, double *frc,
                     double *str, int keep_xyz) {
    int *off, *order, total = 0, s;
    size_t at = 0, up, b_nat, b_off, b_order, b_spc, b_lat, b_x, b_H, b_iters, b_status, b_frc, b_str, b_ev, down;
    char *h, *d;
    float ms = 0.0f;
    const mb_model *m;
    mb_batch_ws *ws;
    cudaStream_t st;
    cudaError_t e;
    if (!pot || S < 1 || !nat || !atmn || !lat || !x || !H || !iters || !status || !(fmax > 0) || mitr < 0)
        return mb_handle_fail(MB_ERR_ARG, "bad arguments");
    if (!(rlxt == 2 || rlxt == 3)) return mb_handle_fail(MB_ERR_ARG, "batched relax supports RLXT 2 and 3");
    m = mb_handle_model(pot);
    for (s = 0; s < S; s++) {
        if (nat[s] < 1 || nat[s] > 64) return mb_handle_fail(MB_ERR_ARG, "batched relax takes 1..64 atoms per structure");
        total += nat[s];
    }
    for (s = 0; s < total; s++)
        if (atmn[s] < 0 || atmn[s] >= m->nspc) return mb_handle_fail(MB_ERR_ARG, "species index out of range");
    /* one block for the call's data, the same offsets on the device and in
     * pinned memory: inputs first, what is both in the middle, results last */
#define PUT(name, bytes) (name = at, at += ((size_t)(bytes) + 15) & ~(size_t)15)
    PUT(b_nat, sizeof(int) * S);
    PUT(b_off, sizeof(int) * (S + 1));
    PUT(b_order, sizeof(int) * S);
    PUT(b_spc, sizeof(int) * total);
    PUT(b_lat, sizeof(double) * 9 * S);
    PUT(b_x, sizeof(double) * 3 * total);
    up = at;
    PUT(b_ev, 4 * sizeof(long long)); /* evaluations, atom evaluations, pairs, triplets */
    PUT(b_H, sizeof(double) * S);
    PUT(b_iters, sizeof(int) * S);
    PUT(b_status, sizeof(int) * S);
    PUT(b_frc, frc ? sizeof(double) * 3 * total : 0);
    PUT(b_str, frc ? sizeof(double) * 6 * S : 0);
#undef PUT
    cudaSetDevice(mb_handle_device(pot));
    st = (cudaStream_t)mb_handle_stream(pot);
    ws = mb_handle_batch(pot);
    e = (cudaError_t)mb_ws_grow(&ws->io, at, at);
    if (e) return mb_handle_fail(MB_ERR_CUDA, cudaGetErrorString(e));
    h = (char *)ws->io.host;
    d = (char *)ws->io.dev;
    off = (int *)(h + b_off);
    order = (int *)(h + b_order);
    memcpy(h + b_nat, nat, sizeof(int) * S);
    for (s = 0, off[0] = 0; s < S; s++) off[s + 1] = off[s] + nat[s];
    /* the persistent CTAs take structures largest first, so that the last
     * ones to start are small and the population finishes evenly */
    {
        int first[66] = {0}, n;
        for (s = 0; s < S; s++) first[64 - nat[s] + 1]++;
        for (n = 1; n < 66; n++) first[n] += first[n - 1];
        for (s = 0; s < S; s++) order[first[64 - nat[s]]++] = s;
    }
    memcpy(h + b_spc, atmn, sizeof(int) * total);
    memcpy(h + b_lat, lat, sizeof(double) * 9 * S);
    memcpy(h + b_x, x, sizeof(double) * 3 * total);
    memset(h + b_ev, 0, 4 * sizeof(long long));
    e = cudaMemcpyAsync(d, h, b_ev + 4 * sizeof(long long), cudaMemcpyHostToDevice, st);
    if (!e)
        e = (cudaError_t)mbk_relax_batch(m, ws, S, (int *)(d + b_nat), (int *)(d + b_off), (int *)(d + b_spc),
                                         (int *)(d + b_order), (double *)(d + b_lat), (double *)(d + b_x),
                                         p_gpa / MB_EV2GPA, urep > 0 ? urep : 0.0, rlxt, mitr, fmax,
                                         (double *)(d + b_H), (int *)(d + b_iters), (int *)(d + b_status),
                                         frc ? (double *)(d + b_frc) : NULL, frc ? (double *)(d + b_str) : NULL,
                                         (long long *)(d + b_ev), st);
    if (e == cudaErrorInvalidValue)
        return mb_handle_fail(MB_ERR_MODEL, "batched relax needs a basis with <= 7 G4 exponents, zeta in {integers}, "
                                            "2 lambdas, <= 16 G2 functions and D <= 288");
    /* results: from the lattices on when they are wanted back, else past the inputs */
    down = keep_xyz ? b_lat : up;
    if (!e) e = cudaMemcpyAsync(h + down, d + down, at - down, cudaMemcpyDeviceToHost, st);
    if (!e) e = cudaStreamSynchronize(st);
    if (e) return mb_handle_fail(MB_ERR_CUDA, cudaGetErrorString(e));
    if (keep_xyz) {
        memcpy(lat, h + b_lat, sizeof(double) * 9 * S);
        memcpy(x, h + b_x, sizeof(double) * 3 * total);
    }
    if (frc) memcpy(frc, h + b_frc, sizeof(double) * 3 * total);
    if (frc && str) memcpy(str, h + b_str, sizeof(double) * 6 * S);
    memcpy(H, h + b_H, sizeof(double) * S);
    memcpy(iters, h + b_iters, sizeof(int) * S);
    memcpy(status, h + b_status, sizeof(int) * S);
    cudaEventElapsedTime(&ms, (cudaEvent_t)ws->e0, (cudaEvent_t)ws->e1);
    mb_handle_set_batch_stats(pot, (long long *)(h + b_ev), ms);
    return MB_OK;
}

int mb_relax_batch(mb_potential *pot, int S, const int *nat, const int *atmn, double *lat, double *x, double p_gpa,
                   double urep, int rlxt, int mitr, double fmax, double *H, int *iters, int *status) {
    return batch_run(pot, S, nat, atmn, lat, x, p_gpa, urep, rlxt, mitr, fmax, H, iters, status, NULL, NULL, 1);
}

int mb_efs_batch(mb_potential *pot, int S, const int *nat, const int *atmn, const double *lat, const double *x,
                 double p_gpa, double urep, double *H, double *frc, double *str) {
    int *iters, *status, rc;
    if (!frc || !H || S < 1) return mb_handle_fail(MB_ERR_ARG, "bad arguments");
    iters = (int *)malloc(sizeof(int) * S);
    status = (int *)malloc(sizeof(int) * S);
    /* no iterations: the kernel evaluates each structure once; the
     * positions and lattices are read, not written back */
    rc = batch_run(pot, S, nat, atmn, (double *)lat, (double *)x, p_gpa, urep, 3, 0, 1.0, H, iters, status, frc, str,
                   0);
    if (!rc)
        for (int s = 0; s < S; s++)
            if (status[s] == 2) {
                rc = mb_handle_fail(MB_ERR_NEIGHBOURS, "a structure has more than 96 neighbours per atom");
                break;
            }
    free(iters);
    free(status);
    return rc;
}

int mb_evos_write(const char *evos_dir, int gen, int member, int N, int nspc, const int *spcz, const int *atmn,
                  const double *lat0, const double *x0, const double *lat, const double *x, double H, double E,
                  double p_gpa, const double *frc, const double *str, int iters);

int mb_evos_relax(mb_potential *pot, const char *evos_dir, int gen, int p0, int S, const int *nat, const int *atmn,
                  double *lat, double *x, double p_gpa, double urep, int rlxt, int mitr, double fmax, double *H,
                  int *iters, int *status) {
    const mb_model *m;
    double *lat0, *x0, *frc, *str;
    int total = 0, s, rc, off = 0;
    if (!pot || !evos_dir || S < 1 || !nat || !atmn || !lat || !x || !H || !iters || !status || p0 < 0 || gen < 0)
        return mb_handle_fail(MB_ERR_ARG, "bad arguments");
    for (s = 0; s < S; s++) total += nat[s] > 0 ? nat[s] : 0;
    m = mb_handle_model(pot);
    lat0 = (double *)malloc(sizeof(double) * 9 * S);
    x0 = (double *)malloc(sizeof(double) * 3 * total);
    frc = (double *)malloc(sizeof(double) * 3 * total);
    str = (double *)malloc(sizeof(double) * 6 * S);
    if (!lat0 || !x0 || !frc || !str) {
        free(lat0); free(x0); free(frc); free(str);
        return mb_handle_fail(MB_ERR_ARG, "out of memory");
    }
    memcpy(lat0, lat, sizeof(double) * 9 * S);
    memcpy(x0, x, sizeof(double) * 3 * total);
    rc = batch_run(pot, S, nat, atmn, lat, x, p_gpa, urep, rlxt, mitr, fmax, H, iters, status, frc, str, 1);
    for (s = 0; s < S && rc == MB_OK; s++) {
        const double *L = lat + 9 * s;
        const double V = fabs(L[0] * L[4] * L[8] + L[2] * L[3] * L[7] + L[1] * L[5] * L[6] - L[0] * L[5] * L[7] -
                              L[1] * L[3] * L[8] - L[2] * L[4] * L[6]);
        const double E = H[s] - p_gpa / MB_EV2GPA * V;
        rc = mb_evos_write(evos_dir, gen, p0 + s, nat[s], m->nspc, m->spcz, atmn + off, lat0 + 9 * s, x0 + 3 * off,
                           L, x + 3 * off, H[s], E, p_gpa, frc + 3 * off, str + 6 * s, iters[s]);
        off += nat[s];
    }
    free(lat0); free(x0); free(frc); free(str);
    return rc;
}
