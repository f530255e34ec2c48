/* mb_batch.h -- launcher of the persistent population relax (mb_batch.cu). */
#ifndef MB_BATCH_H
#define MB_BATCH_H
#include "../mb_internal.h"
#ifdef __cplusplus
extern "C" {
#endif
/* What a handle keeps for its batched calls. */
typedef struct {
    void *model; /* FP32 weights on the device (uploaded once) */
    void *params; /* FP32 parameters, passed to the kernel by value */
    mb_ws io;    /* inputs and results of a call, staged through pinned memory */
    mb_ws scratch; /* per-CTA inverse Hessians and neighbour lists */
    void *e0, *e1; /* events around the launch */
} mb_batch_ws;
int mbk_relax_batch(const mb_model *m, mb_batch_ws *ws, int S, const int *d_nat, const int *d_off, const int *d_spc,
                    const int *d_order, double *d_lat, double *d_x, double p_ev, double urep, int rlxt, int mitr, double fmax, double *d_H, int *d_iters,
                    int *d_status, double *d_frc, double *d_str, long long *d_evals, void *stream);
void mbk_batch_free(mb_batch_ws *ws);
int mbk_batch_clusters(int S, int mitr, int sms); /* CTAs per structure */
#ifdef __cplusplus
}
#endif
#endif
