/* Arguments of the one-launch decode step (step_persistent.cu).  Plain C: model_kquant.c fills them. */
#ifndef CKB200_STEP_PERSISTENT_H
#define CKB200_STEP_PERSISTENT_H

#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

enum { PS_FMT_Q4K = 0, PS_FMT_Q6K_PLANAR = 1, PS_FMT_Q50_PLANAR = 2 };

typedef struct {
    const uint8_t *W;       /* Q4_K rows as in the reference; Q6_K and Q5_0 rows in their row-planar layouts */
    int M, nb;              /* rows; blocks per row (256 elements, Q5_0: 32) */
    int row_bytes;
    int fmt;
    int lanes;              /* lanes that share a row */
    int split;              /* the passes of a row pair go to different warps of a CTA */
    int passes, items;      /* loads of a lane per row; row pairs (or groups of them) of the matrix */
    int cta0, ncta;         /* the shares [cta0, cta0 + ncta) of the deal work on this matrix */
    int pad[2];
} PsSeg;

enum { PS_Q = 0, PS_K, PS_V, PS_O, PS_W1, PS_W2, PS_SEGS };

typedef struct {
    PsSeg seg[PS_SEGS];
    const float *ln1, *ln2;
    void *kc, *vc;          /* this layer's caches, [kv heads][max_seq][head_dim] */
} PsLayer;

#define PS_MAX_GROUP 8      /* query heads per kv head */

typedef struct {
    const PsLayer *layers;  /* device */
    int num_layers;
    PsSeg head;
    const float *final_gamma;
    const float *x;         /* embedded token, Da values */
    float *q, *att, *o, *mf, *prev, *logits;       /* rows between the phases, widths rounded up to 256 with zero tails */
    float *part;            /* partial attention results: ckb_step_persistent_scratch_bytes() */
    unsigned *sync;         /* zeroed once; ckb_step_persistent_sync_bytes() */
    const float *cos_cache, *sin_cache;
    int *pos;
    int D, Da, H, Hkv, head_dim, max_seq, kv_f16;
    int ctas;               /* CTAs that rows and keys are dealt to */
    int extra_arrivals;     /* 0 */
    float eps;
    size_t smem;            /* ckb_step_persistent_smem() */
} PsParams;

/* shared memory of a matrix's staged input row */
size_t ckb_step_persistent_stage_bytes(int fmt, int nb);
/* dynamic shared memory for rows of Da elements and staged inputs of at most `stage` bytes; 0: does not fit */
size_t ckb_step_persistent_smem(int Da, size_t stage, int head_dim, int kv_f16);
size_t ckb_step_persistent_scratch_bytes(int head_dim);
size_t ckb_step_persistent_sync_bytes(void);
/* the fields from `row_bytes` on, of a matrix whose format, shape and CTAs are given */
void ckb_step_persistent_plan(PsSeg *s);
int ckb_launch_step_persistent(const PsParams *p, void *stream);

#ifdef __cplusplus
}
#endif
#endif
