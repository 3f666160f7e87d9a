/* Descriptors of stu_token_step (see include/stu_b200.h); plain C. */
#ifndef STU_STEP_H
#define STU_STEP_H

#define STU_STEP_MAX_LAYERS 40
#define STU_STEP_STU 0
#define STU_STEP_ATTENTION 1

typedef struct {
  int kind;            /* STU_STEP_STU or STU_STEP_ATTENTION */
  int Lh;              /* STU: positions per parity row of the history */
  int W;               /* attention: slots of the key / value rings */
  float eps1, eps2;    /* of the two norms */
  int reserved;
  const void* norm1;   /* [d] */
  const void* w1;      /* STU: M_inputs^T [d][d]; attention: c_attn [3d][d] */
  const void* wo;      /* attention: c_proj [d][d] */
  const void* norm2;   /* [d] */
  const void* wg;      /* [I][d] */
  const void* wu;      /* [I][d] */
  const void* wd;      /* [d][I] */
  void* hist;          /* STU: [B][d][2][Lh] */
  const void* taps;    /* STU: fp32 [d][Lh]; bf16 the reversed tables [8][d][Lh + 8] */
  void* k_ring;        /* attention: [B][W][d] */
  void* v_ring;
  const float* slopes; /* attention: [H] */
  int* pos;            /* [B][2] */
} StuStepLayer;

typedef struct {
  int n_layers, B, d, I, H, window, V;
  float softcap, eps_final;
  int reserved;
  const long long* ids; /* token of sequence b at ids[b * ids_stride], or NULL: x holds the input rows */
  long long ids_stride;
  const void* embedding; /* [V][d] */
  void* x;               /* [B][d] residual stream, input (ids NULL) and output */
  const void* norm_final; /* with lm_head */
  const void* lm_head;    /* [V][d], or NULL: stop after the last layer */
  void* logits;           /* [B] rows of V */
  long long ld_logits;
  void* workspace;        /* stu_token_step_workspace_bytes, 256-byte aligned, zeroed once */
  long long workspace_bytes;
  int* status;
} StuStepArgs;

#endif
