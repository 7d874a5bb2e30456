/* One block-sparse attention problem: what ftk_attn_fwd, ftk_attn_bwd_dq and
 * ftk_attn_bwd_dkv take (see ftk_api.h for the conventions on pointers). */
#ifndef FTK_ATTN_H_
#define FTK_ATTN_H_

#include <stdint.h>

typedef struct ftk_attn {
  const void *q, *k, *v;        /* 16-bit, element [b][n][h][d] at the strides below, d dense */
  int dtype;                    /* FTK_F16 or FTK_BF16 */
  int out_f32;                  /* 1: o, dq, dk, dv are float (the 16-bit results, widened) */
  int64_t B, H, Hkv, N, D;      /* H % Hkv == 0; D a multiple of 8 up to 256 */
  int64_t sq_b, sq_n, sq_h, sk_b, sk_n, sk_h, sv_b, sv_n, sv_h;
  const int32_t* lists;         /* [B*H][list_rows][W] block ids, negative = none */
  int list_rows, W;             /* list_rows * q_block >= q_pad_head + N */
  int q_block, kv_block;        /* rows per listed block, up to 128 */
  int q_pad_head, kv_pad_head;  /* virtual rows before token 0 of either grid */
  float scale;
} ftk_attn;

#endif
