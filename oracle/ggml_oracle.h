/* oracle/ggml_oracle.h -- TEST INFRASTRUCTURE, NOT PRODUCT CODE.
 *
 * CPU restatement of the reference's algorithm for the hot path (GGML MUL_MAT / MUL_MAT_ID over
 * Q4_0, Q8_0, Q4_K, Q5_K, Q6_K and FLASH_ATTN_EXT over an f16 / q8_0 KV cache).
 * Only tests/, __graft_entry__.smoke() and bench.py's cpu_baseline / --impl reference legs may
 * load this library; the product (koboldcpp_b200/) never does.
 *
 * Parity status: PINNED.  Every function here is checked bit-for-bit (integer/byte outputs and
 * block dequantisation) or to <= 2 ulp-of-sum (float dot products, where only the summation
 * order of the SIMD reference differs) against the reference itself compiled from
 * /root/reference into oracle/_ref/libggml_ref*.so -- see tests/test_oracle_vs_ref.py and the
 * committed vectors in tests/golden/ (generated by tests/golden/make_golden.py).
 *
 * All citations are file:line under /root/reference/.
 */
#ifndef GGML_ORACLE_H
#define GGML_ORACLE_H

#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

/* ggml type ids used on this path (ggml/include/ggml.h:361-398) */
enum {
    ORC_TYPE_F32  = 0,
    ORC_TYPE_F16  = 1,
    ORC_TYPE_Q4_0 = 2,
    ORC_TYPE_Q4_1 = 3,
    ORC_TYPE_Q5_0 = 6,
    ORC_TYPE_Q5_1 = 7,
    ORC_TYPE_Q8_0 = 8,
    ORC_TYPE_Q8_1 = 9,
    ORC_TYPE_Q2_K = 10,
    ORC_TYPE_Q3_K = 11,
    ORC_TYPE_Q4_K = 12,
    ORC_TYPE_Q5_K = 13,
    ORC_TYPE_Q6_K = 14,
    ORC_TYPE_Q8_K = 15,
    ORC_TYPE_IQ4_NL = 20, /* non-linear 4-bit: 32 values, codebook of 16 int8 levels   ggml.h:383 */
    ORC_TYPE_IQ4_XS = 23, /* the same codebook in 256-value super-blocks with 6-bit scales  ggml.h:386 */
};

/* block geometry: ggml/src/ggml-common.h:144-335 */
int    orc_blck_size(int type);            /* values per block (1, 32 or 256)          */
size_t orc_type_size(int type);            /* bytes per block                           */
size_t orc_row_size(int type, int64_t ne); /* ggml_row_size, ggml/src/ggml.c:3580-3583  */

/* fp16 <-> fp32, IEEE round-to-nearest-even (ggml/src/ggml-impl.h:80-170) */
float    orc_fp16_to_fp32(uint16_t h);
uint16_t orc_fp32_to_fp16(float f);

/* block -> f32, bit-exact with dequantize_row_* (ggml-quants.c:1523,1617,2556,2764,2978) */
int orc_dequantize_row(int type, const void *src, float *dst, int64_t k);

/* f32 -> activation blocks, bit-exact with quantize_row_q8_0_ref / q8_1_ref / q8_K_ref
 * (ggml-quants.c:849-872, 1160-1193, 3786-3823) and f32 -> q4_0 weights (:669-704) */
int orc_quantize_row(int type, const float *src, void *dst, int64_t k);

/* scalar dot products, the `#else` branches of ggml_vec_dot_{q4_0_q8_0, q8_0_q8_0,
 * q4_K_q8_K, q5_K_q8_K, q6_K_q8_K} (ggml-quants.c:4484-4500, 5846-5858, 8223-8278,
 * 8855-8914, 9524-9566). `wtype` selects the weight type; activations are in that type's
 * vec_dot_type (q8_0 for Q4_0/Q8_0, q8_K for K-quants; ggml.c:793-808, 873-889, 924-959). */
float orc_vec_dot(int wtype, int64_t n, const void *w, const void *act);

/* The integer arithmetic the GPU path performs: weights x 32-wide q8_1 activation blocks
 * (reference CUDA vecdotq.cuh:23-42,151-163,357-379,413-442,476-496),
 * accumulated in double. Used for tight-tolerance kernel checks. */
double orc_vec_dot_q8_1(int wtype, int64_t n, const void *w, const void *act_q8_1);

/* MUL_MAT as the CPU backend computes it (ggml.c:12486-12707): each src1 column is quantised
 * to vec_dot_type, dst[n*M + m] = vec_dot(W row m, col n).  W: M rows of K values, row stride
 * `w_row_bytes`; X: f32 [N][K] contiguous; dst f32 [N][M]. nthreads<=0 -> all cores. */
int orc_mul_mat(int wtype, const void *w, size_t w_row_bytes, const float *x, float *dst,
                int64_t K, int64_t M, int64_t N, int nthreads);

/* Same contraction with the GPU path's activation format (q8_1); dst in double. */
int orc_mul_mat_q8_1(int wtype, const void *w, size_t w_row_bytes, const float *x, double *dst,
                     int64_t K, int64_t M, int64_t N, int nthreads);

/* MUL_MAT_ID (ggml.c:12711-12916, constructor ggml.c:5693-5729):
 *   dst[t][e][:] = as[ids[t][e]] (M x K) . b[t][e % n_b_rows][:]
 * as: n_expert matrices of M rows, expert stride `w_expert_bytes`; ids: i32 [T][n_used];
 * b: f32 [T][n_b_rows][K]; dst: f32 [T][n_used][M]. */
int orc_mul_mat_id(int wtype, const void *as, size_t w_row_bytes, size_t w_expert_bytes,
                   const int32_t *ids, const float *b, float *dst,
                   int64_t K, int64_t M, int64_t n_expert, int64_t n_used, int64_t n_b_rows,
                   int64_t T, int nthreads);

/* FLASH_ATTN_EXT as ggml_compute_forward_flash_attn_ext_f16 computes it (ggml.c:15667-15877):
 * one pass over the KV rows per (q row, head) with scalar online softmax; Q converted to K's
 * vec_dot_type (f16 or q8_0); V accumulated in f16 when V is f16, else f32 after dequant.
 *   q    f32  [n_head][N][D]      (element strides given in bytes: q_nb1 = per-row, q_nb2 = per-head)
 *   k,v  type [n_head_kv][n_kv][D-row]  (k_nb1 per-row bytes, k_nb2 per-head bytes; same for v)
 *   mask f16  [N_pad][n_kv] or NULL (mask_nb1 = bytes per q row)
 *   dst  f32  [N][n_head][D]      (the op's permuted output layout)
 */
typedef struct {
    int64_t D, N, n_head, n_head_kv, n_kv;
    int     type_k, type_v;
    size_t  q_nb1, q_nb2, k_nb1, k_nb2, v_nb1, v_nb2, mask_nb1;
    float   scale, max_bias, logit_softcap;
} orc_fattn_params;
int orc_flash_attn_ext(const orc_fattn_params *p, const void *q, const void *k, const void *v,
                       const void *mask, float *dst, int nthreads);

/* double-precision softmax(QK^T*scale+mask)V on dequantised K/V -- the "ground truth" both the
 * CPU reference and the GPU kernel are measured against. Same layouts as above; dst f64. */
int orc_flash_attn_f64(const orc_fattn_params *p, const void *q, const void *k, const void *v,
                       const void *mask, double *dst, int nthreads);

#ifdef __cplusplus
}
#endif
#endif
