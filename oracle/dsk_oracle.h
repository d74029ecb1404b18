/* oracle/dsk_oracle.h — CPU restatement of the reference decode path.  TEST INFRASTRUCTURE ONLY.
 *
 * Only tests/, __graft_entry__.smoke() and bench.py's cpu_baseline/reference legs may load this
 * library.  The product (deepseek.cpp_b200/) never links or calls it.
 *
 * Parity pinning: every function here is checked against oracle/_ref/libdsref.so (the UNMODIFIED
 * reference compiled, see oracle/Makefile) by tests/test_oracle_vs_ref.py and
 * against the committed golden vectors in tests/golden/ (generated by tests/golden/make_golden.py
 * from that same library, plus the known answers of the reference's own src/test.cpp:128-186).
 *
 * All file:line citations are relative to the reference at commit 8db9e56.
 */
#ifndef DSK_ORACLE_H
#define DSK_ORACLE_H
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

enum { ORK_F32 = 0, ORK_F16 = 1, ORK_F8E5M2 = 2, ORK_Q2_K = 3, ORK_Q3_K = 4 }; /* src/codec.h:79-85 */

#define ORK_QK_K 256
#pragma pack(push, 1)
typedef struct { uint8_t scales[16]; uint8_t qs[64]; uint16_t d; uint16_t dmin; } ork_block_q2_K; /* quant.h:41-52 */
typedef struct { uint8_t hmask[32]; uint8_t qs[64]; uint8_t scales[12]; uint16_t d; } ork_block_q3_K; /* quant.h:70-76 */
typedef struct { float d; int8_t qs[256]; int16_t bsums[16]; } ork_block_q8_K;                        /* quant.h:104-109 */
#pragma pack(pop)

/* A weight matrix (or expert stack) as the reference's QTensor (src/codec.h:107-120). */
typedef struct {
  int quant;          /* ORK_* */
  int n_experts;      /* 0 for a plain (rows, cols) matrix */
  int rows, cols;     /* d, n */
  const void* data;
  const float* scale; /* F8E5M2 only: (ceil(rows/bs0), ceil(cols/bs1)) per expert */
} ork_tensor;

typedef struct { /* src/model.h:47-96 */
  int dim, hidden_dim, n_layers, n_heads, vocab_size, max_seq_len;
  float rope_theta, norm_eps;
  int act_silu; /* 1 silu, 0 gelu */
  int first_k_dense_replace;
  int n_shared_experts, n_routed_experts, n_active_routed, moe_intermediate_size;
  float routed_scaling_factor;
  int n_group, norm_topk_prob, scoring_sigmoid, topk_group, topk_method; /* 0 greedy, 1 group_limited_greedy */
  int is_v3; /* has_moegate_bias: arch == DeepseekV3ForCausalLM */
  int kv_lora_rank, q_lora_rank, qk_nope_head_dim, qk_rope_head_dim, v_head_dim, head_dim;
  int quant;
  int bs0, bs1;
  int original_max_position;
  int use_mla; /* true-MLA blocks (BlockMLA, src/model.h:366-453) */
} ork_config;

typedef struct {
  const float *rms_att, *rms_ffn, *rms_q_a, *rms_kv_a;
  ork_tensor wq, wq_a, wq_b, wkv_a, wkv_b, wo;
  ork_tensor wc, wq_rope_b, wv_b;    /* use_mla: (n_heads*kv_lora_rank, q_lora_rank), (n_heads*qk_rope_head_dim, q_lora_rank),
                                        n_heads stacked (v_head_dim, kv_lora_rank) slabs (src/model.cpp:569-580) */
  int is_moe;
  ork_tensor w1, w2, w3;             /* dense, or expert stacks when is_moe */
  ork_tensor sw1, sw2, sw3;          /* shared experts */
  const float *moegate, *moegate_bias;
  uint16_t *key_cache, *value_cache; /* fp16 (max_seq_len, n_heads*head_dim) / (max_seq_len, n_heads*v_head_dim);
                                        use_mla: kv_nope_cache (max_seq_len, kv_lora_rank) / kv_rope_cache (max_seq_len, qk_rope_head_dim) */
} ork_layer;

typedef struct {
  ork_config cfg;
  ork_layer* layers;
  ork_tensor embed;
  const float* rms_final;
  ork_tensor wcls;
} ork_model;

typedef struct { /* src/model.h:101-179 */
  float *x, *xb, *xb2, *hb, *hb2, *q_a, *q, *kv_a, *kv_b, *att, *moe_weights, *active_experts_weights, *logits;
  int* active_experts;
  float *q_c, *q_rope; /* use_mla: (n_heads*kv_lora_rank), (n_heads*qk_rope_head_dim) (src/model.h:166-167) */
} ork_state;

/* scalar helpers */
float ork_half_to_float(uint16_t h);
uint16_t ork_float_to_half(float f);
float ork_f8e5m2_to_float(uint8_t b);

/* quant.cpp */
void ork_quantize_row_q8_K(const float* x, ork_block_q8_K* y, long k);
void ork_dequantize_row_q2_K(const ork_block_q2_K* x, float* y, long k);
void ork_dequantize_row_q3_K(const ork_block_q3_K* x, float* y, long k);
float ork_vec_dot_q2_K_q8_K(int n, const ork_block_q2_K* x, const ork_block_q8_K* y);
float ork_vec_dot_q3_K_q8_K(int n, const ork_block_q3_K* x, const ork_block_q8_K* y);

/* infer.cpp */
void ork_matmul(float* xout, const float* x, const ork_tensor* w, int expert, int bs0, int bs1);
void ork_softmax(float* o, const float* x, int size);
void ork_moe_gate(float* moe_weights, const float* bias, int* active_experts, float* x, int n_routed, int n_active,
                  int norm_topk_prob, float routed_scaling_factor, int scoring_sigmoid, int topk_method, int n_group,
                  int topk_group);
void ork_rmsnorm(float* o, const float* x, const float* w, int size, float eps);
void ork_rope(float* vec, int d, int head_dim, int pos, float theta);
void ork_rope_v3(float* vec, int d, int head_dim, int pos, float theta);
void ork_rope_f16(uint16_t* vec, int d, int head_dim, int pos, float theta);
void ork_rope_v3_f16(uint16_t* vec, int d, int head_dim, int pos, float theta);
float ork_silu(float x);
float ork_gelu(float x);
void ork_attn(float* xout, float* atth, const float* qh, const uint16_t* kh, const uint16_t* vh, int head_dim,
              int v_head_dim, int n_heads, int kv_len);
void ork_attn_mla(float* xout, float* atth, const float* qh_c, const float* qh_rope, const uint16_t* ckv, const uint16_t* k_rope,
                  int head_dim, int kv_lora_rank, int qk_rope_head_dim, int kv_len);
void ork_copy_embedding(const ork_model* m, ork_state* s, int token);
void ork_block(const ork_model* m, ork_state* s, int layer, int pos, int kv_sink, int kv_pos, int kv_len);
void ork_forward(const ork_model* m, ork_state* s, int token, int pos, int output_logits);
int ork_argmax(const float* logits, int n);
void ork_set_num_threads(int n);

#ifdef __cplusplus
}
#endif
#endif
