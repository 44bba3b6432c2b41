// Layers of a prompt portion as one host call (fk_llama_prompt_layers): nothing but the calls of
// the entry points.  A launch costs the host 20 us where each goes through Python and ctypes, and
// about 5 here; a short prompt's kernels take 9 on average (61 tokens, 8 layers: 1740 -> 960 us a
// prompt).  Both structs are read between the launches: the caller keeps them until the call
// returns.
#include "fk_common.cuh"

using namespace fk;

extern "C" int fk_llama_prompt_layers(const fk_llama_layer* layers, int num_layers, int first,
                                      const fk_llama_prompt* prompt, fk_stream_t stream) {
  FK_REQUIRE(num_layers >= 0 && (layers || num_layers == 0) && prompt, FK_ERR_INVALID_ARG,
             "fk_llama_prompt_layers: bad arguments");
  const fk_llama_prompt& p = *prompt;
  FK_REQUIRE(p.tokens >= 0 && p.hidden > 0 && p.ff > 0 && p.num_q_heads > 0 &&
                 p.num_kv_heads > 0 && p.head_dim > 0 && p.block_size > 0 && p.num_blocks > 0 &&
                 p.num_seqs > 0 && p.workspace_bytes >= 0,
             FK_ERR_INVALID_ARG, "fk_llama_prompt_layers: bad sizes");
  if (p.tokens == 0 || num_layers == 0) return FK_OK;
  FK_REQUIRE(p.residual && p.x && p.qkv && p.attn && p.act && p.positions && p.cos_sin_cache &&
                 p.slots && p.cu_seqlens_q && p.cu_seqlens_k && p.block_table,
             FK_ERR_INVALID_ARG, "fk_llama_prompt_layers: null pointer");
  const int64_t m = p.tokens, q = p.num_q_heads * p.head_dim, kv = p.num_kv_heads * p.head_dim;
  const int64_t qkv = q + 2 * kv;
  const size_t ws = (size_t)p.workspace_bytes;
  const bool few = fk_gemm_bf16_silu_mul_fusable(m, 2 * p.ff, p.hidden) != 0;
#define FK_TRY(call)           \
  do {                         \
    const int rc__ = (call);   \
    if (rc__ != FK_OK) return rc__; \
  } while (0)
  for (int i = 0; i < num_layers; ++i) {
    const fk_llama_layer& l = layers[i];
    if (first && i == 0)
      FK_TRY(fk_rmsnorm(p.residual, p.hidden, 0, 1, p.x, p.hidden, 0, l.input_norm,
                        (float)l.input_eps, m, p.hidden, stream));
    else
      FK_TRY(fk_fused_add_rmsnorm(p.x, p.hidden, p.residual, p.hidden, l.input_norm,
                                  (float)l.input_eps, m, p.hidden, stream));
    FK_TRY(fk_gemm_bf16(p.x, p.hidden, l.qkv, l.qkv_bias, p.qkv, qkv, m, qkv, p.hidden, p.workspace,
                        ws, p.status, stream));
    FK_TRY(fk_qkv_rope_store(p.qkv, qkv, (int)p.num_q_heads, (int)p.num_kv_heads, (int)p.head_dim,
                             p.positions, p.cos_sin_cache, 0, p.max_position, l.q_norm, l.k_norm,
                             (float)l.qk_eps, l.k_cache, l.v_cache, p.slots,
                             p.num_blocks * p.block_size, (int)p.block_size, (int)p.kv_layout, m,
                             p.status, stream));
    FK_TRY(fk_prefill_attn(p.qkv, qkv, p.attn, q, nullptr, l.k_cache, l.v_cache, p.kv_block_stride,
                           p.num_blocks, (int)p.block_size, (int)p.kv_layout, p.cu_seqlens_q,
                           p.cu_seqlens_k, p.block_table, p.block_table_stride, (int)p.num_seqs, m,
                           0, (int)p.max_seqlen_q, (int)p.num_q_heads, (int)p.num_kv_heads,
                           (int)p.head_dim, (float)l.softmax_scale, 1, l.attn_status, stream));
    FK_TRY(fk_gemm_bf16(p.attn, q, l.o, l.o_bias, p.x, p.hidden, m, p.hidden, q, p.workspace, ws,
                        p.status, stream));
    FK_TRY(fk_fused_add_rmsnorm(p.x, p.hidden, p.residual, p.hidden, l.post_norm,
                                (float)l.post_eps, m, p.hidden, stream));
    if (few)
      FK_TRY(fk_gemm_bf16_silu_mul(p.x, p.hidden, l.gate_up, l.gate_up_bias, p.act, p.ff, m,
                                   2 * p.ff, p.hidden, p.workspace, ws, p.status, stream));
    else
      FK_TRY(fk_gemm_bf16_act_mul_many(p.x, p.hidden, l.gate_up, l.gate_up_bias, p.act, p.ff, m,
                                       2 * p.ff, p.hidden, FK_ACT_SILU, p.status, stream));
    FK_TRY(fk_gemm_bf16(p.act, p.ff, l.down, l.down_bias, p.x, p.hidden, m, p.hidden, p.ff,
                        p.workspace, ws, p.status, stream));
  }
#undef FK_TRY
  return FK_OK;
}
