// Vector-sparse flash attention: launch parameters from the C ABI's argument struct, and the choice of the
// kernel by query-tile height (q_pooling_size 64: va_attn64.cu, 128: va_attn128.cu; dense rows: va_dense128.cu).
#include "va_common.cuh"
#include "va_attn.cuh"

namespace va {

int launch_attn64(const AttnParams& p, int dtype, int batch, cudaStream_t stream);   // va_attn64.cu
int launch_attn128(const AttnParams& p, int dtype, int batch, cudaStream_t stream);  // va_attn128.cu
bool launch_dense128(const AttnParams& p, int dtype, int batch, cudaStream_t stream, int* rc);  // va_dense128.cu

// own_blocks: the tables' place is taken by the operator's own rule (see AttnParams)
int sparse_attn(const va_attn_args& a, cudaStream_t stream, bool own_blocks, int first_tile, int seq_len) {
  AttnParams p;
  p.q = a.q.ptr; p.k = a.k.ptr; p.v = a.v.ptr; p.out = a.out.ptr;
  p.q_sb = a.q.stride_b; p.q_sh = a.q.stride_h; p.q_ss = a.q.stride_s;
  p.k_sb = a.k.stride_b; p.k_sh = a.k.stride_h; p.k_ss = a.k.stride_s;
  p.v_sb = a.v.stride_b; p.v_sh = a.v.stride_h; p.v_ss = a.v.stride_s;
  p.o_sb = a.out.stride_b; p.o_sh = a.out.stride_h; p.o_ss = a.out.stride_s;
  auto row_bytes = [](int64_t ss) { return ss >= -(1 << 30) && ss < (1 << 30) ? (int)(ss * 2) : 0; };
  p.k_row_bytes = row_bytes(p.k_ss);
  p.v_row_bytes = row_bytes(p.v_ss);
  p.blk_count = a.blk_idx ? a.blk_count : nullptr;
  p.blk_idx = a.blk_idx; p.blk_stride = a.blk_stride;
  p.own_blocks = own_blocks; p.first_tile = first_tile; p.seq_len = seq_len;
  p.col_count = a.col_count; p.col_idx = a.col_idx; p.col_stride = a.col_stride;
  p.status = a.status;
  p.lse = a.lse;
  p.heads = a.heads; p.rep = a.heads / a.kv_heads; p.sq = a.sq; p.sk = a.sk;
  p.vis_on = a.vision_mode != 0; p.vis_begin = a.vision_begin; p.vis_end = a.vision_end;
  p.nq = ((p.vis_on ? a.vision_end : a.sq) + a.pq - 1) / a.pq;
  p.causal = a.causal; p.q_offset = a.q_offset;
  const float scale = a.softmax_scale > 0.f ? a.softmax_scale : 0.08838834764831845f;
  p.scale_log2 = scale * 1.4426950408889634f;
  // Heads whose K and V together fit half of L2 are listed together, tile by tile: no head's longest causal tiles start
  // last, and the SMs gather from several heads at a time.  Whole calls, head by head and so, with the K and V of one group:
  // 28 query heads on 4 KV heads, causal, 9001 tokens (all heads, 18 MB) 389 -> 350 us, 20011 with a vision span (41 MB) 984 -> 854,
  // 64 K (2 KV heads, 64 MB) 6069 -> 5912; 32 heads, 48 K, causal (2, 48 MB) 4290 -> 4096; not causal, 8 heads x 16 000 (33 MB)
  // 320 -> 286, 32 x 32 K (3, 50 MB) 3299 -> 3235.  Groups of up to 100 MB are slower where the keys are spread over the
  // sequence: 32 x 32 K 3383, 16 x 100 K not causal 14 002 -> 14 833; of up to 24 MB: 3291 and 4280.
  const int64_t kv_bytes = (int64_t)a.sk * kHeadDim * 2 * 2;
  const int64_t fit = kv_bytes < (64 << 20) ? (64 << 20) / kv_bytes : 1;
  const int groups = (int)((a.kv_heads + fit - 1) / fit);
  p.group = (a.kv_heads + groups - 1) / groups * p.rep;
  if (p.vis_on && p.vis_begin >= p.vis_end) {  // every row is dense: 128-row tiles on streamed K and V take 0.47 ms where
    // gathered 64-row tiles took 0.86 (28 query heads on 4 KV heads, 8192 tokens).  A composition with sparse rows keeps its
    // dense tiles in the 64-row launch: they are few, and a launch of their own would leave most SMs idle.
    int rc;
    if (launch_dense128(p, a.dtype, a.batch, stream, &rc)) return rc;
  }
  return a.pq == 64 ? launch_attn64(p, a.dtype, a.batch, stream) : launch_attn128(p, a.dtype, a.batch, stream);
}

}  // namespace va
