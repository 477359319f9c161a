// Vector-sparse flash attention: launch parameters from the C ABI's argument struct, and the choice of the
// kernel by query-tile height (q_pooling_size 64: va_attn64.cu, 128: va_attn128.cu).
#include "va_common.cuh"
#include "va_attn.cuh"

namespace va {

int launch_attn64(const AttnParams& p, int dtype, int batch, cudaStream_t stream);   // va_attn64.cu
int launch_attn128(const AttnParams& p, int dtype, int batch, cudaStream_t stream);  // va_attn128.cu
bool launch_dense128(const AttnParams& p, int dtype, int batch, cudaStream_t stream, int* rc);

int sparse_attn(const va_attn_args& a, cudaStream_t stream) {
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
  p.col_count = a.col_count; p.col_idx = a.col_idx; p.col_stride = a.col_stride;
  p.status = a.status;
  p.lse = a.lse;
  p.heads = a.heads; p.rep = a.heads / a.kv_heads; p.sq = a.sq; p.sk = a.sk;
  p.vis_on = a.vision_mode != 0; p.vis_begin = a.vision_begin; p.vis_end = a.vision_end;
  p.nq = ((p.vis_on ? a.vision_end : a.sq) + a.pq - 1) / a.pq;
  p.causal = a.causal; p.q_offset = a.q_offset;
  const float scale = a.softmax_scale > 0.f ? a.softmax_scale : 0.08838834764831845f;
  p.scale_log2 = scale * 1.4426950408889634f;
  // One head after another keeps a head's K and V in L2 while its tiles run; where those of all heads fit half of it,
  // the tiles of all heads are listed by length instead, so that no head's longest tiles start last: 28 query heads on 4 KV
  // heads, 9001 tokens (18 MB) 0.403 -> 0.370 ms, 20011 tokens with a vision span (41 MB) 1.02 -> 0.87 ms.  The line is not where
  // the two meet: listed by length, whole calls with 64 / 96 / 128 / 256 MB of K and V run 1.08-1.17 / 1.09-1.14 / 1.05-1.13 /
  // 1.04-1.13 times as fast with 64-row tiles, 1.00-1.04 times with 128-row ones (16 to 32 heads, 8 K to 64 K tokens).
  p.by_length = a.causal && (int64_t)a.batch * a.kv_heads * a.sk * kHeadDim * 2 * 2 <= (64 << 20);
  if (p.vis_on && p.vis_begin >= p.vis_end) {  // every row is dense: 128-row tiles on streamed K and V take 0.50 ms where
    // gathered 64-row tiles took 0.86 (28 query heads on 4 KV heads, 8192 tokens).  A composition with sparse rows keeps its
    // dense tiles in the 64-row launch: they are few, and a launch of their own would leave most SMs idle.
    int rc;
    if (launch_dense128(p, a.dtype, a.batch, stream, &rc)) return rc;
  }
  return a.pq == 64 ? launch_attn64(p, a.dtype, a.batch, stream) : launch_attn128(p, a.dtype, a.batch, stream);
}

}  // namespace va
