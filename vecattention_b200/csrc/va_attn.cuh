// Launch parameters shared by the sparse-attention kernels.
#pragma once

#include <stdint.h>

namespace va {

struct AttnParams {
  const void* q;
  const void* k;
  const void* v;
  void* out;
  int64_t q_sb, q_sh, q_ss, k_sb, k_sh, k_ss, v_sb, v_sh, v_ss, o_sb, o_sh, o_ss;
  int k_row_bytes, v_row_bytes;  // k_ss, v_ss in bytes; 0: 32 bits do not hold them (or they are 0)
  const int32_t* blk_count;
  const int32_t* blk_idx;
  int64_t blk_stride;
  const int32_t* col_count;
  const int32_t* col_idx;
  int64_t col_stride;
  int32_t* status;
  float* lse;  // optional (B,H,sq): natural-log sum of exp over the row's keys
  int heads, rep, sq, sk, nq;
  int causal, q_offset;
  float scale_log2;  // softmax_scale * log2(e)
  // Vision-slice composition (64-row kernel only): rows [0, vis_begin) and [vis_end, sq) get full causal attention
  // from tiles that need no tables, rows [vis_begin, vis_end) the sparse attention of their tile; `nq` then counts
  // the table tiles (rows [0, vis_end)) and the grid has the dense tiles behind them.
  int vis_on, vis_begin, vis_end;
  // The operator's own dense blocks, which follow from the tile's number and need no table: under the causal rule the first
  // tile's and the tile's own, else none.  Tile t of this launch is tile first_tile + t of a sequence of seq_len rows.
  int own_blocks, first_tile, seq_len;
  int group;  // heads whose tiles are listed together: tile 0 of each of them, then tile 1 of each, ...
};

// The tile and head of CTA (x, y) of a grid of (tiles, heads): one group of heads after another.  Causal tiles grow with
// their index; the longest are started first, so that a group's tail is made of short ones.
__device__ __forceinline__ void place(const AttnParams& p, int tiles, uint32_t x, uint32_t y, int& tile, int& head) {
  const uint32_t at = y * (uint32_t)tiles + x, first = at / ((uint32_t)tiles * p.group) * p.group;  // the group's first head
  const uint32_t in_group = at - first * tiles, n = min((uint32_t)p.group, p.heads - first);       // (the last group may be smaller)
  head = (int)(first + in_group % n);
  x = in_group / n;
  tile = p.causal ? tiles - 1 - (int)x : (int)x;
}

// The operator's dense 64-key blocks of query tile t (of PQ rows): how many, and where block j starts.
template <int PQ>
__device__ __forceinline__ int own_block_count(const AttnParams& p, int t) {
  constexpr int n = PQ / 64;
  if (!p.causal) return 0;
  t += p.first_tile;
  if (t == 0) return (min(p.seq_len, PQ) + 63) / 64;
  return n + min(n, (p.seq_len - t * PQ + 63) / 64);
}
template <int PQ>
__device__ __forceinline__ int own_block_start(const AttnParams& p, int t, int j) {
  constexpr int n = PQ / 64;
  return j < n ? j * 64 : (p.first_tile + t) * PQ + (j - n) * 64;
}

}  // namespace va
