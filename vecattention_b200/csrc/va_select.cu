// Important-vector selection: pooled-Q . K^T estimate + streaming MinP threshold + compaction,
// with the estimate on tcgen05 tensor cores and the accumulator in tensor memory.
//
// Two kernels.
//
// 1. select_mask_kernel: estimate, running maximum and keep test; its result is one keep BIT per
//    (pooled row, key), written row-major to scratch memory.  The pooled rows of all query heads that
//    share one KV head form one row list (row R -> head hkv*rep + R%rep, tile R/rep, so that neighbours see about as many
//    keys under the causal rule); a CTA owns 128 consecutive rows of that list and walks the keys of its KV head once, 128 keys per tile, in
//    ascending order, so the running (prefix) maximum of a key-block group is a per-thread register.
//    Warp roles (352 threads, one CTA per SM):
//      warps 0-7  row walkers, by turns: warp w can reach TMEM lane quarter w % 4 (32 pooled rows) and takes
//                 every other key tile (tiles n with n % 2 == w / 4), so the two
//                 warps of a scheduler work on different tiles.  A thread walks its row's whole tile:
//                 it takes the 128 estimates into registers, which frees the accumulator buffer, and forms the maxima of the
//                 tile's key blocks, receives the
//                 row's running maximum after the previous tile from the warp that walked it (one float
//                 per row through shared memory, an mbarrier per warp pair), forms the running maximum
//                 entering every block and hands the one after its tile on at once; then it
//                 builds the 128 keep bits fp32(s + gap) >= m and stores them as one
//                 16-byte piece of the row's mask.  Where every tile is a whole number of key-block groups nothing is
//                 handed on.  The key range is cut into segments, one CTA each, where that lets the SMs finish
//                 together (make_plan): a CTA starts its walk where the group of key blocks starts that its segment begins in,
//                 for the maxima, and writes keep bits only for its own segment.
//      warp 8     one thread streams K: a TMA tensor-map copy per 128-key tile (two boxes of 128 rows
//                 x 128 bytes, 128-byte swizzle) into a 4-stage ring; rows past the sequence read as zeros.
//      warps 9,10 one thread each issues S_t = Q~ K_t^T for alternate tiles, 128 x 128 x 128 as eight
//                 tcgen05.mma, into one of four 128-column accumulator buffers in tensor memory.
//    What bounds it: the walkers' instructions, some 500 a tile and scheduler beside 518 clk of tensor arithmetic, of which the
//    ALU takes two clk each (64 three-input maxima, 64 byte permutes and logic operations).  A tile takes about 1060 clk.
//    Sixteen warps that read their estimates from tensor memory twice, 96 registers each, spilled.  What eight that hold their row gave,
//    by themselves: k_local_size 128 (32 heads x 32 K, causal) 210 -> 122 us; 16: 32 heads x 32 K 168 -> 153, 28/4 heads x 64 K causal
//    316 -> 286, 9001 tokens, groups of one block, 48 -> 42.  With the work cut by make_plan besides, a launch takes 69, 151, 276 and 15 us.
//    (A funnel shift per estimate in place of conversion, permute and logic: 1-3 % slower.)
//    All hand-offs are mbarriers with bounded waits; a timeout sets VA_STATUS_TIMEOUT.
//
// 2. select_expand_kernel: one warp per pooled row turns the row's keep bits into its ascending
//    index list (population counts, a warp scan, staging in shared memory, coalesced stores) and
//    writes the row's count.  Lists are deterministic; nothing is zero-filled; no atomics.
#include "va_common.cuh"
#include "va_sm100.cuh"
#include "va_tmap.cuh"

#include <type_traits>

namespace va {

using namespace sm100;

// How a launch's work is cut into CTAs.  A CTA has one block of 128 pooled rows and one segment of its keys: tiles
// [cut[s], cut[s + 1]) from the walk's first tile on.  CTAs below `whole` have all keys of their block; the others are listed in
// runs of one segment each, run r being CTAs whole + start[r] and up.
constexpr int kMaxSegments = 32;
struct Plan {
  int whole, runs, segments, ctas;
  int heads;   // KV heads of all batch entries
  int period;  // tiles after which a group of key blocks starts with a tile again
  int cut[kMaxSegments + 1];
  // not causal: run s has segment s of the blocks from number `whole` on.  Causal: run s has segment s of the blocks that fill it,
  // run segments + s that of the blocks that end inside it, so that the longest walks come first; top: the last block of a run.
  int start[2 * kMaxSegments], top[2 * kMaxSegments];
};

struct SelectParams {
  const void* avg_q;  // (B,H,nq,D)
  const float* gaps;
  int64_t gaps_sb;
  float gap;
  int32_t* col_count;
  int32_t* col_idx;
  int64_t capacity;
  int32_t* status;
  uint32_t* mask;     // keep bits, [(b * kv_heads + hkv) * rows_pad + R][wpad] 32-bit words, bit j of word w = key 32 w + j
  int rows_pad;       // pooled rows per KV head, rounded up to the CTA height
  int wpad;           // words per mask row (whole groups of four key tiles)
  int heads, kv_heads, rep, nq, sk;
  int pq, group_k_block;
  uint32_t starts;    // see WalkArgs
  Plan plan;
  int causal, wo_initial, compat_bsq, tile_offset, chunk_tiles;
};

namespace {

constexpr int kRows = 128;   // pooled rows per CTA
constexpr int kTile = 128;   // keys per tile
constexpr int kTileBytes = 128 * 256;
constexpr int kStages = 4;   // K ring
constexpr int kSBufs = 4;    // accumulator buffers in tensor memory (4 x 128 columns = all of it)
constexpr int kTurns = 2;      // walker warps of a lane quarter, which take key tiles by turns
constexpr int kWalkerWarps = 4 * kTurns;
constexpr int kThreads = 32 * (kWalkerWarps + 3);  // the walkers, the K producer, two MMA issuers
constexpr size_t kSmem = 1024 + (size_t)kTileBytes * (1 + kStages);

struct Barriers {
  uint64_t kfull[kStages], kempty[kStages], sfull[kSBufs], sempty[kSBufs];
  uint64_t hand[4][kTurns];  // [lane quarter][turn]: that warp has published the rows' running maximum after its tile
};

// End (exclusive) of the keys pooled row `tile` of the chunk may select, spattn/src/kernels/
// vecattention_kernels.py:231-233,260: all keys, or under the causal rule the keys before the row's
// diagonal tile; the first row of every compat_bsq rows of a chunk also loses the key blocks that
// start inside the tile before it, except the first (the reference's truncating division).
__device__ __forceinline__ int row_key_limit(const SelectParams& p, int tile, int bk) {
  if (!p.causal) return p.sk;
  const int64_t g = (int64_t)p.tile_offset + tile;
  int64_t lim = g * p.pq;
  const int tile_in_chunk = p.chunk_tiles > 0 ? tile % p.chunk_tiles : tile;
  if (p.compat_bsq > 0 && (tile_in_chunk % p.compat_bsq) == 0) {
    const int64_t q1 = (g - 1) * p.pq + bk;
    lim = q1 < lim ? q1 : lim;
  }
  lim = lim < p.sk ? lim : p.sk;
  return lim > 0 ? (int)lim : 0;
}

// three-input maximum (one instruction)
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// maximum of N estimates (N = 16 or 32) as two chains of three-input maxima
template <int N>
__device__ __forceinline__ float max_of(const uint32_t* v) {
  float a = __uint_as_float(v[0]), b = __uint_as_float(v[1]);
  int i = 2;
#pragma unroll
  for (; i + 3 < N; i += 4) {
    a = fmax3(a, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
    b = fmax3(b, __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
  }
  if (i + 1 < N) a = fmax3(a, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
  return fmaxf(a, b);
}

// two fp32 additions in one instruction (round to nearest, no flush: each half is an IEEE add)
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t pack2u(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t x, uint32_t& lo, uint32_t& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(x));
}

// ---- the row walkers ------------------------------------------------------------------------------
// Eight warps; warp (qtr, turn) = (w % 4, w / 4) owns the pooled rows of TMEM lane quarter qtr (a warp
// reaches only the quarter w % 4) on every other key tile.  A thread handles its row's whole tile: first the maxima of the
// tile's key blocks (independent of earlier tiles), then, once the warp of the previous tile has handed over the rows'
// running maximum, the running maximum entering every block, which it hands on at once, and last the
// keep bits of the 128 keys, from the estimates it still holds.
struct WalkShared {
  float rmx[4][kTurns][32];  // [lane quarter][turn][lane]: running maximum after that warp's latest tile
};

// what a walker thread knows about its CTA and its row
struct WalkArgs {
  uint32_t tmem;       // first accumulator buffer
  int t_lo, t_hi;      // key tiles the CTA walks
  int t_keep;          // first tile whose keep bits this CTA writes (earlier tiles only feed the running maximum)
  int lo, k_hi;        // key range the CTA walks
  int sk, hi;          // sequence length; end of this thread's row
  int G;               // key blocks per group
  uint32_t starts;     // groups inside a tile: bit k is set if block k of a tile starts one
  float gap;
  uint32_t* mrow;      // this thread's mask row
};

// one wait, cheap when the phase is already complete
__device__ __forceinline__ bool wait_fast(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait(bar, parity);
}

// Keep bits of 32 estimates: fp32(s + gap) >= m  <=>  fp32(s + gap) - m is not negative (the difference of
// two floats has the exact sign).  m_lo applies to estimates 0..15, m_hi to 16..31.  Two packed additions per
// pair of estimates.  A difference keeps its sign when it is converted to a 16-bit float, two in one instruction; a byte
// permute turns the signs of keys g, 8 + g, 16 + g and 24 + g into four bytes of zeros or ones, and one logic
// operation files bit g of each of them: key c ends up in bit c.
__device__ __forceinline__ uint32_t keep_bits(const uint32_t (&v)[32], uint64_t gap2, float m_lo, float m_hi) {
  const uint64_t nm2[2] = {pack2(-m_lo, -m_lo), pack2(-m_hi, -m_hi)};
  uint32_t neg = 0u;
#pragma unroll
  for (int g = 0; g < 8; g += 2) {
    uint32_t d[2][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      unpack2(add2(add2(pack2u(v[q * 8 + g], v[q * 8 + g + 1]), gap2), nm2[q >> 1]), d[0][q], d[1][q]);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      uint32_t a, b, spread;
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(a) : "f"(__uint_as_float(d[e][1])), "f"(__uint_as_float(d[e][0])));
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(b) : "f"(__uint_as_float(d[e][3])), "f"(__uint_as_float(d[e][2])));
      asm("prmt.b32 %0, %1, %2, 0xfdb9;" : "=r"(spread) : "r"(a), "r"(b));  // bytes 1 and 3 of both, the sign eight times
      neg |= spread & (0x01010101u << (g + e));
    }
  }
  return ~neg;
}

// Where groups of key blocks begin.
enum Groups {
  kAnywhere,  // any block of a tile
  kAtTiles,   // only at a tile's first block (a group is a whole number of tiles)
  kInTiles,   // at every tile's first block, and perhaps inside it (a tile is a whole number of groups): tiles are independent
};

// Walk every kTurns-th key tile of the CTA for the rows of lane quarter `qtr`.  Returns false if a wait ran
// out.  BK = k_local_size.
template <int BK, Groups GROUPS>
__device__ __forceinline__ bool walk_rows(const WalkArgs& a, Barriers& bars, WalkShared& sh, int qtr, int turn, int lane) {
  constexpr int NBT = kTile / BK;  // key blocks per tile
  const uint32_t taddr0 = a.tmem + ((uint32_t)(qtr * 32) << 16);
  const uint64_t gap2 = pack2(a.gap, a.gap);
  const int before = (turn + kTurns - 1) % kTurns;  // the turn that has the tile before this warp's
  uint64_t* const hand_in = &bars.hand[qtr][before];
  uint64_t* const hand_out = &bars.hand[qtr][turn];
  const float* rm_in = &sh.rmx[qtr][before][lane];
  float* rm_out = &sh.rmx[qtr][turn][lane];
  const int ntiles = a.t_hi - a.t_lo;
  const unsigned tpg = GROUPS == kAtTiles ? (unsigned)(((int64_t)a.G * BK) / kTile) : 1u;  // tiles per group of key blocks
  unsigned tg = GROUPS == kAtTiles ? (unsigned)(a.t_lo + turn) % tpg : 0u;                 // the tile's place in its group
  const uint32_t starts = GROUPS == kInTiles ? a.starts : 1u;  // blocks of a tile with which a group starts
  const int t_in_lo = (a.lo + kTile - 1) / kTile;  // first tile wholly at or after lo
  const int t_in_hi = min(a.k_hi, a.sk) / kTile;   // tiles before this one end at or before k_hi

  for (int n = turn; n < ntiles; n += kTurns) {
    const int t = a.t_lo + n, key_t = t * kTile, sb = n % kSBufs;
    const bool inner = GROUPS != kAnywhere && t >= t_in_lo && t < t_in_hi;  // no range tests
    if (!wait_fast(&bars.sfull[sb], (uint32_t)(n / kSBufs) & 1u)) return false;
    tc_fence_after();
    // ---- the row's 128 estimates; the accumulator buffer is free again ----
    uint32_t v[4][32];
#pragma unroll
    for (int c4 = 0; c4 < 4; ++c4) tmem_ld32(taddr0 + (uint32_t)(sb * 128 + c4 * 32), v[c4]);
    tmem_wait_ld();
    tc_fence_before();
    mbar_arrive(&bars.sempty[sb]);
    // ---- maxima of the tile's key blocks (keys past the sequence end never count) ----
    float pm[NBT];
    if (inner || key_t + kTile <= a.sk) {
#pragma unroll
      for (int k = 0; k < NBT; ++k) {
        if constexpr (BK == 16) {
          pm[k] = max_of<16>(v[k / 2] + (k & 1) * 16);
        } else {
          pm[k] = max_of<32>(v[k * (BK / 32)]);
#pragma unroll
          for (int i = 1; i < BK / 32; ++i) pm[k] = fmaxf(pm[k], max_of<32>(v[k * (BK / 32) + i]));
        }
      }
    } else {
#pragma unroll
      for (int k = 0; k < NBT; ++k) pm[k] = -INFINITY;
#pragma unroll
      for (int j = 0; j < kTile; ++j)
        if (key_t + j < a.sk) pm[j / BK] = fmaxf(pm[j / BK], __uint_as_float(v[j / 32][j % 32]));
    }
    // ---- the rows' running maximum after the previous tile, from the warp that walked it ----
    float run = -INFINITY;
    if (GROUPS != kInTiles && n > 0) {
      if (!wait_fast(hand_in, (uint32_t)((n - 1) / kTurns) & 1u)) return false;
      run = *rm_in;
    }
    // ---- running maximum entering / after every block; handed on before the keep bits are formed ----
    float rm[NBT];
    uint32_t on_bits = 0xffffffffu;  // bit k: block k lies inside the walked key range
    if (inner) {
      if (tg == 0u) run = -INFINITY;  // a new group of key blocks starts with this tile
#pragma unroll
      for (int k = 0; k < NBT; ++k) {
        if (GROUPS == kInTiles && k > 0 && (starts >> k & 1u)) run = -INFINITY;
        run = fmaxf(run, pm[k]);
        rm[k] = run;
      }
    } else {
      int gp = (int)((unsigned)(key_t / BK) % (unsigned)a.G);  // position of the tile's first block inside its group
      on_bits = 0u;
#pragma unroll
      for (int k = 0; k < NBT; ++k) {
        const int key0 = key_t + k * BK;
        if (key0 >= a.lo && key0 < a.k_hi) {
          if (gp == 0) run = -INFINITY;  // a new group of key blocks starts
          run = fmaxf(run, pm[k]);
          on_bits |= 1u << k;
        }
        gp = gp + 1 == a.G ? 0 : gp + 1;
        rm[k] = run;
      }
    }
    if (GROUPS != kInTiles) {
      *rm_out = run;
      mbar_arrive(hand_out);
    }
    if (GROUPS == kAtTiles) {
      tg += kTurns;
      while (tg >= tpg) tg -= tpg;
    }
    if (t < a.t_keep) continue;  // another CTA writes this tile's keep bits: only the running maximum was needed
    // ---- keep bits of the 128 keys ----
    uint32_t w[4];
#pragma unroll
    for (int c4 = 0; c4 < 4; ++c4)
      w[c4] = keep_bits(v[c4], gap2, rm[c4 * 32 / BK], rm[(c4 * 32 + 16) / BK]);
    if (!inner) {
#pragma unroll
      for (int c4 = 0; c4 < 4; ++c4) {
        if (!((on_bits >> (c4 * 32 / BK)) & 1u)) w[c4] &= 0xffff0000u;
        if (!((on_bits >> ((c4 * 32 + 16) / BK)) & 1u)) w[c4] &= 0x0000ffffu;
      }
    }
    if (key_t + kTile > a.hi) {  // keys at or past the row's limit are cut off
#pragma unroll
      for (int c4 = 0; c4 < 4; ++c4) {
        const int room = a.hi - (key_t + c4 * 32);
        if (room < 32) w[c4] = room <= 0 ? 0u : (w[c4] & ((1u << room) - 1u));
      }
    }
    *reinterpret_cast<uint4*>(a.mrow + (size_t)t * 4) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  return true;
}

// BK = k_local_size.
template <int DT, int BK, Groups GROUPS>
__global__ void __launch_bounds__(kThreads, 1) select_mask_kernel(const __grid_constant__ CUtensorMap kmap, const SelectParams p) {
  using T = typename Elem<DT>::T;
  extern __shared__ unsigned char smem_raw[];
  __shared__ Barriers bars;
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_khi;
  __shared__ WalkShared wsh;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  wait_for_previous();
  let_next_start();
  const int nrows = p.rep * p.nq;
  // ---- this CTA's row block and segment ----
  const int blocks = p.rows_pad / kRows;
  int at = (int)blockIdx.x, seg_from = 0, seg_to = 0x7fffffff, run = 0;
  if (at >= p.plan.whole) {
    at -= p.plan.whole;
    while (run + 1 < p.plan.runs && at >= p.plan.start[run + 1]) ++run;
    at -= p.plan.start[run];
    const int s = run < p.plan.segments ? run : run - p.plan.segments;
    seg_from = p.plan.cut[s];
    seg_to = p.plan.cut[s + 1];
    if (!p.causal) at += p.plan.whole;
  }
  int bx, head_at;  // row block; KV head and batch entry
  if (p.causal) {   // the later the rows the longer the walk
    bx = p.plan.top[run] - at / p.plan.heads;
    head_at = at % p.plan.heads;
  } else {          // the row blocks of a head side by side: they walk the same keys
    bx = at % blocks;
    head_at = at / blocks;
  }
  const int row_base = bx * kRows, hkv = head_at % p.kv_heads, b = head_at / p.kv_heads;

  // ---- per-row limits: walker threads own row (warp % 4) * 32 + lane ----
  const bool is_walker = warp < kWalkerWarps;
  const int wrow = (warp & 3) * 32 + lane;
  const int R = row_base + wrow;
  const bool row_ok = is_walker && R < nrows;
  const int h = hkv * p.rep + (row_ok ? R % p.rep : 0);
  const int lo = p.wo_initial ? p.pq : 0;
  const int hi = row_ok ? row_key_limit(p, R / p.rep, BK) : 0;

  if (tid == 0) s_khi = 0;
  __syncthreads();
  if (warp < 4) {
    int whi = hi;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) whi = max(whi, __shfl_xor_sync(0xffffffffu, whi, o));
    if (lane == 0) atomicMax(&s_khi, whi);
  }
  __syncthreads();
  const int k_hi = s_khi;                       // CTA-wide end of the key walk
  int t_lo = lo / kTile;
  int t_hi = (k_hi + kTile - 1) / kTile;  // exclusive
  // The CTA writes the keep bits of its segment only.  The running maximum is that of a group of key blocks up to here, so
  // the walk starts where the segment's first group does.
  const int t_keep = t_lo + seg_from;
  if (seg_to < t_hi - t_lo) t_hi = t_lo + seg_to;
  if (k_hi <= lo || t_keep >= t_hi) return;  // nothing selectable here (the expansion writes the counts)
  t_lo = max(t_lo, t_keep / p.plan.period * p.plan.period);

  unsigned char* smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
  unsigned char* q_s = smem;
  unsigned char* k_s = smem + kTileBytes;

  // ---- scaled pooled Q -> shared operand tile (q~ = round(fp32(q_bar) * fp32(1/sqrt(D)))) ----
  {
    const float scale = 0.08838834764831845f;  // fp32(1/sqrt(128))
    const T* aq = static_cast<const T*>(p.avg_q);
    for (int i = tid; i < kRows * 16; i += kThreads) {
      const int r = i >> 4, c = i & 15;
      const int RR = row_base + r;
      uint4 w = make_uint4(0, 0, 0, 0);
      if (RR < nrows) {
        const int hh = hkv * p.rep + RR % p.rep, tt = RR / p.rep;
        w = *reinterpret_cast<const uint4*>(aq + (((int64_t)b * p.heads + hh) * p.nq + tt) * kHeadDim + c * 8);
        uint32_t* ww = reinterpret_cast<uint32_t*>(&w);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = Elem<DT>::unpack(ww[j]);
          ww[j] = Elem<DT>::pack(__fmul_rn(f.x, scale), __fmul_rn(f.y, scale));
        }
      }
      *reinterpret_cast<uint4*>(q_s + tile_off(128, r, c)) = w;
    }
    fence_proxy_async();
  }
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bars.kfull[s], 1);   // the producer's arrival; the copies complete it by byte count
      mbar_init(&bars.kempty[s], 1);
    }
    for (int s = 0; s < kSBufs; ++s) {
      mbar_init(&bars.sfull[s], 1);
      mbar_init(&bars.sempty[s], 4 * 32);  // four warps, one per lane quarter, read a tile
    }
    for (int s = 0; s < 4 * kTurns; ++s) mbar_init(&bars.hand[s / kTurns][s % kTurns], 32);
    fence_proxy_async();
  }
  if (warp == kWalkerWarps + 1) {
    tmem_alloc(&tmem_base_s, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  bool timed_out = false;

  if (warp == kWalkerWarps) {
    // ======================= K tile producer (one thread, TMA) =======================
    if (lane == 0) {
      int issued = 0, s = 0;
      uint32_t epar = 1;  // phase parity of the stage's "empty" barrier
      const uint32_t k_base = smem_addr(k_s);
      for (int t = t_lo; t < t_hi; ++t) {
        if (!wait_fast(&bars.kempty[s], epar)) { timed_out = true; break; }
        mbar_expect_tx(&bars.kfull[s], kTileBytes);
        const uint32_t dst = k_base + (uint32_t)s * kTileBytes;
        tma_load_4d(dst, &kmap, 0, t * kTile, hkv, b, &bars.kfull[s]);                    // elements 0..63 of the 128 rows
        tma_load_4d(dst + kTileBytes / 2, &kmap, 64, t * kTile, hkv, b, &bars.kfull[s]);  // elements 64..127
        issued = t - t_lo + 1;
        if (++s == kStages) { s = 0; epar ^= 1u; }
      }
      if (timed_out) {  // no copy of this CTA may still be in flight when it retires
        for (int n = max(0, issued - kStages); n < issued; ++n) mbar_wait(&bars.kfull[n % kStages], (n / kStages) & 1);
      }
    }
  } else if (warp > kWalkerWarps) {
    // ======================= MMA issuers =======================
    // Two threads take alternate tiles: while one is held by the tensor pipe's queue, the
    // other has already passed the barrier waits of the next tile, so the pipe never runs dry between tiles.
    if (lane == 0) {
      constexpr uint32_t in16 = DT == VA_BF16 ? 1u : 0u;
      constexpr uint32_t idesc = umma_idesc(128, 128, in16, 0, 0);
      const uint64_t qd = umma_desc(smem_addr(q_s), 16, 1024), kd0 = umma_desc(smem_addr(k_s), 16, 1024);
      int s = warp - kWalkerWarps - 1, sb = s;
      uint32_t kpar = 0, spar = 1;  // phase parities of the stage's "full" and the buffer's "empty" barrier
      for (int t = t_lo + s; t < t_hi; t += 2) {
        if (!wait_fast(&bars.kfull[s], kpar) || !wait_fast(&bars.sempty[sb], spar)) { timed_out = true; break; }
        tc_fence_after();
        umma_k128_rows128(tmem + (uint32_t)sb * 128, qd, kd0 + (uint64_t)(s * (kTileBytes >> 4)), idesc);
        umma_commit(&bars.kempty[s]);
        umma_commit(&bars.sfull[sb]);
        if ((s += 2) >= kStages) { s -= kStages; kpar ^= 1u; }
        if ((sb += 2) >= kSBufs) { sb -= kSBufs; spar ^= 1u; }
      }
    }
  } else {
    // ======================= row walkers =======================
    WalkArgs a;
    a.tmem = tmem;
    a.t_lo = t_lo;
    a.t_hi = t_hi;
    a.t_keep = t_keep;
    a.lo = lo;
    a.k_hi = k_hi;
    a.sk = p.sk;
    a.hi = hi;
    a.G = p.group_k_block;
    a.starts = p.starts;
    a.gap = p.gaps ? p.gaps[b * p.gaps_sb + h] : p.gap;
    a.mrow = p.mask + ((size_t)(b * p.kv_heads + hkv) * p.rows_pad + row_base + wrow) * p.wpad;
    timed_out = !walk_rows<BK, GROUPS>(a, bars, wsh, warp & 3, warp >> 2, lane);
  }
  if (timed_out && p.status) atomicOr(p.status, VA_STATUS_TIMEOUT);
  tc_fence_before();
  __syncthreads();
  if (warp == kWalkerWarps + 1) tmem_dealloc(tmem, 512);
}

// ---- keep bits -> ascending index lists ---------------------------------------------------------
// One warp per pooled row (b, h, tile).  Per step the lanes take 32 consecutive mask words (1024
// keys), a warp scan of their population counts gives every lane the place of its keys, and the keys are
// staged in shared memory.  Whole groups of 128 staged keys leave as one 16-byte store per lane; the rest stays for the
// next steps.  The mask kernel has already cleared every bit outside the row's key range.
// Bound by instruction issue: about 10 % of the bits are set, and the rounds below follow the fullest of 32 words.  With a loop
// per lane (find the lowest bit, branch) and 4-byte stores after every step it took 148 us for 32 heads x 32 K tokens (16 384 rows,
// 85 % of the issue slots), now 105; 28 heads x 64 K causal 279 -> 200; 5 heads x 75 600 tokens 126 -> 88 (161 MB of lists out
// and 56 MB of masks in).
constexpr int kExpandWarps = 8;
constexpr int kFlush = 128;              // keys that leave together
constexpr int kFlushFrom = 2 * kFlush;   // staged keys from which on they leave

// inclusive sum over the lanes up to this one
__device__ __forceinline__ int warp_prefix_sum(int x) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
    asm volatile("{\n\t.reg .pred p;\n\t.reg .s32 u;\n\tshfl.sync.up.b32 u|p, %0, %1, 0, 0xffffffff;\n\t@p add.s32 %0, %0, u;\n\t}" : "+r"(x) : "r"(o));
  return x;
}

template <int BK>
__global__ void __launch_bounds__(kExpandWarps * 32) select_expand_kernel(const SelectParams p, int64_t total_rows) {
  __shared__ __align__(16) int32_t stage_s[kExpandWarps][1024 + kFlushFrom];
  wait_for_previous();
  let_next_start();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row = (int64_t)blockIdx.x * kExpandWarps + warp;  // = (b * heads + h) * nq + tile
  if (row >= total_rows) return;
  const int tile = (int)(row % p.nq);
  const int64_t bh = row / p.nq;
  const int h = (int)(bh % p.heads), b = (int)(bh / p.heads);
  const int hkv = h / p.rep;
  const int R = tile * p.rep + h % p.rep;
  const int lo = p.wo_initial ? p.pq : 0;
  const int hi = row_key_limit(p, tile, BK);
  const int32_t* mrow = reinterpret_cast<const int32_t*>(p.mask) + ((size_t)(b * p.kv_heads + hkv) * p.rows_pad + R) * p.wpad;
  int32_t* out = p.col_idx + row * p.capacity;
  int32_t* stage = stage_s[warp];
  const bool wide = ((p.capacity & 3) | (reinterpret_cast<uintptr_t>(p.col_idx) & 15)) == 0;  // 16-byte stores are possible
  const int room = (int)min(p.capacity, (int64_t)0x7fffffff);
  int cnt = 0;   // keys that have left
  int held = 0;  // keys staged
  // the first n staged keys leave (n a multiple of 128, or all that are left)
  auto flush = [&](int n, bool whole) {
    if (whole && wide && cnt + n <= room) {
      for (int i = lane * 4; i < n; i += kFlush) *reinterpret_cast<int4*>(out + cnt + i) = *reinterpret_cast<const int4*>(stage + i);
    } else {
      for (int i = lane; i < n; i += 32)
        if (cnt + i < room) out[cnt + i] = stage[i];
    }
    cnt += n;
  };
  if (hi > lo) {
    const int w_hi = (hi + 31) >> 5;
    int w = (lo >> 5) + lane;  // this lane's word
    uint32_t cur = w < w_hi ? (uint32_t)load_here(mrow + w) : 0u;
    for (; w - lane < w_hi; w += 32) {
      const uint32_t nxt = w + 32 < w_hi ? (uint32_t)load_here(mrow + w + 32) : 0u;  // the next step's words, fetched early
      uint32_t word = cur;
      const int c = __popc(word), incl = warp_prefix_sum(c);
      // The lane's keys, last one first: the highest set bit is one instruction of the special-function unit, the lowest
      // one two.  All lanes make as many rounds as the fullest word needs, four at a time (a lane whose word is empty
      // stores nothing): branches per lane cost more than the rounds they save.
      const int rounds = (int)__reduce_max_sync(0xffffffffu, (unsigned)c);
      int32_t* end = stage + held + incl;
      const int key0 = w << 5;
      for (int i = 0; i < rounds; i += 4) {
#pragma unroll
        for (int u = 1; u <= 4; ++u) {
          uint32_t at, bit;
          asm("bfind.u32 %0, %1;" : "=r"(at) : "r"(word));
          asm("shl.b32 %0, 1, %1;" : "=r"(bit) : "r"(at));  // no bit at all: bfind gives 2^32 - 1, and the shift 0
          if (word) end[-u] = key0 + (int)at;
          word ^= bit;
        }
        end -= 4;
      }
      held += __shfl_sync(0xffffffffu, incl, 31);
      __syncwarp();
      if (held >= kFlushFrom) {
        const int n = held / kFlush * kFlush;
        flush(n, true);
        held -= n;
        const int4 rest = *reinterpret_cast<const int4*>(stage + n + lane * 4);  // at most 127 keys
        __syncwarp();
        *reinterpret_cast<int4*>(stage + lane * 4) = rest;
        __syncwarp();
      }
      cur = nxt;
    }
  }
  flush(held, false);
  if (lane == 0) {
    p.col_count[row] = cnt;
    if (cnt > p.capacity && p.status) atomicOr(p.status, VA_STATUS_OVERFLOW);
  }
}

template <int DT, int BK>
int launch_bk(const SelectParams& p, const CUtensorMap& kmap, int batch, cudaStream_t stream) {
  const int64_t group = (int64_t)p.group_k_block * BK;
  auto kern = select_mask_kernel<DT, BK, kAnywhere>;
  if (kTile % group == 0) kern = select_mask_kernel<DT, BK, kInTiles>;
  else if (group % kTile == 0) kern = select_mask_kernel<DT, BK, kAtTiles>;
  // per-device attribute; setting it on every launch keeps multi-device processes correct
  if (!succeeded(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem))) return VA_ERR_CUDA;
  if (p.plan.ctas > 0) {
    if (!launch_after(kern, dim3(p.plan.ctas), kThreads, kSmem, stream, kmap, p)) return VA_ERR_CUDA;
  }
  const int64_t total_rows = (int64_t)batch * p.heads * p.nq;
  const dim3 grid((unsigned)((total_rows + kExpandWarps - 1) / kExpandWarps));
  return launch_after(select_expand_kernel<BK>, grid, kExpandWarps * 32, 0, stream, p, total_rows) ? VA_OK : VA_ERR_CUDA;
}

template <int DT>
int launch_dt(const SelectParams& p, const CUtensorMap& kmap, int bk, int batch, cudaStream_t stream) {
  switch (bk) {
    case 16: return launch_bk<DT, 16>(p, kmap, batch, stream);
    case 32: return launch_bk<DT, 32>(p, kmap, batch, stream);
    case 64: return launch_bk<DT, 64>(p, kmap, batch, stream);
    case 128: return launch_bk<DT, 128>(p, kmap, batch, stream);
    default: return VA_ERR_SHAPE;
  }
}

}  // namespace

// mask rows per KV head and words per mask row for a selection of nq pooled rows per head over sk keys
static inline void mask_geometry(int heads, int kv_heads, int nq, int sk, int& rows_pad, int& wpad) {
  const int nrows = (heads / kv_heads) * nq;
  rows_pad = (nrows + kRows - 1) / kRows * kRows;
  const int tiles = (sk + kTile - 1) / kTile;
  wpad = (tiles + 3) / 4 * 16;
}

size_t select_workspace_bytes(int batch, int heads, int kv_heads, int nq, int sk) {
  int rows_pad, wpad;
  mask_geometry(heads, kv_heads, nq, sk, rows_pad, wpad);
  return (size_t)batch * kv_heads * rows_pad * wpad * 4;
}

// Cut the work into CTAs so that the SMs finish together: the number of segments per row block is the one with the least
// estimated time, in tiles.  A tile that only feeds the running maximum costs kFeed of one with keep bits (more than its
// instructions' share: with many segments the CTAs stream K from L2 at the same time), a CTA kSetUp tiles
// (it loads its rows, fills and drains its pipeline: 3 us).
// Each constant here and below was timed against others, selections alone, on shapes of 1 to 40 heads and 2 to 120 K tokens that the
// other value cuts differently; time with it / with this one, mean and worst:
//   kFeed 0.55: 0.98, 1.46 and 0.62: 0.98, 1.47 (some 450 shapes; level from 200 us on; the worst are 40 heads x 9001 and 20 011 tokens,
//     causal, one group), 0.85: 1.07, 1.14.  Whole calls, not causal, one group, 3 x 55 000 to 3 x 118 800 tokens: level with all three, runs differ by 3-5 %.
//   kSetUp 2: 1.03, 1.22; 10: 0.99, 1.05 (this and the rest: 14 shapes each).
//   Another cut is taken if it wins by 3 %, which is what the estimate is good for: by anything 1.04, 1.49; by 10 % 1.01, 1.06.
//   Work that is spread over the SMs ends 0.2 of the longest CTA after an even share: 0 of it 1.11, 1.29; 0.5 1.01, 1.14.
//   Segments are whole groups if that makes them at most a quarter longer: only if not at all 1.42, 3.5; up to twice as long 1.02, 1.22.
static void make_plan(SelectParams& p, int batch, int bk) {
  constexpr double kFeed = 0.70, kSetUp = 5.0;
  Plan& pl = p.plan;
  int sms = 148, dev = 0;
  if (!succeeded(cudaGetDevice(&dev)) || !succeeded(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev))) sms = 148;
  const int blocks = p.rows_pad / kRows, t0 = (p.wo_initial ? p.pq : 0) / kTile;
  const int all = (p.sk + kTile - 1) / kTile;
  pl.heads = p.kv_heads * batch;
  const int64_t group = (int64_t)p.group_k_block * bk;  // a divisor or a multiple of the tile, or anything
  int64_t common = group, rest = kTile;                 // greatest common divisor
  while (rest) {
    const int64_t r = common % rest;
    common = rest;
    rest = r;
  }
  pl.period = (int)(group / common < all ? group / common : all);
  // tiles walked by a row block: all, or under the causal rule those before its last row's own
  auto length = [&](int block) {
    int64_t end = p.sk;
    if (p.causal) {
      const int last = (block + 1) * kRows < p.rep * p.nq ? (block + 1) * kRows - 1 : p.rep * p.nq - 1;
      const int64_t before = ((int64_t)p.tile_offset + last / p.rep) * p.pq;
      end = before < end ? before : end;
    }
    const int n = (int)((end + kTile - 1) / kTile) - t0;
    return n > 0 ? n : 0;
  };
  const int longest = length(blocks - 1);
  const int64_t ctas = (int64_t)blocks * pl.heads;
  // With eight uncut blocks and more for every SM there is nothing to gain.  The search is made on every call: it takes the blocks'
  // lengths from their sums, not block by block (causal, host time: 28/4 heads x 64 K, 56 blocks a KV head, 20 -> 4 us; 64/1 x 131 072, 1024 blocks, 244 -> 9).
  constexpr int kMostBlocks = 2048;
  const bool search = ctas < 8 * (int64_t)sms && blocks <= kMostBlocks;
  int64_t total[kMostBlocks + 1];  // tiles of the blocks before
  if (search && p.causal) {
    total[0] = 0;
    for (int i = 0; i < blocks; ++i) total[i + 1] = total[i] + length(i);
  }
  // (lengths grow with the block) the first block, not before `from`, of at least n tiles
  auto first_of = [&](int n, int from) {
    int lo = from, hi = blocks;
    while (lo < hi) {
      const int mid = (lo + hi) / 2;
      if ((search ? (int)(total[mid + 1] - total[mid]) : length(mid)) < n) lo = mid + 1;
      else hi = mid;
    }
    return lo;
  };
  // segment s of a block that is cut into n: equal ones where a group starts every few tiles; else each is shorter than the
  // one before by what it walks again, so that all take the same time
  auto set_cuts = [&](int n) {
    const int step = (longest + n - 1) / n, whole = (step + pl.period - 1) / pl.period * pl.period;
    pl.segments = n;
    pl.cut[0] = 0;
    if (4 * (whole - step) <= step) {
      for (int s = 1; s <= n; ++s) pl.cut[s] = (int64_t)s * whole < longest ? s * whole : longest;
    } else {
      double left = 1.0, at = 0.0;
      for (int s = 0; s < n; ++s) left *= 1.0 - kFeed;
      const double first = longest * kFeed / (1.0 - left);
      for (int s = 1; s <= n; ++s) {
        at += first - kFeed * at;
        pl.cut[s] = (int)(at + 0.999);
        if (pl.cut[s] > longest) pl.cut[s] = longest;
      }
    }
    pl.cut[n] = longest;
    while (pl.segments > 1 && pl.cut[pl.segments - 1] >= longest) --pl.segments;
  };
  auto segment_cost = [&](int s, int tiles) {  // of a block with that many tiles
    const int to = tiles < pl.cut[s + 1] ? tiles : pl.cut[s + 1], again = (t0 + pl.cut[s]) % pl.period;
    return to - pl.cut[s] + kFeed * (again < pl.cut[s] ? again : pl.cut[s]) + kSetUp;
  };
  auto cost = [&](int64_t first_block) {  // of the segments as they are cut, first_block: in the order of the heads' blocks
    double most = 0.0, sum = 0.0;
    int64_t n = 0;
    if (!p.causal) {
      for (int s = 0; s < pl.segments; ++s) {
        const double c = segment_cost(s, longest);
        most = c > most ? c : most;
      }
      n = (ctas - first_block) * pl.segments;
      return (double)((n + sms - 1) / sms) * most;
    }
    int64_t filled = 0;
    for (int s = 0, reach = 0, fill = 0; s < pl.segments; ++s) {
      reach = first_of(pl.cut[s] + 1, fill);  // the first block that reaches into the segment, and the first that fills it
      fill = first_of(pl.cut[s + 1], reach);
      n += (int64_t)(blocks - reach) * pl.heads;
      if (fill < blocks) {
        const double c = segment_cost(s, pl.cut[s + 1]);
        most = c > most ? c : most;
        sum += c * (blocks - fill) * pl.heads;
        filled += (int64_t)(blocks - fill) * pl.heads;
      }
      if (reach < fill) {
        const double c = segment_cost(s, length(fill - 1));
        most = c > most ? c : most;
        sum += ((double)(total[fill] - total[reach]) + (segment_cost(s, pl.cut[s]) - pl.cut[s]) * (fill - reach)) * pl.heads;
      }
    }
    // the segments that are filled come first, the others fill the gaps
    const double waves = (double)((filled + sms - 1) / sms) * most, spread = sum / sms + 0.2 * most;
    return n <= sms ? most : waves > spread ? waves : spread;
  };
  static const int kTry[] = {1, 2, 3, 4, 5, 6, 7, 8, 10, 12, 16, 24, 32};
  int best = 1;
  int64_t best_whole = 0;
  double least = 0.0;
  for (const int n : kTry) {
    if (!search || (n > 1 && n > longest)) break;
    set_cuts(n);
    const double c = cost(0);
    if (n == 1 || c < 0.97 * least) {
      least = c;
      best = n;
    }
    const int64_t full = ctas / sms * sms;
    if (!p.causal && full > 0 && full < ctas) {  // whole waves of uncut blocks, and the rest cut
      const double w = (double)(full / sms) * (longest + kSetUp) + cost(full);
      if (w < 0.97 * least) {
        least = w;
        best = n;
        best_whole = full;
      }
    }
  }
  set_cuts(best);
  pl.whole = (int)best_whole;
  int n = 0;
  pl.runs = 0;
  auto run_of = [&](int count, int top) {
    pl.start[pl.runs] = n;
    pl.top[pl.runs++] = top;
    n += count * (p.causal ? pl.heads : 1);
  };
  if (!p.causal) {
    for (int s = 0; s < pl.segments; ++s) run_of((int)(ctas - best_whole), 0);
  } else {
    int reach[kMaxSegments], fill[kMaxSegments];  // the first block that reaches into segment s, and the first that fills it
    for (int s = 0; s < pl.segments; ++s) {
      reach[s] = first_of(pl.cut[s] + 1, 0);
      fill[s] = first_of(pl.cut[s + 1], 0);
      run_of(blocks - fill[s], blocks - 1);
    }
    for (int s = 0; s < pl.segments; ++s) run_of(fill[s] - reach[s], fill[s] - 1);
  }
  pl.ctas = pl.whole + n;
}

int select(const va_select_args& a, cudaStream_t stream) {
  SelectParams p;
  p.avg_q = a.avg_q;
  p.gaps = a.gaps;
  p.gaps_sb = a.gaps_stride_b;
  p.gap = a.gap;
  p.col_count = a.col_count;
  p.col_idx = a.col_idx;
  p.capacity = a.capacity;
  p.status = a.status;
  p.heads = a.heads;
  p.kv_heads = a.kv_heads;
  p.rep = a.heads / a.kv_heads;
  p.nq = a.nq;
  p.sk = a.sk;
  p.pq = a.pq;
  p.group_k_block = a.group_k_block;
  p.starts = 0;
  for (int k = 0; k < 8; k += a.group_k_block < 8 ? a.group_k_block : 8) p.starts |= 1u << k;
  p.causal = a.causal;
  p.wo_initial = a.wo_initial;
  p.compat_bsq = a.compat_bsq;
  p.tile_offset = a.tile_offset;
  p.chunk_tiles = a.chunk_tiles;
  mask_geometry(a.heads, a.kv_heads, a.nq, a.sk, p.rows_pad, p.wpad);
  make_plan(p, a.batch, a.bk);
  if (!a.workspace) return VA_ERR_NULL;
  if (a.workspace_bytes < select_workspace_bytes(a.batch, a.heads, a.kv_heads, a.nq, a.sk)) return VA_ERR_CAPACITY;
  if ((reinterpret_cast<uintptr_t>(a.workspace) & 15u) != 0) return VA_ERR_ALIGN;
  p.mask = static_cast<uint32_t*>(a.workspace);
  CUtensorMap kmap;
  if (!encode_rows_map(&kmap, a.dtype == VA_BF16, a.k.ptr, a.batch, a.kv_heads, a.sk, a.k.stride_b, a.k.stride_h, a.k.stride_s,
                       kTile))
    return VA_ERR_CUDA;
  return a.dtype == VA_BF16 ? launch_dt<VA_BF16>(p, kmap, a.bk, a.batch, stream) : launch_dt<VA_FP16>(p, kmap, a.bk, a.batch, stream);
}

}  // namespace va
