// Dense causal flash attention (one sequence for queries and keys) with 128-row query tiles on tcgen05 MMAs with M = 128.
//
// Keys are taken 128 at a time, from key 0 up to the tile's last row: contiguous tiles of K and V, streamed by TMA.  S = Q K^T and
// O += P V are tcgen05.mma with M = 128, N = 128: accumulator row r lives in TMEM lane r.  P is the PV product's A operand
// in tensor memory, so it never passes through shared memory.  As in the 64-row kernel a running CTA takes over further tiles
// (cluster launch control) and its pipeline never drains between them.
//
// Warp roles (512 threads, one CTA per SM):
//   warps 0-7  softmax: two groups of four warps (0-3, 4-7) take alternate chunks, a thread owns a whole row of its
//              group's chunk.  It forms the row maximum, raises the running maximum lazily (only when a chunk exceeds
//              it by more than 2^8; the value is shared by both groups through shared memory), writes
//              P = exp2(S*scale - m) in the input dtype into its group's P buffer in tensor memory and rescales the row
//              of O in the rare chunks where the maximum moved.  At a tile's end it leaves its row sums and goes on.
//   warps 8-11  copy the Q tiles and write the results.
//   warp 12    one thread takes tiles over, describes them and streams K; warp 13: one thread streams V.
//   warps 14,15  MMA issuers (one thread each): warp 14 issues S_j = Q K_j^T into one of two S
//              buffers, warp 15 issues O += P_j V_j; the tensor pipe works on S_{j+1} while the
//              softmax of chunk j runs.
// Warps 8-15 give registers to the softmax warpgroups (setmaxnreg), so that a thread holds a whole row of scores.
// Every wait is a bounded mbarrier wait; a timeout sets VA_STATUS_TIMEOUT and unwinds the CTA.
//
// What bounds it: the softmax groups (64 + 128 special-function and fp32 issue slots per score pair and the tensor-memory
// latencies between them; both groups of a scheduler share its special-function unit).  28 query heads on 4 KV heads, 8192 tokens,
// whole call: 0.855 ms on gathered 64-row tiles, 0.487-0.503 with a CTA per tile, which set up, filled and drained its pipeline 12 times
// per SM and whose softmax warps wrote the results, now 0.45-0.47; 16 heads x 500 tokens 42.2 -> 29.8 us, 32/8 heads x 3000 104 -> 84,
// 16 heads x 16 384 1070 -> 1042.
#include "va_common.cuh"
#include "va_sm100.cuh"
#include "va_attn.cuh"
#include "va_tmap.cuh"

namespace va {

using namespace sm100;

namespace {

constexpr int kChunk = 128;
constexpr int kTileBytes = 128 * 256;  // 128 rows of 256 bytes: Q, one K or V stage
constexpr int kRing = 2;               // stages of the K ring and of the V ring
constexpr int kInfo = 4;               // tiles described ahead
constexpr int kThreads = 512;
// Registers per thread: launched with 128, 256 * 168 + 256 * 88 = 512 * 128.  The softmax warps can only take what the others
// hand back: the sum must fit the launch allocation.
constexpr int kOtherRegs = 88, kSoftmaxRegs = 168;
static_assert(256 * kOtherRegs + 256 * kSoftmaxRegs <= kThreads * 128, "setmaxnreg pool");
constexpr size_t kSmem = 1024 + (size_t)kTileBytes * (2 + 2 * kRing);  // Q x2, K ring, V ring
constexpr float kRescaleThreshold = 8.0f;                               // log2 units

struct Barriers {
  uint64_t qfull[2], qempty[2], kfull[kRing], kempty[kRing], vfull[kRing], vempty[kRing], ifull[kInfo], iempty[kInfo], clc;
  uint64_t sfull[2], sempty[2], pfull[2], pempty[2], ofull[2], oempty[2], dec[2], fin[2];
};

// A query tile: rows [row0, row_end) of head h, batch b; nchunks < 0: no tile left.
struct Tile {
  int row0, row_end, h, b, nchunks;
};

// Tensor maps of K and V (rows of 128 elements, boxes of 128 rows by 64 elements).
struct DenseMaps {
  CUtensorMap k, v;
};

// umma_ts that leaves lanes 0 to 63 of the accumulator as they are
__device__ __forceinline__ void umma_ts_upper(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.eq.b32 p, %3, %3;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%4, %4, %5, %5}, p;\n\t}" ::"r"(
          d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(0xffffffffu), "r"(0u)
      : "memory");
}

template <int N>
__device__ __forceinline__ void reg_alloc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void reg_dealloc() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

template <int DT>
__global__ void __launch_bounds__(kThreads, 1) dense128_kernel(const AttnParams p, const __grid_constant__ DenseMaps maps) {
  using T = typename Elem<DT>::T;
  constexpr int PQ = 128;
  extern __shared__ unsigned char smem_raw[];
  __shared__ Barriers bars;
  __shared__ uint32_t tmem_base_s;
  __shared__ __align__(16) uint4 clc_s;
  __shared__ Tile info_s[kInfo];
  __shared__ float m_row_s[2][128];                 // [chunk parity][row]: the rows' shared reference maxima (exp2 domain)
  __shared__ float fin_s[2][256], fin_m_s[2][256];  // [tile parity][group * 128 + row]: row sums, and the reference they are scaled to

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char* smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
  unsigned char* q_s = smem;                              // two buffers
  unsigned char* k_s = smem + 2 * kTileBytes;             // K ring
  unsigned char* v_s = k_s + (size_t)kRing * kTileBytes;  // V ring

  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars.qfull[s], 128);  // per copying thread: one arrival, made by the hardware when the thread's copies have landed
      mbar_init(&bars.qempty[s], 1);
      mbar_init(&bars.kfull[s], 1);
      mbar_init(&bars.kempty[s], 1);
      mbar_init(&bars.vfull[s], 1);
      mbar_init(&bars.vempty[s], 1);
      mbar_init(&bars.sfull[s], 1);
      mbar_init(&bars.sempty[s], 128);
      mbar_init(&bars.pfull[s], 128);
      mbar_init(&bars.pempty[s], 1);
      mbar_init(&bars.ofull[s], 1);
      mbar_init(&bars.oempty[s], 128);
      mbar_init(&bars.dec[s], 128);
      mbar_init(&bars.fin[s], 256);
    }
    for (int s = 0; s < kInfo; ++s) {
      mbar_init(&bars.ifull[s], 1);
      mbar_init(&bars.iempty[s], 15);  // one lane of every softmax warp and of warps 8-11, V, the two issuers
    }
    mbar_init(&bars.clc, 1);
    fence_proxy_async();
  }
  static_assert(kRing == 2, "initialised above");
  if (warp == 14) {
    tmem_alloc(&tmem_base_s, 512);
    tmem_relinquish();
  }
  wait_for_previous();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  // S buffers at columns 0 and 128, O at 256 (128 columns each), P buffers at 384 and 448 (64 columns of 16-bit pairs).  The
  // one O buffer is read by warps 8-11 right after a tile's last product, while the softmax works on the next tile.
  const uint32_t t_s0 = tmem, t_o = tmem + 256, t_p0 = tmem + 384;

  bool timed_out = false;

  // Tile number `it` of this CTA.  In every role g counts the chunks and n (or `it`) the tiles, over all tiles of the CTA; ring
  // positions, S and P buffers and the softmax group of a chunk follow from g, the Q buffer of a tile from n.
  auto tile_info = [&](int it) -> const Tile* { return mbar_wait(&bars.ifull[it % kInfo], (it / kInfo) & 1) ? &info_s[it % kInfo] : nullptr; };

  // O / l -> global: warp w reads TMEM lane quarter w % 4
  auto write_tile = [&](uint32_t n, int row0, int rows, int h, int b) -> bool {
    const uint32_t ob = n & 1, par = (n >> 1) & 1;
    const int row = tid & 127;
    if (!mbar_wait(&bars.fin[ob], par) || !mbar_wait(&bars.ofull[ob], par)) return false;
    tc_fence_after();
    const float *fl = fin_s[ob], *fm = fin_m_s[ob];
    const float m_fin = fmaxf(fm[row], fm[128 + row]);  // the last decision's: the reference is only ever raised
    auto sum = [&](int i) { return fm[i] != m_fin ? fl[i] * ex2_approx(fm[i] - m_fin) : fl[i]; };  // 0 from a group without a chunk
    const float l = sum(row) + sum(128 + row);
    const float inv = l > 0.f ? 1.f / l : 0.f;
    if (p.lse && row < rows)  // m is in the exp2 domain
      p.lse[((int64_t)b * p.heads + h) * p.sq + row0 + row] = l > 0.f ? (m_fin + log2f(l)) * 0.6931471805599453f : -INFINITY;
    T* orow = static_cast<T*>(p.out) + b * p.o_sb + h * p.o_sh + (int64_t)(row0 + (row < rows ? row : 0)) * p.o_ss;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {
      uint32_t o[16];
      tmem_ld16(t_o + lane_base + c * 16, o);
      tmem_wait_ld();
      if (c == 7) {  // O may be written again
        tc_fence_before();
        mbar_arrive(&bars.oempty[ob]);
      }
      if (row < rows) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          uint4 x;
          x.x = Elem<DT>::pack(__uint_as_float(o[i * 8 + 0]) * inv, __uint_as_float(o[i * 8 + 1]) * inv);
          x.y = Elem<DT>::pack(__uint_as_float(o[i * 8 + 2]) * inv, __uint_as_float(o[i * 8 + 3]) * inv);
          x.z = Elem<DT>::pack(__uint_as_float(o[i * 8 + 4]) * inv, __uint_as_float(o[i * 8 + 5]) * inv);
          x.w = Elem<DT>::pack(__uint_as_float(o[i * 8 + 6]) * inv, __uint_as_float(o[i * 8 + 7]) * inv);
          *reinterpret_cast<uint4*>(orow + c * 16 + i * 8) = x;
        }
      }
    }
    return true;
  };

  if (warp >= 8 && warp < 12) {
    // ======================= Q tiles and results =======================
    reg_dealloc<kOtherRegs>();
    const int pt = tid - 256;
    int row0 = 0, rows = 0, h = 0, b = 0;  // the tile before, whose result is due
    for (int it = 0;; ++it) {
      const Tile* t = tile_info(it);
      if (t == nullptr) { timed_out = true; break; }
      const int nchunks = t->nchunks, next_row0 = t->row0, next_rows = t->row_end - t->row0, next_h = t->h, next_b = t->b;
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.iempty[it % kInfo]);
      if (nchunks >= 0) {
        // the Q buffer is free once the last S product of the tile before the previous one has been computed
        if (!mbar_wait(&bars.qempty[it & 1], ((it >> 1) & 1) ^ 1)) { timed_out = true; break; }
        const T* qb = static_cast<const T*>(p.q) + next_b * p.q_sb + next_h * p.q_sh;
        unsigned char* qt = q_s + (it & 1) * kTileBytes;
#pragma unroll
        for (int i = 0; i < 16; ++i) {  // rows beyond the sequence are zero
          const int pce = pt + i * 128, r = pce >> 4, c = pce & 15;
          const bool ok = r < next_rows;
          cp_async16(smem_addr(qt + tile_off(128, r, c)), qb + (int64_t)(ok ? next_row0 + r : 0) * p.q_ss + c * 8, ok);
        }
        cp_async_arrive_noinc(&bars.qfull[it & 1]);
      }
      if (it > 0 && !write_tile(it - 1, row0, rows, h, b)) { timed_out = true; break; }
      if (nchunks < 0) break;
      row0 = next_row0; rows = next_rows; h = next_h; b = next_b;
    }
    cp_async_commit();
    cp_async_wait<0>();  // nothing of this thread may still be in flight when the CTA retires
  } else if (warp >= 12) {
    reg_dealloc<kOtherRegs>();
    if (lane == 0 && warp == 12) {
      // ======================= tiles and K =======================
      uint3 id = {blockIdx.x, blockIdx.y, blockIdx.z};
      bool more = true;
      int g = 0, stage = 0;
      uint32_t round = 0;
      for (int it = 0; !timed_out; ++it) {
        if (!mbar_wait(&bars.iempty[it % kInfo], ((it / kInfo) & 1) ^ 1)) { timed_out = true; break; }
        Tile* t = &info_s[it % kInfo];
        if (!more) {
          t->nchunks = -1;
          mbar_arrive(&bars.ifull[it % kInfo]);
          break;
        }
        int tile, h;
        place(p, (int)gridDim.x, id.x, id.y, tile, h);
        const int row_end = min(p.sq, (tile + 1) * PQ), nchunks = (row_end + kChunk - 1) / kChunk, b = (int)id.z, hkv = h / p.rep;
        t->row0 = tile * PQ; t->row_end = row_end; t->h = h; t->b = b; t->nchunks = nchunks;
        mbar_arrive(&bars.ifull[it % kInfo]);
        bool asked = false;
        for (int j = 0; j < nchunks; ++j, ++g) {
          if (j == max(nchunks - 3, 0)) {  // asked for when this tile ends: a tile queued here would be missing elsewhere
            fence_proxy_async();
            mbar_expect_tx(&bars.clc, 16);
            clc_try_cancel(&clc_s, &bars.clc);
            asked = true;
          }
          if (!mbar_wait(&bars.kempty[stage], round ^ 1)) { timed_out = true; break; }
          mbar_expect_tx(&bars.kfull[stage], kTileBytes);
          const uint32_t dst = smem_addr(k_s) + (uint32_t)stage * kTileBytes;
          tma_load_4d(dst, &maps.k, 0, j * kChunk, hkv, b, &bars.kfull[stage]);
          tma_load_4d(dst + kTileBytes / 2, &maps.k, 64, j * kChunk, hkv, b, &bars.kfull[stage]);
          if (++stage == kRing) { stage = 0; round ^= 1; }
        }
        if (asked && !mbar_wait(&bars.clc, it & 1)) timed_out = true;  // (also after a timeout: the answer must land before the CTA ends)
        if (timed_out) break;
        more = clc_answer(&clc_s, id);
      }
      if (timed_out)  // copies still in flight must land before the CTA's memory is given back
        for (int i = max(0, g - kRing); i < g; ++i) mbar_wait(&bars.kfull[i % kRing], (i / kRing) & 1);
    } else if (lane == 0 && warp == 13) {
      // ======================= V =======================
      int g = 0, stage = 0;
      uint32_t round = 0;
      for (int it = 0; !timed_out; ++it) {
        const Tile* t = tile_info(it);
        if (t == nullptr) { timed_out = true; break; }
        const int nchunks = t->nchunks, hkv = t->h / p.rep, b = t->b;
        mbar_arrive(&bars.iempty[it % kInfo]);
        for (int j = 0; j < nchunks; ++j, ++g) {
          if (!mbar_wait(&bars.vempty[stage], round ^ 1)) { timed_out = true; break; }
          mbar_expect_tx(&bars.vfull[stage], kTileBytes);
          const uint32_t dst = smem_addr(v_s) + (uint32_t)stage * kTileBytes;
          tma_load_4d(dst, &maps.v, 0, j * kChunk, hkv, b, &bars.vfull[stage]);
          tma_load_4d(dst + kTileBytes / 2, &maps.v, 64, j * kChunk, hkv, b, &bars.vfull[stage]);
          if (++stage == kRing) { stage = 0; round ^= 1; }
        }
        if (nchunks < 0) break;
      }
      if (timed_out)
        for (int i = max(0, g - kRing); i < g; ++i) mbar_wait(&bars.vfull[i % kRing], (i / kRing) & 1);
    } else if (lane == 0) {
      // ======================= MMA issuers =======================
      constexpr uint32_t in16 = DT == VA_BF16 ? 1u : 0u;
      constexpr uint32_t idesc_s = umma_idesc(128, 128, in16, 0, 0), idesc_pv = umma_idesc(128, 128, in16, 0, 1);
      const uint64_t qd0 = umma_desc(smem_addr(q_s), 16, 1024), kd0 = umma_desc(smem_addr(k_s), 16, 1024);
      const uint64_t vd0 = umma_desc(smem_addr(v_s), 128 * 128, 1024);
      bool ok = true;
      uint32_t g = 0;
      for (uint32_t n = 0; ok; ++n) {
        const Tile* t = tile_info(n);
        if (t == nullptr) { ok = false; break; }
        const int nchunks = t->nchunks;
        mbar_arrive(&bars.iempty[n % kInfo]);
        if (nchunks < 0) break;
        if (warp == 14) {
          const uint64_t qd = qd0 + (n & 1) * (kTileBytes >> 4);
          ok = mbar_wait(&bars.qfull[n & 1], (n >> 1) & 1);
          for (int j = 0; j < nchunks && ok; ++j, ++g) {
            const uint32_t s = g % kRing, u = g / kRing, sb = g & 1, ub = g >> 1;
            ok = mbar_wait(&bars.kfull[s], u & 1) && mbar_wait(&bars.sempty[sb], (ub & 1) ^ 1);
            if (!ok) break;
            fence_proxy_async();  // the Q tile's cp.async writes (generic proxy) -> visible to the MMA's operand reads
            tc_fence_after();
            umma_k128_rows128(t_s0 + sb * 128, qd, kd0 + s * (kTileBytes >> 4), idesc_s);
            umma_commit(&bars.kempty[s]);
            umma_commit(&bars.sfull[sb]);
            if (j == nchunks - 1) umma_commit(&bars.qempty[n & 1]);
          }
        } else {
          // the result of the tile before has been read
          if (n > 0) ok = mbar_wait(&bars.oempty[(n - 1) & 1], ((n - 1) >> 1) & 1);
          for (int j = 0; j < nchunks && ok; ++j, ++g) {
            const uint32_t s = g % kRing, u = g / kRing, pb = g & 1;
            ok = mbar_wait(&bars.vfull[s], u & 1) && mbar_wait(&bars.pfull[pb], (g >> 1) & 1);
            if (!ok) break;
            tc_fence_after();
            // a K16 step is 2048 bytes further down the V tile (descriptor addresses count 16 bytes)
            const uint64_t vd = vd0 + s * (kTileBytes >> 4);
            const uint32_t a = t_p0 + pb * 64;
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) umma_ts(t_o, a + ks * 8, vd + ks * 128, idesc_pv, (j > 0 || ks > 0) ? 1u : 0u);
            if (j < nchunks - 1) {
#pragma unroll
              for (int ks = 4; ks < 8; ++ks) umma_ts(t_o, a + ks * 8, vd + ks * 128, idesc_pv, 1u);
            } else {
              // The first 64 rows of the tile see none of the last 64 keys, and their weights for them, exact zeros, would
              // still turn an Inf or NaN in V into a NaN: that half of the product leaves those rows alone.
#pragma unroll
              for (int ks = 4; ks < 8; ++ks) umma_ts_upper(t_o, a + ks * 8, vd + ks * 128, idesc_pv);
            }
            umma_commit(&bars.vempty[s]);
            umma_commit(&bars.pempty[pb]);
            if (j == nchunks - 1) umma_commit(&bars.ofull[n & 1]);
          }
        }
      }
      timed_out |= !ok;
    }
  } else {
    // ======================= softmax / correction =======================
    // Two groups of four warps work on alternate chunks (counted over all tiles), so the latencies of one chunk's softmax
    // overlap the other's.  Accumulator row r lives in TMEM lane r: a thread of either group owns a whole row.  The reference
    // maximum of a row is one value shared by both groups (m_row_s): the decision for chunk j starts from the value left by
    // chunk j - 1, so all P tiles and O stay on one scale.
    reg_alloc<kSoftmaxRegs>();
    const int grp = warp >> 2, qtr = warp & 3;
    const uint32_t lane_base = (uint32_t)(qtr * 32) << 16;
    const int row = qtr * 32 + lane;
    const float sc = p.scale_log2;
    uint32_t g0 = 0, n = 0;  // g0: number of the tile's first chunk
    for (int it = 0; !timed_out; ++it) {
      const Tile* t = tile_info(it);
      if (t == nullptr) { timed_out = true; break; }
      const int nchunks = t->nchunks, row0 = t->row0;
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.iempty[it % kInfo]);
      if (nchunks < 0) break;
      const uint32_t last_key = (uint32_t)(p.q_offset + row0 + row);  // that the row may see
      float m_seen = -INFINITY, l = 0.f;  // reference this thread's row sum is currently scaled to
      for (int j = (int)((g0 ^ (uint32_t)grp) & 1); j < nchunks; j += 2) {  // the chunks whose number has this group's parity
        const uint32_t g = g0 + j, ub = g >> 1;
        if (!mbar_wait(&bars.sfull[grp], ub & 1)) { timed_out = true; break; }
        tc_fence_after();
        const bool masked = (j + 1) * kChunk - 1 > row0;
        // ---- the row's 128 scores and their maximum ----
        const uint32_t t_s = t_s0 + (uint32_t)(grp * 128) + lane_base;
        uint32_t v[4][32];
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        auto hide = [&](int c) {
          if (!masked) return;  // kept out of the arithmetic loops: a branch per element would serialise them
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if ((uint32_t)(j * kChunk + c * 32 + i) > last_key) v[c][i] = 0xff800000u;  // -inf
        };
        auto top = [&](int c) {
#pragma unroll
          for (int i = 0; i < 32; i += 2)
            m4[(i >> 1) & 3] = max3(m4[(i >> 1) & 3], __uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1]));
        };
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(t_s + c * 32, v[c]);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive(&bars.sempty[grp]);  // the S buffer has been read
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          hide(c);
          top(c);
        }
        const float mx_s = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * sc;
        // ---- the row's reference maximum: continue from what the previous chunk (other group) left; raised only when
        // this chunk exceeds it by more than the threshold.  (The wait also at a tile's start, where nothing is read: the
        // other group must have read what this chunk overwrites.) ----
        if (g > 0 && !mbar_wait(&bars.dec[grp ^ 1], ((g - 1) >> 1) & 1)) { timed_out = true; break; }
        const float m_prev = j > 0 ? m_row_s[grp ^ 1][row] : -INFINITY;
        const bool grow = mx_s > m_prev + kRescaleThreshold || (m_prev == -INFINITY && mx_s > -INFINITY);
        const float m_new = grow ? mx_s : m_prev;
        m_row_s[grp][row] = m_new;
        mbar_arrive(&bars.dec[grp]);
        const bool rescale = __any_sync(0xffffffffu, grow && j > 0);
        // P buffer free <=> the PV product that read it two chunks ago has completed
        if (!mbar_wait(&bars.pempty[grp], (ub & 1) ^ 1)) { timed_out = true; break; }
        if (rescale) {
          // O must be quiescent: wait for the PV product of the previous chunk
          if (!mbar_wait(&bars.pempty[grp ^ 1], ((g - 1) >> 1) & 1)) { timed_out = true; break; }
          tc_fence_after();
          const float alpha = grow ? ex2_approx(m_prev - m_new) : 1.f;  // 2^-inf = 0 when nothing was accumulated yet
#pragma unroll 1
          for (int qd = 0; qd < 8; ++qd) {
            uint32_t o[16];
            tmem_ld16(t_o + lane_base + qd * 16, o);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st16(t_o + lane_base + qd * 16, o);
          }
        }
        tc_fence_after();
        if (m_seen != m_new) {  // bring this thread's row sum to the current scale (also after the other group moved it)
          l *= ex2_approx(m_seen - m_new);
          m_seen = m_new;
        }
        const float mref = m_new == -INFINITY ? 0.f : m_new;
        // ---- P = exp2(S * scale - m) -> tensor memory (the A operand of the PV product), row sum ----
        const uint64_t sc2 = pair2(sc, sc), nm2 = pair2(-mref, -mref);
        uint64_t ls[2] = {0, 0};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            uint32_t pk[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const int i = q * 16 + e * 2;
              const float2 x = halves(fma2(pair2(__uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1])), sc2, nm2));
              const float p0 = ex2_approx(x.x), p1 = ex2_approx(x.y);
              ls[e & 1] = add2(ls[e & 1], pair2(p0, p1));
              pk[e] = Elem<DT>::pack(p0, p1);
            }
            tmem_st8(t_p0 + (uint32_t)(grp * 64 + c * 16 + q * 8) + lane_base, pk);
          }
        }
        const float2 la = halves(ls[0]), lb = halves(ls[1]);
        l += (la.x + la.y) + (lb.x + lb.y);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(&bars.pfull[grp]);
      }
      if (timed_out) break;
      // ---- the row sums go to warps 8-11, which write the result; this group goes on with the next tile ----
      g0 += nchunks;
      if (!mbar_wait(&bars.oempty[n & 1], ((n >> 1) & 1) ^ 1)) { timed_out = true; break; }  // the sums two tiles ago have been read
      fin_s[n & 1][grp * 128 + row] = l;
      fin_m_s[n & 1][grp * 128 + row] = m_seen;
      mbar_arrive(&bars.fin[n & 1]);
      ++n;
    }
  }
  if (timed_out && p.status) atomicOr(p.status, VA_STATUS_TIMEOUT);
  tc_fence_before();
  __syncthreads();
  if (warp == 14) tmem_dealloc(tmem, 512);
}

template <int DT>
int launch(const AttnParams& p, const DenseMaps& maps, int tiles, int batch, cudaStream_t stream) {
  // per-device attribute; setting it on every launch keeps multi-device processes correct
  auto kern = dense128_kernel<DT>;
  if (!succeeded(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem))) return VA_ERR_CUDA;
  return launch_after(kern, dim3(tiles, p.heads, batch), kThreads, kSmem, stream, p, maps) ? VA_OK : VA_ERR_CUDA;
}

}  // namespace

// false: the tensors cannot be described by a tensor map (nothing has been launched)
bool launch_dense128(const AttnParams& p, int dtype, int batch, cudaStream_t stream, int* rc) {
  DenseMaps maps;
  const int kv_heads = p.heads / p.rep, bf16 = dtype == VA_BF16;
  auto forward = [&](int64_t sb, int64_t sh, int64_t ss) { return ss > 0 && (kv_heads == 1 || sh > 0) && (batch == 1 || sb > 0); };
  if (!forward(p.k_sb, p.k_sh, p.k_ss) || !forward(p.v_sb, p.v_sh, p.v_ss)) return false;  // repeated or reversed rows
  if (!encode_rows_map(&maps.k, bf16, p.k, batch, kv_heads, p.sk, p.k_sb, p.k_sh, p.k_ss, kChunk) ||
      !encode_rows_map(&maps.v, bf16, p.v, batch, kv_heads, p.sk, p.v_sb, p.v_sh, p.v_ss, kChunk))
    return false;
  const int tiles = (p.sq + 127) / 128;
  *rc = bf16 ? launch<VA_BF16>(p, maps, tiles, batch, stream) : launch<VA_FP16>(p, maps, tiles, batch, stream);
  return true;
}

}  // namespace va
