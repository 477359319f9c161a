// Vector-sparse flash attention for q_pooling_size 64 on tcgen05 weight-stationary MMAs.
//
// A query tile has 64 rows; keys are taken 128 at a time from the tile's dense 64-key
// blocks and then from its selected-column list (row gather).  Both products use
// tcgen05.mma.ws with M = 64, N = 128, whose accumulator occupies all 128 TMEM lanes: row r of
// the 64 x 128 result lives in lane r (columns 0..63 of the result) and lane 64 + r (columns
// 64..127), 64 TMEM columns each.  So every accumulator row is owned by two threads, each holding
// half of it, and all four softmax warps do useful work on a 64-row tile.
//
// The grid has one CTA per tile, but a CTA that is running takes over tiles of CTAs that have not been launched
// (cluster launch control), one ahead of the one it gathers for, and its pipeline never drains between them: rings,
// score buffers and barriers run on over the tiles, the next tile's counts and first indices are in shared memory before
// its turn, its Q tile and first K and V rows are copied while the last chunks are worked on.  A CTA per tile spent 5-6 us a tile
// on set-up, fill and drain, as much as six chunks of 128 keys.  Measured on one B200, whole operator, with the packed
// arithmetic of the softmax: 28 query heads on 4 KV heads, 9001 tokens, causal 0.488 -> 0.368 ms; the same heads, 20011
// tokens around a vision span, 1.23 -> 0.88 ms (both with their tiles listed by length); 64 K tokens 6.7 -> 6.2 ms; 32 heads x 32 K
// tokens 3.6 -> 3.34 ms; 5 heads x 75 600 tokens 2.89 -> 2.72 ms.
//
// Warp roles (608 threads, one CTA per SM):
//   warps 0-7  softmax: two groups of four warps (0-3, 4-7) take alternate chunks; inside a group
//              two threads own half a row (64 scores) each.  Per chunk a thread pulls its scores
//              from tensor memory into registers (which frees the S buffer at once), forms the row
//              maximum with its partner thread through shared memory, raises the running maximum
//              lazily (only when a chunk exceeds it by more than 2^8; the value is shared by both
//              groups), writes P = exp2(S*scale - m) in the input dtype into a double-buffered
//              operand tile and rescales its part of the row of O in the rare chunks where the
//              maximum moved.
//   warps 8-11  K gather producers, warps 12-15 V gather producers: cp.async 16-byte pieces of the
//              selected rows into rings of 128-byte-swizzled operand tiles (2 stages each);
//              copy completion is reported to the stage's mbarrier asynchronously; index
//              loads run two chunks ahead and are exchanged inside the warp through shared memory.
//   warps 16,17  MMA issuers (one thread each): warp 16 issues S_j = Q K_j^T, warp 17 issues
//              O += P_j V_j; S, P, Q and O are double buffered, so the tensor pipe works on S_{j+1} and
//              O += P_{j-1} V_{j-1} while softmax j runs.
//   warp 18    scheduler: takes tiles over and describes them.
// The producer warpgroups give registers to the softmax warpgroups (setmaxnreg).
// Every wait is a bounded mbarrier wait; a timeout sets VA_STATUS_TIMEOUT and unwinds the CTA.
#include "va_common.cuh"
#include "va_sm100.cuh"
#include "va_attn.cuh"

#include <type_traits>

namespace va {

using namespace sm100;

namespace {

constexpr int kChunk = 128;
constexpr int kKvTile = 128 * 256;  // 128 gathered rows
constexpr int kQTile = 64 * 256;    // 64 query rows / 64 rows of P
constexpr int kKStages = 2;
constexpr int kVStages = 2;
constexpr int kThreads = 608;
constexpr int kInfo = 4;     // tiles described ahead: the producers may be several short tiles ahead of the softmax
// Registers per thread: the kernel is launched with 96 (the most 19 warps can all have); the two
// producer warpgroups hand 40 each back and the two softmax warpgroups take them:
// 256 * 56 + 256 * 136 + 96 * 96 = 608 * 96.
constexpr int kProducerRegs = 56, kSoftmaxRegs = 136;
// The softmax warps can only take what the producer warps hand back (the CTA's own allocation is the pool); if the
// sum exceeded the launch allocation they would wait for registers nobody releases.
static_assert(256 * kProducerRegs + 256 * kSoftmaxRegs + 96 * 96 <= kThreads * 96, "setmaxnreg pool");
constexpr size_t kSmem = 1024 + (size_t)kQTile * 4 + (size_t)kKvTile * (kKStages + kVStages);  // Q x2, P x2, K ring, V ring
constexpr float kRescaleThreshold = 8.0f;                                            // log2 units

struct Barriers {
  uint64_t qfull[2], qempty[2], kfull[kKStages], kempty[kKStages], vfull[kVStages], vempty[kVStages];
  uint64_t sfull[2], sempty[2], pfull[2], pempty[2], ofull, xch[4], dec[4], fin, ifull[kInfo], iempty[kInfo], begun, clc;
};
// Expected arrivals, in the order of the members above (thread i initialises barrier i).  The "full" barriers of
// the gathered tiles count one arrival per producer thread, made by the hardware when the thread's copies have landed.
constexpr int kNumBarriers = sizeof(Barriers) / sizeof(uint64_t);
__device__ __forceinline__ uint32_t barrier_count(int i) {
  constexpr int qe = 2, kf = qe + 2, ke = kf + kKStages, vf = ke + kKStages, ve = vf + kVStages, sf = ve + kVStages;
  constexpr int se = sf + 2, pf = se + 2, pe = pf + 2, of = pe + 2, xc = of + 1, dc = xc + 4, fn = dc + 4, fi = fn + 1;
  constexpr int ie = fi + kInfo, be = ie + kInfo;
  static_assert(be + 2 == kNumBarriers, "barrier table out of step with struct Barriers");
  if (i < qe) return 128;              // qfull
  if (i < kf) return 1;                // qempty
  if (i < ke) return 128;              // kfull
  if (i < vf) return 1;                // kempty
  if (i < ve) return 128;              // vfull
  if (i < se) return 1;                // vempty, sfull
  if (i < pe) return 128;              // sempty, pfull
  if (i < xc) return 1;                // pempty, ofull
  if (i < fn) return 64;               // xch, dec: the two warps of a group that share 32 rows
  if (i < fi) return 256;              // fin
  if (i < ie) return 32;               // ifull: the lanes of the scheduling warp
  if (i < be) return 18;               // iempty: one lane of every producer and softmax warp, the two issuers
  return 1;                            // begun, clc
}

// A query tile: rows [row0, row_end) of head h, batch b; nchunks < 0: no tile left.  raw: the first 256 slots' entries.
struct Tile {
  int row0, row_end, h, b, nblk, ncol, nchunks, dense;
  int64_t trow;
  int raw[2 * kChunk];
};

// Register hand-over between warpgroups (four consecutive warps, all of which execute it).
template <int N>
__device__ __forceinline__ void reg_alloc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void reg_dealloc() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// D[tmem] (+)= A[smem] * B[smem], weight-stationary form (M = 64 uses all 128 lanes)
__device__ __forceinline__ void umma_ws(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.ws.cta_group::1.kind::f16.collector::b0::discard [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// VIS: the vision-slice composition (a kernel of its own, so that the ordinary one carries none of its bookkeeping)
template <int DT, bool VIS>
__global__ void __launch_bounds__(kThreads, 1) sparse_attn64_kernel(const AttnParams p) {
  using T = typename Elem<DT>::T;
  constexpr int PQ = 64;
  extern __shared__ unsigned char smem_raw[];
  __shared__ Barriers bars;
  __shared__ uint32_t tmem_base_s;
  __shared__ __align__(16) uint4 clc_s;
  __shared__ __align__(16) Tile info_s[kInfo];
  __shared__ __align__(16) int keys_s[8][kChunk];  // ring deep enough that a slot is rewritten long after its last reader
  __shared__ __align__(16) int xk_s[8][2][32];  // per producer warp: the lanes' key indices of a chunk, for the exchange
  __shared__ __align__(16) int mask_s[8][4];  // per chunk and K producer warp: does any of its keys need masking?
  __shared__ float xch_s[2][256];   // [group][phase][TMEM lane]: chunk maxima swapped by a row's two owners
  __shared__ float m_row_s[2][64];   // [chunk parity][row]: the rows' shared reference maxima (exp2 domain)
  __shared__ float fin_s[2][256];    // [tile parity][group][TMEM lane]: row sums, added in the epilogue

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char* smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
  unsigned char* q_s = smem;                                       // two buffers
  unsigned char* p_s = smem + 2 * kQTile;                          // two buffers
  unsigned char* k_s = smem + 4 * kQTile;                          // K ring
  unsigned char* v_s = k_s + (size_t)kKStages * kKvTile;           // V ring

  if (tid < kNumBarriers) {
    mbar_init(reinterpret_cast<uint64_t*>(&bars) + tid, barrier_count(tid));
    fence_proxy_async();
  }
  if (warp == 16) {
    tmem_alloc(&tmem_base_s, 256);
    tmem_relinquish();
  }
  wait_for_previous();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  const uint32_t t_s0 = tmem, t_o0 = tmem + 128;  // S buffers at columns 0 and 64, O buffers at 128 and 192 (64 columns each)

  bool timed_out = false;

  // Tile number `it` of this CTA, as the scheduling warp described it.  In every role: g counts the chunks and n the
  // tiles that have any, over all tiles of the CTA; ring positions, S and P buffers and the softmax group of a chunk
  // follow from g, the Q and O buffers of a tile from n, so no role ever drains between tiles.
  auto tile_info = [&](int it) -> const Tile* {
    if (!mbar_wait(&bars.ifull[it % kInfo], (it / kInfo) & 1)) {
      timed_out = true;
      return nullptr;
    }
    return &info_s[it % kInfo];
  };

  if (warp == 18) {
    // ======================= scheduler =======================
    // Describes this CTA's own tile and then, one after another, tiles taken over from CTAs that have not been
    // launched, with the tile's counts and its first two chunks' column indices, so that the memory latencies at the
    // start of a tile pass while the tile before it is being worked on.
    uint3 id = {blockIdx.x, blockIdx.y, blockIdx.z};
    uint32_t asked = 0;
    bool more = true;
    for (int it = 0; !timed_out;) {
      bool have = more;
      int row0 = 0, row_end = p.sq, tile = 0, head = 0, dense = 0;
      if (more) {
        place(p, (int)gridDim.x, id.x, id.y, tile, head);
        // The tile's rows [row0, row_end).  Ordinarily tile t has rows 64 t ... ; in the vision-slice composition the
        // first p.nq tiles are the sparse tiles of rows [0, vis_end), cut to the rows from vis_begin on, and behind
        // them come dense tiles for rows [0, vis_begin) and for rows [vis_end, sq): all 64-key blocks up to the
        // tile's last row, no tables.
        row0 = tile * PQ;
        if constexpr (VIS) {
          row_end = min(row0 + PQ, p.sq);
          if (tile < p.nq) {
            row_end = min(row0 + PQ, p.vis_end);
            row0 = max(row0, p.vis_begin);
          } else {
            dense = 1;
            const int e = tile - p.nq, n_before = (p.vis_begin + PQ - 1) / PQ;
            if (e < n_before) {
              row0 = e * PQ;
              row_end = min(row0 + PQ, p.vis_begin);
            } else {
              row0 = p.vis_end + (e - n_before) * PQ;
              row_end = min(row0 + PQ, p.sq);
            }
          }
          have = row_end > row0;  // otherwise every row of this sparse tile belongs to the dense part before it
        }
      }
      if (have || !more) {
        Tile* t = &info_s[it % kInfo];
        if (!mbar_wait(&bars.iempty[it % kInfo], ((it / kInfo) & 1) ^ 1)) { timed_out = true; break; }
        if (more) {
          const int64_t trow = dense ? 0 : ((int64_t)id.z * p.heads + head) * p.nq + tile;
          const int32_t* col = p.col_idx + trow * p.col_stride;
          int raw[8];
          // requested before the counts are known; a tile with dense blocks, which come first in slot order, fetches again
#pragma unroll
          for (int i = 0; i < 8; ++i) raw[i] = !dense && i * 32 + lane < p.col_stride ? load_here(col + i * 32 + lane) : 0;
          const int nblk = dense ? (row_end - 1) / 64 + 1
                                 : (p.own_blocks ? own_block_count<PQ>(p, tile) : (p.blk_count ? load_here(p.blk_count + trow) : 0));
          const int ncol = dense ? 0 : load_here(p.col_count + trow);
          if (nblk > 0) {
            const int32_t* blk = dense ? nullptr : p.blk_idx + trow * p.blk_stride;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int slot = i * 32 + lane, ci = slot - nblk * 64;
              if (slot < nblk * 64)
                raw[i] = dense ? (slot >> 6) << 6 : (p.own_blocks ? own_block_start<PQ>(p, tile, slot >> 6) : load_here(blk + (slot >> 6)));
              else raw[i] = ci < ncol ? load_here(col + ci) : 0;
            }
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) t->raw[i * 32 + lane] = raw[i];
          if (lane == 0) {
            t->row0 = row0; t->row_end = row_end; t->h = head; t->b = (int)id.z;
            t->nblk = nblk; t->ncol = ncol; t->nchunks = (nblk * 64 + ncol + kChunk - 1) / kChunk; t->dense = dense;
            t->trow = trow;
          }
        } else if (lane == 0) {
          t->nchunks = -1;
        }
        mbar_arrive(&bars.ifull[it % kInfo]);
        ++it;
      }
      if (!more) break;
      // A tile is only taken over when the gather has begun with the one before it: tiles queued in a CTA that is
      // behind would be missing elsewhere at the end of the grid.
      if (it > 0 && !mbar_wait(&bars.begun, (it - 1) & 1)) { timed_out = true; break; }
      __syncwarp();  // every lane has read the previous answer
      if (lane == 0) {
        fence_proxy_async();
        mbar_expect_tx(&bars.clc, 16);
        clc_try_cancel(&clc_s, &bars.clc);
      }
      if (!mbar_wait(&bars.clc, asked & 1)) { timed_out = true; break; }
      ++asked;
      more = clc_answer(&clc_s, id);
    }
  } else if (warp >= 8 && warp < 16) {
    // ======================= gather producers (warps 8-11: K and the Q tile, warps 12-15: V) =======================
    reg_dealloc<kProducerRegs>();
    // One body, compiled for K and for V: the loop has few registers and sets the pace of the kernel.  With the choice made
    // at run time and 64-bit row offsets it spilled: 5 heads x 75 600 tokens 2.92 ms instead of 2.72, 32 heads x 32 K tokens
    // 3.46 instead of 3.34.
    auto produce = [&](auto is_v_c) {
      constexpr bool is_v = decltype(is_v_c)::value;
      const int pt = is_v ? tid - 384 : tid - 256;
      // Copy geometry.  A warp covers two key rows per instruction: lanes 0-15 the sixteen 16-byte
      // pieces of row rbase + 8 i, lanes 16-31 those of the next row.  Because the rows of one thread
      // differ by multiples of 8, its swizzled piece position is the same in all of them and the
      // shared-memory destinations are one base address plus i * 1024.
      // Each lane fetches ONE key index per chunk (that of row rbase + 8 * (lane & 15)), two chunks
      // ahead; the sixteen indices a thread needs are then exchanged through shared memory.
      const int pw = (pt >> 5), hi = lane >> 4, c = lane & 15;
      const int rbase = 2 * pw + hi;
      const uint32_t dst_off = tile_off(128, rbase, c);
      const int my_slot = rbase + 8 * c;
      // All sixteen keys of this thread's rows, from the lanes that fetched them: through a small exchange array of
      // the warp (one store and four 16-byte loads per thread instead of sixteen shuffles; two buffers, so the
      // next chunk's stores cannot overtake this chunk's loads).
      int* xk = xk_s[warp - 8][0];
      uint32_t g = 0, n = 0;
      int stage = 0;           // ring position of the chunk, and how often the ring has gone round (mod 2)
      uint32_t round = 0;
      for (int it = 0; !timed_out; ++it) {
        const Tile* t = tile_info(it);
        if (t == nullptr) break;
        const int nchunks = t->nchunks, nblk = t->nblk, ncol = t->ncol, row0 = t->row0, row_end = t->row_end, h = t->h, b = t->b;
        const bool dense = VIS && t->dense;
        const int64_t trow = t->trow;
        int raw0 = t->raw[my_slot], raw1 = t->raw[kChunk + my_slot];
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&bars.iempty[it % kInfo]);
          if (warp == 8) mbar_arrive(&bars.begun);
        }
        if (nchunks < 0) break;
        if (nchunks == 0) continue;
        const int hkv = h / p.rep;
        const char* src = reinterpret_cast<const char*>((is_v ? static_cast<const T*>(p.v) + b * p.v_sb + hkv * p.v_sh
                                                              : static_cast<const T*>(p.k) + b * p.k_sb + hkv * p.k_sh) + c * 8);
        const int32_t* blk = dense ? nullptr : p.blk_idx + trow * p.blk_stride;  // no table: blocks 0, 64, 128, ...
        const int32_t* col = p.col_idx + trow * p.col_stride;
        if (!is_v) {
          // the Q buffer is free once the last S product of the tile before the previous one has been computed
          if (!mbar_wait(&bars.qempty[n & 1], ((n >> 1) & 1) ^ 1)) { timed_out = true; break; }
          const T* qb = static_cast<const T*>(p.q) + b * p.q_sb + h * p.q_sh;
          unsigned char* qt = q_s + (n & 1) * kQTile;
#pragma unroll
          for (int i = 0; i < 8; ++i) {  // Q tile: rows beyond the sequence are zero
            const int pce = pt + i * 128, r = pce >> 4, cq = pce & 15;
            const bool ok = row0 + r < row_end;
            cp_async16(smem_addr(qt + tile_off(64, r, cq)), qb + (int64_t)(ok ? row0 + r : 0) * p.q_ss + cq * 8, ok);
          }
          cp_async_arrive_noinc(&bars.qfull[n & 1]);
        }
        // K and V have producer warps of their own, so neither copy waits behind the other's stage:
        // a K stage is free as soon as S has been computed from it, a V stage only after the PV
        // product.  Raw index loads run two chunks ahead and are only interpreted at the top of a
        // later iteration, so the in-order warp never stalls on them.
        // a tile without dense blocks (every non-causal tile): slot s is entry s of the column list
        const bool plain = nblk == 0;
        for (int j = 0; j < nchunks; ++j, ++g) {
          const int slot = j * kChunk + my_slot;
          int key;
          if (plain) {
            key = (slot < ncol && (unsigned)raw0 < (unsigned)p.sk) ? raw0 : -1;
            raw0 = raw1;
            if (j + 2 < nchunks) raw1 = load_here(col + min(slot + 2 * kChunk, ncol - 1));
          } else {
            key = slot < nblk * 64 ? raw0 + (slot & 63) : (slot < nblk * 64 + ncol ? raw0 : -1);
            if ((unsigned)key >= (unsigned)p.sk) key = -1;
            raw0 = raw1;
            if (j + 2 < nchunks) {
              const int s2 = slot + 2 * kChunk;
              if (VIS && s2 < nblk * 64 && blk == nullptr) {
                raw1 = (s2 >> 6) << 6;  // a dense tile: block i starts at key 64 i
              } else {
                const int ci = min(max(s2 - nblk * 64, 0), max(ncol - 1, 0));
                raw1 = load_here(s2 < nblk * 64 ? blk + (s2 >> 6) : col + ci);
              }
            }
          }
          if (!is_v) {
            keys_s[g & 7][my_slot] = key;
            // unused slots, and keys that some row of the tile may not see, make the chunk take the masking pass
            const bool flag = key < 0 || (p.causal && key > p.q_offset + row0);
            const int any = __any_sync(0xffffffffu, flag);
            if (lane == 0) mask_s[g & 7][pw] = any;
          }
          int keys[16];
          {
            int* buf = xk + (g & 1) * 32;
            buf[lane] = max(key, 0);  // an unused slot copies row 0: its scores are masked and its P is zero
            __syncwarp();
            const int4* x4 = reinterpret_cast<const int4*>(buf + (lane & 16));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int4 q4 = x4[i];
              keys[4 * i] = q4.x; keys[4 * i + 1] = q4.y; keys[4 * i + 2] = q4.z; keys[4 * i + 3] = q4.w;
            }
          }
          uint64_t* full = is_v ? &bars.vfull[stage] : &bars.kfull[stage];
          if (!mbar_wait(is_v ? &bars.vempty[stage] : &bars.kempty[stage], round ^ 1)) { timed_out = true; break; }
          const uint32_t dst = smem_addr(is_v ? v_s : k_s) + (uint32_t)stage * kKvTile + dst_off;
          const int row_bytes = is_v ? p.v_row_bytes : p.k_row_bytes;
          if (row_bytes != 0) {  // one 32-bit multiplication into the 64-bit address per row
#pragma unroll
            for (int i = 0; i < 16; ++i) cp_async16_full(dst + i * 1024, src + (int64_t)keys[i] * row_bytes);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) cp_async16_full(dst + i * 1024, src + (int64_t)keys[i] * ((is_v ? p.v_ss : p.k_ss) * 2));
          }
          cp_async_arrive_noinc(full);
          static_assert(kKStages == kVStages, "one ring position for both kinds of producer");
          if (++stage == kKStages) { stage = 0; round ^= 1; }
        }
        ++n;
      }
    };
    if (warp < 12) produce(std::false_type{});
    else produce(std::true_type{});
    cp_async_commit();
    cp_async_wait<0>();  // nothing of this thread may still be in flight when the CTA retires
  } else if (warp >= 16) {
    // ======================= MMA issuers =======================
    // Two independent issuing threads, so that neither product waits behind the other's barriers:
    // warp 16 issues S_j = Q K_j^T, warp 17 issues O += P_j V_j.
    if (lane == 0) {
      constexpr uint32_t in16 = DT == VA_BF16 ? 1u : 0u;
      constexpr uint32_t idesc_s = umma_idesc(64, 128, in16, 0, 0), idesc_pv = umma_idesc(64, 128, in16, 0, 1);
      const uint64_t qd0 = umma_desc(smem_addr(q_s), 16, 1024), kd0 = umma_desc(smem_addr(k_s), 16, 1024);
      const uint64_t pd0 = umma_desc(smem_addr(p_s), 16, 1024), vd0 = umma_desc(smem_addr(v_s), 128 * 128, 1024);
      // (descriptor addresses count 16 bytes; a K16 step is 32 bytes further along a K-major row, 16 rows of V)
      bool ok = true;
      uint32_t g = 0, n = 0;
      for (int it = 0; ok; ++it) {
        const Tile* t = tile_info(it);
        if (t == nullptr) break;
        const int nchunks = t->nchunks;
        mbar_arrive(&bars.iempty[it % kInfo]);
        if (nchunks < 0) break;
        if (nchunks == 0) continue;
        if (warp == 16) {
          const uint64_t qd = qd0 + (n & 1) * (kQTile >> 4);
          ok = mbar_wait(&bars.qfull[n & 1], (n >> 1) & 1);
          for (int j = 0; j < nchunks && ok; ++j, ++g) {
            const uint32_t s = g % kKStages, u = g / kKStages, sb = g & 1, ub = g >> 1;
            ok = mbar_wait(&bars.kfull[s], u & 1) && mbar_wait(&bars.sempty[sb], (ub & 1) ^ 1);
            if (!ok) break;
            fence_proxy_async();  // the producers' cp.async writes (generic proxy) -> visible to the MMA's operand reads
            tc_fence_after();
            const uint64_t kd = kd0 + s * (kKvTile >> 4);
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)
              umma_ws(t_s0 + sb * 64, qd + (ks >> 2) * (64 * 128 >> 4) + (ks & 3) * 2, kd + (ks >> 2) * (128 * 128 >> 4) + (ks & 3) * 2,
                      idesc_s, ks > 0);
            umma_commit(&bars.kempty[s]);
            umma_commit(&bars.sfull[sb]);
            if (j == nchunks - 1) umma_commit(&bars.qempty[n & 1]);
          }
        } else {
          const uint32_t t_o = t_o0 + (n & 1) * 64;
          for (int j = 0; j < nchunks && ok; ++j, ++g) {
            const uint32_t s = g % kVStages, u = g / kVStages, pb = g & 1, upb = g >> 1;
            ok = mbar_wait(&bars.vfull[s], u & 1) && mbar_wait(&bars.pfull[pb], upb & 1);
            if (!ok) break;
            fence_proxy_async();
            tc_fence_after();
            const uint64_t vd = vd0 + s * (kKvTile >> 4), pd = pd0 + pb * (kQTile >> 4);
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)
              umma_ws(t_o, pd + (ks >> 2) * (64 * 128 >> 4) + (ks & 3) * 2, vd + ks * (16 * 128 >> 4), idesc_pv,
                      (j > 0 || ks > 0) ? 1u : 0u);
            umma_commit(&bars.vempty[s]);
            umma_commit(&bars.pempty[pb]);
            if (j == nchunks - 1) umma_commit(&bars.ofull);
          }
        }
        ++n;
      }
      timed_out |= !ok;
    }
  } else {
    // ======================= softmax / correction / epilogue =======================
    // Two groups of four warps work on alternate chunks (group 0 = warps 0-3 the even ones, group 1
    // = warps 4-7 the odd ones, counted over all tiles), so the latencies of one chunk's softmax (tensor-memory load,
    // maximum exchange, exponentials, shared-memory stores) overlap the other's.  Inside a group,
    // accumulator row r lives in TMEM lanes r and 64 + r (64 columns each; a warp reaches the lane
    // quarter warp % 4): two threads own half a row each and meet through shared memory.
    // The reference maximum of a row is one value shared by both groups (m_row_s): the decision for
    // chunk j starts from the value left by chunk j - 1, so all P tiles and O stay on one scale.
    reg_alloc<kSoftmaxRegs>();
    const int grp = warp >> 2;
    const int qtr = warp & 3;
    const uint32_t lane_base = (uint32_t)(qtr * 32) << 16;
    const int tl = qtr * 32 + lane;           // TMEM lane
    const int row = tl & 63, half = tl >> 6;  // query row, which 64-key half of the chunk
    const int pair = qtr & 1;                 // rows 0..31 / 32..63: the two warps of the group that share them
    const float sc = p.scale_log2;
    float* xbuf = xch_s[grp];                 // [2 phases][128]
    uint32_t xc = 0, g0 = 0, n = 0;           // g0: number of the tile's first chunk
    for (int it = 0; !timed_out; ++it) {
      const Tile* t = tile_info(it);
      if (t == nullptr) break;
      const int nchunks = t->nchunks, row0 = t->row0, row_end = t->row_end, h = t->h, b = t->b;
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.iempty[it % kInfo]);
      if (nchunks < 0) break;
      T* ob = static_cast<T*>(p.out) + b * p.o_sb + h * p.o_sh;
      if (nchunks == 0) {  // no key at all: the tile's output is zero
        for (int i = tid; i < PQ * 16; i += 256) {
          const int r = i >> 4, c = i & 15;
          if (row0 + r < row_end) *reinterpret_cast<uint4*>(ob + (int64_t)(row0 + r) * p.o_ss + c * 8) = make_uint4(0, 0, 0, 0);
        }
        if (p.lse && tid < PQ && row0 + tid < row_end) p.lse[((int64_t)b * p.heads + h) * p.sq + row0 + tid] = -INFINITY;
        continue;
      }
      const uint32_t t_o = t_o0 + (n & 1) * 64;
      const uint32_t last_key = p.causal ? (uint32_t)(p.q_offset + row0 + row) : 0x7fffffffu;  // that the row may see
      float m_seen = -INFINITY, l = 0.f;        // reference this thread's row sum is currently scaled to
      for (int j = (int)((g0 ^ (uint32_t)grp) & 1); j < nchunks; j += 2) {  // the chunks whose number has this group's parity
        const uint32_t g = g0 + j, sb = grp, ub = g >> 1;
        const int* keys = keys_s[g & 7] + half * 64;
        if (!mbar_wait(&bars.sfull[sb], ub & 1)) { timed_out = true; break; }
        tc_fence_after();
        const int4 mk = *reinterpret_cast<const int4*>(mask_s[g & 7]);
        const bool masked = (mk.x | mk.y | mk.z | mk.w) != 0;
        // ---- this thread's 64 scores -> registers; the S buffer is free again right away ----
        uint32_t v[64];
        {
          uint32_t lo[32], hi[32];
          tmem_ld32(t_s0 + sb * 64 + lane_base, lo);
          tmem_ld32(t_s0 + sb * 64 + lane_base + 32, hi);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            v[i] = lo[i];
            v[32 + i] = hi[i];
          }
        }
        tc_fence_before();
        mbar_arrive(&bars.sempty[sb]);
        if (masked) {  // kept out of the arithmetic loops: a branch per element would serialise them
#pragma unroll
          for (int i = 0; i < 64; i += 4) {
            const int4 k4 = *reinterpret_cast<const int4*>(keys + i);  // an unused slot's key is -1
            if ((uint32_t)k4.x > last_key) v[i] = 0xff800000u;  // -inf
            if ((uint32_t)k4.y > last_key) v[i + 1] = 0xff800000u;
            if ((uint32_t)k4.z > last_key) v[i + 2] = 0xff800000u;
            if ((uint32_t)k4.w > last_key) v[i + 3] = 0xff800000u;
          }
        }
        // ---- row maximum of the chunk: own half, then the partner's through shared memory ----
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 64; i += 2) m4[(i >> 1) & 3] = max3(m4[(i >> 1) & 3], __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
        float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
        xbuf[(xc & 1) * 128 + tl] = mx;
        mbar_arrive(&bars.xch[grp * 2 + pair]);
        if (!mbar_wait(&bars.xch[grp * 2 + pair], xc & 1)) { timed_out = true; break; }
        mx = fmaxf(mx, xbuf[(xc & 1) * 128 + (tl ^ 64)]);
        ++xc;
        // ---- the row's reference maximum: continue from what the previous chunk (other group) left ----
        if (j > 0 && !mbar_wait(&bars.dec[(grp ^ 1) * 2 + pair], ((g - 1) >> 1) & 1)) { timed_out = true; break; }
        const float m_prev = j > 0 ? m_row_s[grp ^ 1][row] : -INFINITY;
        const float mx_s = mx * sc;
        const bool grow = mx_s > m_prev + kRescaleThreshold || (m_prev == -INFINITY && mx_s > -INFINITY);
        const float m_new = grow ? mx_s : m_prev;
        // Written to the slot of this chunk's parity, never to the one just read: the row's other owner
        // (in another warp) may not have read it yet.  Both owners write the same value.  A tile's first chunk reads
        // nothing, but its group has been through the previous tile's epilogue, which waited for the last decision.
        m_row_s[grp][row] = m_new;
        mbar_arrive(&bars.dec[grp * 2 + pair]);
        const bool rescale = __any_sync(0xffffffffu, grow && j > 0);  // same rows, hence the same outcome, in the partner warp
        // P buffer free <=> the PV product that read it two chunks ago has completed
        if (!mbar_wait(&bars.pempty[sb], (ub & 1) ^ 1)) { timed_out = true; break; }
        if (rescale) {
          // O must be quiescent: wait for the PV product of the previous chunk
          if (!mbar_wait(&bars.pempty[sb ^ 1], ((g - 1) >> 1) & 1)) { timed_out = true; break; }
          tc_fence_after();
          const float alpha = grow ? ex2_approx(m_prev - m_new) : 1.f;  // 2^-inf = 0 when nothing was accumulated yet
#pragma unroll 1
          for (int qd = 0; qd < 2; ++qd) {
            uint32_t o[32];
            tmem_ld32(t_o + lane_base + qd * 32, o);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st32(t_o + lane_base + qd * 32, o);
          }
          tmem_wait_st();
        }
        if (m_seen != m_new) {  // bring this thread's row sum to the current scale (also after the other group moved it)
          l *= ex2_approx(m_seen - m_new);
          m_seen = m_new;
        }
        const float mref = m_new == -INFINITY ? 0.f : m_new;
        // ---- P = exp2(S * scale - m), row sum, P -> shared memory (K-major operand, this thread's 64 keys) ----
        unsigned char* pdst = p_s + (size_t)sb * kQTile;
        const uint64_t sc2 = pair2(sc, sc), nm2 = pair2(-mref, -mref);
        uint64_t sums = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint32_t pk[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = c * 8 + e * 2;
            const float2 x = halves(fma2(pair2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), sc2, nm2));
            const float p0 = ex2_approx(x.x), p1 = ex2_approx(x.y);
            sums = add2(sums, pair2(p0, p1));
            pk[e] = Elem<DT>::pack(p0, p1);
          }
          *reinterpret_cast<uint4*>(pdst + tile_off(64, row, half * 8 + c)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        }
        const float2 ls = halves(sums);
        l += ls.x + ls.y;
        tc_fence_before();
        fence_proxy_async();
        mbar_arrive(&bars.pfull[sb]);
      }
      if (timed_out) break;
      // ---- epilogue: O / l -> global.  Every thread first brings its row sum to the final scale
      // (the last chunk's decision), then the four owners of a row add their sums. ----
      g0 += nchunks;
      const uint32_t jl = g0 - 1;  // the tile's last chunk, decided by group (jl & 1)
      if (!mbar_wait(&bars.dec[(jl & 1) * 2 + pair], (jl >> 1) & 1) || !mbar_wait(&bars.ofull, n & 1)) { timed_out = true; break; }
      tc_fence_after();
      const float m_fin = m_row_s[jl & 1][row];
      if (m_seen != m_fin) l *= ex2_approx(m_seen - m_fin);  // l == 0 when m_seen == -inf
      float* fin = fin_s[n & 1];
      fin[grp * 128 + tl] = l;
      mbar_arrive(&bars.fin);
      // the two groups split the 64 columns of a lane: group 0 takes the lower 32, group 1 the upper
      uint32_t o[32];
      tmem_ld32(t_o + lane_base + grp * 32, o);
      tmem_wait_ld();
      tc_fence_before();  // read before this thread's next arrival: the O buffer is written again two tiles from here
      if (!mbar_wait(&bars.fin, n & 1)) { timed_out = true; break; }
      ++n;
      l = (fin[tl] + fin[tl ^ 64]) + (fin[128 + tl] + fin[128 + (tl ^ 64)]);
      const float inv = l > 0.f ? 1.f / l : 0.f;
      if (row0 + row < row_end) {
        if (p.lse && grp == 0 && half == 0)  // one of the row's four owners; m is in the exp2 domain
          p.lse[((int64_t)b * p.heads + h) * p.sq + row0 + row] = l > 0.f ? (m_fin + log2f(l)) * 0.6931471805599453f : -INFINITY;
        T* orow = ob + (int64_t)(row0 + row) * p.o_ss + half * 64 + grp * 32;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint4 w;
          w.x = Elem<DT>::pack(__uint_as_float(o[c * 8 + 0]) * inv, __uint_as_float(o[c * 8 + 1]) * inv);
          w.y = Elem<DT>::pack(__uint_as_float(o[c * 8 + 2]) * inv, __uint_as_float(o[c * 8 + 3]) * inv);
          w.z = Elem<DT>::pack(__uint_as_float(o[c * 8 + 4]) * inv, __uint_as_float(o[c * 8 + 5]) * inv);
          w.w = Elem<DT>::pack(__uint_as_float(o[c * 8 + 6]) * inv, __uint_as_float(o[c * 8 + 7]) * inv);
          *reinterpret_cast<uint4*>(orow + c * 8) = w;
        }
      }
    }
  }
  if (timed_out && p.status) atomicOr(p.status, VA_STATUS_TIMEOUT);
  tc_fence_before();
  __syncthreads();
  if (warp == 16) tmem_dealloc(tmem, 256);
}

template <int DT>
int launch(const AttnParams& p, int batch, cudaStream_t stream) {
  // per-device attribute; setting it on every launch keeps multi-device processes correct
  auto kern = p.vis_on ? sparse_attn64_kernel<DT, true> : sparse_attn64_kernel<DT, false>;
  if (!succeeded(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem))) return VA_ERR_CUDA;
  int tiles = p.nq;
  if (p.vis_on) tiles += (p.vis_begin + 63) / 64 + (p.sq - p.vis_end + 63) / 64;  // the dense tiles before and after
  dim3 grid(tiles, p.heads, batch);
  return launch_after(kern, grid, kThreads, kSmem, stream, p) ? VA_OK : VA_ERR_CUDA;
}

}  // namespace


int launch_attn64(const AttnParams& p, int dtype, int batch, cudaStream_t stream) {
  return dtype == VA_BF16 ? launch<VA_BF16>(p, batch, stream) : launch<VA_FP16>(p, batch, stream);
}

}  // namespace va
