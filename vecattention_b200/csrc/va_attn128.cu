// Vector-sparse flash attention for q_pooling_size 128 on tcgen05 MMAs with M = 128.
//
// One CTA per query tile of 128 rows; keys are taken 128 at a time, from the tile's dense 64-key blocks and then its
// selected-column list (row gather).  S = Q K^T and
// O += P V are tcgen05.mma with M = 128, N = 128: accumulator row r lives in TMEM lane r.  P is the PV product's A operand
// in tensor memory, so it never passes through shared memory: of the traffic of a chunk (K and V written 64 KB, Q and K
// read by S 64 KB, V read by PV 32 KB) the 64 KB that P's store and operand read were are gone.
//
// Warp roles (576 threads, one CTA per SM):
//   warps 0-7  softmax: two groups of four warps (0-3, 4-7) take alternate chunks, a thread owns a whole row of its
//              group's chunk.  It forms the row maximum, raises the running maximum lazily (only when a chunk exceeds
//              it by more than 2^8; the value is shared by both groups through shared memory), writes
//              P = exp2(S*scale - m) in the input dtype into its group's P buffer in tensor memory and rescales the row
//              of O in the rare chunks where the maximum moved.
//   warps 8-15  K (8-11) and V (12-15) gather producers, cp.async 16-byte pieces of the selected rows into rings
//              of 128-byte-swizzled operand tiles (3 K stages, 2 V stages).  Warps 8-11 copy the Q tile too.
//   warps 16,17  MMA issuers (one thread each): warp 16 issues S_j = Q K_j^T into one of two S
//              buffers, warp 17 issues O += P_j V_j; the tensor pipe works on S_{j+1} while the
//              softmax of chunk j runs.
// The producer warpgroups give registers to the softmax warpgroups (setmaxnreg).
// Every wait is a bounded mbarrier wait; a timeout sets VA_STATUS_TIMEOUT and unwinds the CTA.
//
// What bounds it: the softmax groups, three quarters of whose time is work (64 + 128 special-function and fp32 issue slots
// and the tensor-memory latencies between them; both groups of a scheduler share its special-function unit), then
// the gather beside them.  Measured on one B200 with the former kernel (P in shared memory, eight warps in
// lockstep on one chunk): 32 heads x 32 K tokens causal at the reference's default
// arguments 1.97 -> 1.69 ms for the whole operator (1.75 while the gather multiplied 64-bit row offsets).
// Tiles that run on in a CTA, as with 64 rows, with two K stages and the one O buffer that tensor memory has room for: 1.53 -> 1.64 ms.
#include "va_common.cuh"
#include "va_sm100.cuh"
#include "va_attn.cuh"

namespace va {

using namespace sm100;

namespace {

constexpr int kChunk = 128;
constexpr int kTileBytes = 128 * 256;  // 128 rows of 256 bytes: Q, one K or V stage
constexpr int kKStages = 3;
constexpr int kVStages = 2;
constexpr int kThreads = 576;
// Registers per thread: the kernel is launched with 96 (the most 18 warps can all have); the two producer warpgroups
// hand 40 each back and the two softmax warpgroups take them: 256 * 56 + 256 * 136 + 64 * 96 = 576 * 96.
constexpr int kLaunchRegs = 96;
constexpr int kProducerRegs = 56, kSoftmaxRegs = 136;
// the softmax warps can only take what the producer warps hand back: the sum must fit the launch allocation
static_assert(256 * kProducerRegs + 256 * kSoftmaxRegs + 64 * kLaunchRegs <= kThreads * kLaunchRegs, "setmaxnreg pool");
constexpr size_t kSmem = 1024 + (size_t)kTileBytes * (1 + kKStages + kVStages);  // Q, K ring, V ring
constexpr float kRescaleThreshold = 8.0f;                                        // log2 units

struct Barriers {
  uint64_t qfull, kfull[kKStages], kempty[kKStages], vfull[kVStages], vempty[kVStages];
  uint64_t sfull[2], sempty[2], pfull[2], pempty[2], ofull, dec[2], fin;
};

template <int N>
__device__ __forceinline__ void reg_alloc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void reg_dealloc() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

template <int DT>
__global__ void __launch_bounds__(kThreads, 1) attn128_kernel(const AttnParams p) {
  using T = typename Elem<DT>::T;
  constexpr int PQ = 128;
  extern __shared__ unsigned char smem_raw[];
  __shared__ Barriers bars;
  __shared__ uint32_t tmem_base_s;
  __shared__ __align__(16) int keys_s[8][kChunk];           // ring deep enough that a slot is rewritten long after its last reader
  __shared__ __align__(16) int xk_s[8][2][32];  // per producer warp: the lanes' key indices of a chunk, for the exchange
  __shared__ __align__(16) int mask_s[8][4];  // per chunk and K producer warp: does any of its keys need masking?
  __shared__ float m_row_s[2][128];           // [chunk parity][row]: the rows' shared reference maxima (exp2 domain)
  __shared__ float fin_s[256];                // [group * 128 + row]: row sums, added in the epilogue

  wait_for_previous();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int tile, h;
  place(p, (int)gridDim.x, blockIdx.x, blockIdx.y, tile, h);
  const int b = blockIdx.z;
  const int hkv = h / p.rep;
  const int row0 = tile * PQ, row_end = p.sq;  // rows at or past row_end do not exist
  const int64_t trow = ((int64_t)b * p.heads + h) * p.nq + tile;
  const int nblk = p.own_blocks ? own_block_count<PQ>(p, tile) : (p.blk_count ? load_here(p.blk_count + trow) : 0);
  const int ncol = load_here(p.col_count + trow);
  const int nslots = nblk * 64 + ncol;
  const int nchunks = (nslots + kChunk - 1) / kChunk;
  T* ob = static_cast<T*>(p.out) + b * p.o_sb + h * p.o_sh;

  if (nchunks == 0) {  // no key at all: the tile's output is zero
    for (int i = tid; i < PQ * 16; i += kThreads) {
      const int r = i >> 4, c = i & 15;
      if (row0 + r < row_end) *reinterpret_cast<uint4*>(ob + (int64_t)(row0 + r) * p.o_ss + c * 8) = make_uint4(0, 0, 0, 0);
    }
    if (p.lse && tid < PQ && row0 + tid < row_end) p.lse[((int64_t)b * p.heads + h) * p.sq + row0 + tid] = -INFINITY;
    return;
  }

  unsigned char* smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
  unsigned char* q_s = smem;
  unsigned char* k_s = smem + kTileBytes;                     // K ring
  unsigned char* v_s = k_s + (size_t)kKStages * kTileBytes;   // V ring

  if (tid == 0) {
    mbar_init(&bars.qfull, 128);  // per producer thread: one arrival, made by the hardware when the thread's copies have landed
    for (int s = 0; s < kKStages; ++s) {
      mbar_init(&bars.kfull[s], 128);
      mbar_init(&bars.kempty[s], 1);
    }
    for (int s = 0; s < kVStages; ++s) {
      mbar_init(&bars.vfull[s], 128);
      mbar_init(&bars.vempty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars.sfull[s], 1);
      mbar_init(&bars.sempty[s], 128);
      mbar_init(&bars.pfull[s], 128);
      mbar_init(&bars.pempty[s], 1);
      mbar_init(&bars.dec[s], 128);
    }
    mbar_init(&bars.fin, 256);
    mbar_init(&bars.ofull, 1);
    fence_proxy_async();
  }
  if (warp == 16) {
    tmem_alloc(&tmem_base_s, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  // S buffers at columns 0 and 128, O at 256 (128 columns each), P buffers at 384 and 448 (64 columns of 16-bit pairs)
  const uint32_t t_s0 = tmem, t_o = tmem + 256, t_p0 = tmem + 384;

  bool timed_out = false;

  if (warp >= 8 && warp < 16) {
    // ======================= gather producers (warps 8-11: K and the Q tile, warps 12-15: V) =======================
    reg_dealloc<kProducerRegs>();
    const bool is_v = warp >= 12;
    const int pt = is_v ? tid - 384 : tid - 256;
    const T* qb = static_cast<const T*>(p.q) + b * p.q_sb + h * p.q_sh;
    const T* kb = static_cast<const T*>(p.k) + b * p.k_sb + hkv * p.k_sh;
    const T* vb = static_cast<const T*>(p.v) + b * p.v_sb + hkv * p.v_sh;
    const int32_t* blk = p.blk_idx + trow * p.blk_stride;
    const int32_t* col = p.col_idx + trow * p.col_stride;
    if (!is_v) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {  // Q tile: rows beyond the sequence are zero
        const int pce = pt + i * 128, r = pce >> 4, c = pce & 15;
        const bool ok = row0 + r < row_end;
        cp_async16(smem_addr(q_s + tile_off(128, r, c)), qb + (int64_t)(ok ? row0 + r : 0) * p.q_ss + c * 8, ok);
      }
      cp_async_arrive_noinc(&bars.qfull);
    }
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
    auto fetch_raw = [&](int j) -> int {
      const int slot = j * kChunk + my_slot;
      const int ci = min(max(slot - nblk * 64, 0), max(ncol - 1, 0));
      if (p.own_blocks && slot < nblk * 64) return own_block_start<PQ>(p, tile, slot >> 6);
      return load_here(slot < nblk * 64 ? blk + (slot >> 6) : col + ci);
    };
    auto decode = [&](int j, int raw) -> int {
      const int slot = j * kChunk + my_slot;
      const int key = slot < nblk * 64 ? raw + (slot & 63) : (slot < nslots ? raw : -1);
      return (key >= 0 && key < p.sk) ? key : -1;
    };
    // through a small exchange array of the warp: one store and four 16-byte loads per thread instead of sixteen
    // shuffles; two buffers, so the next chunk's stores cannot overtake this chunk's loads
    int* xk = xk_s[warp - 8][0];
    auto spread = [&](int j, int key, int (&out)[16]) {
      int* buf = xk + (j & 1) * 32;
      buf[lane] = max(key, 0);  // an unused slot copies row 0: its scores are masked and its P is zero
      __syncwarp();
      const int4* src = reinterpret_cast<const int4*>(buf + (lane & 16));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int4 q4 = src[i];
        out[4 * i] = q4.x; out[4 * i + 1] = q4.y; out[4 * i + 2] = q4.z; out[4 * i + 3] = q4.w;
      }
    };
    auto copy_tile = [&](unsigned char* tile_s, const T* base, int64_t stride, int row_bytes, const int (&keys)[16], uint64_t* full) {
      const uint32_t dst = smem_addr(tile_s) + dst_off;
      const char* src = reinterpret_cast<const char*>(base + c * 8);
      if (row_bytes != 0) {  // one 32-bit multiplication into the 64-bit address per row
#pragma unroll
        for (int i = 0; i < 16; ++i) cp_async16_full(dst + i * 1024, src + (int64_t)keys[i] * row_bytes);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) cp_async16_full(dst + i * 1024, src + (int64_t)keys[i] * (stride * 2));
      }
      cp_async_arrive_noinc(full);
    };
    int keys[16];
    int raw0 = fetch_raw(0), raw1 = nchunks > 1 ? fetch_raw(1) : 0;
    for (int j = 0; j < nchunks && !timed_out; ++j) {
      const int key = decode(j, raw0);
      raw0 = raw1;
      if (j + 2 < nchunks) raw1 = fetch_raw(j + 2);
      if (!is_v) {
        keys_s[j & 7][my_slot] = key;
        // unused slots, and keys that some row of the tile may not see, make the chunk take the masking pass
        const bool flag = key < 0 || (p.causal && key > p.q_offset + row0);
        const int any = __any_sync(0xffffffffu, flag);
        if (lane == 0) mask_s[j & 7][pw] = any;
      }
      spread(j, key, keys);
      if (!is_v) {
        const int ks = j % kKStages, ku = j / kKStages;
        if (!mbar_wait(&bars.kempty[ks], (ku & 1) ^ 1)) { timed_out = true; break; }
        copy_tile(k_s + (size_t)ks * kTileBytes, kb, p.k_ss, p.k_row_bytes, keys, &bars.kfull[ks]);
      } else {
        const int vs = j % kVStages, vu = j / kVStages;
        if (!mbar_wait(&bars.vempty[vs], (vu & 1) ^ 1)) { timed_out = true; break; }
        copy_tile(v_s + (size_t)vs * kTileBytes, vb, p.v_ss, p.v_row_bytes, keys, &bars.vfull[vs]);
      }
    }
    cp_async_commit();
    cp_async_wait<0>();  // nothing of this thread may still be in flight when the CTA retires
  } else if (warp >= 16) {
    // ======================= MMA issuers =======================
    if (lane == 0) {
      constexpr uint32_t in16 = DT == VA_BF16 ? 1u : 0u;
      bool ok = true;
      if (warp == 16) {
        constexpr uint32_t idesc_s = umma_idesc(128, 128, in16, 0, 0);
        const uint64_t qd = umma_desc(smem_addr(q_s), 16, 1024), kd0 = umma_desc(smem_addr(k_s), 16, 1024);
        ok = mbar_wait(&bars.qfull, 0);
        for (int j = 0; j < nchunks && ok; ++j) {
          const int s = j % kKStages, u = j / kKStages, sb = j & 1, ub = j >> 1;
          ok = mbar_wait(&bars.kfull[s], u & 1) && mbar_wait(&bars.sempty[sb], (ub & 1) ^ 1);
          if (!ok) break;
          fence_proxy_async();  // the producers' cp.async writes (generic proxy) -> visible to the MMA's operand reads
          tc_fence_after();
          umma_k128_rows128(t_s0 + (uint32_t)sb * 128, qd, kd0 + (uint64_t)(s * (kTileBytes >> 4)), idesc_s);
          umma_commit(&bars.kempty[s]);
          umma_commit(&bars.sfull[sb]);
        }
      } else {
        constexpr uint32_t idesc_pv = umma_idesc(128, 128, in16, 0, 1);
        const uint64_t vd0 = umma_desc(smem_addr(v_s), 128 * 128, 1024);
        for (int j = 0; j < nchunks && ok; ++j) {
          const int s = j % kVStages, u = j / kVStages, pb = j & 1;
          ok = mbar_wait(&bars.vfull[s], u & 1) && mbar_wait(&bars.pfull[pb], (j >> 1) & 1);
          if (!ok) break;
          fence_proxy_async();
          tc_fence_after();
          // a K16 step is 2048 bytes further down the V tile (descriptor addresses count 16 bytes)
          const uint64_t vd = vd0 + (uint64_t)(s * (kTileBytes >> 4));
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            umma_ts(t_o, t_p0 + (uint32_t)(pb * 64 + ks * 8), vd + ks * 128, idesc_pv, (j > 0 || ks > 0) ? 1u : 0u);
          umma_commit(&bars.vempty[s]);
          umma_commit(&bars.pempty[pb]);
          if (j == nchunks - 1) umma_commit(&bars.ofull);
        }
      }
      timed_out = !ok;
    }
  } else {
    // ======================= softmax / correction / epilogue =======================
    // Two groups of four warps work on alternate chunks (group 0 = warps 0-3 the even ones, group 1 = warps 4-7 the
    // odd ones), so the latencies of one chunk's softmax overlap the other's.  Accumulator row r lives in TMEM lane r:
    // a thread of either group owns a whole row.  The reference maximum of a row is one value shared by both groups
    // (m_row_s): the decision for chunk j starts from the value left by chunk j - 1, so all P tiles and O stay on one
    // scale.
    reg_alloc<kSoftmaxRegs>();
    const int grp = warp >> 2, qtr = warp & 3;
    const uint32_t lane_base = (uint32_t)(qtr * 32) << 16;
    const int row = qtr * 32 + lane;
    const uint32_t last_key = p.causal ? (uint32_t)(p.q_offset + row0 + row) : 0x7fffffffu;  // that the row may see
    float m_seen = -INFINITY, l = 0.f;  // reference this thread's row sum is currently scaled to
    const float sc = p.scale_log2;
    for (int j = grp; j < nchunks && !timed_out; j += 2) {
      const int ub = j >> 1;
      const int* keys = keys_s[j & 7];
      if (!mbar_wait(&bars.sfull[grp], ub & 1)) { timed_out = true; break; }
      tc_fence_after();
      const int4 mk = *reinterpret_cast<const int4*>(mask_s[j & 7]);
      const bool masked = (mk.x | mk.y | mk.z | mk.w) != 0;
      // ---- the row's maximum.  Beside the gather producers a whole row of 128 scores does not fit the registers: the
      // first 32 are then read again below, the other 96 stay (v[1..3]) ----
      const uint32_t t_s = t_s0 + (uint32_t)(grp * 128) + lane_base;
      uint32_t v[4][32];
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      auto hide = [&](int c) {
        if (!masked) return;  // kept out of the arithmetic loops: a branch per element would serialise them
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const int4 k4 = *reinterpret_cast<const int4*>(keys + c * 32 + i);
          if ((uint32_t)k4.x > last_key) v[c][i] = 0xff800000u;  // -inf; an unused slot's key is -1
          if ((uint32_t)k4.y > last_key) v[c][i + 1] = 0xff800000u;
          if ((uint32_t)k4.z > last_key) v[c][i + 2] = 0xff800000u;
          if ((uint32_t)k4.w > last_key) v[c][i + 3] = 0xff800000u;
        }
      };
      auto top = [&](int c) {
#pragma unroll
        for (int i = 0; i < 32; i += 2)
          m4[(i >> 1) & 3] = max3(m4[(i >> 1) & 3], __uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1]));
      };
      tmem_ld32(t_s, v[0]);
      tmem_ld32(t_s + 32, v[1]);
      tmem_wait_ld();
      hide(0);
      top(0);
      tmem_ld32(t_s + 64, v[2]);
      tmem_ld32(t_s + 96, v[3]);
      hide(1);
      top(1);
      tmem_wait_ld();
      hide(2);
      hide(3);
      top(2);
      top(3);
      const float mx_s = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * sc;
      // ---- the row's reference maximum: continue from what the previous chunk (other group) left; raised only when
      // this chunk exceeds it by more than the threshold ----
      if (j > 0 && !mbar_wait(&bars.dec[grp ^ 1], ((j - 1) >> 1) & 1)) { timed_out = true; break; }
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
        if (!mbar_wait(&bars.pempty[grp ^ 1], ((j - 1) >> 1) & 1)) { timed_out = true; break; }
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
      auto expo = [&](int c) {
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
      };
      expo(1);
      tmem_ld32(t_s, v[0]);
      expo(2);
      tmem_wait_ld();
      tc_fence_before();
      mbar_arrive(&bars.sempty[grp]);  // the S buffer has been read
      hide(0);
      expo(3);
      expo(0);
      const float2 la = halves(ls[0]), lb = halves(ls[1]);
      l += (la.x + la.y) + (lb.x + lb.y);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&bars.pfull[grp]);
    }
    // ---- epilogue: O / l -> global.  Every thread first brings its row sum to the final scale (the last chunk's
    // decision), then the two owners of a row add their sums. ----
    const int jl = nchunks - 1;  // decided by group (jl & 1)
    if (!timed_out && (!mbar_wait(&bars.dec[jl & 1], (jl >> 1) & 1) || !mbar_wait(&bars.ofull, 0))) timed_out = true;
    if (!timed_out) {
      tc_fence_after();
      const float m_fin = m_row_s[jl & 1][row];
      if (m_seen != m_fin) l *= ex2_approx(m_seen - m_fin);  // l == 0 when m_seen == -inf
      fin_s[grp * 128 + row] = l;
      mbar_arrive(&bars.fin);
      if (mbar_wait(&bars.fin, 0)) {
        l = fin_s[row] + fin_s[128 + row];
        const float inv = l > 0.f ? 1.f / l : 0.f;
        const bool row_ok = row0 + row < row_end;
        if (p.lse && row_ok && grp == 0)  // one of the row's two owners; m is in the exp2 domain
          p.lse[((int64_t)b * p.heads + h) * p.sq + row0 + row] = l > 0.f ? (m_fin + log2f(l)) * 0.6931471805599453f : -INFINITY;
        // the two groups split the row's 128 columns
        T* orow = ob + (int64_t)(row0 + (row_ok ? row : 0)) * p.o_ss + grp * 64;
        uint32_t o[2][32];
        tmem_ld32(t_o + lane_base + grp * 64, o[0]);
        tmem_ld32(t_o + lane_base + grp * 64 + 32, o[1]);
        tmem_wait_ld();
        if (row_ok) {
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const uint32_t* x = &o[c >> 2][(c & 3) * 8];
            uint4 w;
            w.x = Elem<DT>::pack(__uint_as_float(x[0]) * inv, __uint_as_float(x[1]) * inv);
            w.y = Elem<DT>::pack(__uint_as_float(x[2]) * inv, __uint_as_float(x[3]) * inv);
            w.z = Elem<DT>::pack(__uint_as_float(x[4]) * inv, __uint_as_float(x[5]) * inv);
            w.w = Elem<DT>::pack(__uint_as_float(x[6]) * inv, __uint_as_float(x[7]) * inv);
            *reinterpret_cast<uint4*>(orow + c * 8) = w;
          }
        }
      } else {
        timed_out = true;
      }
    }
  }
  if (timed_out && p.status) atomicOr(p.status, VA_STATUS_TIMEOUT);
  tc_fence_before();
  __syncthreads();
  if (warp == 16) tmem_dealloc(tmem, 512);
}

template <int DT>
int launch(const AttnParams& p, int batch, cudaStream_t stream) {
  // per-device attribute; setting it on every launch keeps multi-device processes correct
  auto kern = attn128_kernel<DT>;
  if (!succeeded(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem))) return VA_ERR_CUDA;
  return launch_after(kern, dim3(p.nq, p.heads, batch), kThreads, kSmem, stream, p) ? VA_OK : VA_ERR_CUDA;
}

}  // namespace

int launch_attn128(const AttnParams& p, int dtype, int batch, cudaStream_t stream) {
  return dtype == VA_BF16 ? launch<VA_BF16>(p, batch, stream) : launch<VA_FP16>(p, batch, stream);
}

}  // namespace va
