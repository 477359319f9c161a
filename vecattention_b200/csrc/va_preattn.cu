// What a video-DiT attention layer does to Q and K between the projections and the operator, in one pass:
// RMSNorm over the hidden dimension, the rotary embedding on interleaved (even, odd) element pairs, and no
// layout change at all, because the operator reads (B, S, H, D) storage in place through strides.
//
// Reference (eval/DiTEvalKit/models/wan/attention.py:108-136): a Triton RMSNorm kernel (read + write),
// three transposed copies to (B, H, S, D) (read + write each) and an in-place rotary kernel (read + write).
// Here every element of Q and K is read once and written once; V is not touched.
//
// A token row of one tensor (grid.y: 0 = Q, 1 = K) is taken by one, two or four warps, whose lanes own 16-byte
// pieces (8 elements) of it: sum of squares in fp32 (per lane in piece order, a fixed shuffle tree, a fixed sum over
// the row's warps), y = round16(x * rstd * w) as the norm kernel stores it
// (eval/DiTEvalKit/kernels/triton/rmsnorm.py:30-47), then out = round16(double(y0) * cos - double(y1) * sin),
// round16(double(y1) * cos + double(y0) * sin) for every pair, in double precision as the rotary kernel
// computes it (eval/DiTEvalKit/kernels/include/rope/rope_enc_complex.cuh:27-45).
// A second kernel serves models whose tensors are (B, H, L, 128) already, with a per-head norm and the text tokens
// last (HunyuanVideo).
#include "va_common.cuh"

namespace va {

namespace {

template <int DT>
__device__ __forceinline__ typename Elem<DT>::T from_double(double x) {
  if constexpr (DT == VA_BF16) return __double2bfloat16(x);
  else return __double2half(x);
}

// ---- the rotation of a pair, rounded once ----
// x = a c - b s rounded once to the 16-bit type is what the double-precision expression gives.  Its conversions and the
// rounding from double cost the kernel, which is bound by issue slots, more than the norm did, so nearly all pairs are
// done in fp32 with the same result (40 heads, 75 600 tokens: 0.995 -> 0.82 ms; a branch per pair instead of
// one per piece of four: 0.886):
//  * Kahan's product sum (w = b s; f = a c - w; t = f + (w - b s), both fma exact to their last rounding) is within
//    1.5 units in the last place of x (Jeannerod, Louvet, Muller, "Further analysis of Kahan's algorithm for the accurate
//    computation of 2 x 2 determinants", 2013) unless something over- or underflows: an overflow leaves an infinity or a
//    NaN in t, and what an underflow can lose, 2^-149, is nothing beside an x of 2^-100 or more.
//  * x then lies between t (1 - 2^-22) and t (1 + 2^-22) (2 to 4 units in the last place away, more where t is just
//    below a power of two and x above it); if both round to the same 16-bit value, so does x.
//  * Otherwise (a rounding boundary lies in between: one value in 10000 in bf16, in 1400 in fp16), or if some |t| is not between
//    2^-100 and 2^100, the double-precision expression decides, in one call for the piece.
//  * A piece of zeros (rows of padding) needs no decision unless a table holds an infinity or a NaN, which shows in the
//    result: f is then the sum of its two products, signs of zero included, and w - b s is +0.  All rows zero, 40 heads,
//    75 600 tokens: 0.86 ms; 1.23 when each pair of them went to the double-precision branch, 1.03 with no other.
constexpr float kTiny = 7.8886091e-31f, kHuge = 1.2676506e30f;  // 2^-100, 2^100
// the pairs of a piece that `which` has a bit for; the others stay as fp32 gave them (`out`)
template <int DT>
__device__ __noinline__ uint4 turn_exactly(float4 y0, float4 y1, float4 c4, float4 s4, uint4 out, uint32_t which) {
  using T = typename Elem<DT>::T;
  const float y[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w}, c[4] = {c4.x, c4.y, c4.z, c4.w}, s[4] = {s4.x, s4.y, s4.z, s4.w};
  uint32_t r[4] = {out.x, out.y, out.z, out.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if ((which >> j & 1) == 0) continue;
    const double ed = y[2 * j], od = y[2 * j + 1], cd = c[j], sd = s[j];
    const T r0 = from_double<DT>(ed * cd + (-od) * sd), r1 = from_double<DT>(od * cd + ed * sd);
    r[j] = (uint32_t) * reinterpret_cast<const uint16_t*>(&r0) | ((uint32_t) * reinterpret_cast<const uint16_t*>(&r1) << 16);
  }
  return make_uint4(r[0], r[1], r[2], r[3]);
}
// the four pairs (y[2 j], y[2 j + 1]) of a piece, turned by the angles with cosines c[j] and sines s[j], packed; one
// branch for all of them
template <int DT>
__device__ __forceinline__ void turn(const float (&y)[8], const float (&c)[4], const float (&s)[4], uint32_t (&out)[4]) {
  const uint64_t down = pair2(1.f - 2.38418579e-7f, 1.f - 2.38418579e-7f), up = pair2(1.f + 2.38418579e-7f, 1.f + 2.38418579e-7f);
  uint32_t differ = 0, other[4];
  float least = INFINITY, total = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float e = y[2 * j], o = y[2 * j + 1];
    const uint64_t oe = pair2(o, e), ss = pair2(-s[j], s[j]), ns = pair2(s[j], -s[j]);
    const uint64_t w = mul2(oe, ss), f = fma2(pair2(e, o), pair2(c[j], c[j]), w), over = fma2(oe, ns, w);  // over: w minus the exact product
    const float2 fh = halves(f), oh = halves(over);
    const float t0 = fh.x - oh.x, t1 = fh.y - oh.y;
    least = fminf(fminf(least, fabsf(t0)), fabsf(t1));
    total += fabsf(t0);
    total += fabsf(t1);
    const uint64_t t = pair2(t0, t1);
    const float2 lo = halves(mul2(t, down)), hi = halves(mul2(t, up));
    out[j] = Elem<DT>::pack(lo.x, lo.y);
    other[j] = Elem<DT>::pack(hi.x, hi.y);
    differ |= out[j] ^ other[j];
  }
  const bool plain = least >= kTiny && total <= kHuge;  // (false for a NaN)
  if (differ != 0 || !plain) {
    uint32_t which = 0;
    if (!plain) {
      float most = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) most = fmaxf(most, fabsf(y[i]));
      if (most == 0.f && ((out[0] | out[1] | out[2] | out[3]) & 0x7fff7fffu) == 0) return;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) which |= out[j] != other[j] || !plain ? 1u << j : 0u;
    const uint4 r = turn_exactly<DT>(make_float4(y[0], y[1], y[2], y[3]), make_float4(y[4], y[5], y[6], y[7]),
                                     make_float4(c[0], c[1], c[2], c[3]), make_float4(s[0], s[1], s[2], s[3]),
                                     make_uint4(out[0], out[1], out[2], out[3]), which);
    out[0] = r.x; out[1] = r.y; out[2] = r.z; out[3] = r.w;
  }
}

// ---- the hidden-size form: W warps per token row ------------------------------------------------------------------
// A row is taken by W = ceil(hidden / 1024) warps; a lane keeps its (up to) four 16-byte pieces packed in registers,
// so every warp has its whole share of the row in flight at once, and the W warps add their partial sums through
// shared memory (one block barrier).  Few registers, hence some thirty warps resident per SM: enough outstanding
// memory, which one CTA per row with one piece or two per thread in flight was not (2.4 TB/s).  A CTA holds as many
// whole rows as fit eight warps.
// Bound by issue slots (71 %), and a row has only sixteen pairs per lane: what is done once a row counts.  With a 64-bit remainder, two
// divisions by W and a loop over the row's partial sums it took 0.814-0.818 ms at 40 heads x 75 600 tokens in bf16, without
// them 0.713-0.741 (eight runs on several GPUs), 4.2-4.4 TB/s; fp16 0.843 -> 0.725, 12 heads x 30 000 tokens 0.114 -> 0.103 (one run each).
constexpr int NP = 4;  // pieces per lane
// ROTATE: the call has tables.  The norm alone is a kernel of its own: with the rotation's registers and branches around it,
// it took 0.612 ms (0.579 before the rotation was done in fp32), alone 0.521 (40 heads, 75 600 tokens).
template <int DT, bool ROTATE>
__global__ void __launch_bounds__(256, 4) qk_norm_rope_rows_kernel(const va_norm_rope_args a, uint32_t rows) {
  using T = typename Elem<DT>::T;
  __shared__ __align__(16) float part[8][8];  // [row of the CTA][warp of the row], zeros behind the last
  const bool is_k = blockIdx.y == 1;
  // a block is 32 W x rows threads: no division by W, and 32-bit arithmetic up to the addresses
  const int lane = threadIdx.x & 31, W = blockDim.x >> 5, wsub = threadIdx.x >> 5, rsub = threadIdx.y;
  const uint32_t at = blockIdx.x * blockDim.y + rsub;  // b * seq_len + s
  const bool live = at < rows;
  const uint32_t token = live ? at : 0;
  const int hidden = (is_k ? a.kv_heads : a.heads) * kHeadDim;
  const T* x = static_cast<const T*>(is_k ? a.k : a.q) + (int64_t)token * (is_k ? a.k_row_stride : a.q_row_stride);
  T* y = static_cast<T*>(is_k ? a.k_out : a.q_out) + (int64_t)token * (is_k ? a.k_out_row_stride : a.q_out_row_stride);
  const T* w = static_cast<const T*>(is_k ? a.k_weight : a.q_weight);
  const int pieces = live ? hidden / 8 : 0;

  uint4 raw[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const int pc = wsub * 32 + lane + 32 * W * i;
    raw[i] = pc < pieces ? __ldg(reinterpret_cast<const uint4*>(x + pc * 8)) : make_uint4(0, 0, 0, 0);
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const uint32_t ww[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = Elem<DT>::unpack(ww[j]);
      ss = fmaf(f.x, f.x, ss);
      ss = fmaf(f.y, f.y, ss);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if (W > 1) {
    if (lane == 0) part[rsub][wsub] = ss;
    if (wsub == 0 && lane >= W && lane < 8) part[rsub][lane] = 0.f;
    __syncthreads();
    const float4 a0 = *reinterpret_cast<const float4*>(part[rsub]), a1 = *reinterpret_cast<const float4*>(part[rsub] + 4);
    ss = ((((((a0.x + a0.y) + a0.z) + a0.w) + a1.x) + a1.y) + a1.z) + a1.w;  // the same order in every warp of the row
  }
  const float rstd = w ? 1.0f / sqrtf(ss / (float)hidden + a.eps) : 1.0f;  // no weight: no normalisation
  const uint64_t rstd2 = pair2(rstd, rstd);

  const int rs = (int)(a.batch == 1 ? token : token % (uint32_t)a.seq_len) - a.rope_skip;  // row of the cos / sin tables; the first rope_skip tokens are not rotated
  const bool rotate = ROTATE && live && rs >= 0;
  float cc[4] = {}, sv[4] = {};
  if (rotate) {  // a lane's pieces lie 32 W pieces apart, whole heads: all of them sit at the same place of their head
    const int64_t at = (int64_t)rs * (kHeadDim / 2) + (lane & 15) * 4;
    const float4 c = __ldg(reinterpret_cast<const float4*>(a.cos + at)), sn = __ldg(reinterpret_cast<const float4*>(a.sin + at));
    cc[0] = c.x; cc[1] = c.y; cc[2] = c.z; cc[3] = c.w;
    sv[0] = sn.x; sv[1] = sn.y; sv[2] = sn.z; sv[3] = sn.w;
  }
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const int pc = wsub * 32 + lane + 32 * W * i;
    if (pc < pieces) {
      const uint32_t xw[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
      float yv[8];
      if (w) {
        const uint4 wr = __ldg(reinterpret_cast<const uint4*>(w + pc * 8));
        const uint32_t ww[4] = {wr.x, wr.y, wr.z, wr.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = Elem<DT>::unpack(ww[j]), v = Elem<DT>::unpack(xw[j]);
          // x_hat = x * rstd, y = x_hat * w, rounded to the 16-bit type as the norm kernel stores it
          const float2 n = halves(mul2(mul2(pair2(v.x, v.y), rstd2), pair2(f.x, f.y)));
          const float2 y = Elem<DT>::unpack(Elem<DT>::pack(n.x, n.y));
          yv[2 * j] = y.x;
          yv[2 * j + 1] = y.y;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 v = Elem<DT>::unpack(xw[j]);
          yv[2 * j] = v.x;
          yv[2 * j + 1] = v.y;
        }
      }
      uint32_t out[4];
      if (rotate) {
        turn<DT>(yv, cc, sv, out);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) out[j] = Elem<DT>::pack(yv[2 * j], yv[2 * j + 1]);
      }
      *reinterpret_cast<uint4*>(y + pc * 8) = make_uint4(out[0], out[1], out[2], out[3]);
    }
  }
}

template <int DT>
int launch_rows_dt(const va_norm_rope_args& a, cudaStream_t stream) {
  const int64_t rows = (int64_t)a.batch * a.seq_len;
  const int pieces = (a.heads > a.kv_heads ? a.heads : a.kv_heads) * kHeadDim / 8;  // of the wider of the two tensors
  const int W = (pieces + 32 * NP - 1) / (32 * NP);                                 // 1 .. 8 (hidden sizes up to 8192)
  const int per = 8 / W;
  dim3 grid((unsigned)((rows + per - 1) / per), 2, 1);
  auto kern = a.cos ? qk_norm_rope_rows_kernel<DT, true> : qk_norm_rope_rows_kernel<DT, false>;
  kern<<<grid, dim3(32 * W, per), 0, stream>>>(a, (uint32_t)rows);
  return cudaGetLastError() == cudaSuccess ? VA_OK : VA_ERR_CUDA;
}

// ---- the per-head form (HunyuanVideo): tensors are (B, H, L, 128) already ---------------------------------------
// RMSNorm over the 128 elements of every (batch, head, token) row (eval/DiTEvalKit/kernels/include/norm/
// narrow_rms_norm.cuh:22-73: sixteen threads per row, eight elements each, sum of squares in element order, xor
// shuffles 8-4-2-1, rsqrtf(sum / 128 + eps), y = T((x * r) * w)), then the rotary embedding on interleaved pairs
// in fp32 with per-element tables, out[i] = y[i] cos[i] + (i even ? -y[i+1] : y[i-1]) sin[i]
// (eval/DiTEvalKit/kernels/include/rope/rope_enc_txtlast.cuh:32-76: tokens from rope_len on are left alone).
// The same sixteen-threads-per-row layout here.
template <int DT>
__global__ void __launch_bounds__(256) qk_head_norm_rope_kernel(const va_head_norm_rope_args a, int64_t tokens) {
  using T = typename Elem<DT>::T;
  // Sixteen lanes per token (b, l); they walk the token's heads, Q's then K's, four at a time, so that the token's
  // 1 KB of cos / sin entries is read once and four rows are in flight per lane.
  const int lane16 = threadIdx.x & 15;
  const int64_t token = (int64_t)blockIdx.x * 16 + (threadIdx.x >> 4);
  const bool live = token < tokens;
  const int l = (int)((live ? token : 0) % a.seq_len);
  const int b = (int)((live ? token : 0) / a.seq_len);
  const bool rotate = a.cos != nullptr && l < a.rope_len;
  float cc[8], sn[8];
  if (rotate) {
    const float* cr = a.cos + (int64_t)l * kHeadDim + lane16 * 8;
    const float* sr = a.sin + (int64_t)l * kHeadDim + lane16 * 8;
    const float4 c0 = __ldg(reinterpret_cast<const float4*>(cr)), c1 = __ldg(reinterpret_cast<const float4*>(cr + 4));
    const float4 s0 = __ldg(reinterpret_cast<const float4*>(sr)), s1 = __ldg(reinterpret_cast<const float4*>(sr + 4));
    cc[0] = c0.x; cc[1] = c0.y; cc[2] = c0.z; cc[3] = c0.w; cc[4] = c1.x; cc[5] = c1.y; cc[6] = c1.z; cc[7] = c1.w;
    sn[0] = s0.x; sn[1] = s0.y; sn[2] = s0.z; sn[3] = s0.w; sn[4] = s1.x; sn[5] = s1.y; sn[6] = s1.z; sn[7] = s1.w;
  }
#pragma unroll 1
  for (int which = 0; which < 2; ++which) {  // 0: Q, 1: K
    const va_tensor4& in = which ? a.k : a.q;
    const va_tensor4_out& out = which ? a.k_out : a.q_out;
    const int heads = which ? a.kv_heads : a.heads;
    const T* w = static_cast<const T*>(which ? a.k_weight : a.q_weight);
    const T* xb = static_cast<const T*>(in.ptr) + b * in.stride_b + (int64_t)l * in.stride_s + lane16 * 8;
    T* yb = static_cast<T*>(out.ptr) + b * out.stride_b + (int64_t)l * out.stride_s + lane16 * 8;
    float wv[8];
    if (w) {
      const uint4 wr = __ldg(reinterpret_cast<const uint4*>(w + lane16 * 8));
      const uint32_t ww[4] = {wr.x, wr.y, wr.z, wr.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = Elem<DT>::unpack(ww[j]);
        wv[2 * j] = f.x;
        wv[2 * j + 1] = f.y;
      }
    }
#pragma unroll 1
    for (int h0 = 0; h0 < heads; h0 += 4) {
      uint4 raw[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        raw[u] = (live && h0 + u < heads) ? __ldg(reinterpret_cast<const uint4*>(xb + (int64_t)(h0 + u) * in.stride_h)) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t xw[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
        float v[8];
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = Elem<DT>::unpack(xw[j]);
          v[2 * j] = f.x;
          v[2 * j + 1] = f.y;
          ss = fmaf(f.x, f.x, ss);
          ss = fmaf(f.y, f.y, ss);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);  // within the token's sixteen lanes
        if (w) {
          const float rs = rsqrtf(ss / (float)kHeadDim + a.eps);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = Elem<DT>::to_float(Elem<DT>::from_float(__fmul_rn(__fmul_rn(v[j], rs), wv[j])));
        }
        uint32_t o4[4];
        if (rotate) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float e = v[2 * j], od = v[2 * j + 1];
            const float r0 = fmaf(-od, sn[2 * j], __fmul_rn(e, cc[2 * j]));        // x[i] cos[i] + (-x[i+1]) sin[i]
            const float r1 = fmaf(e, sn[2 * j + 1], __fmul_rn(od, cc[2 * j + 1]));  // x[i] cos[i] + x[i-1] sin[i]
            o4[j] = Elem<DT>::pack(r0, r1);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) o4[j] = Elem<DT>::pack(v[2 * j], v[2 * j + 1]);
        }
        if (live && h0 + u < heads)
          *reinterpret_cast<uint4*>(yb + (int64_t)(h0 + u) * out.stride_h) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
      }
    }
  }
}

}  // namespace

int qk_head_norm_rope(const va_head_norm_rope_args& a, cudaStream_t stream) {
  const int64_t tokens = (int64_t)a.batch * a.seq_len;
  const unsigned grid = (unsigned)((tokens + 15) / 16);
  if (a.dtype == VA_BF16) qk_head_norm_rope_kernel<VA_BF16><<<grid, 256, 0, stream>>>(a, tokens);
  else qk_head_norm_rope_kernel<VA_FP16><<<grid, 256, 0, stream>>>(a, tokens);
  return cudaGetLastError() == cudaSuccess ? VA_OK : VA_ERR_CUDA;
}

int qk_norm_rope(const va_norm_rope_args& a, cudaStream_t stream) {
  return a.dtype == VA_BF16 ? launch_rows_dt<VA_BF16>(a, stream) : launch_rows_dt<VA_FP16>(a, stream);
}

}  // namespace va
