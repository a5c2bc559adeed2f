// KIVI cache maintenance kernels: quantize-on-append and dense dequantize, sm_100a.
//
// Storage of one layer (caller-owned, preallocated for `cap` tokens, cap % 128 == 0):
//   k_codes [B][H][cap][D*bits/8]            codes packed along CHANNELS: channel c of a token
//                                            sits at bit (c*bits) of the token's row (little endian)
//   k_scale, k_zero [B][H][cap/group][D]     fp32 per (group of `group` tokens, channel); channel c at
//                                            position kmeta_pos(c, D) of the row (common.cuh)
//   v_codes [B][H][cap/128][D][128*bits/8]   codes packed along TOKENS inside blocks of 128 tokens:
//                                            token t of the block sits at bit (t*bits) of row d
//   v_scale, v_zero [B][H][cap][D/v_group]   fp32 per (token, group of v_group channels); v_group == D (one per
//                                            token, the reference's form) or 32
// The two code layouts follow the two contractions of attention: q.K^T contracts channels,
// P.V contracts tokens, so each packs along the axis its consumer reads 128 bits at a time.
//
// Arithmetic restates pare/kv_cache.py:75-156 in IEEE fp32 with the same operation order, so
// codes, scales and zeros are bit-identical to the reference:
//   scale = max((max - min) / qmax, 1e-8)          true division
//   code  = rint(min(max((x - min) / scale, 0), qmax))   true division, clamp, then half-to-even
//   x^    = code * scale + min                     separate multiply and add (no FMA contraction)

#include <type_traits>

#include "common.cuh"

namespace pare {
namespace {

struct CachePtrs {
  uint8_t* k_codes;
  float* k_scale;
  float* k_zero;
  uint8_t* v_codes;
  float* v_scale;
  float* v_zero;
  int B, H, D, bits, group, cap;
  int v_group;   // channels that share a value scale / zero: D, or a multiple of 32 that divides D
};

template <typename T>
__device__ __forceinline__ float load_as_float(const void* base, int64_t idx) {
  return to_float<T>(reinterpret_cast<const T*>(base)[idx]);
}

__device__ __forceinline__ uint8_t affine_code(float x, float lo, float scale, float qmax) {
  const float q = fminf(fmaxf(__fdiv_rn(__fsub_rn(x, lo), scale), 0.f), qmax);
  return (uint8_t)rintf(q);
}

// Eight such codes without a division per element, packed code k at bit k * BITS.  A quotient is approximated by a
// product with the correctly rounded reciprocal (error below 2 units in the last place of a number below 16, i.e. < 4e-6)
// and rounded to the nearest integer by adding 1.5 * 2^23 (round-to-nearest-even, like rintf; the integer then sits in the
// low mantissa bits, and the eight shifted words are added up, the exponent bits taken off once).  Only an approximation
// within 1e-4 of a rounding boundary could round differently from the exact quotient: one branch per eight elements
// sends those (about one set in six hundred) through the division.  x >= lo by construction, so only the upper clamp
// is needed.  Bit-identical to affine_code.
template <int BITS>
__device__ __forceinline__ uint32_t affine_codes8(const float (&x)[8], const float (&lo)[8], const float (&inv)[8], const float (&scale)[8]) {
  constexpr float qmax = (float)((1 << BITS) - 1);
  constexpr uint32_t kMagic = 0x4B400000u;
  uint32_t w = 0, fix = 0;
  float worst = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float q = fminf(__fmul_rn(__fsub_rn(x[k], lo[k]), inv[k]), qmax);
    const float r = __fadd_rn(q, 12582912.f);
    worst = fmaxf(worst, fabsf(__fsub_rn(__fsub_rn(r, 12582912.f), q)));
    w += __float_as_uint(r) << (k * BITS);
    fix += kMagic << (k * BITS);
  }
  w -= fix;
  if (worst > 0.4999f) {
    w = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) w |= (uint32_t)affine_code(x[k], lo[k], scale[k], qmax) << (k * BITS);
  }
  return w;
}

struct SrcStrides {
  int64_t b, h, t;
};

// One CTA per (token group, head, batch); blockDim.x == D.
template <typename T>
__global__ void kivi_append_kernel(const void* k_src, const void* v_src, SrcStrides ks, SrcStrides vs, int t0, CachePtrs c) {
  extern __shared__ unsigned char smem[];
  const int G = c.group, D = c.D, bits = c.bits;
  const int g = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int d = threadIdx.x, warp = d >> 5, lane = d & 31, nwarps = D >> 5;
  const float qmax = (float)((1 << bits) - 1);
  const int tok0 = t0 + g * G;                      // first destination token of this group
  const int64_t k0 = (int64_t)b * ks.b + (int64_t)h * ks.h + (int64_t)g * G * ks.t;
  const int64_t v0 = (int64_t)b * vs.b + (int64_t)h * vs.h + (int64_t)g * G * vs.t;
  const size_t bh = (size_t)b * c.H + h;

  uint8_t* codes = smem;                                                   // [G][D]
  const int VG = D / c.v_group;                                            // value groups per token
  float* v_lo = reinterpret_cast<float*>(smem + (size_t)G * D);            // [G][VG]
  float* v_sc = v_lo + G * VG;                                             // [G][VG]

  // ---- keys: per channel over the G tokens of the group ----
  {
    float lo = INFINITY, hi = -INFINITY;
    for (int t = 0; t < G; ++t) {
      const float x = load_as_float<T>(k_src, k0 + (int64_t)t * ks.t + d);
      lo = fminf(lo, x);
      hi = fmaxf(hi, x);
    }
    const float scale = fmaxf(__fdiv_rn(__fsub_rn(hi, lo), qmax), 1e-8f);
    const size_t mi = (bh * (c.cap / G) + tok0 / G) * D + kmeta_pos(d, D);
    c.k_scale[mi] = scale;
    c.k_zero[mi] = lo;
    for (int t = 0; t < G; ++t) {
      const float x = load_as_float<T>(k_src, k0 + (int64_t)t * ks.t + d);
      codes[t * D + d] = affine_code(x, lo, scale, qmax);
    }
  }
  __syncthreads();
  {
    // pack along channels: every thread emits whole bytes of the [G][D*bits/8] block
    const int row_bytes = D * bits / 8, per_byte = 8 / bits;
    uint8_t* dst = c.k_codes + (bh * c.cap + tok0) * (size_t)row_bytes;
    for (int i = d; i < G * row_bytes; i += D) {
      const int t = i / row_bytes, j = i - t * row_bytes;
      uint32_t v = 0;
      for (int e = 0; e < per_byte; ++e) v |= (uint32_t)codes[t * D + j * per_byte + e] << (e * bits);
      dst[i] = (uint8_t)v;
    }
  }
  __syncthreads();

  // ---- values: per token over each group of v_group channels (all D of them in the reference's form) ----
  for (int t = warp; t < G; t += nwarps) {
    for (int vg = 0; vg < VG; ++vg) {
      float lo = INFINITY, hi = -INFINITY;
      for (int cc = vg * c.v_group + lane; cc < (vg + 1) * c.v_group; cc += 32) {
        const float x = load_as_float<T>(v_src, v0 + (int64_t)t * vs.t + cc);
        lo = fminf(lo, x);
        hi = fmaxf(hi, x);
      }
      lo = warp_min(lo);
      hi = warp_max(hi);
      const float scale = fmaxf(__fdiv_rn(__fsub_rn(hi, lo), qmax), 1e-8f);
      if (lane == 0) {
        v_lo[t * VG + vg] = lo;
        v_sc[t * VG + vg] = scale;
        c.v_scale[(bh * c.cap + tok0 + t) * VG + vg] = scale;
        c.v_zero[(bh * c.cap + tok0 + t) * VG + vg] = lo;
      }
    }
  }
  __syncthreads();
  {
    // pack along tokens: thread d owns row d of the 128-token block(s) this group falls into
    const int row_bytes = 128 * bits / 8, per_byte = 8 / bits;
    for (int tb = 0; tb < G; tb += per_byte) {
      uint32_t v = 0;
      for (int e = 0; e < per_byte; ++e) {
        const int t = tb + e;
        const float x = load_as_float<T>(v_src, v0 + (int64_t)t * vs.t + d);
        v |= (uint32_t)affine_code(x, v_lo[t * VG + d / c.v_group], v_sc[t * VG + d / c.v_group], qmax) << (e * bits);
      }
      const int tok = tok0 + tb;
      uint8_t* row = c.v_codes + ((bh * (c.cap / 128) + tok / 128) * D + d) * (size_t)row_bytes;
      row[(tok % 128) * bits / 8] = (uint8_t)v;
    }
  }
}

// Vectorised quantize-on-append for the attention geometry (D == 128, 2- or 4-bit codes, 16-bit source, groups of up
// to 64 tokens, 16-byte aligned source rows): one CTA of 128 threads per (token group, head, batch).  The group's keys
// and values (G x 256 bytes each) come in with 16-byte loads into shared memory and every later pass reads them from
// there; the codes leave as 16-byte vectors -- a token's key codes in runs of 16 bytes, a channel's value codes of
// the group in pieces of its row.  Same arithmetic, in the same order, as the element-wise kernel above.
// The group size is a template parameter: with run-time trip counts the shared-memory reads of the statistics and of the
// value codes were one round trip each (128 threads, 0.26 of the HBM rate); unrolled they overlap.
__host__ __device__ constexpr int key_pair_slot(int c) {   // (minimum, 1 / scale) of channel c, 8 bytes each: a quarter warp's eight readers (below) hit eight bank groups
  return 2 * ((c >> 5) * 24 + ((c >> 3) & 3) * 4 + 2 * (((c >> 3) & 3) >> 1) + ((c >> 5) & 1) + ((c & 7) >> 1)) + (c & 1);
}
constexpr int kKeyPairs = 192;         // slots, some unused

template <typename T, int BITS, int VG, int G>
__global__ void __launch_bounds__(128) kivi_append128_kernel(const void* k_src, const void* v_src, SrcStrides ks, SrcStrides vs, int t0,
                                                              CachePtrs c) {
  constexpr int D = 128;
  extern __shared__ __align__(16) unsigned char sm[];
  T* kt = reinterpret_cast<T*>(sm);                         // [G][D]
  T* vt = kt + G * D;                                       // [G][D]
  float2* kp_s = reinterpret_cast<float2*>(vt + G * D);     // [key_pair_slot(channel)] (group minimum, 1 / scale)
  float2* vp_s = kp_s + kKeyPairs;                          // [G][VG] (minimum, 1 / scale)
  float* ks_s = reinterpret_cast<float*>(vp_s + G * VG);    // [D] scale
  float* vs_s = ks_s + D;                                   // [G][VG] scale
  const int g = blockIdx.x, h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const float qmax = (float)((1 << BITS) - 1);
  const int tok0 = t0 + g * G;
  const size_t bh = (size_t)b * c.H + h;
  const T* kg = reinterpret_cast<const T*>(k_src) + (int64_t)b * ks.b + (int64_t)h * ks.h + (int64_t)g * G * ks.t;
  const T* vg_ = reinterpret_cast<const T*>(v_src) + (int64_t)b * vs.b + (int64_t)h * vs.h + (int64_t)g * G * vs.t;
#pragma unroll
  for (int i0 = 0; i0 < G * 16; i0 += 128) {
    const int i = i0 + tid, t = i >> 4, part = i & 15;
    reinterpret_cast<uint4*>(kt)[i] = __ldg(reinterpret_cast<const uint4*>(kg + (int64_t)t * ks.t) + part);
    reinterpret_cast<uint4*>(vt)[i] = __ldg(reinterpret_cast<const uint4*>(vg_ + (int64_t)t * vs.t) + part);
  }
  __syncthreads();
  // ---- keys: per channel over the G tokens of the group ----
  {
    const int d = tid;
    float lo = INFINITY, hi = -INFINITY;
#pragma unroll
    for (int t = 0; t < G; ++t) {
      const float x = to_float<T>(kt[t * D + d]);
      lo = fminf(lo, x);
      hi = fmaxf(hi, x);
    }
    const float scale = fmaxf(__fdiv_rn(__fsub_rn(hi, lo), qmax), 1e-8f);
    const size_t mi = (bh * (c.cap / G) + tok0 / G) * D + kmeta_pos(d, D);
    c.k_scale[mi] = scale;
    c.k_zero[mi] = lo;
    ks_s[d] = scale;
    kp_s[key_pair_slot(d)] = make_float2(lo, __frcp_rn(scale));
  }
  // ---- values: per token over each group of D / VG channels (a warp per token, a lane per four channels) ----
#pragma unroll
  for (int t = warp; t < G; t += 4) {
    const uint2 raw = *reinterpret_cast<const uint2*>(vt + t * D + lane * 4);
    const T* e = reinterpret_cast<const T*>(&raw);
    float lo = fminf(fminf(to_float<T>(e[0]), to_float<T>(e[1])), fminf(to_float<T>(e[2]), to_float<T>(e[3])));
    float hi = fmaxf(fmaxf(to_float<T>(e[0]), to_float<T>(e[1])), fmaxf(to_float<T>(e[2]), to_float<T>(e[3])));
    constexpr int kLanes = 32 / VG;                         // lanes that share a value group
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((lane & (kLanes - 1)) == 0) {
      const float scale = fmaxf(__fdiv_rn(__fsub_rn(hi, lo), qmax), 1e-8f);
      vs_s[t * VG + lane / kLanes] = scale;
      vp_s[t * VG + lane / kLanes] = make_float2(lo, __frcp_rn(scale));
    }
  }
  __syncthreads();
  for (int i = tid; i < G * VG; i += 128) {                 // the group's value scales / zeros: contiguous in the cache
    c.v_scale[(bh * c.cap + tok0) * VG + i] = vs_s[i];
    c.v_zero[(bh * c.cap + tok0) * VG + i] = vp_s[i].x;
  }
  // ---- key codes: 16 bytes (32 or 64 channels) of one token per step ----
  {
    constexpr int CPI = 128 / BITS;                         // channels per 16 bytes of codes
    constexpr int IPT = D / CPI;                            // such pieces per token
    constexpr int CH = CPI / 8;                             // 8-channel chunks per piece
    uint8_t* dst = c.k_codes + (bh * c.cap + tok0) * (size_t)(D * BITS / 8);
#pragma unroll
    for (int i0 = 0; i0 < G * IPT; i0 += 128) {
      const int i = i0 + tid;
      if (G * IPT % 128 != 0 && i >= G * IPT) break;
      const int t = i / IPT, q = i % IPT;
      // the pieces of a quarter warp start at different chunks, so that its 16-byte reads fall in different banks
      const int rot = BITS == 4 ? ((q >> 1) + 2 * (t & 1)) & 3 : 0;
      uint32_t cw[CH];
#pragma unroll
      for (int jj = 0; jj < CH; ++jj) {
        const int c0 = q * CPI + ((jj + rot) & (CH - 1)) * 8;
        const uint4 raw = *reinterpret_cast<const uint4*>(kt + t * D + c0);
        const T* e = reinterpret_cast<const T*>(&raw);
        float x[8], lo[8], in[8], sc[8];
        const float4* pr = reinterpret_cast<const float4*>(kp_s + key_pair_slot(c0));
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          const float4 pv = pr[k >> 1];
          lo[k] = pv.x; in[k] = pv.y; lo[k + 1] = pv.z; in[k + 1] = pv.w;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = to_float<T>(e[k]), sc[k] = ks_s[c0 + k];
        cw[jj] = affine_codes8<BITS>(x, lo, in, sc);
      }
      uint32_t w[4];
      if constexpr (BITS == 4) {   // undo the rotation: chunk j was done at place (j - rot) mod 4
        const bool r1 = rot & 1, r2 = rot & 2;
        uint32_t m[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) m[j] = r1 ? cw[(j + 3) & 3] : cw[j];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = r2 ? m[(j + 2) & 3] : m[j];
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = (cw[2 * j] & 0xffffu) | (cw[2 * j + 1] << 16);
      }
      *reinterpret_cast<uint4*>(dst + (size_t)i * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  // ---- value codes: a thread packs half of the group's tokens of two neighbouring channels into their rows ----
  {
    const int d = (tid & 63) * 2, gi = VG == 1 ? 0 : (d >> 5);
    constexpr int HT = G / 2;                               // tokens per thread
    const int th = (tid >> 6) * HT;
    uint32_t w[2][HT / 8];
#pragma unroll
    for (int t8 = 0; t8 < HT; t8 += 8) {
      float x0[8], x1[8], lo[8], in[8], sc[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int t = th + t8 + k;
        const uint32_t raw = *reinterpret_cast<const uint32_t*>(vt + t * D + d);
        const T* e = reinterpret_cast<const T*>(&raw);
        x0[k] = to_float<T>(e[0]);
        x1[k] = to_float<T>(e[1]);
        const float2 pv = vp_s[t * VG + gi];
        lo[k] = pv.x; in[k] = pv.y;
        sc[k] = vs_s[t * VG + gi];
      }
      w[0][t8 / 8] = affine_codes8<BITS>(x0, lo, in, sc);
      w[1][t8 / 8] = affine_codes8<BITS>(x1, lo, in, sc);
    }
    uint8_t* row = c.v_codes + ((bh * (c.cap / 128) + tok0 / 128) * D + d) * (size_t)(128 * BITS / 8) + (tok0 % 128 + th) * BITS / 8;
#pragma unroll
    for (int e = 0; e < 2; ++e, row += 128 * BITS / 8) {
      constexpr int NB = HT * BITS / 8;                     // bytes: 2, 4, 8 or 16
      if constexpr (BITS == 4) {
        if constexpr (NB == 16) *reinterpret_cast<uint4*>(row) = make_uint4(w[e][0], w[e][1], w[e][2], w[e][3]);
        else if constexpr (NB == 8) *reinterpret_cast<uint2*>(row) = make_uint2(w[e][0], w[e][1]);
        else *reinterpret_cast<uint32_t*>(row) = w[e][0];
      } else {
        if constexpr (NB == 8) *reinterpret_cast<uint2*>(row) = make_uint2((w[e][0] & 0xffffu) | (w[e][1] << 16), (w[e][2] & 0xffffu) | (w[e][3] << 16));
        else if constexpr (NB == 4) *reinterpret_cast<uint32_t*>(row) = (w[e][0] & 0xffffu) | (w[e][1] << 16);
        else *reinterpret_cast<uint16_t*>(row) = (uint16_t)w[e][0];
      }
    }
  }
}

// Element-wise form of the dequantize kernel for any supported geometry (head dims other than 128, 8-bit codes):
// one CTA per (128-token block, head, batch); blockDim.x == D.  Writes tokens [0, n_comp).
template <typename T>
__global__ void kivi_dequant_kernel(CachePtrs c, int n_comp, void* out_k, void* out_v, int64_t ob, int64_t oh, int64_t ot) {
  const int D = c.D, bits = c.bits, G = c.group;
  const int blk = blockIdx.x, h = blockIdx.y, b = blockIdx.z, d = threadIdx.x;
  const size_t bh = (size_t)b * c.H + h;
  const uint32_t mask = (1u << bits) - 1u;
  T* ok = reinterpret_cast<T*>(out_k) + (int64_t)b * ob + (int64_t)h * oh;
  T* ov = reinterpret_cast<T*>(out_v) + (int64_t)b * ob + (int64_t)h * oh;
  const int t_end = min(n_comp, (blk + 1) * 128);
  const int k_row_bytes = D * bits / 8, v_row_bytes = 128 * bits / 8;
  const uint8_t* vrow = c.v_codes + ((bh * (c.cap / 128) + blk) * D + d) * (size_t)v_row_bytes;
  for (int t = blk * 128; t < t_end; ++t) {
    const uint8_t kb = c.k_codes[(bh * c.cap + t) * (size_t)k_row_bytes + (d * bits >> 3)];
    const float kq = (float)((kb >> ((d * bits) & 7)) & mask);
    const size_t mi = (bh * (c.cap / G) + t / G) * D + kmeta_pos(d, D);
    ok[(int64_t)t * ot + d] = from_float<T>(__fadd_rn(__fmul_rn(kq, c.k_scale[mi]), c.k_zero[mi]));
    const int tl = t & 127;
    const uint8_t vb = vrow[tl * bits >> 3];
    const float vq = (float)((vb >> ((tl * bits) & 7)) & mask);
    const size_t vi = (bh * c.cap + t) * (D / c.v_group) + d / c.v_group;
    ov[(int64_t)t * ot + d] = from_float<T>(__fadd_rn(__fmul_rn(vq, c.v_scale[vi]), c.v_zero[vi]));
  }
}

// Eight dequantized values (code * scale + zero, separately rounded product and sum) as one 16-byte vector of T, or two of
// them for T = float; called by all lanes of a half warp, whose pieces of a row are neighbours.  Two lanes swap halves of their 32 bytes
// for T = float, so that every store fills 32-byte sectors (4 x 4 x 4096 tokens, 4 bits: 23.1 us with half sectors, 14.7 so).
template <typename T>
__device__ __forceinline__ void store8(T* dst, const float (&v)[8]) {
  if constexpr (sizeof(T) == 2) {
    uint4 o;
    T* e = reinterpret_cast<T*>(&o);
#pragma unroll
    for (int j = 0; j < 8; ++j) e[j] = from_float<T>(v[j]);
    *reinterpret_cast<uint4*>(dst) = o;
  } else {
    const bool odd = threadIdx.x & 1;
    const unsigned half = 0xffffu << (threadIdx.x & 16);
    float got[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) got[i] = __shfl_xor_sync(half, odd ? v[i] : v[4 + i], 1);
    const float4 mine = odd ? make_float4(v[4], v[5], v[6], v[7]) : make_float4(v[0], v[1], v[2], v[3]);
    const float4 theirs = make_float4(got[0], got[1], got[2], got[3]);
    T* const first = odd ? dst - 4 : dst;
    *reinterpret_cast<float4*>(first) = odd ? theirs : mine;
    *reinterpret_cast<float4*>(first + 8) = odd ? mine : theirs;
  }
}

// (2^23 + q 2^p) - 2^23 for two codes at once (exact), then times scale plus zero, each rounded separately.  Product and
// sum are scalar on purpose: the compiler contracts a packed multiply and add into one fused operation.
__device__ __forceinline__ void affine_pair(float& a, float& b, float s0, float s1, float z0, float z1) {
  asm("{\n\t.reg .b64 x, m;\n\t"
      "mov.b64 x, {%0, %1};\n\t"
      "mov.b64 m, {%2, %2};\n\t"
      "add.rn.f32x2 x, x, m;\n\t"
      "mov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a), "+f"(b)
      : "f"(-8388608.f));
  a = __fadd_rn(__fmul_rn(a, s0), z0);
  b = __fadd_rn(__fmul_rn(b, s1), z1);
}

// What update() returns beside the reconstructed tokens: the full-precision window, and tokens that are only now arriving
struct WindowArgs {
  void* res_k;              // [B][H][..][128] window, n_old tokens of it in use
  void* res_v;
  const void* new_k;        // n_new tokens that are copied into the window and the result on the way
  const void* new_v;
  SrcStrides r, nk, nv;
  int n_old, n_new;
};

// Vectorised dequantize for the attention geometry (D == 128, 2- or 4-bit codes, 16-byte aligned output rows): one
// CTA of 256 threads per (128-token block, head, batch).  The block's codes and metadata (about 21 KB) come in with
// 16-byte loads into shared memory; a thread then produces EIGHT TOKENS of eight consecutive channels: one code word per
// token (keys) or channel (values) and the keys' scales and zeros in registers for all eight, sixteen 16-byte stores,
// a token's 256 output bytes contiguous across 16 threads.  (One token at a time took a shared-memory byte read per
// value code and an integer-to-float conversion per element: 0.44 - 0.51 of the HBM rate.)  A code left in place at bit p
// of a float's mantissa under the exponent of 2^23 is 2^23 + code * 2^p; taking 2^23 off is exact, and the 2^p goes into
// the scale, which a power of two leaves exact: the product rounds like code * scale.
// CTAs beyond the compressed blocks copy 128 tokens of the window each (WindowArgs).
template <typename T, int BITS, int VG>
__global__ void __launch_bounds__(256) kivi_dequant128_kernel(CachePtrs c, int n_comp, int n_blocks, void* out_k, void* out_v, int64_t ob,
                                                               int64_t oh, int64_t ot, const WindowArgs win) {
  constexpr int D = 128, KROW = D * BITS / 8, VROW = 128 * BITS / 8;
  extern __shared__ __align__(16) unsigned char sm[];
  const int G = c.group, ngr = 128 / G;
  const int blk = blockIdx.x, h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x;
  T* okp = reinterpret_cast<T*>(out_k) + (int64_t)b * ob + (int64_t)h * oh;
  T* ovp = reinterpret_cast<T*>(out_v) + (int64_t)b * ob + (int64_t)h * oh;
  if (blk >= n_blocks) {
    constexpr int kVec = 16 / (int)sizeof(T), kPer = D / kVec;   // 16-byte pieces per row
    const int w0 = (blk - n_blocks) * 128, n = min(128, win.n_old + win.n_new - w0);
    T* rk = reinterpret_cast<T*>(win.res_k) + (int64_t)b * win.r.b + (int64_t)h * win.r.h;
    T* rv = reinterpret_cast<T*>(win.res_v) + (int64_t)b * win.r.b + (int64_t)h * win.r.h;
    const T* nk = reinterpret_cast<const T*>(win.new_k) + (int64_t)b * win.nk.b + (int64_t)h * win.nk.h;
    const T* nv = reinterpret_cast<const T*>(win.new_v) + (int64_t)b * win.nv.b + (int64_t)h * win.nv.h;
    for (int i = tid; i < n * kPer; i += 256) {
      const int t = w0 + i / kPer, at = (i % kPer) * kVec;
      const bool fresh = t >= win.n_old;
      const uint4 kq = *reinterpret_cast<const uint4*>(fresh ? nk + (int64_t)(t - win.n_old) * win.nk.t + at : rk + (int64_t)t * win.r.t + at);
      const uint4 vq = *reinterpret_cast<const uint4*>(fresh ? nv + (int64_t)(t - win.n_old) * win.nv.t + at : rv + (int64_t)t * win.r.t + at);
      *reinterpret_cast<uint4*>(okp + (int64_t)(n_comp + t) * ot + at) = kq;
      *reinterpret_cast<uint4*>(ovp + (int64_t)(n_comp + t) * ot + at) = vq;
      if (fresh) {
        *reinterpret_cast<uint4*>(rk + (int64_t)t * win.r.t + at) = kq;
        *reinterpret_cast<uint4*>(rv + (int64_t)t * win.r.t + at) = vq;
      }
    }
    return;
  }
  // rows of eight tokens (keys) / channels (values) are skewed so that a warp's word reads fall in different banks
  constexpr int KSKEW = KROW, VSKEW = 8;
  unsigned char* kc = sm;                                              // [128][KROW], + KSKEW every 8 rows
  unsigned char* vc = kc + 128 * KROW + 16 * KSKEW;                    // [D][VROW], + VSKEW every 8 rows
  float* ks = reinterpret_cast<float*>(vc + D * VROW + 16 * VSKEW);    // [ngr][D] in kmeta_pos order
  float* kz = ks + ngr * D;
  float* vs = kz + ngr * D;                                            // [128][VG]
  float* vz = vs + 128 * VG;
  const size_t bh = (size_t)b * c.H + h;
  const int t0 = blk * 128, valid = min(128, n_comp - t0);             // a multiple of G
  const int vgroups = valid / G;
  {
    const uint4* src = reinterpret_cast<const uint4*>(c.k_codes + (bh * c.cap + t0) * (size_t)KROW);
    for (int i = tid; i < valid * KROW / 16; i += 256) {
      const int row = i / (KROW / 16);
      *reinterpret_cast<uint4*>(kc + i * 16 + (row >> 3) * KSKEW) = __ldg(src + i);
    }
    const uint4* vsrc = reinterpret_cast<const uint4*>(c.v_codes + (bh * (c.cap / 128) + blk) * (size_t)(D * VROW));
    for (int i = tid; i < D * VROW / 16; i += 256) {
      const uint4 v = __ldg(vsrc + i);
      const int row = i / (VROW / 16);
      uint2* dst = reinterpret_cast<uint2*>(vc + i * 16 + (row >> 3) * VSKEW);   // 8-byte aligned
      dst[0] = make_uint2(v.x, v.y);
      dst[1] = make_uint2(v.z, v.w);
    }
    const size_t grow = (bh * (c.cap / G) + t0 / G) * D;
    for (int i = tid; i < vgroups * D / 4; i += 256) {
      reinterpret_cast<float4*>(ks)[i] = __ldg(reinterpret_cast<const float4*>(c.k_scale + grow) + i);
      reinterpret_cast<float4*>(kz)[i] = __ldg(reinterpret_cast<const float4*>(c.k_zero + grow) + i);
    }
    const size_t vrow0 = (bh * c.cap + t0) * VG;
    for (int i = tid; i < valid * VG / 4; i += 256) {
      reinterpret_cast<float4*>(vs)[i] = __ldg(reinterpret_cast<const float4*>(c.v_scale + vrow0) + i);
      reinterpret_cast<float4*>(vz)[i] = __ldg(reinterpret_cast<const float4*>(c.v_zero + vrow0) + i);
    }
  }
  __syncthreads();
  const int tg = tid >> 4, r = tid & 15, c8 = r * 8, tl = tg * 8;      // tokens tl .. tl + 7 (one group: groups are multiples of 16)
  if (tl >= valid) return;
  constexpr uint32_t kMagic = 0x4B000000u;
  // code j of a word as 2^23 + code * 2^(shift_of(j)); 4-bit words are read in two halves
  auto place = [](uint32_t w, int j) -> float {
    if constexpr (BITS == 4) return __uint_as_float(and_or(j < 4 ? w : w >> 16, 0xFu << (4 * (j & 3)), kMagic));
    else return __uint_as_float(and_or(w, 0x3u << (2 * j), kMagic));
  };
  auto unit = [](int j) -> float {   // 2^-shift_of(j)
    return __int_as_float((127 - (BITS == 4 ? 4 * (j & 3) : 2 * j)) << 23);
  };
  {  // ---- keys ----
    const int mp = (tl / G) * D + kmeta_pos(c8, D);          // the eight channels of a run are adjacent in the stored order
    const float4 s0 = *reinterpret_cast<const float4*>(ks + mp), s1 = *reinterpret_cast<const float4*>(ks + mp + 4);
    const float4 z0 = *reinterpret_cast<const float4*>(kz + mp), z1 = *reinterpret_cast<const float4*>(kz + mp + 4);
    float sv[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    const float zv[8] = {z0.x, z0.y, z0.z, z0.w, z1.x, z1.y, z1.z, z1.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) sv[j] *= unit(j);
    T* dst = okp + (int64_t)(t0 + tl) * ot + c8;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const unsigned char* at = kc + (tl + t) * KROW + tg * KSKEW + r * BITS;
      const uint32_t w = BITS == 4 ? *reinterpret_cast<const uint32_t*>(at) : *reinterpret_cast<const uint16_t*>(at);
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = place(w, j);
#pragma unroll
      for (int j = 0; j < 8; j += 2) affine_pair(v[j], v[j + 1], sv[j], sv[j + 1], zv[j], zv[j + 1]);
      store8<T>(dst + (int64_t)t * ot, v);
    }
  }
  {  // ---- values: word j holds the eight tokens of channel c8 + j ----
    const int vgi = VG == 1 ? 0 : (c8 >> 5);
    uint32_t w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const unsigned char* at = vc + (c8 + j) * VROW + r * VSKEW + tg * BITS;
      w[j] = BITS == 4 ? *reinterpret_cast<const uint32_t*>(at) : *reinterpret_cast<const uint16_t*>(at);
    }
    T* dst = ovp + (int64_t)(t0 + tl) * ot + c8;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const float s = vs[(tl + t) * VG + vgi] * unit(t), z = vz[(tl + t) * VG + vgi];
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = place(w[j], t);
#pragma unroll
      for (int j = 0; j < 8; j += 2) affine_pair(v[j], v[j + 1], s, s, z, z);
      store8<T>(dst + (int64_t)t * ot, v);
    }
  }
}

int check_cache(const CachePtrs& c) {
  PARE_REQUIRE(c.B > 0 && c.H > 0 && c.D > 0 && c.cap > 0, PARE_ERR_SHAPE);
  PARE_REQUIRE(c.D % 32 == 0 && c.D <= 256, PARE_ERR_UNSUPPORTED);
  PARE_REQUIRE(c.bits == 2 || c.bits == 4 || c.bits == 8, PARE_ERR_UNSUPPORTED);
  PARE_REQUIRE(c.group == 16 || c.group == 32 || c.group == 64 || c.group == 128, PARE_ERR_UNSUPPORTED);
  PARE_REQUIRE(c.cap % 128 == 0, PARE_ERR_SHAPE);
  PARE_REQUIRE(c.v_group > 0 && c.v_group % 32 == 0 && c.D % c.v_group == 0, PARE_ERR_UNSUPPORTED);
  PARE_REQUIRE(c.k_codes && c.k_scale && c.k_zero && c.v_codes && c.v_scale && c.v_zero, PARE_ERR_SHAPE);
  return PARE_OK;
}

}  // namespace
}  // namespace pare

using pare::CachePtrs;

extern "C" {

int pare_kivi_append_kv(const void* k_src, const void* v_src, int src_dtype, int64_t k_stride_b, int64_t k_stride_h, int64_t k_stride_t,
                        int64_t v_stride_b, int64_t v_stride_h, int64_t v_stride_t, int n_tokens, int t0, uint8_t* k_codes,
                        float* k_scale, float* k_zero, uint8_t* v_codes, float* v_scale, float* v_zero, int B, int H, int D, int bits,
                        int group, int v_group, int cap, void* stream) {
  CachePtrs c{k_codes, k_scale, k_zero, v_codes, v_scale, v_zero, B, H, D, bits, group, cap, v_group > 0 ? v_group : D};
  const int rc = pare::check_cache(c);
  if (rc != PARE_OK) return rc;
  PARE_REQUIRE(k_src && v_src && n_tokens > 0, PARE_ERR_SHAPE);
  PARE_REQUIRE(n_tokens % group == 0 && t0 >= 0 && t0 % group == 0 && t0 + n_tokens <= cap, PARE_ERR_SHAPE);
  const dim3 grid(n_tokens / group, H, B);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const pare::SrcStrides ks{k_stride_b, k_stride_h, k_stride_t}, vst{v_stride_b, v_stride_h, v_stride_t};
  const int vg = D / c.v_group;
  bool vec = true;
  for (int64_t st : {k_stride_b, k_stride_h, k_stride_t, v_stride_b, v_stride_h, v_stride_t}) vec = vec && st % 8 == 0;
  if (vec && D == 128 && (bits == 2 || bits == 4) && (vg == 1 || vg == 4) && group <= 64 && (src_dtype == PARE_F16 || src_dtype == PARE_BF16) &&
      pare::aligned16(k_src) && pare::aligned16(v_src) && pare::aligned16(k_codes) && pare::aligned16(v_codes)) {
    const size_t smem = (size_t)2 * group * 128 * 2 + pare::kKeyPairs * sizeof(float2) + 128 * sizeof(float) + 3 * (size_t)group * vg * sizeof(float);
    auto launch = [&](auto t_tag, auto bits_tag, auto vg_tag) -> int {
      using T = decltype(t_tag);
      constexpr int BITS = decltype(bits_tag)::value, VG = decltype(vg_tag)::value;
      if (group == 16) pare::kivi_append128_kernel<T, BITS, VG, 16><<<grid, 128, smem, s>>>(k_src, v_src, ks, vst, t0, c);
      else if (group == 32) pare::kivi_append128_kernel<T, BITS, VG, 32><<<grid, 128, smem, s>>>(k_src, v_src, ks, vst, t0, c);
      else pare::kivi_append128_kernel<T, BITS, VG, 64><<<grid, 128, smem, s>>>(k_src, v_src, ks, vst, t0, c);
      return pare::launch_status();
    };
    using std::integral_constant;
    auto pick = [&](auto t_tag) -> int {
      if (bits == 4) return vg == 1 ? launch(t_tag, integral_constant<int, 4>{}, integral_constant<int, 1>{}) : launch(t_tag, integral_constant<int, 4>{}, integral_constant<int, 4>{});
      return vg == 1 ? launch(t_tag, integral_constant<int, 2>{}, integral_constant<int, 1>{}) : launch(t_tag, integral_constant<int, 2>{}, integral_constant<int, 4>{});
    };
    return src_dtype == PARE_F16 ? pick(__half{}) : pick(__nv_bfloat16{});
  }
  const size_t smem = (size_t)group * D + 2 * group * (D / c.v_group) * sizeof(float);
  switch (src_dtype) {
    case PARE_F16:
      pare::kivi_append_kernel<__half><<<grid, D, smem, s>>>(k_src, v_src, ks, vst, t0, c);
      break;
    case PARE_BF16:
      pare::kivi_append_kernel<__nv_bfloat16><<<grid, D, smem, s>>>(k_src, v_src, ks, vst, t0, c);
      break;
    case PARE_F32:
      pare::kivi_append_kernel<float><<<grid, D, smem, s>>>(k_src, v_src, ks, vst, t0, c);
      break;
    default:
      return PARE_ERR_DTYPE;
  }
  return pare::launch_status();
}

int pare_kivi_append(const void* k_src, const void* v_src, int src_dtype, int64_t stride_b, int64_t stride_h,
                     int64_t stride_t, int n_tokens, int t0, uint8_t* k_codes, float* k_scale, float* k_zero,
                     uint8_t* v_codes, float* v_scale, float* v_zero, int B, int H, int D, int bits, int group, int v_group,
                     int cap, void* stream) {
  return pare_kivi_append_kv(k_src, v_src, src_dtype, stride_b, stride_h, stride_t, stride_b, stride_h, stride_t, n_tokens, t0, k_codes,
                             k_scale, k_zero, v_codes, v_scale, v_zero, B, H, D, bits, group, v_group, cap, stream);
}

static int dequant128(const CachePtrs& c, int n_comp, void* out_k, void* out_v, int out_dtype, int64_t stride_b, int64_t stride_h,
                      int64_t stride_t, const pare::WindowArgs& win, void* stream) {
  const int vg = c.D / c.v_group, bits = c.bits;
  const size_t esz = out_dtype == PARE_F32 ? 4 : 2;
  const bool fast = c.D == 128 && (bits == 2 || bits == 4) && (vg == 1 || vg == 4) && pare::aligned16(out_k) && pare::aligned16(out_v) &&
                    (stride_b * esz) % 16 == 0 && (stride_h * esz) % 16 == 0 && (stride_t * esz) % 16 == 0 &&
                    pare::aligned16(c.k_codes) && pare::aligned16(c.v_codes) && pare::aligned16(c.k_scale) && pare::aligned16(c.k_zero) &&
                    pare::aligned16(c.v_scale) && pare::aligned16(c.v_zero);
  if (!fast) return PARE_ERR_UNSUPPORTED;
  const int n_blocks = (n_comp + 127) / 128;
  const dim3 grid(n_blocks + (win.n_old + win.n_new + 127) / 128, c.H, c.B);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const size_t row = 128 * bits / 8;
  const size_t smem = 128 * row + 16 * row + 128 * row + 16 * 8 + 2 * (size_t)(128 / c.group) * 128 * 4 + 2 * (size_t)128 * vg * 4;
  auto launch = [&](auto kern) -> int {
    if (smem > 48 * 1024 && !pare::ensure_smem_attr(reinterpret_cast<const void*>(kern), 64 * 1024)) return PARE_ERR_CUDA;
    kern<<<grid, 256, smem, s>>>(c, n_comp, n_blocks, out_k, out_v, stride_b, stride_h, stride_t, win);
    return pare::launch_status();
  };
#define PARE_DQ(T)                                                                                        \
  (bits == 4 ? (vg == 1 ? launch(pare::kivi_dequant128_kernel<T, 4, 1>) : launch(pare::kivi_dequant128_kernel<T, 4, 4>)) \
             : (vg == 1 ? launch(pare::kivi_dequant128_kernel<T, 2, 1>) : launch(pare::kivi_dequant128_kernel<T, 2, 4>)))
  switch (out_dtype) {
    case PARE_F16: return PARE_DQ(__half);
    case PARE_BF16: return PARE_DQ(__nv_bfloat16);
    case PARE_F32: return PARE_DQ(float);
    default: return PARE_ERR_DTYPE;
  }
#undef PARE_DQ
}

int pare_kivi_dense(const uint8_t* k_codes, const float* k_scale, const float* k_zero, const uint8_t* v_codes, const float* v_scale,
                    const float* v_zero, int B, int H, int D, int bits, int group, int v_group, int cap, int n_comp, void* out_k,
                    void* out_v, int dtype, int64_t out_stride_b, int64_t out_stride_h, int64_t out_stride_t, void* res_k, void* res_v,
                    int64_t res_stride_b, int64_t res_stride_h, int64_t res_stride_t, int n_res, const void* new_k, const void* new_v,
                    int64_t new_k_stride_b, int64_t new_k_stride_h, int64_t new_k_stride_t, int64_t new_v_stride_b,
                    int64_t new_v_stride_h, int64_t new_v_stride_t, int n_new, void* stream) {
  CachePtrs c{const_cast<uint8_t*>(k_codes), const_cast<float*>(k_scale), const_cast<float*>(k_zero),
              const_cast<uint8_t*>(v_codes), const_cast<float*>(v_scale), const_cast<float*>(v_zero),
              B, H, D, bits, group, cap, v_group > 0 ? v_group : D};
  const int rc = pare::check_cache(c);
  if (rc != PARE_OK) return rc;
  PARE_REQUIRE(out_k && out_v && n_comp >= 0 && n_comp <= cap && n_comp % group == 0 && n_res >= 0 && n_new >= 0, PARE_ERR_SHAPE);
  PARE_REQUIRE(n_res + n_new == 0 || (res_k && res_v), PARE_ERR_SHAPE);
  PARE_REQUIRE(n_new == 0 || (new_k && new_v), PARE_ERR_SHAPE);
  PARE_REQUIRE(B <= 65535 && H <= 65535, PARE_ERR_UNSUPPORTED);   // the launch grid
  if (n_comp + n_res + n_new == 0) return PARE_OK;
  const size_t esz = dtype == PARE_F32 ? 4 : 2;
  for (int64_t st : {res_stride_b, res_stride_h, res_stride_t, new_k_stride_b, new_k_stride_h, new_k_stride_t, new_v_stride_b,
                     new_v_stride_h, new_v_stride_t})
    PARE_REQUIRE((st * (int64_t)esz) % 16 == 0, PARE_ERR_UNSUPPORTED);
  PARE_REQUIRE(pare::aligned16(res_k) && pare::aligned16(res_v) && pare::aligned16(new_k) && pare::aligned16(new_v), PARE_ERR_UNSUPPORTED);
  const pare::WindowArgs win{res_k, res_v, new_k, new_v, {res_stride_b, res_stride_h, res_stride_t},
                             {new_k_stride_b, new_k_stride_h, new_k_stride_t}, {new_v_stride_b, new_v_stride_h, new_v_stride_t}, n_res, n_new};
  return dequant128(c, n_comp, out_k, out_v, dtype, out_stride_b, out_stride_h, out_stride_t, win, stream);
}

int pare_kivi_dequant(const uint8_t* k_codes, const float* k_scale, const float* k_zero, const uint8_t* v_codes,
                      const float* v_scale, const float* v_zero, int B, int H, int D, int bits, int group, int v_group,
                      int cap, int n_comp, void* out_k, void* out_v, int out_dtype, int64_t stride_b, int64_t stride_h,
                      int64_t stride_t, void* stream) {
  CachePtrs c{const_cast<uint8_t*>(k_codes), const_cast<float*>(k_scale), const_cast<float*>(k_zero),
              const_cast<uint8_t*>(v_codes), const_cast<float*>(v_scale), const_cast<float*>(v_zero),
              B, H, D, bits, group, cap, v_group > 0 ? v_group : D};
  const int rc = pare::check_cache(c);
  if (rc != PARE_OK) return rc;
  PARE_REQUIRE(out_k && out_v && n_comp >= 0 && n_comp <= cap && n_comp % group == 0, PARE_ERR_SHAPE);
  if (n_comp == 0) return PARE_OK;
  const int fast = dequant128(c, n_comp, out_k, out_v, out_dtype, stride_b, stride_h, stride_t, pare::WindowArgs{}, stream);
  if (fast != PARE_ERR_UNSUPPORTED) return fast;
  const dim3 grid((n_comp + 127) / 128, H, B);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  switch (out_dtype) {
    case PARE_F16:
      pare::kivi_dequant_kernel<__half><<<grid, D, 0, s>>>(c, n_comp, out_k, out_v, stride_b, stride_h, stride_t);
      break;
    case PARE_BF16:
      pare::kivi_dequant_kernel<__nv_bfloat16><<<grid, D, 0, s>>>(c, n_comp, out_k, out_v, stride_b, stride_h, stride_t);
      break;
    case PARE_F32:
      pare::kivi_dequant_kernel<float><<<grid, D, 0, s>>>(c, n_comp, out_k, out_v, stride_b, stride_h, stride_t);
      break;
    default:
      return PARE_ERR_DTYPE;
  }
  return pare::launch_status();
}

}  // extern "C"
