// Prefill attention over full-precision K / V (fp16 / bf16), sm_100a: the attention of a prompt's tokens
// before the cache compresses them.  The reference leaves this to its caller
// (scaled_dot_product_attention on update()'s return, pare/kv_cache.py:183-186, 205-252); for a prompt
// that return is mostly a lossy reconstruction, so this kernel attends to the tokens as they were given.
//
//   out[b][hq][i][:] = softmax_j(q[b][hq][i] . k[b][hq / rep][j] * scale) . v[b][hq / rep][j]
//   causal: key j is visible to query i iff j <= i + (Tk - Tq)   (the queries are the newest Tq tokens)
//
// Two kernels: tensor-memory tiles of 128 queries x 128 keys (further down) and, for very short prompts and what those do not
// take, warp-level tiles of 64 x 64:
// One CTA per (64-query tile, query head, batch), four warps of 16 query rows.  K / V stream through shared
// memory in 64-key tiles, two buffers, cp.async; S = Q K^T and O += P V on warp-level tensor-core steps
// (m16n8k16, fp32 accumulate) with ldmatrix operand loads; softmax statistics online in registers, so the
// score matrix never exists.  head_dim 128.
#include <limits.h>

#include "tcgen05.cuh"

namespace pare {
namespace {

constexpr int kPD = 128;                 // head_dim
constexpr int kPQ = 64;                  // query rows per CTA
constexpr int kPK = 64;                  // keys per tile
constexpr int kPWarps = 4;
constexpr int kPThreads = kPWarps * 32;
constexpr int kPPitch = kPD * 2 + 16;    // bytes per staged row: 16-byte skew keeps ldmatrix conflict-free
constexpr size_t kPSmem = (size_t)(kPQ + 4 * kPK) * kPPitch;   // Q tile + two (K, V) buffers

struct PrefillParams {
  const void* q;
  const void* k;
  const void* v;
  void* out;
  int64_t q_sb, q_sh, q_st;
  int64_t k_sb, k_sh, k_st;
  int64_t v_sb, v_sh, v_st;
  int64_t o_sb, o_sh, o_st;
  int B, Hq, H, rep, Tq, Tk;
  float scale_log2;    // softmax scale * log2(e)
  int causal;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool pred) {
  const int n = pred ? 16 : 0;   // zero-fill rows beyond the sequence
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

template <typename T>
__device__ __forceinline__ uint32_t pack2(float a, float b);
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// 16-bit pair of (a, b) minus what the pair `packed` already holds: the second term of a two-term expansion
template <typename T>
__device__ __forceinline__ uint32_t residual2(float a, float b, uint32_t packed);
template <>
__device__ __forceinline__ uint32_t residual2<__nv_bfloat16>(float a, float b, uint32_t packed) {
  return pack2<__nv_bfloat16>(a - __uint_as_float(packed << 16), b - __uint_as_float(packed & 0xffff0000u));
}
template <>
__device__ __forceinline__ uint32_t residual2<__half>(float a, float b, uint32_t packed) {
  const __half2 h = *reinterpret_cast<const __half2*>(&packed);
  return pack2<__half>(a - __low2float(h), b - __high2float(h));
}

// rows [row0, row0 + rows) of a [T][128] tensor (row stride st elements) into a staged tile; rows >= T are zeros
template <typename T>
__device__ __forceinline__ void stage_rows(uint32_t dst, const T* src, int64_t st, int row0, int rows, int T_total) {
  for (int i = threadIdx.x; i < rows * (kPD / 8); i += kPThreads) {
    const int r = i >> 4, c = i & 15;
    const bool ok = row0 + r < T_total;
    cp_async16(dst + r * kPPitch + c * 16, src + (int64_t)(ok ? row0 + r : 0) * st + c * 8, ok);
  }
}

template <typename T>
__global__ void __launch_bounds__(kPThreads) prefill_attn_kernel(const PrefillParams p) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int qt = gridDim.x - 1 - blockIdx.x;   // the longest (latest) query tiles start first
  const int hq = blockIdx.y, b = blockIdx.z, h = hq / p.rep;
  const T* qg = reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_sb + (int64_t)hq * p.q_sh;
  const T* kg = reinterpret_cast<const T*>(p.k) + (int64_t)b * p.k_sb + (int64_t)h * p.k_sh;
  const T* vg = reinterpret_cast<const T*>(p.v) + (int64_t)b * p.v_sb + (int64_t)h * p.v_sh;
  T* og = reinterpret_cast<T*>(p.out) + (int64_t)b * p.o_sb + (int64_t)hq * p.o_sh;
  const int q0 = qt * kPQ;
  const int off = p.Tk - p.Tq;                                   // key index of query 0's own token
  const int k_end = p.causal ? min(p.Tk, q0 + kPQ + off) : p.Tk;  // keys [0, k_end) can be visible to this tile
  const int n_tiles = (k_end + kPK - 1) / kPK;

  const uint32_t qs = (uint32_t)__cvta_generic_to_shared(smem);
  auto kbuf = [&](int buf) { return qs + (kPQ + buf * 2 * kPK) * kPPitch; };
  auto vbuf = [&](int buf) { return kbuf(buf) + kPK * kPPitch; };

  stage_rows<T>(qs, qg, p.q_st, q0, kPQ, p.Tq);
  stage_rows<T>(kbuf(0), kg, p.k_st, 0, kPK, p.Tk);
  stage_rows<T>(vbuf(0), vg, p.v_st, 0, kPK, p.Tk);
  cp_async_commit();

  uint32_t qf[kPD / 16][4];
  float o[kPD / 8][4];
#pragma unroll
  for (int ct = 0; ct < kPD / 8; ++ct)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[ct][e] = 0.f;
  float m_i[2] = {-INFINITY, -INFINITY}, l_i[2] = {0.f, 0.f};   // rows gid and gid + 8 of this warp's 16
  const int row_lo = q0 + warp * 16 + gid;                      // query index of the first of them

  int buf = 0;
  for (int t = 0; t < n_tiles; ++t) {
    cp_async_wait<0>();
    __syncthreads();   // tile t is in shared memory, and every warp has finished with the other buffer
    if (t + 1 < n_tiles) {
      stage_rows<T>(kbuf(buf ^ 1), kg, p.k_st, (t + 1) * kPK, kPK, p.Tk);
      stage_rows<T>(vbuf(buf ^ 1), vg, p.v_st, (t + 1) * kPK, kPK, p.Tk);
      cp_async_commit();
    }
    if (t == 0) {
#pragma unroll
      for (int ks = 0; ks < kPD / 16; ++ks)
        ldsm_x4(qf[ks], qs + (warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * kPPitch + (ks * 16 + (lane >> 4) * 8) * 2);
    }

    // ---- S = Q K^T for 16 query rows x 64 keys ----
    float s[kPK / 8][4];
#pragma unroll
    for (int nt = 0; nt < kPK / 8; ++nt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) s[nt][e] = 0.f;
#pragma unroll
      for (int ks = 0; ks < kPD / 16; ks += 2) {
        uint32_t kb[4];
        ldsm_x4(kb, kbuf(buf) + (nt * 8 + (lane & 7)) * kPPitch + (ks * 16 + (lane >> 3) * 8) * 2);
        mma16816<T>(s[nt], qf[ks][0], qf[ks][1], qf[ks][2], qf[ks][3], kb[0], kb[1]);
        mma16816<T>(s[nt], qf[ks + 1][0], qf[ks + 1][1], qf[ks + 1][2], qf[ks + 1][3], kb[2], kb[3]);
      }
    }

    // ---- scale, mask, online softmax ----
    const int key0 = t * kPK;
    const bool need_mask = key0 + kPK > p.Tk || (p.causal && key0 + kPK - 1 > q0 + warp * 16 + off);
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int nt = 0; nt < kPK / 8; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float x = s[nt][e] * p.scale_log2;
        if (need_mask) {
          const int key = key0 + nt * 8 + tig * 2 + (e & 1);
          const int row = row_lo + (e >> 1) * 8;
          if (key >= p.Tk || (p.causal && key > row + off)) x = -INFINITY;
        }
        s[nt][e] = x;
        mx[e >> 1] = fmaxf(mx[e >> 1], x);
      }
    float alpha[2], m_use[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
      const float m_new = fmaxf(m_i[r], mx[r]);
      m_use[r] = m_new == -INFINITY ? 0.f : m_new;      // a row with nothing visible yet
      alpha[r] = exp2f(m_i[r] - m_use[r]);              // exp2(-inf) = 0 on the first tile
      m_i[r] = m_new;
      l_i[r] *= alpha[r];
    }
#pragma unroll
    for (int nt = 0; nt < kPK / 8; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float pe = exp2f(s[nt][e] - m_use[e >> 1]);
        s[nt][e] = pe;
        l_i[e >> 1] += pe;
      }
#pragma unroll
    for (int ct = 0; ct < kPD / 8; ++ct) {
      o[ct][0] *= alpha[0]; o[ct][1] *= alpha[0];
      o[ct][2] *= alpha[1]; o[ct][3] *= alpha[1];
    }

    // ---- O += P V ----
#pragma unroll
    for (int kk = 0; kk < kPK / 16; ++kk) {
      const uint32_t a0 = pack2<T>(s[2 * kk][0], s[2 * kk][1]), a1 = pack2<T>(s[2 * kk][2], s[2 * kk][3]);
      const uint32_t a2 = pack2<T>(s[2 * kk + 1][0], s[2 * kk + 1][1]), a3 = pack2<T>(s[2 * kk + 1][2], s[2 * kk + 1][3]);
      // a 16-bit probability keeps 8 (bf16) or 11 (fp16) bits; where the output is small by cancellation that shows.
      // A second operand with the rounding residuals keeps P.V at fp32-level accuracy.
      const uint32_t r0 = residual2<T>(s[2 * kk][0], s[2 * kk][1], a0), r1 = residual2<T>(s[2 * kk][2], s[2 * kk][3], a1);
      const uint32_t r2 = residual2<T>(s[2 * kk + 1][0], s[2 * kk + 1][1], a2), r3 = residual2<T>(s[2 * kk + 1][2], s[2 * kk + 1][3], a3);
#pragma unroll
      for (int ct = 0; ct < kPD / 8; ct += 2) {
        uint32_t vb[4];
        ldsm_x4_trans(vb, vbuf(buf) + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * kPPitch + (ct * 8 + (lane >> 4) * 8) * 2);
        mma16816<T>(o[ct], a0, a1, a2, a3, vb[0], vb[1]);
        mma16816<T>(o[ct + 1], a0, a1, a2, a3, vb[2], vb[3]);
        mma16816<T>(o[ct], r0, r1, r2, r3, vb[0], vb[1]);
        mma16816<T>(o[ct + 1], r0, r1, r2, r3, vb[2], vb[3]);
      }
    }
    buf ^= 1;
  }

  // ---- normalise and store ----
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    l_i[r] += __shfl_xor_sync(0xffffffffu, l_i[r], 1);
    l_i[r] += __shfl_xor_sync(0xffffffffu, l_i[r], 2);
  }
  const float inv0 = l_i[0] > 0.f ? 1.f / l_i[0] : 0.f, inv1 = l_i[1] > 0.f ? 1.f / l_i[1] : 0.f;
#pragma unroll
  for (int ct = 0; ct < kPD / 8; ++ct) {
    const int col = ct * 8 + tig * 2;
    if (row_lo < p.Tq) *reinterpret_cast<uint32_t*>(og + (int64_t)row_lo * p.o_st + col) = pack2<T>(o[ct][0] * inv0, o[ct][1] * inv0);
    if (row_lo + 8 < p.Tq)
      *reinterpret_cast<uint32_t*>(og + (int64_t)(row_lo + 8) * p.o_st + col) = pack2<T>(o[ct][2] * inv1, o[ct][3] * inv1);
  }
}

// ---- tensor-memory path -------------------------------------------------------------------------------------------------
// One CTA works on two 128-query tiles ("halves") of one KV head: two query heads that share the KV head at the same
// tokens, or -- where the heads per KV head are odd -- also the last head at two neighbouring tiles.  K and V tiles of 128 keys come by
// TMA once for both.  Per half and key tile
//     S = Q K^T        tcgen05.mma, both operands in shared memory, 128 x 128 fp32 in tensor memory
//     P = exp2(S - m)  four warps, a thread per query row: read S, write P over it as TWO 16-bit terms (value and rounding
//                      residual, interleaved per 16 keys: exactly the space S took)
//     O += P V         tcgen05.mma, A = P in tensor memory, both terms against the same V tile (read with its rows as K)
// and the two halves take turns: while one's softmax runs, the other's products do.  The running maximum is only raised (and O
// rescaled) when a row's maximum grew by more than 2^8: the probabilities stay below 256, well inside fp16, and l and O
// carry the same factor, so nothing is lost and almost all rescaling passes over O fall away.
// Bound: the tensor pipe, 512 cycles for S and 2 x 512 for the two-term P V per half and tile (of a whole CTA's time about 55 %
// at 8192 tokens; the rest is the softmax that does not overlap and, for short prompts, the first loads).  Measured, 32 / 8
// heads, bf16, causal flops: 4999 tokens 1329 -> 268 us (154 -> 763 TFLOP/s), 8192 tokens 3247 -> 640 us (859 TFLOP/s).
constexpr int kTQ = 128;                       // query rows per half
constexpr int kTK = 128;                       // keys per tile
constexpr int kTRing = 5;                      // K and V tiles in flight (32 KB each), in the order K0 V0 K1 V1 ...
constexpr uint32_t kTTile = 32768;             // 128 rows of 128 16-bit elements: two 64-element swizzled blocks
constexpr int kTThreads = 320;                 // warps 0-3 / 4-7: softmax of half 0 / 1; warp 8: TMA; warp 9: MMA
constexpr size_t kTSmem = 1024 + (2 + kTRing) * (size_t)kTTile + 256;
constexpr float kTLazy = 8.f;

struct TcParams {
  void* out;
  int64_t o_sb, o_sh, o_st;
  int H, rep, Tq, Tk, n_qt;
  int ranks;           // work items per (batch, KV head), longest first
  float scale_log2;
  int causal;
  int loads;           // K and V tiles that a CTA loads at most: all, except in the self test, where the rest never comes
  uint64_t wait_ns;    // after which a wait gives up
};

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ bool not_finite(float x) { return x - x != 0.f; }

// A query whose stored output is not finite everywhere.  A key that it does not see counts with a probability of 0 within its tile, which
// an infinity or a NaN among that key's values survives: channels for which that is the only cause are summed again over the keys
// that it sees (m_ref and 1 / l are as they should be: hidden scores are masked).  Rare, so one thread by itself.  (Looking every
// tile with hidden keys through before the products read it took 1.3 us of a block, 7 - 10 % of short prompts; the check at the end
// takes 0.1 - 0.3 us.)
template <typename T>
__device__ __noinline__ void attend_again(const PrefillParams& p, int b, int h, int hq, int row, int key_lim, int key_end, float m_ref, float inv) {
  const T* q = reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_sb + (int64_t)hq * p.q_sh + (int64_t)row * p.q_st;
  const T* k = reinterpret_cast<const T*>(p.k) + (int64_t)b * p.k_sb + (int64_t)h * p.k_sh;
  T* out = reinterpret_cast<T*>(p.out) + (int64_t)b * p.o_sb + (int64_t)hq * p.o_sh + (int64_t)row * p.o_st;
  for (int c = 0; c < kPD; c += 8) {
    const T* v = reinterpret_cast<const T*>(p.v) + (int64_t)b * p.v_sb + (int64_t)h * p.v_sh + c;
    auto any_bad = [&](int e, int from, int to) {
      for (int j = from; j < to; ++j)
        if (not_finite(to_float<T>(v[(int64_t)j * p.v_st + e]))) return true;
      return false;
    };
    uint32_t again = 0;
    for (int e = 0; e < 8; ++e)
      if (not_finite(to_float<T>(out[c + e])) && any_bad(e, key_lim + 1, key_end) && !any_bad(e, 0, key_lim + 1)) again |= 1u << e;
    if (again == 0) continue;
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    for (int j = 0; j <= key_lim; ++j) {
      float s = 0.f;
      for (int d = 0; d < kPD; ++d) s = fmaf(to_float<T>(q[d]), to_float<T>(k[(int64_t)j * p.k_st + d]), s);
      const float pr = ex2_approx(fmaf(s, p.scale_log2, -m_ref));
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = fmaf(pr, to_float<T>(v[(int64_t)j * p.v_st + e]), acc[e]);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (again >> e & 1) out[c + e] = from_float<T>(acc[e] * inv);
  }
}

template <typename T>
__global__ void __launch_bounds__(kTThreads, 1) prefill_attn_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                                                                      const __grid_constant__ CUtensorMap tm_v, const TcParams p,
                                                                      const __grid_constant__ PrefillParams again) {
  extern __shared__ unsigned char smem_dyn[];
  // There is no status word on this path, so a wait that ran out must show in the result: the warp that gave up says so here and
  // stops (nothing that follows from its data is committed or arrived at, so the others run out as well), and rows that
  // are stored after that are NaN.  The CTA ends when its copies and products in flight have ended.
  __shared__ int s_failed;
  const uint32_t base = (tc::s_u32(smem_dyn) + 1023u) & ~1023u;
  const uint32_t q_s = base, ring = base + 2 * kTTile, bars = ring + kTRing * kTTile;
  const uint32_t q_full = bars, kv_full = bars + 8, kv_empty = kv_full + kTRing * 8, s_full = kv_empty + kTRing * 8, p_full = s_full + 16,
                 mma_done = p_full + 16, tmem_slot = mma_done + 8;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // warp-uniform, and known to be
  bool dead = false;

  // ---- which work ----
  const int n_hb = gridDim.x / p.ranks, hb = blockIdx.x % n_hb, rank = blockIdx.x / n_hb;   // the longest tiles of all heads first
  const int h = hb % p.H, b = hb / p.H;
  int hq0, hq1, qt0, qt1;
  if ((p.rep & 1) == 0) {
    const int per = p.rep / 2;
    qt0 = qt1 = p.n_qt - 1 - rank / per;
    hq0 = 2 * (rank % per);
    hq1 = hq0 + 1;
  } else {
    const int j = rank / p.rep, i = rank - j * p.rep, half = (p.rep - 1) / 2, hi = p.n_qt - 1 - 2 * j;
    if (i < half) {
      qt0 = qt1 = hi;
      hq0 = 2 * i, hq1 = hq0 + 1;
    } else if (i == half) {
      qt0 = hi, qt1 = hi - 1;            // qt1 = -1: nothing for the second half
      hq0 = hq1 = p.rep - 1;
    } else {
      qt0 = qt1 = hi - 1;
      hq0 = 2 * (i - half - 1), hq1 = hq0 + 1;
    }
  }
  hq0 += h * p.rep;
  hq1 += h * p.rep;
  const int off = p.Tk - p.Tq;
  auto tiles_of = [&](int qt) {
    if (qt < 0) return 0;
    const int k_end = p.causal ? min(p.Tq, (qt + 1) * kTQ) + off : p.Tk;
    return (k_end + kTK - 1) / kTK;
  };
  const int nk0 = tiles_of(qt0), nk1 = tiles_of(qt1);   // nk0 >= nk1

  if (threadIdx.x == 0) {
    s_failed = 0;
    tc::bar_init(q_full, 1);
    tc::bar_init(mma_done, 1);
    for (int i = 0; i < kTRing; ++i) {
      tc::bar_init(kv_full + i * 8, 1);
      tc::bar_init(kv_empty + i * 8, 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::bar_init(s_full + i * 8, 1);
      tc::bar_init(p_full + i * 8, 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {   // one CTA per SM (its shared memory sees to that): it takes all of tensor memory
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot));
  tmem = __shfl_sync(0xffffffffu, tmem, 0);
  // columns: S / P of half 0, of half 1, O of half 0, of half 1, 128 each

  if (warp == 8) {
    // ================= loads =================
    if (lane == 0) {
      tc::bar_expect(q_full, (nk1 > 0 ? 2 : 1) * kTTile);
      tc::tma_tile4(q_s, &tm_q, 0, qt0 * kTQ, hq0, b, q_full);
      tc::tma_tile4(q_s + kTTile / 2, &tm_q, 64, qt0 * kTQ, hq0, b, q_full);
      if (nk1 > 0) {
        tc::tma_tile4(q_s + kTTile, &tm_q, 0, qt1 * kTQ, hq1, b, q_full);
        tc::tma_tile4(q_s + kTTile + kTTile / 2, &tm_q, 64, qt1 * kTQ, hq1, b, q_full);
      }
      int slot = 0, i = 0;
      uint32_t par = 1;
      for (const int n = min(2 * nk0, p.loads); i < n; ++i) {
        tc::bar_wait(kv_empty + slot * 8, par, &s_failed, dead, p.wait_ns);
        if (dead) break;
        tc::bar_expect(kv_full + slot * 8, kTTile);
        const CUtensorMap* map = (i & 1) ? &tm_v : &tm_k;
        tc::tma_tile4(ring + slot * kTTile, map, 0, (i >> 1) * kTK, h, b, kv_full + slot * 8);
        tc::tma_tile4(ring + slot * kTTile + kTTile / 2, map, 64, (i >> 1) * kTK, h, b, kv_full + slot * 8);
        if (++slot == kTRing) slot = 0, par ^= 1;
      }
      bool late = false;
      tc::bar_wait(q_full, 0, &s_failed, late);
      for (int j = max(0, i - kTRing); j < i; ++j) tc::bar_wait(kv_full + (j % kTRing) * 8, (j / kTRing) & 1, &s_failed, late);
    }
    __syncwarp();
  } else if (warp == 9) {
    // ================= products =================
    {
      const uint32_t me = tc::elect_one();
      constexpr uint32_t kFmt = tc::Pair<T>::kFmt;
      constexpr uint32_t kIdescQK = (1u << 4) | (kFmt << 7) | (kFmt << 10) | ((kTK / 8) << 17) | ((kTQ / 16) << 24);
      constexpr uint32_t kIdescPV = kIdescQK | (1u << 16);   // B = V with the contraction along its rows
      auto qk = [&](int half, uint32_t k_smem) {
        const uint64_t da = tc::umma_desc(q_s + half * kTTile), db = tc::umma_desc(k_smem);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint64_t o = (uint64_t)((j >> 2) * (kTTile / 2 >> 4) + (j & 3) * 2);
          tc::umma_f16_ss(tmem + half * 128, da + o, db + o, kIdescQK, j != 0, me);
        }
      };
      auto pv = [&](int half, uint32_t v_smem, bool first) {
        const uint64_t db = tc::umma_desc_mn(v_smem, kTTile / 2);
        const uint32_t pa = tmem + half * 128, o = tmem + 256 + half * 128;
#pragma unroll
        for (int j = 0; j < 8; ++j) {   // 16 keys: 2048 bytes of V rows; 8 columns of values, then 8 of residuals
          tc::umma_f16(o, pa + j * 16, db + (uint64_t)(j * 128), kIdescPV, !(first && j == 0), me);
          tc::umma_f16(o, pa + j * 16 + 8, db + (uint64_t)(j * 128), kIdescPV, 1u, me);
        }
      };
      int slot = 0;
      uint32_t par = 0;
      auto wait = [&](uint32_t bar, uint32_t parity) {   // for the whole warp; dead if a lane gave up
        tc::bar_wait(bar, parity, &s_failed, dead, p.wait_ns);
        dead = __any_sync(0xffffffffu, dead);
      };
      auto take = [&](uint32_t& bar_empty) {   // next tile of the ring, in load order
        wait(kv_full + slot * 8, par);
        const uint32_t addr = ring + slot * kTTile;
        bar_empty = kv_empty + slot * 8;
        if (++slot == kTRing) slot = 0, par ^= 1;
        return addr;
      };
      wait(q_full, 0);
      uint32_t k_empty, v_empty;
      uint32_t ks = take(k_empty);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (!dead) {
        qk(0, ks);
        tc::umma_commit(s_full, me);
        if (nk1 > 0) {
          qk(1, ks);
          tc::umma_commit(s_full + 8, me);
        }
        tc::umma_commit(k_empty, me);
      }
      for (int t = 0; t < nk0; ++t) {
        const uint32_t vs = take(v_empty);
        const bool more = t + 1 < nk0;
        wait(p_full, t & 1);
        if (dead) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        pv(0, vs, t == 0);
        if (more) {
          ks = take(k_empty);
          if (dead) break;
          qk(0, ks);
        }
        tc::umma_commit(s_full, me);       // S of the next tile (or, after the last, O) is complete -- and with it P V so far
        if (t < nk1) {
          wait(p_full + 8, t & 1);
          if (dead) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          pv(1, vs, t == 0);
          if (t + 1 < nk1) qk(1, ks);
          tc::umma_commit(s_full + 8, me);
        }
        tc::umma_commit(v_empty, me);
        if (more) tc::umma_commit(k_empty, me);
      }
      tc::umma_commit(mma_done, me);
      bool late = false;
      tc::bar_wait(mma_done, 0, &s_failed, late);
    }
    __syncwarp();
  } else {
    // ================= softmax: a thread per query row =================
    const int half = warp >> 2, nk = half ? nk1 : nk0, qt = half ? qt1 : qt0, hq = half ? hq1 : hq0;
    const int row = (nk ? qt : 0) * kTQ + (warp & 3) * 32 + lane;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t ts = tmem + half * 128 + lanes, to = tmem + 256 + half * 128 + lanes;
    const float sc = p.scale_log2;
    const int key_lim = p.causal ? min(p.Tk - 1, row + off) : p.Tk - 1;   // last visible key of this row
    float m_ref = 0.f, l = 0.f;
    bool seen = false;   // m_ref is the scaled maximum of something visible
    for (int t = 0; t < nk; ++t) {
      tc::bar_wait(s_full + half * 8, t & 1, &s_failed, dead, p.wait_ns);
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int key0 = t * kTK;
      const bool mask = __any_sync(0xffffffffu, key0 + kTK - 1 > key_lim);
      float mx = -INFINITY;
#pragma unroll
      for (int c = 0; c < kTK; c += 64) {
        uint32_t a[32], bb[32];
        tc::tmem_ld32(ts + c, a);
        tc::tmem_ld32(ts + c + 32, bb);
        tc::tmem_ld_wait(a);
        tc::tmem_ld_wait(bb);
        if (mask) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (key0 + c + i <= key_lim) mx = fmaxf(mx, __uint_as_float(a[i]));
            if (key0 + c + 32 + i <= key_lim) mx = fmaxf(mx, __uint_as_float(bb[i]));
          }
        } else {
          float m4[4] = {mx, mx, mx, mx};
#pragma unroll
          for (int i = 0; i < 32; i += 4)
#pragma unroll
            for (int e = 0; e < 4; ++e) m4[e] = fmaxf(m4[e], fmaxf(__uint_as_float(a[i + e]), __uint_as_float(bb[i + e])));
          mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
        }
      }
      mx *= sc;
      const bool raise = mx != -INFINITY && (!seen || mx > m_ref + kTLazy);
      if (__any_sync(0xffffffffu, raise)) {
        float alpha = 1.f;
        if (raise) {
          alpha = seen ? ex2_approx(m_ref - mx) : 0.f;
          m_ref = mx;
          seen = true;
          l *= alpha;
        }
        if (t > 0) {   // O exists (the products up to tile t - 1 completed before S of tile t)
          if (!raise) alpha = 1.f;
#pragma unroll 1
          for (int c = 0; c < 128; c += 32) {
            uint32_t o[32];
            tc::tmem_ld32(to + c, o);
            tc::tmem_ld_wait(o);
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tc::tmem_st32(to + c, o);
          }
        }
      }
      float l4[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t sbuf[2][32];
      tc::tmem_ld32(ts, sbuf[0]);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t (&s)[32] = sbuf[c & 1];
        tc::tmem_ld_wait(s);
        if (c < 3) tc::tmem_ld32(ts + (c + 1) * 32, sbuf[(c + 1) & 1]);
        uint32_t w[32];   // [values of 16 keys][residuals], twice
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float x0 = fmaf(__uint_as_float(s[i]), sc, -m_ref), x1 = fmaf(__uint_as_float(s[i + 1]), sc, -m_ref);
          if (mask) {
            if (key0 + c * 32 + i > key_lim) x0 = -INFINITY;
            if (key0 + c * 32 + i + 1 > key_lim) x1 = -INFINITY;
          }
          const float p0 = ex2_approx(x0), p1 = ex2_approx(x1);
          l4[i & 3] += p0;
          l4[(i + 1) & 3] += p1;
          const uint32_t hi = pack2<T>(p0, p1);
          const int at = (i >> 4) * 16 + ((i & 15) >> 1);
          w[at] = hi;
          w[at + 8] = residual2<T>(p0, p1, hi);
        }
        tc::tmem_st32(ts + c * 32, w);
      }
      l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      // (leaving the loop instead when a wait ran out cost 2 % of the kernel: 8192 tokens 733 us, 711 so)
      if (!__any_sync(0xffffffffu, dead) && lane == 0) tc::bar_arrive(p_full + half * 8);
    }
    if (nk > 0) {
      tc::bar_wait(s_full + half * 8, nk & 1, &s_failed, dead, p.wait_ns);
      dead = __any_sync(0xffffffffu, dead || *const_cast<volatile int*>(&s_failed) != 0);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float inv = dead ? __int_as_float(0x7fffffff) : (l > 0.f ? 1.f / l : (l == 0.f ? 0.f : l));
      T* og = reinterpret_cast<T*>(p.out) + (int64_t)b * p.o_sb + (int64_t)hq * p.o_sh + (int64_t)row * p.o_st;
      float z4[4] = {0.f, 0.f, 0.f, 0.f};   // NaN if an output is not finite
#pragma unroll 1
      for (int c = 0; c < 128; c += 32) {
        uint32_t o[32];
        tc::tmem_ld32(to + c, o);
        tc::tmem_ld_wait(o);
#pragma unroll
        for (int i = 0; i < 32; ++i) z4[i & 3] = fmaf(__uint_as_float(o[i]), 0.f, z4[i & 3]);
        if (row < p.Tq) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 v;
            v.x = pack2<T>(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv);
            v.y = pack2<T>(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv);
            v.z = pack2<T>(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv);
            v.w = pack2<T>(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv);
            *reinterpret_cast<uint4*>(og + c + i) = v;
          }
        }
      }
      if ((z4[0] + z4[1]) + (z4[2] + z4[3]) != 0.f && row < p.Tq && !not_finite(inv)) attend_again<T>(again, b, h, hq, row, key_lim, min(nk * kTK, p.Tk), m_ref, inv);
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 9) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}


// Tensor map of [B][heads][T][128] with 64-element x 128-row boxes.  False: the strides are not what one can describe
// (zero strides of broadcast tensors, more than 2^40 bytes), or the encoder refuses.
bool tc_map(CUtensorMap* map, const void* base, int dtype, int64_t sb, int64_t sh, int64_t st, int B, int heads, int T) {
  tc::EncodeTiledFn enc = tc::encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)kPD, (cuuint64_t)T, (cuuint64_t)heads, (cuuint64_t)B};
  const int64_t want[3] = {st, sh, sb};
  cuuint64_t strides[3];
  for (int i = 0; i < 3; ++i) {
    int64_t s = want[i];
    if (dims[i + 1] == 1) s = kPD;      // never used: any legal value
    if (s < kPD || s >= ((int64_t)1 << 39)) return false;
    strides[i] = (cuuint64_t)s * 2;
  }
  const cuuint32_t box[4] = {64u, (cuuint32_t)kTQ, 1u, 1u}, estr[4] = {1, 1, 1, 1};
  return enc(map, dtype == PARE_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims,
             strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The tensor-memory kernel; PARE_ERR_UNSUPPORTED where no tensor map describes the operands.
int prefill_tc(const PrefillParams& p, int dtype, int loads, uint64_t wait_ns, cudaStream_t s) {
  TcParams tp{};
  tp.out = p.out; tp.o_sb = p.o_sb; tp.o_sh = p.o_sh; tp.o_st = p.o_st;
  tp.H = p.H; tp.rep = p.rep; tp.Tq = p.Tq; tp.Tk = p.Tk;
  tp.n_qt = (p.Tq + kTQ - 1) / kTQ;
  tp.ranks = (p.rep & 1) ? tp.n_qt / 2 * p.rep + (tp.n_qt & 1) * ((p.rep + 1) / 2) : tp.n_qt * (p.rep / 2);
  tp.scale_log2 = p.scale_log2;
  tp.causal = p.causal;
  tp.loads = loads;
  tp.wait_ns = wait_ns;
  CUtensorMap mq, mk, mv;
  const int64_t ctas = (int64_t)tp.ranks * p.H * p.B;
  if (ctas >= ((int64_t)1 << 31) || !tc_map(&mq, p.q, dtype, p.q_sb, p.q_sh, p.q_st, p.B, p.Hq, p.Tq) ||
      !tc_map(&mk, p.k, dtype, p.k_sb, p.k_sh, p.k_st, p.B, p.H, p.Tk) || !tc_map(&mv, p.v, dtype, p.v_sb, p.v_sh, p.v_st, p.B, p.H, p.Tk))
    return PARE_ERR_UNSUPPORTED;
  auto launch = [&](auto kern) -> int {
    if (!ensure_smem_attr(reinterpret_cast<const void*>(kern), (int)kTSmem)) return PARE_ERR_CUDA;
    kern<<<(unsigned)ctas, kTThreads, kTSmem, s>>>(mq, mk, mv, tp, p);
    return launch_status();
  };
  return dtype == PARE_F16 ? launch(prefill_attn_tc_kernel<__half>) : launch(prefill_attn_tc_kernel<__nv_bfloat16>);
}

}  // namespace
}  // namespace pare

extern "C" int pare_selftest_prefill_wait(const void* q, const void* k, const void* v, void* out, int B, int Hq, int H, int T, int loads,
                                          unsigned int wait_us, void* stream) {
  using namespace pare;
  PARE_REQUIRE(q && k && v && out && B > 0 && Hq > 0 && H > 0 && Hq % H == 0 && T > 0 && loads >= 0, PARE_ERR_SHAPE);
  PARE_REQUIRE(wait_us <= 10000, PARE_ERR_SHAPE);   // short waits by construction
  PARE_REQUIRE(aligned16(q) && aligned16(k) && aligned16(v) && aligned16(out), PARE_ERR_ALIGN);
  PrefillParams p{};
  p.q = q; p.k = k; p.v = v; p.out = out;
  p.q_st = p.k_st = p.v_st = p.o_st = kPD;
  p.q_sh = p.k_sh = p.v_sh = p.o_sh = (int64_t)T * kPD;
  p.q_sb = p.o_sb = p.q_sh * Hq;
  p.k_sb = p.v_sb = p.k_sh * H;
  p.B = B; p.Hq = Hq; p.H = H; p.rep = Hq / H; p.Tq = p.Tk = T;
  p.scale_log2 = 0.08838834764831845f * 1.4426950408889634f;
  p.causal = 1;
  return prefill_tc(p, PARE_F16, loads, 1000ull * wait_us, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int pare_prefill_attn(const void* q, const void* k, const void* v, void* out, int dtype, int64_t q_stride_b,
                                 int64_t q_stride_h, int64_t q_stride_t, int64_t k_stride_b, int64_t k_stride_h,
                                 int64_t k_stride_t, int64_t v_stride_b, int64_t v_stride_h, int64_t v_stride_t,
                                 int64_t out_stride_b, int64_t out_stride_h, int64_t out_stride_t, int B, int Hq, int H,
                                 int Tq, int Tk, int D, float softmax_scale, int causal, void* stream) {
  using namespace pare;
  PARE_REQUIRE(B > 0 && Hq > 0 && H > 0 && Hq % H == 0 && Tq > 0 && Tk >= Tq, PARE_ERR_SHAPE);
  PARE_REQUIRE(D == kPD, PARE_ERR_UNSUPPORTED);
  PARE_REQUIRE(dtype == PARE_F16 || dtype == PARE_BF16, PARE_ERR_DTYPE);
  PARE_REQUIRE(q && k && v && out, PARE_ERR_SHAPE);
  PARE_REQUIRE(aligned16(q) && aligned16(k) && aligned16(v) && aligned16(out), PARE_ERR_ALIGN);
  for (int64_t s : {q_stride_b, q_stride_h, q_stride_t, k_stride_b, k_stride_h, k_stride_t, v_stride_b, v_stride_h, v_stride_t,
                    out_stride_b, out_stride_h, out_stride_t})
    PARE_REQUIRE(s % 8 == 0, PARE_ERR_ALIGN);
  PARE_REQUIRE(Hq <= 65535 && B <= 65535, PARE_ERR_UNSUPPORTED);
  PrefillParams p{};
  p.q = q; p.k = k; p.v = v; p.out = out;
  p.q_sb = q_stride_b; p.q_sh = q_stride_h; p.q_st = q_stride_t;
  p.k_sb = k_stride_b; p.k_sh = k_stride_h; p.k_st = k_stride_t;
  p.v_sb = v_stride_b; p.v_sh = v_stride_h; p.v_st = v_stride_t;
  p.o_sb = out_stride_b; p.o_sh = out_stride_h; p.o_st = out_stride_t;
  p.B = B; p.Hq = Hq; p.H = H; p.rep = Hq / H; p.Tq = Tq; p.Tk = Tk;
  p.scale_log2 = softmax_scale * 1.4426950408889634f;
  p.causal = causal ? 1 : 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  // The tensor-memory kernel wherever a softmax scale is positive (its running maximum is taken before scaling), the strides can be
  // described by a tensor map, and there is more than one 64-key tile (kernel alone, 32 query / 8 KV heads, bf16: 64 tokens
  // 9.0 us there, 6.6 us here; 128 tokens 10.3 / 9.5; 4 x 200 tokens 13.1 / 32.0; 512 tokens 18.5 / 33.9; 8192 tokens
  // 640 / 3250).  The kernel above serves the rest.
  // Up to one key tile and query heads that share a KV head: two of them take turns on an SM there, 64-query tiles of all heads run
  // at once here as long as there are SMs (128 tokens, batch 1 / 2 / 4 / 8: 10.5 / 10.6 / 10.8 / 11.3 there, 9.8 / 9.8 / 12.2 / 22.3 here;
  // 8 heads that share nothing, batch 1: 8.4 / 9.5).
  const bool all_at_once = Tk <= kTK && p.rep > 1 && (int64_t)((Tq + kPQ - 1) / kPQ) * Hq * B <= sm_count();
  if (softmax_scale > 0.f && Tk > kPK && !all_at_once) {
    const int rc = prefill_tc(p, dtype, INT_MAX, tc::kWaitNs, s);
    if (rc != PARE_ERR_UNSUPPORTED) return rc;
  }
  const dim3 grid((Tq + kPQ - 1) / kPQ, Hq, B);
  auto launch = [&](auto kern) -> int {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPSmem) != cudaSuccess) return PARE_ERR_CUDA;
    kern<<<grid, kPThreads, kPSmem, s>>>(p);
    return launch_status();
  };
  return dtype == PARE_F16 ? launch(prefill_attn_kernel<__half>) : launch(prefill_attn_kernel<__nv_bfloat16>);
}
