// W4A16 tensor-core path for M > 16 (prefill), sm_100a: dequantize into tensor memory, tcgen05.mma
// with weights and accumulator there.
//
// Replaces the Triton tile kernel of the reference (pare/kernels/matmul_int4.py:54-176) where
// tiles are worth it.  Orientation: the 128 rows of a weight tile sit on the MMA M axis (the 128
// TMEM lanes), the activation rows on the MMA N axis, so a 64-row batch does not waste half of
// every instruction:   Y^T[n][m] = sum_k W[n][k] * X[m][k].
//
// A persistent grid, one CTA per SM.  The work is the list of (128-row weight tile, activation tile, 256-column unit)
// in that nesting order (the first two exchanged for very large activations); a CTA takes one contiguous run of units, so a
// run may begin and end inside a tile.  Tiles that lie in several runs are finished by the CTA that arrives last, which adds
// the fp32 partial sums in K order.
// Warp roles:
//   warps 0-7    dequantize (two groups of four warps, one per 64-column block of a 128-column stage, one thread per
//                weight row): codes from shared memory, 16-bit weights into TENSOR MEMORY (tcgen05.st), where the MMA
//                reads its A operand.  Shared memory then carries only the codes and the activations.
//   warp 8       codes by TMA (cp.async.bulk.tensor.2d over the [N][K/2] byte matrix, one 128-row x 128-byte box per
//                256-column unit, 128B swizzle) into a ring of 2-8 units
//   warp 9       activation tiles by TMA (128B swizzle) into a ring of 3-4 stages of 128 columns
//   warp 10      one elected thread issues tcgen05.mma (UMMA 128 x mt x 16, A in tensor memory, fp32 accumulate)
//   warp 11      allocates tensor memory
//   warps 12-15  epilogue: accumulator -> output or partial sums, while the other warps are already in the next tile
// Per 64-column block a dequantizing thread reads 32 bytes of codes, computes (q - zero) * scale in fp32 (packed
// two-wide fp32 instructions, codes read in place as subnormal floats: dequant_word below) and rounds to the 16-bit
// type.  Weights therefore reach the tensor core as exactly dtype(fp32((q - zero) * scale)),
// bit for bit what the reference's own dequantize-then-matmul path feeds its GEMM (pare/layers/linear.py:112-118, 129).
// All mbarrier waits are bounded; on expiry the CTA records PARE_ERR_TIMEOUT, stops waiting and loading, lets its copies and
// products in flight end (bounded again), frees its tensor memory and returns.

#include "tcgen05.cuh"

namespace pare {
namespace {

using namespace tc;

constexpr int kRows = 128;             // weight rows per CTA (UMMA M)
constexpr int kBlockK = 64;            // columns per swizzle row: 128 bytes of 16-bit elements
constexpr int kStageK = 128;           // columns per operand stage: two blocks, one barrier round
constexpr int kUnitK = 256;            // columns per unit of work: one tensor-map box of packed codes, two stages
constexpr int kRawBytes = kRows * 128; // bytes of a unit's codes: 128 rows x 128 bytes, 128B swizzle
constexpr int kMaxStages = 4;          // operand stages: 4 x 64 tensor-memory columns of weights beside the accumulators
constexpr int kMaxRaw = 8;
constexpr uint32_t kTmemCols = 512;    // accumulators: columns 0-255 (two of up to 128, or one of up to 256)
constexpr uint32_t kTmemA = 256;       // weights: columns 256-511
constexpr int kDequantThreads = 256;
constexpr int kGemmThreads = 512;
constexpr size_t kCounterInts = 16384;
constexpr size_t kCounterBytes = kCounterInts * sizeof(int);
constexpr size_t kStatusIndex = kCounterInts - 1;

struct GemmParams {
  const float* scale;
  const float* zero;
  const void* bias;
  void* y;
  int64_t ldy;
  int M, N, ngroups, group_size;
  int mt;               // activation rows per tile (UMMA N): a multiple of 16, 32 .. 256
  int inner;            // tiles of the inner direction of the tile order
  int rows_inner;       // 1: weight tiles are the inner direction (activation tiles the outer), 0: the other way round
  int tile_units;       // units per tile: K / 256
  int total_units;      // units of the whole product
  int run_units;        // units per CTA
  int stages, raw_stages;
  float* partial;       // [CTA][2][mt / 4][128][4] fp32: a run's first tile (begun by another CTA) and its last (not finished)
  int* counters;        // [CTA]: arrivals at the tile that is begun by this CTA and continued by others
};

// ---- activations for the tensor-core path when they need work: the act-order gather and / or the run-time input
// scale, into a dense [M][K] copy in column order.  Plain layers skip this launch: the activation tiles are then
// fetched by TMA straight from the caller's tensor. ----
// Eight columns per thread: their sources and scales in two or four 16-byte loads, all eight gathers in flight, one
// 16-byte store.  (A column per thread and a 64-bit division each took 5 us for 64 x 14336.)
template <typename T>
__global__ void __launch_bounds__(128) w4a16_gemm_prep_kernel(const T* x, int64_t ldx, const int32_t* col_perm, const float* input_scale, T* xq,
                                                              int K) {
  const int k = (blockIdx.y * 128 + threadIdx.x) * 8, m = blockIdx.x;
  if (k >= K) return;   // K % 8 == 0
  const T* row = x + (int64_t)m * ldx;
  int src[8];
  if (col_perm && (reinterpret_cast<uintptr_t>(col_perm) & 15u) == 0) {
    const int4 a = __ldg(reinterpret_cast<const int4*>(col_perm + k)), b = __ldg(reinterpret_cast<const int4*>(col_perm + k + 4));
    src[0] = a.x; src[1] = a.y; src[2] = a.z; src[3] = a.w; src[4] = b.x; src[5] = b.y; src[6] = b.z; src[7] = b.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) src[i] = col_perm ? __ldg(col_perm + k + i) : k + i;
  }
  T v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = row[src[i]];
  if (input_scale) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = from_float<T>(__fdiv_rn(to_float<T>(v[i]), __ldg(input_scale + src[i])));
  }
  *reinterpret_cast<uint4*>(xq + (int64_t)m * K + k) = *reinterpret_cast<const uint4*>(v);
}

// Packed fp32 pairs (two independent IEEE operations per instruction).
__device__ __forceinline__ void fma_pair2(float& a, float& b, float m, float c0, float c1) {   // (a, b) = (a, b) * m + (c0, c1)
  asm("{\n\t.reg .b64 x, y, z;\n\t"
      "mov.b64 x, {%0, %1};\n\t"
      "mov.b64 y, {%2, %2};\n\t"
      "mov.b64 z, {%3, %4};\n\t"
      "fma.rn.f32x2 x, x, y, z;\n\t"
      "mov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a), "+f"(b)
      : "f"(m), "f"(c0), "f"(c1));
}
__device__ __forceinline__ void mul_pair2(float& a, float& b, float m0, float m1) {   // (a, b) = (a, b) * (m0, m1)
  asm("{\n\t.reg .b64 x, y;\n\t"
      "mov.b64 x, {%0, %1};\n\t"
      "mov.b64 y, {%2, %3};\n\t"
      "mul.rn.f32x2 x, x, y;\n\t"
      "mov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a), "+f"(b)
      : "f"(m0), "f"(m1));
}

// Per (weight row, group) constants of the dequantization below.
struct DqConst {
  float zc[4];   // -zero * 2^(4k - 22)
  float sc[4];   // scale * 2^(22 - 4k)
  __device__ __forceinline__ void set(float scale, float zero) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      zc[k] = -zero * __int_as_float((127 + 4 * k - 22) << 23);
      sc[k] = scale * __int_as_float((127 + 22 - 4 * k) << 23);
    }
  }
};

// One 32-bit word of codes -> 8 dequantized 16-bit values in COLUMN ORDER as four words of two, each EXACTLY
// dtype(fp32((q - zero) * scale)): the weight the reference's eager path feeds its GEMM
// (pare/layers/linear.py:112-118, 129: fp32 subtract, fp32 multiply, cast).  A code nibble left in place at bits
// 4k .. 4k+3 (k = 0..3; the upper four codes after one shift by 16) and read as a float's bit pattern is the subnormal
// q * 2^(4k - 149); one fused multiply-add by 2^127 with -zero * 2^(4k - 22) gives (q - zero) * 2^(4k - 22) with the
// single rounding of the reference's fp32 subtraction (powers of two do not change a rounding; no rounding at all for
// the integer zero-points of the reference's quantizers), one multiply by scale * 2^(22 - 4k) its fp32 product, one
// conversion per pair the cast.  The two lanes of a packed instruction are neighbouring columns (positions k, k + 1),
// each with its own constants, so the operand tile is in the activations' own column order and the activations need
// no re-ordering pass.
template <typename T>
__device__ __forceinline__ void dequant_word(uint32_t w, const DqConst& c, uint32_t* o) {
  const uint32_t t = w >> 16;
  constexpr float kTwo127 = 1.7014118346046923e38f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {   // columns 2j, 2j + 1
    const uint32_t src = j < 2 ? w : t;
    const int k = (2 * j) & 3;
    float a = __uint_as_float(src & (0xFu << (4 * k)));
    float b = __uint_as_float(src & (0xFu << (4 * k + 4)));
    fma_pair2(a, b, kTwo127, c.zc[k], c.zc[k + 1]);
    mul_pair2(a, b, c.sc[k], c.sc[k + 1]);
    o[j] = Pair<T>::pack(a, b);
  }
}

// What bounds it, and why this shape (one B200, bf16): with the dequantized weights in shared memory that memory had to
// carry 208 KB per 128 columns at 256 activation rows (weights written and read, activations written and read, codes), 1.6
// times what it moves in the 1024 cycles of the MMAs.  With the weights in tensor memory 144 KB remain, and the freed 64 KB
// hold one more activation stage.  Few rows are bound by the dequantizing warps (about 750 cycles per 128 columns);
// four stages instead of two keep the MMA's round trip off their path, and equal runs of units instead of whole tiles per
// CTA keep all SMs busy to the end.  28672 x 4096: 64 rows 65.9 -> 33.7 us, 256 rows 74.5 -> 52.7, 2048 rows 473 -> 356 us
// (1350 TFLOP/s); 4096 x 4096: 64 rows 23.6 -> 13.6, 128 rows 35.0 -> 16.2; 3584 x 18944, 1531 rows 294 -> 182 us.
template <typename T>
__global__ void __launch_bounds__(kGemmThreads, 1) w4a16_gemm_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                                                                    const GemmParams p) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ int s_flag;
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t b_blk = (uint32_t)p.mt * 128u, b_stage = 2 * b_blk;
  const int stages = p.stages, rstages = p.raw_stages;
  const uint32_t b_ring = s_u32(smem), raw = b_ring + stages * b_stage;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + stages * b_stage + rstages * kRawBytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kMaxRaw + 2 * kMaxStages + 5);
  const uint32_t raw_full = s_u32(bars), raw_empty = raw_full + kMaxRaw * 8, ab_full = raw_empty + kMaxRaw * 8,
                 ab_empty = ab_full + kMaxStages * 8, acc_full = ab_empty + kMaxStages * 8, acc_empty = acc_full + 16, mma_done = acc_empty + 16;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // warp-uniform, and known to be
  const int ku = p.tile_units;
  const int u0 = blockIdx.x * p.run_units, u1 = min(u0 + p.run_units, p.total_units);
  auto row_tile = [&](int t) { return p.rows_inner ? t % p.inner : t / p.inner; };
  auto act_tile = [&](int t) { return p.rows_inner ? t / p.inner : t % p.inner; };
  const bool two_acc = p.mt <= 128;   // two accumulators: a tile's epilogue overlaps the next tile's products
  int* status = p.counters + kStatusIndex;
  bool dead = false;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kMaxRaw; ++i) {
      bar_init(raw_full + i * 8, 1);
      bar_init(raw_empty + i * 8, kDequantThreads / 32);
    }
    for (int i = 0; i < kMaxStages; ++i) {
      // one barrier per operand stage for both operands: the eight dequantizing warps that write A (one group per
      // 64-column block) and the producer's expect-tx arrival for the two activation tiles
      bar_init(ab_full + i * 8, kDequantThreads / 32 + 1);
      bar_init(ab_empty + i * 8, 1);
    }
    bar_init(mma_done, 1);
    for (int i = 0; i < 2; ++i) {
      bar_init(acc_full + i * 8, 1);
      bar_init(acc_empty + i * 8, 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 11) {  // one CTA per SM (its shared memory sees to that): it takes all of tensor memory
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp < 8) {
    // ================= dequantize =================
    // Group g writes block g of every stage.
    const int r = threadIdx.x & 127, grp = threadIdx.x >> 7;
    const int spg = p.group_size / kStageK;                 // stages per quantization group
    const uint32_t a_dst = tmem + kTmemA + ((uint32_t)((warp & 3) * 32) << 16) + grp * 32;
    float sc[2], zc[2], sc_n[2], zc_n[2];
    // scale / zero of a unit's two stages: a row-strided (one line per thread) read that often comes from DRAM, so the
    // next unit's values are requested a whole unit before they are needed.  Position of the next request, kept by
    // counting: the divisions that derive it from the unit's number cost a third of a unit's dequantization.
    int mt = u0 / ku, mk = u0 - mt * ku, m_out = mt / p.inner, m_in = mt - m_out * p.inner, mg = 2 * mk / spg, mr = 2 * mk - mg * spg;
    size_t mrow = (size_t)min((p.rows_inner ? m_in : m_out) * kRows + r, p.N - 1) * p.ngroups;
    auto load_meta = [&] {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        sc_n[i] = __ldg(p.scale + mrow + mg);
        zc_n[i] = __ldg(p.zero + mrow + mg);
        if (++mr == spg) mr = 0, ++mg;
      }
      if (++mk == ku) {
        mk = mg = mr = 0;
        if (++m_in == p.inner) m_in = 0, ++m_out;
        mrow = (size_t)min((p.rows_inner ? m_in : m_out) * kRows + r, p.N - 1) * p.ngroups;
      }
    };
    load_meta();
    int slot = 0, s = 0;
    uint32_t rpar = 0, spar = 1;
    for (int u = u0; u < u1; ++u) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        sc[i] = sc_n[i];
        zc[i] = zc_n[i];
      }
      if (u + 1 < u1) load_meta();
      bar_wait(raw_full + slot * 8, rpar, status, dead);
      const uint32_t raw_row = raw + slot * kRawBytes + r * 128;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        // 16-byte chunks of row r where the 128B swizzle put them
        const uint4 codes0 = ld_s128(raw_row + (((4 * j + 2 * grp) ^ (r & 7)) << 4));
        const uint4 codes1 = ld_s128(raw_row + (((4 * j + 2 * grp + 1) ^ (r & 7)) << 4));
        DqConst dq;
        dq.set(sc[j], zc[j]);
        const uint32_t wv[8] = {codes0.x, codes0.y, codes0.z, codes0.w, codes1.x, codes1.y, codes1.z, codes1.w};
        uint32_t v[32];
#pragma unroll
        for (int wi = 0; wi < 8; ++wi) dequant_word<T>(wv[wi], dq, v + 4 * wi);
        bar_wait(ab_empty + s * 8, spar, status, dead);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_st32(a_dst + s * 64, v);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          bar_arrive(ab_full + s * 8);
          // only now: the stores above have used what was read.  Reads still in flight do not hold this arrival back, and with
          // the load pipe congested the next unit's codes were seen to land before them.
          if (j == 1) bar_arrive(raw_empty + slot * 8);
        }
        if (++s == stages) s = 0, spar ^= 1;
      }
      if (++slot == rstages) slot = 0, rpar ^= 1;
    }
  } else if (warp == 8) {
    // ================= packed codes =================
    if (lane == 0) {
      int slot = 0, u = u0;
      uint32_t par = 1;
      for (; u < u1; ++u) {
        const int t = u / ku, k = u - t * ku;
        bar_wait(raw_empty + slot * 8, par, status, dead);
        if (dead) break;
        bar_expect(raw_full + slot * 8, kRawBytes);
        tma_tile(raw + slot * kRawBytes, &tm_w, k * (kUnitK / 2), row_tile(t) * kRows, raw_full + slot * 8);
        if (++slot == rstages) slot = 0, par ^= 1;
      }
      bool late = false;
      for (int j = max(0, u - u0 - rstages); j < u - u0; ++j) bar_wait(raw_full + (j % rstages) * 8, (j / rstages) & 1, status, late);
    }
    __syncwarp();
  } else if (warp == 9) {
    // ================= activations =================
    if (lane == 0) {
      int s = 0, issued = 0;
      uint32_t par = 1;
      for (int u = u0; u < u1 && !dead; ++u) {
        const int t = u / ku, k = u - t * ku, m0 = act_tile(t) * p.mt;
        for (int j = 0; j < 2; ++j, ++issued) {
          bar_wait(ab_empty + s * 8, par, status, dead);
          if (dead) break;
          bar_expect(ab_full + s * 8, b_stage);
          tma_tile(b_ring + s * b_stage, &tm_x, k * kUnitK + j * kStageK, m0, ab_full + s * 8);
          tma_tile(b_ring + s * b_stage + b_blk, &tm_x, k * kUnitK + j * kStageK + kBlockK, m0, ab_full + s * 8);
          if (++s == stages) s = 0, par ^= 1;
        }
      }
      bool late = false;
      for (int i = max(0, issued - stages); i < issued; ++i) bar_wait(ab_full + (i % stages) * 8, (i / stages) & 1, status, late);
    }
    __syncwarp();
  } else if (warp == 10) {
    // ================= MMA issuer =================
    const uint32_t me = elect_one();
    const uint32_t idesc = (1u << 4) | (Pair<T>::kFmt << 7) | (Pair<T>::kFmt << 10) | ((uint32_t)(p.mt >> 3) << 17) |
                           ((uint32_t)(kRows >> 4) << 24);
    const uint64_t b_desc0 = umma_desc(b_ring);
    int s = 0, seg = 0;
    uint32_t par = 0;
    for (int u = u0; u < u1; ++seg) {
      const int nst = 2 * min(ku - u % ku, u1 - u);   // stages of this tile in this run
      const int buf = two_acc ? (seg & 1) : 0;
      const uint32_t acc = tmem + buf * 128;
      bar_wait(acc_empty + buf * 8, (two_acc ? (seg >> 1) & 1 : seg & 1) ^ 1, status, dead);
      for (int i = 0; i < nst; ++i) {
        bar_wait(ab_full + s * 8, par, status, dead);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t b_desc = b_desc0 + (uint64_t)(s * (b_stage >> 4));
        const uint32_t a = tmem + kTmemA + s * 64;
#pragma unroll
        for (int j = 0; j < 8; ++j)   // the second block's activations start one block after the first's
          umma_f16(acc, a + j * 8, b_desc + (uint64_t)((j >> 2) * (b_blk >> 4) + (j & 3) * 2), idesc, (i | j) != 0, me);
        umma_commit(ab_empty + s * 8, me);  // frees the operand stage when these MMAs have read it
        if (++s == stages) s = 0, par ^= 1;
      }
      umma_commit(acc_full + buf * 8, me);
      u += nst / 2;
    }
    umma_commit(mma_done, me);
    bool late = false;
    bar_wait(mma_done, 0, status, late);
    __syncwarp();
  } else if (warp >= 12) {
    // ================= epilogue: tensor memory -> registers -> global =================
    const int q4 = warp & 3, te = threadIdx.x - 12 * 32;
    T* yg = reinterpret_cast<T*>(p.y);
    const T* bias = reinterpret_cast<const T*>(p.bias);
    const bool pair_out = (reinterpret_cast<uintptr_t>(p.y) & 3u) == 0 && (p.ldy & 1) == 0 && (p.N & 1) == 0;
    auto epi_sync = [] { asm volatile("bar.sync 1, 128;" ::: "memory"); };
    int seg = 0;
    for (int u = u0; u < u1; ++seg) {
      const int t = u / ku, k0 = u - t * ku, len = min(ku - k0, u1 - u);
      u += len;
      const int row0 = row_tile(t) * kRows, m0 = act_tile(t) * p.mt;
      const int n = row0 + q4 * 32 + lane, mrows = min(p.mt, p.M - m0);
      const int buf = two_acc ? (seg & 1) : 0;
      const uint32_t acc = tmem + buf * 128 + ((uint32_t)(q4 * 32) << 16);
      const float bv = (bias && n < p.N) ? to_float<T>(bias[n]) : 0.f;
      // a lane holds ONE output column n for 16 rows m; neighbouring lanes swap so that each stores two columns of
      // every other row: 4 bytes per lane, 64 contiguous bytes per row and instruction.  The row's address is carried along:
      // with a 64-bit product in front of every store these four warps paced the kernel, 0.035 us a row beside the dequantizing
      // warps (28672 x 4096, bf16: 512 rows 128.7 -> 105.7 us, 128 rows 39.3 -> 36.8; 18944 x 512, 1024 rows 44.4 -> 25.8).
      // 16-byte stores after two more exchanges between lanes were slower (113.7, 38.0, 31.0 us).
      const int odd = lane & 1;
      T* const mine_at = yg + (size_t)(m0 + odd) * p.ldy + (n & ~1);
      auto store16 = [&](const float (&f)[16], int c) {
        if (dead) return;
        if (pair_out) {
          T* at = mine_at + (size_t)c * p.ldy;
#pragma unroll
          for (int i = 0; i < 16; i += 2, at += 2 * p.ldy) {
            const float mine = (odd ? f[i + 1] : f[i]) + bv, give = odd ? f[i] : f[i + 1];
            const float got = __shfl_xor_sync(0xffffffffu, give + bv, 1);
            // the partner added its own column's bias to what it gave
            const uint32_t w = odd ? Pair<T>::pack(got, mine) : Pair<T>::pack(mine, got);
            if (c + i + odd < mrows && n < p.N) *reinterpret_cast<uint32_t*>(at) = w;
          }
        } else if (n < p.N) {
          T* at = yg + (size_t)(m0 + c) * p.ldy + n;
#pragma unroll
          for (int i = 0; i < 16; ++i, at += p.ldy)
            if (c + i < mrows) *at = from_float<T>(f[i] + bv);
        }
      };
      bar_wait(acc_full + buf * 8, two_acc ? (seg >> 1) & 1 : seg & 1, status, dead);
      dead = __any_sync(0xffffffffu, dead);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (len == ku) {
        for (int c = 0; c < mrows; c += 16) {
          uint32_t v[16];
          float f[16];
          tmem_ld16(acc + c, v);
#pragma unroll
          for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(v[i]);
          store16(f, c);
        }
      } else {
        // ---- the tile spans the runs of CTAs first .. last; whoever arrives last adds the parts in that (K) order ----
        const int first = (int)((int64_t)t * ku / p.run_units), last = (int)(((int64_t)t * ku + ku - 1) / p.run_units), me = blockIdx.x;
        const size_t slot_floats = (size_t)p.mt * kRows;
        int* counter = p.counters + first;
        // a slot is [mt / 4][128 n][4 m]: four rows of this thread's column per 16-byte access
        auto slot_of = [&](int cta) {
          return reinterpret_cast<float4*>(p.partial + ((size_t)cta * 2 + (cta == first ? 1 : 0)) * slot_floats) + q4 * 32 + lane;
        };
        epi_sync();
        if (te == 0) {
          int have;
          asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(have) : "l"(counter) : "memory");
          s_flag = have == last - first;
        }
        epi_sync();
        const bool in_tmem = s_flag != 0;   // all others are there already: this CTA's part need not leave tensor memory
        bool finish = in_tmem;
        if (!in_tmem) {
          float4* dst = slot_of(me);
          for (int c = 0; c < mrows; c += 16) {
            uint32_t v[16];
            tmem_ld16(acc + c, v);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              __stcg(dst + (c / 4 + i) * kRows, make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]),
                                                            __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3])));
          }
          __threadfence();
          epi_sync();
          if (te == 0) s_flag = atomicAdd(counter, 1) == last - first;
          epi_sync();
          finish = s_flag != 0;
        }
        if (finish) {
          __threadfence();
          for (int c = 0; c < mrows; c += 16) {
            float f[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) f[i] = 0.f;
            // two parts requested before the first is added: what counts is how many loads share an L2 round trip
            for (int base = first; base <= last; base += 2) {
              float4 t[2][4];
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const int cta = base + e;
                if (cta <= last && !(in_tmem && cta == me)) {
                  const float4* src = slot_of(cta) + c / 4 * kRows;
#pragma unroll
                  for (int i = 0; i < 4; ++i) t[e][i] = __ldcg(src + i * kRows);
                }
              }
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const int cta = base + e;
                if (cta > last) continue;
                if (in_tmem && cta == me) {
                  uint32_t v[16];
                  tmem_ld16(acc + c, v);
#pragma unroll
                  for (int i = 0; i < 16; ++i) f[i] += __uint_as_float(v[i]);
                } else {
#pragma unroll
                  for (int i = 0; i < 4; ++i) {
                    f[4 * i] += t[e][i].x;
                    f[4 * i + 1] += t[e][i].y;
                    f[4 * i + 2] += t[e][i].z;
                    f[4 * i + 3] += t[e][i].w;
                  }
                }
              }
            }
            store16(f, c);
          }
          if (te == 0) *counter = 0;
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(acc_empty + buf * 8);
    }
  }

  // ---- teardown: everyone done with tensor memory, then free it ----
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 11) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// ---- host side --------------------------------------------------------------------------
// activation ring + packed-code ring; in front the alignment slack, behind the barriers and the TMEM slot
constexpr int kMaxSmem = 226 * 1024;   // dynamic; the flag word is static
constexpr int kRingBytes = kMaxSmem - 1024 - 512;

struct GemmPlan {
  int mt, mtiles, mpad, tiles, ku, run, ctas, stages, raw_stages;
  bool split;   // some tile lies in more than one run
  int rows_inner;
};

// Heights of the activation tiles (a multiple of 16, what the MMA's N takes, all tiles alike) and runs (a CTA's share in
// units of 256 columns) by a cost in microseconds, fitted to a sweep over 32 - 512 rows, 4096 / 6144 / 28672 x 4096 and
// 4096 x 14336 (bf16), with an epilogue that took longer than the present one: a unit takes 1.0 at 32 - 128 rows and 1.5 - 1.7 at
// 256, so tall tiles win once they fill the SMs; below that, more tiles of fewer rows beat cutting K (4096 x 4096, 128 rows: 64
// tiles of 64 rows in two parts 16.9, 32 tiles of 128 rows in four parts 17.9; 512 rows: 128 tiles of 128 rows 21.3, 64 of 256
// in two parts 26.6).  A tile above 128 rows has a single accumulator, so its epilogue stalls the next tile's products.  Parts are
// written and read again by one CTA (about 14 ns per row and part), more of them where a run does not end with its tile.
GemmPlan gemm_plan(int M, int N, int K) {
  GemmPlan best_plan{};
  double best = 1e30;
  const int sms = sm_count();
  int seen = 0;
  for (int target : {256, 192, 128, 96, 64, 32}) {
    GemmPlan g{};
    g.mtiles = (M + target - 1) / target;
    g.mt = ((M + g.mtiles - 1) / g.mtiles + 15) / 16 * 16;
    if (g.mt < 32) g.mt = 32;
    g.mtiles = (M + g.mt - 1) / g.mt;
    if (g.mt == seen) continue;
    seen = g.mt;
    g.mpad = g.mtiles * g.mt;
    g.tiles = (N + kRows - 1) / kRows * g.mtiles;
    g.ku = K / kUnitK;
    const int64_t units = (int64_t)g.tiles * g.ku;
    const double unit_us = 1.05 + 0.002 * (g.mt - 32), stall_us = g.mt > 128 ? 0.02 * g.mt : 0.0;
    auto consider = [&](int64_t run) {
      if (run < 1 || (units + run - 1) / run > sms) return;
      double cost = run * unit_us + (double)((run + g.ku - 1) / g.ku) * stall_us + 0.02 * g.mt;
      if (run % g.ku) {
        const bool ragged = g.ku % run != 0;
        const int64_t parts = (g.ku + run - 1) / run + (ragged ? 1 : 0);
        cost += 1.0 + 0.014 * g.mt * parts + (ragged ? 1.0 + 0.04 * g.mt + stall_us : 0.0);
      }
      if (cost < best - 1e-9) {
        best = cost;
        g.run = (int)run;
        best_plan = g;
      }
    };
    consider((int64_t)((g.tiles + sms - 1) / sms) * g.ku);    // whole tiles
    consider((units + sms - 1) / sms);                        // equal runs
    for (int parts = 2; parts <= 16; ++parts) consider((g.ku + parts - 1) / parts);
  }
  GemmPlan& g = best_plan;
  g.stages = (kRingBytes - 2 * kRawBytes) / (g.mt * 256);
  if (g.stages > kMaxStages) g.stages = kMaxStages;
  g.raw_stages = (kRingBytes - g.stages * g.mt * 256) / kRawBytes;
  if (g.raw_stages > kMaxRaw) g.raw_stages = kMaxRaw;
  g.ctas = (int)(((int64_t)g.tiles * g.ku + g.run - 1) / g.run);
  g.split = g.run % g.ku != 0;
  // Tile order.  Activation tiles inner: a CTA stays with its weight rows, codes are read once.  When runs cut tiles, the CTAs are
  // at different depths of different activation tiles, and activations that do not fit L2 then come from DRAM over and over
  // (4999 x 14336 for 4096 rows: 4.6 GB in 600 us); with the weight tiles inner, neighbouring CTAs walk the same activation
  // tile together (measured with the epilogue before the present one): 636 -> 531 us, 8192 x 28672 with 3000 / 4999 rows
  // 1545 / 2879 -> 1252 / 2246 us.  Whole tiles per CTA keep step by themselves, smaller activations stay in L2 (28672 x 4096,
  // 1531 rows: 293 us, 309 the other way), and codes larger than the activations would be the ones re-read (57344 x 8192,
  // 1000 rows: 1052 / 1418 us).
  const double act = 2.0 * M * K, codes = 0.5 * N * K;
  g.rows_inner = g.split && act > (double)l2_bytes() && codes < act;
  return g;
}

size_t gemm_partial_bytes(const GemmPlan& g) { return g.split ? (size_t)g.ctas * 2 * g.mt * kRows * sizeof(float) : 0; }
size_t gemm_xq_bytes(const GemmPlan& g, int K) { return ((size_t)g.mpad * K * 2 + 255) / 256 * 256; }

}  // namespace

bool gemm_supported(int M, int K, int G, const float* scale, const float* zero) {
  // 512 rather than the raw stage's 256: shapes between the two keep the streaming kernel's fp32-weight semantics
  return M > 16 && (K % 512) == 0 && (G % 128) == 0 && scale != nullptr && zero != nullptr;
}

size_t gemm_workspace_bytes(int M, int N, int K) {
  const GemmPlan g = gemm_plan(M, N, K);
  return kCounterBytes + gemm_xq_bytes(g, K) + gemm_partial_bytes(g);   // gemm_forward checks for the same
}

int gemm_forward(const void* x, int x_dtype, int64_t ldx, const uint8_t* packed, const float* scale, const float* zero,
                 const int32_t* col_perm, const float* input_scale, const void* bias, void* y, int64_t ldy, int M, int N,
                 int K, int G, void* workspace, size_t workspace_bytes, cudaStream_t stream) {
  const GemmPlan g = gemm_plan(M, N, K);
  const size_t xq_bytes = gemm_xq_bytes(g, K);
  const size_t need = kCounterBytes + xq_bytes + gemm_partial_bytes(g);
  PARE_REQUIRE(workspace != nullptr && workspace_bytes >= need, PARE_ERR_WORKSPACE);
  PARE_REQUIRE(aligned16(packed), PARE_ERR_ALIGN);
  PARE_REQUIRE((int64_t)g.tiles * g.ku + g.run < (int64_t)1 << 31 && (size_t)g.ctas < kStatusIndex, PARE_ERR_UNSUPPORTED);
  unsigned char* ws = reinterpret_cast<unsigned char*>(workspace);
  void* xq = ws + kCounterBytes;

  // 1) activations: gathered / scaled into the workspace if the layer asks for that (or the caller's rows cannot be
  //    described by a tensor map: 16-byte aligned base and row pitch), otherwise used where they are
  const bool direct = col_perm == nullptr && input_scale == nullptr && aligned16(x) && (ldx % 8) == 0;
  if (!direct) {
    const dim3 blocks(M, (K / 8 + 127) / 128);
    if (x_dtype == PARE_F16)
      w4a16_gemm_prep_kernel<__half><<<blocks, 128, 0, stream>>>((const __half*)x, ldx, col_perm, input_scale, (__half*)xq, K);
    else
      w4a16_gemm_prep_kernel<__nv_bfloat16><<<blocks, 128, 0, stream>>>((const __nv_bfloat16*)x, ldx, col_perm, input_scale,
                                                                        (__nv_bfloat16*)xq, K);
    if (cudaGetLastError() != cudaSuccess) return PARE_ERR_CUDA;
  }

  // 2) tensor map over the activations [M][K] (rows of the last tile beyond M read as zeros), box 64 columns x mt
  //    rows, 128B swizzle
  EncodeTiledFn enc = encode_fn();
  PARE_REQUIRE(enc != nullptr, PARE_ERR_CUDA);
  CUtensorMap tm;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
  const cuuint64_t strides[1] = {(cuuint64_t)(direct ? ldx : K) * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kBlockK, (cuuint32_t)g.mt};
  const cuuint32_t estr[2] = {1, 1};
  PARE_REQUIRE(enc(&tm, x_dtype == PARE_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                   direct ? const_cast<void*>(x) : xq, dims,
                   strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS,
               PARE_ERR_CUDA);

  // tensor map over the packed codes [N][K/2] bytes, box 128 bytes x 128 rows, 128B swizzle (rows beyond N read as zeros)
  CUtensorMap tw;
  const cuuint64_t wdims[2] = {(cuuint64_t)(K / 2), (cuuint64_t)N};
  const cuuint64_t wstrides[1] = {(cuuint64_t)(K / 2)};
  const cuuint32_t wbox[2] = {128u, (cuuint32_t)kRows};
  PARE_REQUIRE(enc(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(packed), wdims, wstrides, wbox, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS,
               PARE_ERR_CUDA);

  GemmParams p{};
  p.scale = scale;
  p.zero = zero;
  p.bias = bias;
  p.y = y;
  p.ldy = ldy;
  p.M = M;
  p.N = N;
  p.ngroups = K / G;
  p.group_size = G;
  p.mt = g.mt;
  p.rows_inner = g.rows_inner;
  p.inner = g.rows_inner ? g.tiles / g.mtiles : g.mtiles;
  p.tile_units = g.ku;
  p.total_units = g.tiles * g.ku;
  p.run_units = g.run;
  p.stages = g.stages;
  p.raw_stages = g.raw_stages;
  p.counters = reinterpret_cast<int*>(ws);
  p.partial = reinterpret_cast<float*>(ws + kCounterBytes + xq_bytes);

  const size_t smem = 1024 + (size_t)g.stages * g.mt * 256 + (size_t)g.raw_stages * kRawBytes + 512;
  auto launch = [&](auto kern) -> int {
    if (!ensure_smem_attr(reinterpret_cast<const void*>(kern), kMaxSmem)) return PARE_ERR_CUDA;
    kern<<<g.ctas, kGemmThreads, smem, stream>>>(tm, tw, p);
    return launch_status();
  };
  return x_dtype == PARE_F16 ? launch(w4a16_gemm_kernel<__half>) : launch(w4a16_gemm_kernel<__nv_bfloat16>);
}

}  // namespace pare
