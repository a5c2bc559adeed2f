// W4A16 linear for a handful of activation rows (batched decode, up to 16 rows), sm_100a: the CODES go to the tensor core.
//
//     y[m][n] = sum over 128-column steps of  scale * g[m] * ( sum_k q[n][k] * x^[m][k]  -  zero * SX[m] )
//
// Same arithmetic as the streaming kernels (w4a16_gemv.cu: activations prepared as scaled fp16 with a step table, prep.cuh;
// zero-point and scale applied in fp32 per step), other machinery: the weight rows sit on the MMA M axis, the activation
// rows on its N axis (16 columns), the unpacked codes are the A operand in TENSOR MEMORY.
//   * a code nibble left in place inside the ten mantissa bits of an fp16 with zero exponent IS the number q * 2^-24
//     (bits 0-3) or q * 2^-20 (bits 4-7; the prepared activation of such a position is divided by 16): one `and` per pair of
//     codes and one shift per eight is all the conversion there is; the step's sum is rescaled by 2^24 in fp32
//   * a step's 128 x 16 sums come back from tensor memory to one thread per weight row, which folds scale and zero of its
//     row in: three fp32 operations per output and step
// Persistent grid, one CTA per SM, equal runs of 256-column units (as in w4a16_gemm.cu: a run may begin and end inside a
// tile of 128 rows; the CTA that arrives last adds the parts in K order).  Warp roles:
//   warps 0-7    unpack: four warps per step, alternating; a thread reads its row's 64 bytes of codes and writes 64 columns
//   warp 8       codes by TMA, up to eight 16 KB units in flight; prefetch of the scale / zero lines of those units into L2
//   warp 9       prepared activations by TMA (16 rows x 128 columns per step)
//   warp 10      tcgen05.mma
//   warp 11      tensor memory allocation
//   warps 12-19  fold: two groups of four warps (a thread per weight row), one per step of a unit; their sums meet in shared
//                memory at the end of a tile, the first group writes the output
#include "gemv_common.cuh"
#include "prep.cuh"
#include "tcgen05.cuh"

namespace pare {
namespace {

using namespace tc;
using gemv::GemvParams;
using gemv::kTabCols;

constexpr int kRows = 128;              // weight rows per tile (UMMA M)
constexpr int kN = 16;                  // activation rows (UMMA N)
constexpr int kUnitK = 256;             // columns per unit: two steps
constexpr int kRawBytes = kRows * 128;
constexpr int kRaw = 8;                 // units of codes in flight: 128 KB per SM
constexpr int kStages = 6;              // unpacked steps: 6 x 64 tensor-memory columns
constexpr int kSums = 8;                // steps' sums: 8 x 16 columns
constexpr uint32_t kTmemSums = kStages * 64;
constexpr uint32_t kBBlk = kN * 128, kBStage = 2 * kBBlk;
constexpr int kThreads = 640;
constexpr int kXchg = kN * kRows * 4;    // bytes: the second fold group's sums of a tile
constexpr int kMaxSmem = 226 * 1024;

struct TcPlan {
  int tiles, ku, run, ctas;
};

struct TcArgs {
  int tile_units, total_units, run_units;
};

// What bounds it (one B200, bf16, kernel alone): the codes arrive at 4.7 TB/s when nothing else is done (12.4 us for 28672 x
// 4096), the unpack - multiply - fold chain of a 256-column unit takes 0.6 us of an SM, and 5 - 6 us are launch, first
// loads and drain.  16 rows: 28672 x 4096 40.2 -> 23.7 us, 4096 x 14336 34.9 -> 13.9, 4096 x 4096 11.0 -> 7.8,
// 57344 x 8192 322 -> 73, 8192 x 28672 242 -> 45 us against the streaming kernels, whose activations (16 rows x 4096
// columns) fill shared memory and whose warp-level operand handling grows with the rows.
template <typename T>
__global__ void __launch_bounds__(kThreads, 1) w4a16_gemv_tc_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                                                                   const GemvParams p, const TcArgs a) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ int s_flag;
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t raw = s_u32(smem), b_ring = raw + kRaw * kRawBytes, bars = b_ring + kStages * kBStage;
  const uint32_t raw_full = bars, raw_empty = raw_full + kRaw * 8, ab_full = raw_empty + kRaw * 8, ab_empty = ab_full + kStages * 8,
                 d_full = ab_empty + kStages * 8, d_empty = d_full + kSums * 8, mma_done = d_empty + kSums * 8, tmem_slot = mma_done + 8;
  float* xchg = reinterpret_cast<float*>(smem + kRaw * kRawBytes + kStages * kBStage + 512);   // [kN][kRows]
  // (SX, g) of every step and activation row
  float2* tab = reinterpret_cast<float2*>(smem + kRaw * kRawBytes + kStages * kBStage + 512 + kXchg);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // warp-uniform, and known to be
  const int ku = a.tile_units;
  const int u0 = blockIdx.x * a.run_units, u1 = min(u0 + a.run_units, a.total_units);
  int* status = p.counters + gemv::kStatusIndex;
  bool dead = false;
  pdl_launch_dependents();

  if (threadIdx.x == 0) {
    bar_init(mma_done, 1);
    for (int i = 0; i < kRaw; ++i) {
      bar_init(raw_full + i * 8, 1);
      bar_init(raw_empty + i * 8, 8);
    }
    for (int i = 0; i < kStages; ++i) {
      bar_init(ab_full + i * 8, 4 + 1);
      bar_init(ab_empty + i * 8, 1);
    }
    for (int i = 0; i < kSums; ++i) {
      bar_init(d_full + i * 8, 1);
      bar_init(d_empty + i * 8, 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 11) {   // one CTA per SM (its shared memory sees to that): it takes all of tensor memory
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot));
  tmem = __shfl_sync(0xffffffffu, tmem, 0);

  if (warp < 8) {
    // ================= unpack: group g takes step g of every unit =================
    const int r = threadIdx.x & 127, grp = threadIdx.x >> 7;
    const uint32_t a_dst = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    int slot = 0, s = grp;
    uint32_t rpar = 0, spar = 1;
    for (int u = u0; u < u1; ++u) {
      bar_wait(raw_full + slot * 8, rpar, status, dead);
      const uint32_t raw_row = raw + slot * kRawBytes + r * 128;
      uint32_t w[16];   // word c = columns 8c .. 8c + 7 of the step
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint4 q = ld_s128(raw_row + (((4 * grp + j) ^ (r & 7)) << 4));
        w[4 * j] = q.x; w[4 * j + 1] = q.y; w[4 * j + 2] = q.z; w[4 * j + 3] = q.w;
      }
      bar_wait(ab_empty + s * 8, spar, status, dead);
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int pos = hf * 8 + i, c = (pos & 3) * 4 + (pos >> 2);   // the chunk that prep.cuh stores at position pos
          const uint32_t lo = w[c], hi = lo >> 8;
          v[4 * i] = lo & 0x000f000fu;
          v[4 * i + 1] = lo & 0x00f000f0u;
          v[4 * i + 2] = hi & 0x000f000fu;
          v[4 * i + 3] = hi & 0x00f000f0u;
        }
        tmem_st32(a_dst + s * 64 + hf * 32, v);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        bar_arrive(ab_full + s * 8);
        // only now: the stores above have used what was read.  Reads still in flight do not hold this arrival back, and with
        // the load pipe congested the next unit's codes were seen to land before them.
        bar_arrive(raw_empty + slot * 8);
      }
      s += 2;
      if (s >= kStages) s -= kStages, spar ^= 1;
      if (++slot == kRaw) slot = 0, rpar ^= 1;
    }
  } else if (warp == 8) {
    // ================= packed codes (weights: no dependency on the kernel before) =================
    int slot = 0;
    uint32_t par = 1;
    const int upl = max(1, 8 * p.steps_per_group / 2);   // units per 32-byte sector of a scale row
    int u = u0;
    for (; u < u1; ++u) {
      const int t = u / ku, k = u - t * ku;
      if (lane == 0) bar_wait(raw_empty + slot * 8, par, status, dead);
      if (__any_sync(0xffffffffu, dead)) break;
      if (lane == 0) {
        bar_expect(raw_full + slot * 8, kRawBytes);
        tma_tile(raw + slot * kRawBytes, &tm_w, k * (kUnitK / 2), t * kRows, raw_full + slot * 8);
      }
      __syncwarp();
      if (k % upl == 0 || u == u0) {
        const int g = 2 * k / p.steps_per_group;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const size_t at = (size_t)min(t * kRows + i * 32 + lane, p.N - 1) * p.ngroups + g;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p.scale + at));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p.zero + at));
        }
      }
      if (++slot == kRaw) slot = 0, par ^= 1;
    }
    if (lane == 0) {   // the block may end only when what it asked for has arrived, also where a wait ran out
      bool late = false;
      for (int j = max(0, u - u0 - kRaw); j < u - u0; ++j) bar_wait(raw_full + (j % kRaw) * 8, (j / kRaw) & 1, status, late);
    }
    __syncwarp();
  } else if (warp == 9) {
    // ================= activations =================
    if (lane == 0) {
      pdl_wait();
      int s = 0, issued = 0;
      uint32_t par = 1;
      for (int u = u0; u < u1 && !dead; ++u) {
        const int k = u % ku;
        for (int j = 0; j < 2; ++j, ++issued) {
          bar_wait(ab_empty + s * 8, par, status, dead);
          if (dead) break;
          bar_expect(ab_full + s * 8, kBStage);
          tma_tile(b_ring + s * kBStage, &tm_x, k * kUnitK + j * 128, 0, ab_full + s * 8);
          tma_tile(b_ring + s * kBStage + kBBlk, &tm_x, k * kUnitK + j * 128 + 64, 0, ab_full + s * 8);
          if (++s == kStages) s = 0, par ^= 1;
        }
      }
      bool late = false;
      for (int i = max(0, issued - kStages); i < issued; ++i) bar_wait(ab_full + (i % kStages) * 8, (i / kStages) & 1, status, late);
    }
    __syncwarp();
  } else if (warp == 10) {
    // ================= MMA issuer =================
    const uint32_t me = elect_one();
    constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(kN >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);   // fp16 x fp16 -> fp32
    const uint64_t b_desc0 = umma_desc(b_ring);
    int s = 0, d = 0;
    uint32_t par = 0, dpar = 1;
    for (int i = 2 * (u1 - u0); i > 0; --i) {
      bar_wait(d_empty + d * 8, dpar, status, dead);
      bar_wait(ab_full + s * 8, par, status, dead);
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t b_desc = b_desc0 + (uint64_t)(s * (kBStage >> 4));
#pragma unroll
      for (int j = 0; j < 8; ++j)
        umma_f16(tmem + kTmemSums + d * kN, tmem + s * 64 + j * 8, b_desc + (uint64_t)((j >> 2) * (kBBlk >> 4) + (j & 3) * 2), idesc, j != 0, me);
      umma_commit(ab_empty + s * 8, me);
      umma_commit(d_full + d * 8, me);
      if (++s == kStages) s = 0, par ^= 1;
      if (++d == kSums) d = 0, dpar ^= 1;
    }
    umma_commit(mma_done, me);
    bool late = false;
    bar_wait(mma_done, 0, status, late);
    __syncwarp();
  } else if (warp >= 12) {
    // ================= fold and output =================
    // One group of four warps was what paced the kernel (1150 of the 1350 cycles that a unit took, a third of them integer
    // divisions for the addresses of scale and zero).
    const int q4 = warp & 3, te = threadIdx.x & 127, grp = warp >= 16;
    T* yg = reinterpret_cast<T*>(p.y);
    const T* bias = reinterpret_cast<const T*>(p.bias);
    auto fold_sync = [] { asm volatile("bar.sync 1, 128;" ::: "memory"); };        // the first group
    auto both_sync = [](int id) { asm volatile("bar.sync %0, 256;" ::"r"(id) : "memory"); };
    // scale / zero of this thread's row at this group's step, requested one unit ahead: position of the next request
    int mt = u0 / ku, mk = u0 - mt * ku, mg = (2 * mk + grp) / p.steps_per_group, mr = (2 * mk + grp) - mg * p.steps_per_group;
    size_t mrow = (size_t)min(mt * kRows + te, p.N - 1) * p.ngroups;
    float sc_n, zc_n;
    auto load_meta = [&] {
      sc_n = __ldg(p.scale + mrow + mg);
      zc_n = __ldg(p.zero + mrow + mg);
      mr += 2;
      while (mr >= p.steps_per_group) mr -= p.steps_per_group, ++mg;
      if (++mk == ku) {
        mk = 0, ++mt;
        mrow = (size_t)min(mt * kRows + te, p.N - 1) * p.ngroups;
        mg = grp / p.steps_per_group;
        mr = grp - mg * p.steps_per_group;
      }
    };
    load_meta();
    pdl_wait();
    for (int i = threadIdx.x - 12 * 32; i < 2 * ku * kN; i += 256) {
      const int m = i & (kN - 1);
      const float4 e = m < p.M ? p.tabg[(size_t)(i / kN) * kTabCols + m] : make_float4(0.f, 0.f, 0.f, 0.f);
      tab[i] = make_float2(e.y, e.z);
    }
    both_sync(2);
    int d = grp;
    uint32_t dpar = 0;
    for (int u = u0; u < u1;) {
      const int t = u / ku, k0 = u - t * ku, len = min(ku - k0, u1 - u);
      float y[kN];
#pragma unroll
      for (int m = 0; m < kN; ++m) y[m] = 0.f;
      const float4* tb = reinterpret_cast<const float4*>(tab + (2 * k0 + grp) * kN);
      for (const int end = u + len; u < end; ++u, tb += kN) {
        const float sc = sc_n, zc = zc_n;
        if (u + 1 < u1) load_meta();
        bar_wait(d_full + d * 8, dpar, status, dead);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t v[16];
        tmem_ld16(tmem + kTmemSums + d * kN + ((uint32_t)(q4 * 32) << 16), v);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) bar_arrive(d_empty + d * 8);
        d += 2;
        if (d >= kSums) d -= kSums, dpar ^= 1;
#pragma unroll
        for (int m = 0; m < kN; m += 2) {
          const float4 e = tb[m >> 1];   // (SX, g) of rows m, m + 1
          y[m] = fmaf(sc * e.y, fmaf(-zc, e.x, __uint_as_float(v[m]) * 16777216.f), y[m]);
          y[m + 1] = fmaf(sc * e.w, fmaf(-zc, e.z, __uint_as_float(v[m + 1]) * 16777216.f), y[m + 1]);
        }
      }
      // even steps + odd steps
      if (grp) {
#pragma unroll
        for (int m = 0; m < kN; ++m) xchg[m * kRows + te] = y[m];
      }
      both_sync(2);
      if (!grp) {
#pragma unroll
        for (int m = 0; m < kN; ++m) y[m] += xchg[m * kRows + te];
      }
      both_sync(3);   // the exchange area may be written again
      if (grp) continue;
      const int n = t * kRows + te;
      bool store = true;
      if (len != ku) {
        // ---- the tile spans the runs of CTAs first .. last; whoever arrives last adds the parts in that (K) order ----
        const int first = (int)((int64_t)t * ku / a.run_units), last = (int)(((int64_t)t * ku + ku - 1) / a.run_units);
        int* counter = p.counters + first;
        auto slot_of = [&](int cta) { return p.partial + ((size_t)cta * 2 + (cta == first ? 1 : 0)) * (kN * kRows) + te; };
        float* dst = slot_of(blockIdx.x);
#pragma unroll
        for (int m = 0; m < kN; ++m)
          if (m < p.M) __stcg(dst + m * kRows, y[m]);
        __threadfence();
        fold_sync();
        if (te == 0) s_flag = atomicAdd(counter, 1) == last - first;
        fold_sync();
        store = s_flag != 0;
        if (store) {
          __threadfence();
#pragma unroll
          for (int m = 0; m < kN; ++m) y[m] = 0.f;
          for (int cta = first; cta <= last; cta += 2) {   // two parts per L2 round trip
            const float* s0 = slot_of(cta);
            const float* s1 = slot_of(min(cta + 1, last));
            float a0[kN], a1[kN];
#pragma unroll
            for (int m = 0; m < kN; ++m) a0[m] = m < p.M ? __ldcg(s0 + m * kRows) : 0.f;
#pragma unroll
            for (int m = 0; m < kN; ++m) a1[m] = m < p.M ? __ldcg(s1 + m * kRows) : 0.f;
#pragma unroll
            for (int m = 0; m < kN; ++m) y[m] += a0[m];
            if (cta < last) {
#pragma unroll
              for (int m = 0; m < kN; ++m) y[m] += a1[m];
            }
          }
          if (te == 0) *counter = 0;
        }
        fold_sync();   // s_flag may be written again
      }
      if (store && n < p.N && !dead) {
        const float bv = bias ? to_float<T>(bias[n]) : 0.f;
#pragma unroll
        for (int m = 0; m < kN; ++m)
          if (m < p.M) yg[(size_t)m * p.ldy + n] = from_float<T>(y[m] + bv);
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 11) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// Runs: whole tiles, equal parts of a tile, or equal shares of all units (which cut tiles at odd places, so that a CTA finishes
// two part tiles one after the other).  Microseconds, fitted to every run length of 19 heights x 10 depths with 8 and 16 rows: a unit
// takes 0.575, a part 0.28, a cut tile 1.8, cuts at odd places 1.2 more (8192 x 4096, 8 rows: 128 CTAs of half a tile 9.9, 147 of
// 7 units 11.1; 3072 x 4096: runs of 4 units 7.3, of 3 units 8.5; 14336 x 4096: whole tiles 12.8, runs of 13 units 14.6).
TcPlan tc_plan(int N, int K) {
  TcPlan g{};
  g.tiles = (N + kRows - 1) / kRows;
  g.ku = K / kUnitK;
  const int sms = sm_count();
  const int64_t units = (int64_t)g.tiles * g.ku;
  double best = 1e30;
  auto consider = [&](int64_t run) {
    if (run < 1 || (units + run - 1) / run > sms) return;
    double cost = run * 0.575;
    if (run % g.ku) {
      const bool odd = g.ku % run != 0;
      cost += (odd ? 3.0 : 1.8) + 0.28 * (double)((g.ku + run - 1) / run + odd);
    }
    if (cost < best - 1e-9) {
      best = cost;
      g.run = (int)run;
    }
  };
  consider((int64_t)((g.tiles + sms - 1) / sms) * g.ku);
  consider((units + sms - 1) / sms);
  for (int s = 2; s <= 16; ++s) consider((g.ku + s - 1) / s);
  g.ctas = (int)((units + g.run - 1) / g.run);
  return g;
}

size_t tc_smem(int K) { return 1024 + kRaw * (size_t)kRawBytes + kStages * (size_t)kBStage + 512 + kXchg + (size_t)(K / 128) * kN * sizeof(float2); }

}  // namespace

size_t gemv_tc_partial_floats(int N, int K) {
  if (K % kUnitK) return 0;
  return (size_t)tc_plan(N, K).ctas * 2 * kN * kRows;
}

bool gemv_tc_supported(int M, int N, int K, int G) {
  return M >= 1 && M <= kN && K % kUnitK == 0 && G % 128 == 0 && tc_smem(K) <= (size_t)kMaxSmem &&
         (int64_t)((N + kRows - 1) / kRows) * (K / kUnitK) < (int64_t)1 << 30;
}

int gemv_tc_launch(const GemvParams& p, int x_dtype, cudaStream_t stream) {
  const TcPlan g = tc_plan(p.N, p.K);
  EncodeTiledFn enc = encode_fn();
  PARE_REQUIRE(enc != nullptr, PARE_ERR_CUDA);
  CUtensorMap tx, tw;
  const cuuint32_t estr[2] = {1, 1};
  const cuuint64_t xdims[2] = {(cuuint64_t)p.K, (cuuint64_t)p.M}, xstr[1] = {(cuuint64_t)p.K * 2};
  const cuuint32_t xbox[2] = {64u, (cuuint32_t)kN};   // rows beyond M read as zeros
  PARE_REQUIRE(enc(&tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p.xp, xdims, xstr, xbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS,
               PARE_ERR_CUDA);
  const cuuint64_t wdims[2] = {(cuuint64_t)(p.K / 2), (cuuint64_t)p.N}, wstr[1] = {(cuuint64_t)(p.K / 2)};
  const cuuint32_t wbox[2] = {128u, (cuuint32_t)kRows};
  PARE_REQUIRE(enc(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(p.packed), wdims, wstr, wbox, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS,
               PARE_ERR_CUDA);
  const TcArgs a{g.ku, g.tiles * g.ku, g.run};
  auto launch = [&](auto kern) -> int {
    if (!ensure_smem_attr(reinterpret_cast<const void*>(kern), kMaxSmem)) return PARE_ERR_CUDA;
    return launch_pdl(kern, dim3(g.ctas), dim3(kThreads), tc_smem(p.K), stream, tx, tw, p, a);
  };
  return x_dtype == PARE_F16 ? launch(w4a16_gemv_tc_kernel<__half>) : launch(w4a16_gemv_tc_kernel<__nv_bfloat16>);
}

}  // namespace pare
