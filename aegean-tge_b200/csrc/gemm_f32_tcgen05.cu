// Float32 matrix product on the 5th-generation tensor cores: out = x . w^T (+ epilogue), every number of x and w as the
// sum of three bfloat16 numbers.
//
// gemm_simt.cu is bound by the FMA pipes and by shared memory in front of them: 7.1 ms for a layer of 233 M weights at 512
// tokens (33 TFLOP/s), and a step of 8 tokens computes its 64-row tile whole and streams the weights at 0.45 TB/s.  A
// float32 number is h + m + l with h, m, l bfloat16 (8 bits of significand each, 24 together, exact down to numbers of
// about 1e-33), and of the nine products of two such sums the three of 2^-24 and below are left out; the other six are
// tensor-core products of 16 times the FMA pipes' rate.  Measured alone (B200), FMA kernel and this one, us:
//   weights           8 tokens           40 tokens        128 tokens        512 tokens
//   3,584 x  3,584      218 ->  17        215 ->  20        221 ->  26        524 ->  75
//   37,888 x 3,584      523 ->  90        528 -> 114      1,048 -> 210      3,912 -> 734  (189 TFLOP/s of float32 work)
//   3,584 x 18,944    1,601 ->  52      1,571 ->  59      1,475 ->  89      2,686 -> 334
//   152,064 x 3,584   2,063 -> 342 (6.4 TB/s of weights)  1 token: 2,065 -> 331
// With few tokens the weights' bytes bound it; with many, the shared memory that feeds the products.
//
// Precision.  A tensor-core product adds into its float32 accumulator with less care than a rounded FMA, so no accumulator
// lives longer than one k-block of 64, is filled from the smallest products to the largest (l h, h l, m m, m h, h m, h h), and is
// added into registers with rounding to nearest: the error against float64 is a tenth of one FMA chain's along k
// (relative, random numbers: 1.1e-7 against 1.07e-6 at K = 3,584, 1.7e-7 against 2.5e-6 at 18,944).
// Numbers that are not finite, or products beyond float32's range, do not survive the split (infinity - infinity), and below about
// 1e-33 the low parts run out of exponents: an output that is not finite, or below 2^-100 without being zero, is computed
// again as one FMA chain along k, so it is what that chain makes of it.  (A part lost below 2^-133 is worth 2^-134 of the other side's
// number: against an output of 2^-100 nothing.  What remains is an output that the chain makes of numbers below 2^-134 alone: zero here.)
//
// An output element depends on its own row of x and of w only: the k-blocks' order, the cut along k (a rule on N and K) and
// the order in which the cuts are added do not depend on how many tokens there are or on the tile a token falls in.
//
// Shape of the kernel (one persistent block per SM, 512 threads, weight rows on the M side as in gemm_tcgen05.cu):
//   warp 0      asks for weight tiles (128 rows x 64 float32, two 128-byte-swizzled halves), warp 3 for the token tiles (BN
//               rows x 64 of each of the three parts, split beforehand by a small kernel: the tokens' bytes are few);
//   warps 4-7   read a weight row each thread, split it and store the parts to tensor memory, from where the product reads its
//               first operand: shared memory, the scarce resource here, then carries a weight twice (in and out) and the token
//               tiles, about 137 bytes a cycle at BN = 128 where parts in shared memory would need 250 (128 is the limit);
//   warp 1      issues the products, warps 8-15 add finished k-blocks into registers while the next is multiplied.
// The weights are split anew for each panel of tokens: a converted copy would cost 6 bytes a weight beside the 4.
// Every wait is bounded, as in gemm_tcgen05.cu.
#include "tcgen05_ptx.cuh"

namespace {

enum F32Epilogue : int { F32_STORE = 0, F32_STORE_F32 = 1, F32_ADD = 2, F32_SWIGLU = 3, F32_GELU = 4, F32_GELU_TANH = 5, F32_GLU_CLAMPED = 6 };

constexpr int BM = 128, BK = 64, PARTS = 3, UMMA_K = 16;
constexpr int W_STAGE_BYTES = BM * BK * 4;
constexpr int SMEM_LIMIT = 227 * 1024;
constexpr int CONVERT_WARPS = 4, EPI_WARPS = 8;
constexpr int THREADS = 512;
constexpr int TMEM_COLS = 512;
constexpr int A_COLS = PARTS * BK / 2;       // tensor-memory columns of one converted weight tile
constexpr int MAX_W_STAGES = 6;

template <int BN>
struct Shape {
  static constexpr int X_STAGES = BN >= 128 ? 2 : BN >= 64 ? 3 : 4;
  static constexpr int X_STAGE_BYTES = PARTS * BN * BK * 2;
  static constexpr int ROOM = (SMEM_LIMIT - 2048 - X_STAGES * X_STAGE_BYTES) / W_STAGE_BYTES;
  static constexpr int W_STAGES = ROOM < MAX_W_STAGES ? ROOM : MAX_W_STAGES;
  static constexpr int A_STAGES = BN >= 128 ? 2 : 4;
  static constexpr int A_FIRST_COL = BN >= 128 ? 2 * BN : 128;
  static constexpr int BARRIERS = 2 * (W_STAGES + X_STAGES + A_STAGES + 2);
  static constexpr size_t SMEM = 1024 + (size_t)W_STAGES * W_STAGE_BYTES + (size_t)X_STAGES * X_STAGE_BYTES + 8 * BARRIERS + 16;
  static_assert(W_STAGES >= 3 && SMEM <= SMEM_LIMIT && A_FIRST_COL >= 2 * BN && A_FIRST_COL + A_STAGES * A_COLS <= TMEM_COLS, "a block's room");
};

struct F32GemmParams {
  const float* x;       // for outputs outside the usual range
  const float* w;
  long long ldx, ldw;
  int M, N, K;
  int k_blocks, splits, tiles_w, tiles_t;
  int epilogue, act_from;
  float alpha;
  const float* bias;
  float* out;
  long long ldo;
  float* partial;       // [splits][M][N] where the product is cut along k
  int* status;
};

__device__ __forceinline__ void tmem_load8(uint32_t taddr, uint32_t r[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

__device__ __noinline__ float fma_chain(const float* x, const float* w, int K) {
  float acc = 0.0f;
  for (int k = 0; k < K; ++k) acc = fmaf(x[k], w[k], acc);
  return acc;
}
__device__ __forceinline__ float usual_or_chain(const F32GemmParams& p, float v, int m, int n) {
  const float size = fabsf(v);
  return (size <= 3.402823466e38f && size >= 7.8886090522e-31f) || size == 0.0f ? v : fma_chain(p.x + (size_t)m * p.ldx, p.w + (size_t)n * p.ldw, p.K);
}

__device__ __forceinline__ float gated(const F32GemmParams& p, float g, float u) {
  if (p.epilogue == F32_GLU_CLAMPED) {
    g = fminf(g, p.alpha);
    u = fminf(fmaxf(u, -p.alpha), p.alpha) + 1.0f;
    g *= 1.702f;
    u *= 1.0f / 1.702f;
  }
  return g / (1.0f + expf(-g)) * u;
}
// the plain epilogues of one element; `v` has its bias
__device__ __forceinline__ void finish(const F32GemmParams& p, float v, int m, int n) {
  float* dst = p.out + (size_t)m * p.ldo + n;
  if (p.epilogue >= F32_GELU) {
    if (n >= p.act_from) v = p.epilogue == F32_GELU ? gelu_erf(v) : gelu_tanh(v);
    *dst = v;
  } else if (p.epilogue == F32_ADD) {
    *dst += v * p.alpha;
  } else {
    *dst = v * p.alpha;
  }
}

// ---- the token rows in three parts: planes [3][M][Kp] of bfloat16, zeros behind column K ----
__global__ void __launch_bounds__(256) split_rows_kernel(const float* x, long long ldx, __nv_bfloat16* __restrict__ planes,
                                                         int M, int K, int Kp, int vec) {
  // Trigger behind the wait: the product then starts once whatever came before this call is done, so its loader may ask for the
  // weights, and the kernel that adds the cuts for the bias, ahead of their own waits, whoever wrote those.
  pdl_wait();
  pdl_trigger();
  const int m = blockIdx.y, k = ((int)blockIdx.x * 256 + (int)threadIdx.x) * 8;
  if (k >= Kp) return;
  const float* src = x + (size_t)m * ldx + k;
  float v[8];
  if (vec && k + 8 <= K) {
    const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = k + i < K ? src[i] : 0.0f;
  }
  uint4 h, mid, l;
  split_pair(v[0], v[1], h.x, mid.x, l.x);
  split_pair(v[2], v[3], h.y, mid.y, l.y);
  split_pair(v[4], v[5], h.z, mid.z, l.z);
  split_pair(v[6], v[7], h.w, mid.w, l.w);
  const size_t plane = (size_t)M * Kp, at = (size_t)m * Kp + k;
  *reinterpret_cast<uint4*>(planes + at) = h;
  *reinterpret_cast<uint4*>(planes + plane + at) = mid;
  *reinterpret_cast<uint4*>(planes + 2 * plane + at) = l;
}

// ---- the product ----
template <int BN>
__global__ void __launch_bounds__(THREADS, 1) gemm_f32_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                      const __grid_constant__ CUtensorMap map_x, const F32GemmParams p) {
  using S = Shape<BN>;
  constexpr int COLS = BN / 2;                 // columns of an epilogue warp
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* generic = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t x_base = base + S::W_STAGES * W_STAGE_BYTES;
  const uint32_t bars = x_base + S::X_STAGES * S::X_STAGE_BYTES;
  const uint32_t w_full = bars, w_empty = w_full + 8 * S::W_STAGES, x_full = w_empty + 8 * S::W_STAGES, x_empty = x_full + 8 * S::X_STAGES;
  const uint32_t a_full = x_empty + 8 * S::X_STAGES, a_empty = a_full + 8 * S::A_STAGES, d_full = a_empty + 8 * S::A_STAGES, d_empty = d_full + 16;
  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::W_STAGES; ++s) { mbar_init(w_full + 8 * s, 1); mbar_init(w_empty + 8 * s, CONVERT_WARPS); }
    for (int s = 0; s < S::X_STAGES; ++s) { mbar_init(x_full + 8 * s, 1); mbar_init(x_empty + 8 * s, 1); }
    for (int s = 0; s < S::A_STAGES; ++s) { mbar_init(a_full + 8 * s, CONVERT_WARPS); mbar_init(a_empty + 8 * s, 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(d_full + 8 * s, 1); mbar_init(d_empty + 8 * s, EPI_WARPS); }
    abort_word = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_trigger();                               // tensor memory is held: the next kernel's blocks can at worst wait for it
  if (warp != 0) pdl_wait();                   // the weights are there (see split_rows_kernel): their loader goes ahead

  const int units = p.tiles_w * p.tiles_t * p.splits;
  // unit -> cut along k, token tile, weight tile (the cuts of a tile and the token tiles of a weight tile side by side)
  auto k_begin = [&](int split) { return (int)((long long)split * p.k_blocks / p.splits); };

  if (warp == 0) {
    // ------------------------------ weight tiles ------------------------------
    if (elect_one()) {
      int stage = 0, issued = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
        const int split = unit % p.splits, tile_w = unit / p.splits / p.tiles_t;
        const int end = k_begin(split + 1);
        for (int kb = k_begin(split); kb < end; ++kb) {
          if (!mbar_wait(w_empty + 8 * stage, phase ^ 1u, p.status, abort_flag)) { ok = false; break; }
          const uint32_t dst = base + stage * W_STAGE_BYTES, bar = w_full + 8 * stage;
          mbar_expect_tx(bar, W_STAGE_BYTES);
          tma_load_2d(dst, &map_w, bar, kb * BK, tile_w * BM);
          tma_load_2d(dst + W_STAGE_BYTES / 2, &map_w, bar, kb * BK + BK / 2, tile_w * BM);
          ++issued;
          if (++stage == S::W_STAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok || *abort_flag) {                // wait (bounded) for the copies already issued
        const int used = issued < S::W_STAGES ? issued : S::W_STAGES;
        for (int back = 1; back <= used; ++back) {
          int s = stage - back;
          uint32_t ph = phase;
          if (s < 0) { s += S::W_STAGES; ph ^= 1u; }
          const unsigned long long start = global_timer();
          while (!mbar_try_wait(w_full + 8 * s, ph) && global_timer() - start < 100000000ull) {}
        }
      }
    }
  } else if (warp == 3) {
    // ------------------------------ token tiles ------------------------------
    if (elect_one()) {
      int stage = 0, issued = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
        const int split = unit % p.splits, tile_t = unit / p.splits % p.tiles_t;
        const int end = k_begin(split + 1);
        for (int kb = k_begin(split); kb < end; ++kb) {
          if (!mbar_wait(x_empty + 8 * stage, phase ^ 1u, p.status, abort_flag)) { ok = false; break; }
          const uint32_t dst = x_base + stage * S::X_STAGE_BYTES, bar = x_full + 8 * stage;
          mbar_expect_tx(bar, S::X_STAGE_BYTES);
          // rows of a part beyond its M are the next part's: their columns of the product are never stored
#pragma unroll
          for (int part = 0; part < PARTS; ++part)
            tma_load_2d(dst + part * (S::X_STAGE_BYTES / PARTS), &map_x, bar, kb * BK, part * p.M + tile_t * BN);
          ++issued;
          if (++stage == S::X_STAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok || *abort_flag) {
        const int used = issued < S::X_STAGES ? issued : S::X_STAGES;
        for (int back = 1; back <= used; ++back) {
          int s = stage - back;
          uint32_t ph = phase;
          if (s < 0) { s += S::X_STAGES; ph ^= 1u; }
          const unsigned long long start = global_timer();
          while (!mbar_try_wait(x_full + 8 * s, ph) && global_timer() - start < 100000000ull) {}
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ products ------------------------------
    if (elect_one()) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      int xs = 0, as = 0, acc = 0;
      uint32_t x_phase = 0, a_phase = 0, d_phase = 0;
      bool ok = true;
      for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
        const int split = unit % p.splits;
        const int end = k_begin(split + 1);
        for (int kb = k_begin(split); kb < end; ++kb) {
          if (!mbar_wait(d_empty + 8 * acc, d_phase ^ 1u, p.status, abort_flag) || !mbar_wait(x_full + 8 * xs, x_phase, p.status, abort_flag) ||
              !mbar_wait(a_full + 8 * as, a_phase, p.status, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d = tmem + (uint32_t)(acc * BN), a = tmem + (uint32_t)(S::A_FIRST_COL + as * A_COLS);
          const uint64_t b = make_smem_desc(x_base + xs * S::X_STAGE_BYTES);
          // parts of (weight, token) from the smallest products to the largest: 0 high, 1 middle, 2 low
          constexpr int of_w[6] = {2, 0, 1, 1, 0, 0}, of_x[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
          for (int product = 0; product < 6; ++product)
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              mma_tmem_a(d, a + of_w[product] * (BK / 2) + k * (UMMA_K / 2),
                         b + ((of_x[product] * (S::X_STAGE_BYTES / PARTS) + k * UMMA_K * 2) >> 4), idesc, (product > 0 || k > 0) ? 1u : 0u);
          tc_commit(a_empty + 8 * as);
          tc_commit(x_empty + 8 * xs);
          tc_commit(d_full + 8 * acc);
          if (++as == S::A_STAGES) { as = 0; a_phase ^= 1u; }
          if (++xs == S::X_STAGES) { xs = 0; x_phase ^= 1u; }
          if (++acc == 2) { acc = 0; d_phase ^= 1u; }
        }
      }
    }
  } else if (warp >= 4 && warp < 4 + CONVERT_WARPS) {
    // ------------------------------ weights into their parts ------------------------------
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    int ws = 0, as = 0;
    uint32_t w_phase = 0, a_phase = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
      const int split = unit % p.splits;
      const int end = k_begin(split + 1);
      for (int kb = k_begin(split); kb < end; ++kb) {
        if (!mbar_wait(w_full + 8 * ws, w_phase, p.status, abort_flag) || !mbar_wait(a_empty + 8 * as, a_phase ^ 1u, p.status, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const unsigned char* src = generic + ws * W_STAGE_BYTES + row * 128;
        const uint32_t dst = tmem + lane_base + (uint32_t)(S::A_FIRST_COL + as * A_COLS);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t h[16], m[16], l[16];
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float4 v = *reinterpret_cast<const float4*>(src + half * (W_STAGE_BYTES / 2) + ((c ^ (row & 7)) << 4));
            split_pair(v.x, v.y, h[2 * c], m[2 * c], l[2 * c]);
            split_pair(v.z, v.w, h[2 * c + 1], m[2 * c + 1], l[2 * c + 1]);
          }
          tmem_store16(dst + half * 16, h);
          tmem_store16(dst + BK / 2 + half * 16, m);
          tmem_store16(dst + 2 * (BK / 2) + half * 16, l);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(w_empty + 8 * ws);
          mbar_arrive(a_full + 8 * as);
        }
        if (++ws == S::W_STAGES) { ws = 0; w_phase ^= 1u; }
        if (++as == S::A_STAGES) { as = 0; a_phase ^= 1u; }
      }
    }
  } else if (warp >= 8) {
    // ------------------------------ sums and epilogue ------------------------------
    const int quarter = warp & 3, c_first = ((warp - 8) >> 2) * COLS;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    int acc = 0;
    uint32_t d_phase = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
      const int split = unit % p.splits, rest = unit / p.splits;
      const int tile_t = rest % p.tiles_t, tile_w = rest / p.tiles_t;
      const int end = k_begin(split + 1);
      float sum[COLS];
#pragma unroll
      for (int c = 0; c < COLS; ++c) sum[c] = 0.0f;
      for (int kb = k_begin(split); kb < end; ++kb) {
        if (!mbar_wait(d_full + 8 * acc, d_phase, p.status, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t src = tmem + lane_base + (uint32_t)(acc * BN + c_first);
        if constexpr (COLS >= 16) {
#pragma unroll
          for (int c = 0; c < COLS; c += 16) {
            uint32_t r[16];
            tc_load16(src + c, r);
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[c + j] += __uint_as_float(r[j]);
          }
        } else {
          uint32_t r[8];
          tmem_load8(src, r);
#pragma unroll
          for (int j = 0; j < 8; ++j) sum[j] += __uint_as_float(r[j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(d_empty + 8 * acc);
        if (++acc == 2) { acc = 0; d_phase ^= 1u; }
      }
      if (!ok) break;
      const int n = tile_w * BM + quarter * 32 + lane, m0 = tile_t * BN + c_first;
      const bool n_ok = n < p.N;
      if (p.splits > 1) {
        float* dst = p.partial + ((size_t)split * p.M + m0) * p.N + n;
#pragma unroll
        for (int c = 0; c < COLS; ++c)
          if (n_ok && m0 + c < p.M) dst[(size_t)c * p.N] = sum[c];
        continue;
      }
      const float bias = p.bias != nullptr && n_ok ? p.bias[n] : 0.0f;
      const bool is_gated = p.epilogue == F32_SWIGLU || p.epilogue == F32_GLU_CLAMPED;
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        const int m = m0 + c;
        if (m >= p.M) continue;                // uniform over the warp
        const float v = (n_ok ? usual_or_chain(p, sum[c], m, n) : 0.0f) + bias;
        if (is_gated) {
          const float up = __shfl_down_sync(0xffffffffu, v, 1);      // N is even: an even row's partner exists
          if (n_ok && !(lane & 1)) p.out[(size_t)m * p.ldo + (n >> 1)] = gated(p, v, up);
        } else if (n_ok) {
          finish(p, v, m, n);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"((uint32_t)TMEM_COLS) : "memory");
  }
}

// ---- the cuts along k added in order, then the epilogue: a thread per pair of neighbouring weight rows ----
__global__ void __launch_bounds__(256) gemm_f32_combine_kernel(const F32GemmParams p) {
  pdl_trigger();
  const int m = blockIdx.y, n = 2 * ((int)blockIdx.x * 256 + (int)threadIdx.x);
  if (n >= p.N) return;
  const bool second = n + 1 < p.N;
  // the bias is there already (see split_rows_kernel)
  const float bias0 = p.bias ? p.bias[n] : 0.0f, bias1 = p.bias && second ? p.bias[n + 1] : 0.0f;
  pdl_wait();
  const float* src = p.partial + (size_t)m * p.N + n;
  const size_t plane = (size_t)p.M * p.N;
  const bool pairs = (p.N & 1) == 0;           // then every row of the partial sums starts on an even float
  float a = 0.0f, b = 0.0f;
  for (int s0 = 0; s0 < p.splits; s0 += 4) {
    float2 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float* at = src + (size_t)(s0 + i) * plane;
      if (s0 + i >= p.splits) v[i] = make_float2(0.0f, 0.0f);
      else if (pairs) v[i] = *reinterpret_cast<const float2*>(at);
      else v[i] = make_float2(at[0], second ? at[1] : 0.0f);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (s0 + i >= p.splits) break;
      a += v[i].x;
      b += v[i].y;
    }
  }
  a = usual_or_chain(p, a, m, n) + bias0;
  if (second) b = usual_or_chain(p, b, m, n + 1) + bias1;
  if (p.epilogue == F32_SWIGLU || p.epilogue == F32_GLU_CLAMPED) {
    p.out[(size_t)m * p.ldo + (n >> 1)] = gated(p, a, b);
    return;
  }
  finish(p, a, m, n);
  if (second) finish(p, b, m, n + 1);
}

// ---- host side ----
// The cut along k: a rule on N and K alone, so that a row's sums never depend on the step it is in.  One token tile of few
// weight tiles leaves SMs idle, so the cuts fill whole waves of 148; a cut costs its partial sums (about four k-blocks' time).
constexpr int SMS = 148;
int cuts_of(int N, int K) {
  const int tiles = (N + BM - 1) / BM, k_blocks = (K + BK - 1) / BK;
  if (tiles >= 2 * SMS) return 1;
  long long best = -1;
  int splits = 1;
  for (int s = 1; s <= 16 && s * 4 <= k_blocks; ++s) {
    const long long waves = ((long long)tiles * s + SMS - 1) / SMS;
    const long long cost = waves * ((k_blocks + s - 1) / s + 4);
    if (best < 0 || cost < best) { best = cost; splits = s; }
  }
  return splits;
}
// Tokens per pass over the weights: the scratch memory of a pass (parts and partial sums) stays within 64 MB
// each, and 512 tokens multiply long enough (0.7 ms a layer of 233 M weights) that reading the weights again hides.
constexpr long long PASS_FLOATS = 16 << 20;
int panel_of(int N, int K, int splits) {
  int panel = 512;
  const long long Kp = (K + 7) / 8 * 8;
  while (panel > 128 && (panel * Kp * PARTS / 2 > PASS_FLOATS || (splits > 1 && (long long)splits * panel * N > PASS_FLOATS))) panel /= 2;
  return panel;
}
long long plane_floats(int rows, int K) { return ((long long)PARTS * rows * ((K + 7) / 8 * 8) / 2 + 3) / 4 * 4; }

// Where the kernel is used: contractions long and wide enough to fill its 128 x 64 tiles several times over (below, the
// launches and the chain copy - split - product - sum cost more than the FMA chain: 64 x 176 takes 8.4 us there),
// by N and K alone, and weights that TMA can copy.  At 1,536 x 1,536 it is 8.9 against 97 us already.
bool f32_tc_takes(const void* w, long long ldw, int N, int K) {
  return N >= 512 && K >= 512 && (ldw * 4) % 16 == 0 && (uintptr_t)w % 16 == 0;
}

template <int BN>
int launch_product(const CUtensorMap& map_w, const CUtensorMap& map_x, const F32GemmParams& p, cudaStream_t stream) {
  cudaError_t err = cudaFuncSetAttribute(gemm_f32_tcgen05_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape<BN>::SMEM);
  const long long units = (long long)p.tiles_w * p.tiles_t * p.splits;
  if (err == cudaSuccess)
    err = tge_launch(gemm_f32_tcgen05_kernel<BN>, dim3((unsigned)(units < tge_sm_count() ? units : tge_sm_count())), dim3(THREADS), Shape<BN>::SMEM, stream,
                     map_w, map_x, p);
  if (err != cudaSuccess) {
    tge_set_error("gemm_f32_tcgen05: launch failed: %s", cudaGetErrorString(err));
    cudaGetLastError();
    return -2;
  }
  return 0;
}

}  // namespace

// Floats of scratch memory for M tokens; negative: not a shape for this kernel.
TGE_API long long tge_gemm_f32_tcgen05_scratch_floats(const void* w, long long ldw, int M, int N, int K) {
  if (M <= 0 || !f32_tc_takes(w, ldw, N, K)) return TGE_UNSUPPORTED;
  const int splits = cuts_of(N, K), panel = panel_of(N, K, splits);
  const int rows = M < panel ? M : panel;
  return plane_floats(rows, K) + (splits > 1 ? (long long)splits * rows * N : 0);
}

// x [M, K] (row stride ldx), w [N, K] (row stride ldw), out as the epilogue says, all float32; epilogues of gemm_simt.cu.
TGE_API int tge_gemm_f32_tcgen05(const float* x, long long ldx, const float* w, long long ldw, const float* bias, float* out, long long ldo,
                                 int M, int N, int K, int epilogue, float* scratch, long long scratch_floats, float alpha, int act_from,
                                 int* status, cudaStream_t stream) {
  TGE_REQUIRE(epilogue >= F32_STORE && epilogue <= F32_GLU_CLAMPED, "gemm: unknown epilogue %d", epilogue);
  TGE_REQUIRE((epilogue != F32_SWIGLU && epilogue != F32_GLU_CLAMPED) || N % 2 == 0, "gemm: the gated epilogue needs an even number of weight rows, got %d", N);
  TGE_REQUIRE(ldx >= K && ldw >= K, "gemm: row strides %lld/%lld shorter than K=%d", ldx, ldw, K);
  const long long need = tge_gemm_f32_tcgen05_scratch_floats(w, ldw, M, N, K);
  if (need < 0) return TGE_UNSUPPORTED;
  TGE_REQUIRE(scratch != nullptr && scratch_floats >= need && (uintptr_t)scratch % 16 == 0, "gemm: %lld floats of aligned scratch memory needed", need);
  CUtensorMap map_w, map_x;
  int rc = make_rows_map(&map_w, w, N, K, ldw, BM, true, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, "gemm_f32_tcgen05");
  if (rc != 0) return rc;
  const int splits = cuts_of(N, K), panel = panel_of(N, K, splits), Kp = (K + 7) / 8 * 8;
  int launched = 0;
  for (int m0 = 0; m0 < M; m0 += panel) {
    const int rows = M - m0 < panel ? M - m0 : panel;
    F32GemmParams p;
    p.x = x + (size_t)m0 * ldx; p.w = w; p.ldx = ldx; p.ldw = ldw; p.M = rows; p.N = N; p.K = K;
    p.k_blocks = (K + BK - 1) / BK; p.splits = splits; p.tiles_w = (N + BM - 1) / BM;
    p.epilogue = epilogue; p.act_from = act_from; p.alpha = alpha; p.bias = bias;
    p.out = out + (size_t)m0 * ldo; p.ldo = ldo; p.status = status;
    __nv_bfloat16* planes = reinterpret_cast<__nv_bfloat16*>(scratch);
    p.partial = scratch + plane_floats(rows, K);
    const int vec = (uintptr_t)p.x % 16 == 0 && (ldx * 4) % 16 == 0;
    cudaError_t err = tge_launch(split_rows_kernel, dim3((Kp / 8 + 255) / 256, rows), dim3(256), 0, stream, p.x, ldx, planes, rows, K, Kp, vec);
    if (err != cudaSuccess) {
      tge_set_error("gemm_f32_tcgen05: launch failed: %s", cudaGetErrorString(err));
      cudaGetLastError();
      return -2;
    }
    const int bn = rows <= 16 ? 16 : rows <= 32 ? 32 : rows <= 64 ? 64 : 128;
    rc = make_rows_map(&map_x, planes, (long long)PARTS * rows, K, Kp, bn, false, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, "gemm_f32_tcgen05");
    if (rc != 0) return rc;
    p.tiles_t = (rows + bn - 1) / bn;
    rc = bn == 16 ? launch_product<16>(map_w, map_x, p, stream) : bn == 32 ? launch_product<32>(map_w, map_x, p, stream)
         : bn == 64 ? launch_product<64>(map_w, map_x, p, stream) : launch_product<128>(map_w, map_x, p, stream);
    if (rc != 0) return rc;
    launched += 2;
    if (splits > 1) {
      err = tge_launch(gemm_f32_combine_kernel, dim3((N + 511) / 512, rows), dim3(256), 0, stream, p);
      if (err != cudaSuccess) {
        tge_set_error("gemm_f32_tcgen05: launch failed: %s", cudaGetErrorString(err));
        cudaGetLastError();
        return -2;
      }
      ++launched;
    }
  }
  return tge_launched("gemm_f32_tcgen05", launched);
}
