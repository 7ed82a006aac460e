// Matrix product on the CUDA cores with float32 accumulation: out = x . w^T (+ epilogue).
//
// This is the float32 path's product (plain FFMA, no reduced-precision matrix
// mode) for weights smaller than 512 x 512 or not aligned for TMA (the others go
// to gemm_f32_tcgen05.cu) and the fallback of the bfloat16 path for shapes the
// tensor-core kernel refuses.  Every output element is accumulated over k in ascending
// order by one thread, so its value depends on neither the tile it falls in
// nor on what else is in the batch.  The formula is the reference's
// row-times-vector product (src/tensor/reference.cpp:29-45) followed by the
// separate bias loop (src/models/qwen2.cpp:2062-2068), SiLU gate
// (src/cpu/scalar/norm_rope_scalar.cpp:43-51) or residual add
// (src/models/qwen2.cpp:2101-2103).
#include "common.cuh"

enum GemmEpilogue : int {
  GEMM_STORE = 0,      // out[m, n] = acc + bias[n], run dtype
  GEMM_STORE_F32 = 1,  // out[m, n] = acc + bias[n], float32
  GEMM_ADD_F32 = 2,    // residual[m, n] += acc + bias[n], float32 in place
  GEMM_SWIGLU = 3,     // w rows interleaved (gate_i, up_i): out[m, i] = silu(g) * u, run dtype
  GEMM_GELU = 4,       // out[m, n] = gelu(acc + bias[n]) for n >= act_from (plain below it), run dtype; the erf form
  GEMM_GELU_TANH = 5,  // the same with the tanh approximation 0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3)))
  GEMM_GLU_CLAMPED = 6,  // gated like 3 with both halves clamped at L = alpha: min(g, L) sigmoid(1.702 min(g, L)) (clamp(u, -L, L) + 1)
};
// `alpha` multiplies acc + bias in the three plain epilogues (store, store float32, add): a residual multiplier or a
// logit scale costs no pass of its own.

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename T>
__device__ __forceinline__ void load4(const T* base, size_t row_stride, int row, int rows, int k, int K, bool vec,
                                      float out[4]);

template <>
__device__ __forceinline__ void load4<float>(const float* base, size_t row_stride, int row, int rows, int k, int K,
                                             bool vec, float out[4]) {
  if (row < rows && vec && k + 3 < K) {
    const float4 v = *reinterpret_cast<const float4*>(base + (size_t)row * row_stride + k);
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) out[i] = (row < rows && k + i < K) ? base[(size_t)row * row_stride + k + i] : 0.0f;
}

template <>
__device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* base, size_t row_stride, int row, int rows,
                                                     int k, int K, bool vec, float out[4]) {
  if (row < rows && vec && k + 3 < K) {
    const uint2 raw = *reinterpret_cast<const uint2*>(base + (size_t)row * row_stride + k);
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&raw.x);
    const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
    out[0] = __low2float(a); out[1] = __high2float(a); out[2] = __low2float(b); out[3] = __high2float(b);
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    out[i] = (row < rows && k + i < K) ? __bfloat162float(base[(size_t)row * row_stride + k + i]) : 0.0f;
}

template <typename T>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const T* __restrict__ x, size_t ldx, const T* __restrict__ w,
                                                        size_t ldw, const float* __restrict__ bias, void* out,
                                                        size_t ldo, int M, int N, int K, int epilogue, int vec,
                                                        float alpha, int act_from) {
  __shared__ float xs[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int load_row = tid >> 2, load_k = (tid & 3) * 4;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    float xv[4], wv[4];
    load4<T>(x, ldx, m0 + load_row, M, k0 + load_k, K, vec != 0, xv);
    load4<T>(w, ldw, n0 + load_row, N, k0 + load_k, K, vec != 0, wv);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      xs[load_k + i][load_row] = xv[i];
      ws[load_k + i][load_row] = wv[i];
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = xs[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = ws[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
  }

#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
    if (epilogue == GEMM_SWIGLU || epilogue == GEMM_GLU_CLAMPED) {
#pragma unroll
      for (int j = 0; j < TN; j += 2) {
        const int n = n0 + tx * TN + j;
        if (n + 1 >= N) continue;
        float g = acc[i][j], u = acc[i][j + 1];
        if (bias) { g += bias[n]; u += bias[n + 1]; }
        if (epilogue == GEMM_GLU_CLAMPED) {
          g = fminf(g, alpha);
          u = fminf(fmaxf(u, -alpha), alpha) + 1.0f;
          g *= 1.702f;                                   // a = (g / 1.702) sigmoid(g) u below
          u *= 1.0f / 1.702f;
        }
        const float a = g / (1.0f + expf(-g)) * u;
        reinterpret_cast<T*>(out)[(size_t)m * ldo + (n >> 1)] = from_float<T>(a);
      }
      continue;
    }
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * TN + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      if (epilogue >= GEMM_GELU) {
        if (n >= act_from) v = epilogue == GEMM_GELU ? gelu_erf(v) : gelu_tanh(v);
        reinterpret_cast<T*>(out)[(size_t)m * ldo + n] = from_float<T>(v);
        continue;
      }
      v *= alpha;
      if (epilogue == GEMM_STORE) {
        reinterpret_cast<T*>(out)[(size_t)m * ldo + n] = from_float<T>(v);
      } else if (epilogue == GEMM_STORE_F32) {
        reinterpret_cast<float*>(out)[(size_t)m * ldo + n] = v;
      } else {
        reinterpret_cast<float*>(out)[(size_t)m * ldo + n] += v;
      }
    }
  }
}

// Few tokens, float32, aligned rows: the same chain of FMAs per element, organised for latency.
//
// The tile above waits for its loads in each of K / 16 rounds and has 64 x 64 elements whatever M is: a tiny model's product
// of 3 rows took 8.4 us at K = 64 and 20 us at K = 384, nearly all of it round trips to L2.  Here a block owns 16 x 32 elements
// (a lane per weight row, a warp per four tokens), so a product spreads over four times the SMs and more, and
// four blocks of 64 k are on their way at once by cp.async.  Measured (B200), the tile above and this kernel, us, at 4 tokens:
// 128 x 64 6.3 -> 2.3, 512 x 96 8.5 -> 2.8, 64 x 176 12.9 -> 3.8, 96 x 256 17.8 -> 5.0, 500 x 3,000 181 -> 48; 512 tokens
// of 384 x 96 4.9 and of 500 x 3,000 104.  (Weights asked for ahead of the wait for the kernel in front were 0.2 to 0.4 us faster, and
// wrong where that kernel had written them.)
constexpr int SKINNY_M = 16, SKINNY_N = 32, SKINNY_K = 64, SKINNY_PITCH = SKINNY_K + 4, SKINNY_STAGES = 4;
constexpr int SKINNY_STAGE = (SKINNY_M + SKINNY_N) * SKINNY_PITCH;

__device__ __forceinline__ void copy16(float* dst, const float* src, bool live) {
  const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
  const int bytes = live ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to), "l"(src), "r"(bytes) : "memory");
}

__global__ void __launch_bounds__(128) gemm_skinny_kernel(const float* x, size_t ldx, const float* w, size_t ldw,
                                                          const float* bias, float* __restrict__ out, size_t ldo, int M,
                                                          int N, int K, int epilogue, float alpha, int act_from) {
  extern __shared__ __align__(16) float ring[];
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = blockIdx.y * SKINNY_M, n0 = blockIdx.x * SKINNY_N;
  const int blocks = (K + SKINNY_K - 1) / SKINNY_K;
  auto fetch_w = [&](int kb) {
    float* stage = ring + (kb % SKINNY_STAGES) * SKINNY_STAGE + SKINNY_M * SKINNY_PITCH;
#pragma unroll
    for (int i = 0; i < SKINNY_N * SKINNY_K / 4 / 128; ++i) {
      const int c = tid + i * 128, row = c >> 4, k = kb * SKINNY_K + (c & 15) * 4;
      const bool live = n0 + row < N && k < K;
      copy16(stage + row * SKINNY_PITCH + (c & 15) * 4, live ? w + (size_t)(n0 + row) * ldw + k : w, live);
    }
  };
  auto fetch_x = [&](int kb) {
    float* stage = ring + (kb % SKINNY_STAGES) * SKINNY_STAGE;
#pragma unroll
    for (int i = 0; i < SKINNY_M * SKINNY_K / 4 / 128; ++i) {
      const int c = tid + i * 128, row = c >> 4, k = kb * SKINNY_K + (c & 15) * 4;
      const bool live = m0 + row < M && k < K;
      copy16(stage + row * SKINNY_PITCH + (c & 15) * 4, live ? x + (size_t)(m0 + row) * ldx + k : x, live);
    }
  };
  auto commit = [] { asm volatile("cp.async.commit_group;\n" ::: "memory"); };
  const int n = n0 + lane;
  pdl_wait();                                           // weights and bias may be the kernel in front's result as well
  const float add = bias != nullptr && n < N ? bias[n] : 0.0f;
#pragma unroll
  for (int kb = 0; kb < SKINNY_STAGES - 1; ++kb) {
    if (kb < blocks) {
      fetch_w(kb);
      fetch_x(kb);
    }
    commit();
  }
  float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  for (int kb = 0; kb < blocks; ++kb) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(SKINNY_STAGES - 2) : "memory");
    __syncthreads();                                    // everyone's part of block kb is there, and block kb - 1 is read
    if (kb + SKINNY_STAGES - 1 < blocks) {
      fetch_w(kb + SKINNY_STAGES - 1);
      fetch_x(kb + SKINNY_STAGES - 1);
    }
    commit();
    if (m0 + warp * 4 >= M) continue;                   // uniform over the warp
    const float* xs = ring + (kb % SKINNY_STAGES) * SKINNY_STAGE + warp * 4 * SKINNY_PITCH;
    const float* ws = ring + (kb % SKINNY_STAGES) * SKINNY_STAGE + (SKINNY_M + lane) * SKINNY_PITCH;
    const int held = min(K - kb * SKINNY_K, SKINNY_K);  // a multiple of four
#pragma unroll 4
    for (int k = 0; k < held; k += 4) {
      const float4 b = *reinterpret_cast<const float4*>(ws + k);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(xs + i * SKINNY_PITCH + k);
        acc[i] = fmaf(a.x, b.x, acc[i]);
        acc[i] = fmaf(a.y, b.y, acc[i]);
        acc[i] = fmaf(a.z, b.z, acc[i]);
        acc[i] = fmaf(a.w, b.w, acc[i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + warp * 4 + i;
    if (m >= M) break;
    float v = acc[i];
    if (bias) v += add;
    if (epilogue == GEMM_SWIGLU || epilogue == GEMM_GLU_CLAMPED) {
      float u = __shfl_down_sync(0xffffffffu, v, 1);    // an even lane's neighbour holds the row above
      if (epilogue == GEMM_GLU_CLAMPED) {
        v = fminf(v, alpha);
        u = fminf(fmaxf(u, -alpha), alpha) + 1.0f;
        v *= 1.702f;
        u *= 1.0f / 1.702f;
      }
      if (!(lane & 1) && n + 1 < N) out[(size_t)m * ldo + (n >> 1)] = v / (1.0f + expf(-v)) * u;
      continue;
    }
    if (n >= N) continue;
    float* dst = out + (size_t)m * ldo + n;
    if (epilogue >= GEMM_GELU) {
      if (n >= act_from) v = epilogue == GEMM_GELU ? gelu_erf(v) : gelu_tanh(v);
      *dst = v;
    } else if (epilogue == GEMM_ADD_F32) {
      *dst = __fadd_rn(*dst, __fmul_rn(v, alpha));      // rounded twice, as above
    } else {
      *dst = v * alpha;
    }
  }
}

}  // namespace

// x [M, K] (row stride ldx), w [N, K] (row stride ldw), both in the run dtype;
// bias float32 [N] or null; out as the epilogue says (row stride ldo, in elements).
TGE_API int tge_gemm_simt(const void* x, long long ldx, const void* w, long long ldw, const float* bias, void* out,
                          long long ldo, int M, int N, int K, int is_bf16, int epilogue, float alpha, int act_from,
                          cudaStream_t stream) {
  TGE_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
  TGE_REQUIRE(epilogue >= GEMM_STORE && epilogue <= GEMM_GLU_CLAMPED, "gemm: unknown epilogue %d", epilogue);
  TGE_REQUIRE((epilogue != GEMM_SWIGLU && epilogue != GEMM_GLU_CLAMPED) || N % 2 == 0, "gemm: the gated epilogue needs an even number of weight rows, got %d", N);
  TGE_REQUIRE(ldx >= K && ldw >= K, "gemm: row strides %lld/%lld shorter than K=%d", ldx, ldw, K);
  if (M == 0) return 0;
  const size_t elem = is_bf16 ? 2 : 4;
  const size_t align = is_bf16 ? 8 : 16;
  const int vec = (K % 4 == 0) && ((ldx * elem) % align == 0) && ((ldw * elem) % align == 0) &&
                  ((uintptr_t)x % align == 0) && ((uintptr_t)w % align == 0);
  // Float32 rows that 16-byte copies can read: up to 64 tokens always, more while the small tiles of all of them fit the
  // chip at once (then latency counts, not the number of shared-memory reads per FMA: 1,000 tokens of 512 x 96, beyond
  // the line, take 8.5 us either way).
  const long long small_tiles = (long long)((N + SKINNY_N - 1) / SKINNY_N) * ((M + SKINNY_M - 1) / SKINNY_M);
  if (!is_bf16 && vec && (M <= 64 || small_tiles <= 4 * tge_sm_count())) {
    constexpr int smem = SKINNY_STAGES * SKINNY_STAGE * (int)sizeof(float);
    cudaError_t err = cudaFuncSetAttribute(gemm_skinny_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err == cudaSuccess)
      err = tge_launch(gemm_skinny_kernel, dim3((N + SKINNY_N - 1) / SKINNY_N, (M + SKINNY_M - 1) / SKINNY_M), dim3(128), smem, stream,
                       (const float*)x, (size_t)ldx, (const float*)w, (size_t)ldw, bias, (float*)out, (size_t)ldo, M, N, K, epilogue,
                       alpha, act_from);
    if (err != cudaSuccess) {
      tge_set_error("gemm_simt: launch failed: %s", cudaGetErrorString(err));
      cudaGetLastError();
      return -2;
    }
    return tge_launched("gemm_simt", 1);
  }
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (is_bf16)
    gemm_simt_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)x, (size_t)ldx,
                                                              (const __nv_bfloat16*)w, (size_t)ldw, bias, out,
                                                              (size_t)ldo, M, N, K, epilogue, vec, alpha, act_from);
  else
    gemm_simt_kernel<float><<<grid, 256, 0, stream>>>((const float*)x, (size_t)ldx, (const float*)w, (size_t)ldw,
                                                      bias, out, (size_t)ldo, M, N, K, epilogue, vec, alpha, act_from);
  return tge_launched("gemm_simt", 1);
}
