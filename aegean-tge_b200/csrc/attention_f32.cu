// Paged causal attention of the float32 path, float32 arithmetic, keys in tiles shared by a block's rows.
//
// attention_simt.cu gives a warp one (token, head) and walks the keys one at a time: a key costs a chain of loads, a
// butterfly over the warp and two exponentials, about 1.4 us a key and nothing to hide it behind, and
// every head of a group fetches the keys for itself.  Bound by that chain, not by bytes: a step of 8 requests of 1,000
// tokens at 28 heads over 4 of 128 took 1,403 us a layer, against 5 us for its 33 MB of keys and values.  Here
//   * a block owns up to 16, 32 or 64 rows, (query, head of the group) pairs of one request and kv head, and 64 keys at a time
//     lie in shared memory for all of them, the next 64 under way (cp.async, two buffers);
//   * 16 x 16 threads hold the scores as a matrix product does (rows by 4 keys each, paired float32 FMAs over the head),
//     so a tile costs one round of maxima, exponentials and sums, not 64;
//   * where the rows are few the keys are cut into runs, each a block of its own, merged by a second kernel.
// Measured in place (B200, float32): that step 1,403 -> 25 us a layer, 512 prompt tokens 639 -> 122 us; 100 prompt tokens at 12
// heads over 2 of 128 56 -> 15 us alone, three single tokens at 4 heads of 16 18 -> 3 us, 7 prompt tokens at 28 heads 5.8 -> 4.9; one to three
// tokens at a request's very beginning lose (28 heads: one 2.3 -> 3.3, three 3.7 -> 4.6: a block's copies and barriers cost more there than they save).
//
// A row's result depends only on its own keys, not on the batch, on how its request was cut into portions or on which of
// the three row counts serves it: keys go in tiles of 64 and runs of RUN_KEYS that start at multiples of these positions, a
// tile that a row does not see changes nothing of its state, every sum over keys or numbers of a head has one order, and
// the runs are merged in order by the same code inside a block and in the merging kernel.
#include "common.cuh"

namespace {

constexpr int TILE_KEYS = 64;
constexpr int RUN_KEYS = 256;          // four tiles: long enough that merging costs little, short enough to fill the chip
constexpr int THREADS = 256;
constexpr int MAX_ROWS_PER_THREAD = 4;

struct F32AttnParams {
  const float* q;
  const float* k_pages;
  const float* v_pages;
  const int* block_table;
  const int* q_start;
  const int* start_pos;
  const int* positions;
  float* out;
  float* partial;          // [runs][tokens][heads][head size + 2]: sums, then maximum and denominator
  int* status;
  int q_stride, out_stride, max_pages, num_pages, page_size, page_shift, num_seqs, tokens, heads, kv_heads, group, window, runs;
  float scale;
};

__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
struct Masked { static constexpr bool value = true; };
struct NoMask { static constexpr bool value = false; };
template <int N>
struct Groups { static constexpr int value = N; };
// 16 bytes into shared memory, zeros when `bytes` is 0
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// One run's state joins the state of the runs before it; the factors for the sums are returned.
__device__ __forceinline__ void merge_run(float& m_all, float& l_all, float m_run, float l_run, float& keep, float& take) {
  const float m_new = fmaxf(m_all, m_run);
  const float base = m_new == -INFINITY ? 0.0f : m_new;
  keep = expf(m_all - base);
  take = expf(m_run - base);
  l_all = __fmaf_rn(l_run, take, __fmul_rn(l_all, keep));
  m_all = m_new;
}
__device__ __forceinline__ float merge_sum(float all, float run, float keep, float take) {
  return __fmaf_rn(run, take, __fmul_rn(all, keep));
}

template <int HD, int TR>
constexpr size_t f32_attn_smem() {
  return sizeof(float) * ((size_t)16 * TR * (HD + 4) + 2 * (size_t)TILE_KEYS * (HD + 4) + 2 * (size_t)TILE_KEYS * HD +
                          (size_t)16 * TR * (TILE_KEYS + 4));
}

// Rows r = ty + 16 i of the block, keys tx + 16 j of the tile, columns of the output in groups of VEC from tx * VEC.
template <int HD, int TR>
__global__ void __launch_bounds__(THREADS) attention_f32_kernel(const F32AttnParams p) {
  constexpr int ROWS = 16 * TR, KP = HD + 4, PP = TILE_KEYS + 4;
  constexpr int COLS = HD / 16, VEC = COLS < 4 ? COLS : 4, GROUPS = COLS / VEC;
  extern __shared__ __align__(16) float smem_f32[];
  float* q_s = smem_f32;                               // [ROWS][KP]
  float* k_s = q_s + ROWS * KP;                        // [2][TILE_KEYS][KP]
  float* v_s = k_s + 2 * TILE_KEYS * KP;               // [2][TILE_KEYS][HD]
  float* p_s = v_s + 2 * TILE_KEYS * HD;               // [ROWS][PP]
  __shared__ int tile_info[2];
  pdl_trigger();
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int kvh = blockIdx.y, run_only = (int)blockIdx.z;
  const int bq = ROWS / p.group;                       // queries per block
  if (tid < 32) {
    // which request and which of its query blocks: 32 requests at a time, one to a lane (a loop of dependent loads by one
    // thread took 0.3 us a request); later queries first, they see the most keys
    int remaining = (int)(gridDim.x - 1 - blockIdx.x), seq = -1, block = 0;
    for (int s0 = 0; s0 < p.num_seqs && seq < 0; s0 += 32) {
      const int s = s0 + tid;
      const int mine = s < p.num_seqs ? (p.q_start[s + 1] - p.q_start[s] + bq - 1) / bq : 0;
      int upto = mine;
#pragma unroll
      for (int offset = 1; offset < 32; offset <<= 1) {
        const int other = __shfl_up_sync(0xffffffffu, upto, offset);
        if (tid >= offset) upto += other;
      }
      const unsigned hit = __ballot_sync(0xffffffffu, remaining < upto);
      if (hit != 0) {
        const int lane = __ffs(hit) - 1;
        seq = s0 + lane;
        block = remaining - __shfl_sync(0xffffffffu, upto - mine, lane);
      } else {
        remaining -= __shfl_sync(0xffffffffu, upto, 31);
      }
    }
    if (tid == 0) {
      tile_info[0] = seq;
      tile_info[1] = block;
    }
  }
  __syncthreads();
  const int seq = tile_info[0];
  if (seq < 0) return;
  const int q_first = tile_info[1] * bq;
  const int q_begin = p.q_start[seq];
  const int q_count = min(bq, p.q_start[seq + 1] - q_begin - q_first);
  const int pos0 = p.start_pos[seq] + q_first;
  const int pos_last = pos0 + q_count - 1;
  // the keys that some row of this block sees, cut down to this block's run if the runs are blocks of their own
  int lo = p.window > 0 ? max(pos0 - p.window + 1, 0) : 0;
  int hi = pos_last + 1;
  const bool one_run = p.runs > 1;
  if (one_run) {
    lo = max(lo, run_only * RUN_KEYS);
    hi = min(hi, (run_only + 1) * RUN_KEYS);
    if (lo >= hi) return;
  }
  pdl_wait();

  int row_pos[TR], row_first[TR];
  bool row_ok[TR];
#pragma unroll
  for (int i = 0; i < TR; ++i) {
    const int r = ty + 16 * i;
    row_ok[i] = r < q_count * p.group;
    row_pos[i] = row_ok[i] ? pos0 + r / p.group : -1;          // a row that is none sees no key
    row_first[i] = p.window > 0 ? max(row_pos[i] - p.window + 1, 0) : 0;
  }
#pragma unroll
  for (int r = tid >> 5; r < ROWS; r += THREADS / 32) {
    const int qi = r / p.group, head = kvh * p.group + r - qi * p.group;
    const float* src = p.q + (size_t)(q_begin + q_first + qi) * p.q_stride + (size_t)head * HD;
#pragma unroll
    for (int d = tid & 31; d < HD; d += 32) q_s[r * KP + d] = qi < q_count ? src[d] : 0.0f;
  }

  const int first_tile = lo / TILE_KEYS, last_tile = (hi - 1) / TILE_KEYS;
  const int* table = p.block_table + (size_t)seq * p.max_pages;
  auto fetch = [&](int tile) {
    const int buffer = tile & 1;
    const uint32_t k_dst = (uint32_t)__cvta_generic_to_shared(k_s + buffer * TILE_KEYS * KP);
    const uint32_t v_dst = (uint32_t)__cvta_generic_to_shared(v_s + buffer * TILE_KEYS * HD);
#pragma unroll 8
    for (int c = tid; c < TILE_KEYS * (HD / 4); c += THREADS) {
      const int key = c / (HD / 4), part = c % (HD / 4);
      const int pos = tile * TILE_KEYS + key;
      const int page_index = p.page_shift >= 0 ? pos >> p.page_shift : pos / p.page_size;
      const int slot = pos - page_index * p.page_size;
      int page = -1;
      if (pos >= lo && pos < hi) {
        page = page_index < p.max_pages ? table[page_index] : -1;
        if (page < 0 || page >= p.num_pages) {
          if (part == 0) atomicOr(p.status, TGE_STATUS_BAD_PAGE);
          page = -1;
        }
      }
      const size_t offset = page < 0 ? 0 : (((size_t)page * p.kv_heads + kvh) * p.page_size + slot) * HD + part * 4;
      const int bytes = page < 0 ? 0 : 16;
      copy16(k_dst + (uint32_t)(key * KP + part * 4) * 4, p.k_pages + offset, bytes);
      copy16(v_dst + (uint32_t)(key * HD + part * 4) * 4, p.v_pages + offset, bytes);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  bool any_row = false;
#pragma unroll
  for (int i = 0; i < TR; ++i) any_row = any_row || row_ok[i];
  const bool idle = !__any_sync(0xffffffffu, any_row);      // a warp without rows only copies

  float acc[TR][COLS], all[TR][COLS];
  float m_run[TR], l_run[TR], m_all[TR], l_all[TR];
#pragma unroll
  for (int i = 0; i < TR; ++i) {
    m_run[i] = m_all[i] = -INFINITY;
    l_run[i] = l_all[i] = 0.0f;
#pragma unroll
    for (int c = 0; c < COLS; ++c) acc[i][c] = all[i][c] = 0.0f;
  }

  fetch(first_tile);
  for (int tile = first_tile; tile <= last_tile; ++tile) {
    if (tile < last_tile) {
      fetch(tile + 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const float* kt = k_s + (tile & 1) * TILE_KEYS * KP;
    const float* vt = v_s + (tile & 1) * TILE_KEYS * HD;
    const int k0 = tile * TILE_KEYS;
    if (!idle) {
    const int held = min(hi - k0, TILE_KEYS);            // keys of the tile that any row sees lie before this
    // scores: four partial sums per pair (numbers 0, 1, 2, 3 mod 4 of the head), added pairwise at the end
    uint64_t dot[TR][4][2];
#pragma unroll
    for (int i = 0; i < TR; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) dot[i][j][0] = dot[i][j][1] = 0ull;
    auto add_scores = [&](auto groups) {
      constexpr int J = decltype(groups)::value;
#pragma unroll 4
      for (int d = 0; d < HD; d += 4) {
        ulonglong2 qv[TR], kv[J];
#pragma unroll
        for (int i = 0; i < TR; ++i) qv[i] = *reinterpret_cast<const ulonglong2*>(q_s + (ty + 16 * i) * KP + d);
#pragma unroll
        for (int j = 0; j < J; ++j) kv[j] = *reinterpret_cast<const ulonglong2*>(kt + (tx + 16 * j) * KP + d);
#pragma unroll
        for (int i = 0; i < TR; ++i)
#pragma unroll
          for (int j = 0; j < J; ++j) {
            dot[i][j][0] = fma2(qv[i].x, kv[j].x, dot[i][j][0]);
            dot[i][j][1] = fma2(qv[i].y, kv[j].y, dot[i][j][1]);
          }
      }
    };
    if (held <= 16) add_scores(Groups<1>());             // the rest of the tile is masked
    else add_scores(Groups<4>());
    bool whole = true;                                  // every row of this thread sees every key of the tile
#pragma unroll
    for (int i = 0; i < TR; ++i) {
      whole = whole && (!row_ok[i] || (k0 >= row_first[i] && k0 + TILE_KEYS - 1 <= row_pos[i]));
      float s[4], mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float a, b, c, d;
        unpack2(dot[i][j][0], a, b);
        unpack2(dot[i][j][1], c, d);
        const int kpos = k0 + tx + 16 * j;
        const bool seen = kpos <= row_pos[i] && kpos >= row_first[i];
        s[j] = seen ? __fmul_rn((a + b) + (c + d), p.scale) : -INFINITY;
        mx = fmaxf(mx, s[j]);
      }
#pragma unroll
      for (int offset = 8; offset > 0; offset >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, offset));
      const float m_new = fmaxf(m_run[i], mx);
      const float base = m_new == -INFINITY ? 0.0f : m_new;
      const float corr = expf(m_run[i] - base);
      float sum = 0.0f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float w = expf(s[j] - base);
        p_s[(ty + 16 * i) * PP + tx + 16 * j] = w;
        sum += w;
      }
#pragma unroll
      for (int offset = 8; offset > 0; offset >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, offset);
      l_run[i] = __fmaf_rn(l_run[i], corr, sum);
      m_run[i] = m_new;
#pragma unroll
      for (int c = 0; c < COLS; ++c) acc[i][c] = __fmul_rn(acc[i][c], corr);
    }
    __syncwarp();                                       // a row's weights are written and read by the same half warp
    auto add_values = [&](auto masked) {
#pragma unroll 2
      for (int j = 0; j < held; j += 4) {
        float4 w[TR];
#pragma unroll
        for (int i = 0; i < TR; ++i) w[i] = *reinterpret_cast<const float4*>(p_s + (ty + 16 * i) * PP + j);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          const float* vrow = vt + (j + jj) * HD;
          const int kpos = k0 + j + jj;
#pragma unroll
          for (int g = 0; g < GROUPS; ++g) {
            float v[VEC];
            if constexpr (VEC == 4) {
              const float4 t = *reinterpret_cast<const float4*>(vrow + g * 64 + tx * 4);
              v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
            } else {
#pragma unroll
              for (int e = 0; e < VEC; ++e) v[e] = vrow[tx * VEC + e];
            }
#pragma unroll
            for (int i = 0; i < TR; ++i) {
              const float wi = jj == 0 ? w[i].x : jj == 1 ? w[i].y : jj == 2 ? w[i].z : w[i].w;
              // a key the row does not see adds nothing, whatever its value holds (0 x infinity is not 0)
              if (decltype(masked)::value && !(kpos <= row_pos[i] && kpos >= row_first[i])) continue;
#pragma unroll
              for (int e = 0; e < VEC; ++e) acc[i][g * VEC + e] = __fmaf_rn(wi, v[e], acc[i][g * VEC + e]);
            }
          }
        }
      }
    };
    if (__all_sync(0xffffffffu, whole)) add_values(NoMask());
    else add_values(Masked());
    }
    if (tile == last_tile || (tile + 1) % (RUN_KEYS / TILE_KEYS) == 0) {
      // the run ends: its state joins the earlier runs' (in a block of its own it is written as it is)
      if (!one_run) {
#pragma unroll
        for (int i = 0; i < TR; ++i) {
          float keep, take;
          merge_run(m_all[i], l_all[i], m_run[i], l_run[i], keep, take);
#pragma unroll
          for (int c = 0; c < COLS; ++c) {
            all[i][c] = merge_sum(all[i][c], acc[i][c], keep, take);
            acc[i][c] = 0.0f;
          }
          m_run[i] = -INFINITY;
          l_run[i] = 0.0f;
        }
      }
    }
    __syncthreads();                                    // the buffer may be filled again
  }

#pragma unroll
  for (int i = 0; i < TR; ++i) {
    if (!row_ok[i]) continue;
    const int r = ty + 16 * i;
    const int token = q_begin + q_first + r / p.group, head = kvh * p.group + r % p.group;
    if (one_run) {
      float* dst = p.partial + (((size_t)run_only * p.tokens + token) * p.heads + head) * (HD + 2);
#pragma unroll
      for (int c = 0; c < COLS; ++c) dst[(c / VEC) * 64 + tx * VEC + c % VEC] = acc[i][c];
      if (tx == 0) {
        dst[HD] = m_run[i];
        dst[HD + 1] = l_run[i];
      }
    } else {
      const float inv = l_all[i] > 0.0f ? 1.0f / l_all[i] : 0.0f;
      float* dst = p.out + (size_t)token * p.out_stride + (size_t)head * HD;
#pragma unroll
      for (int c = 0; c < COLS; ++c) dst[(c / VEC) * 64 + tx * VEC + c % VEC] = __fmul_rn(all[i][c], inv);
    }
  }
}

// The runs of a row in order: one block per (token, run of heads), one thread per number of a head.
template <int HD>
__global__ void __launch_bounds__(128) attention_f32_merge_kernel(const F32AttnParams p) {
  pdl_trigger();
  const int token = blockIdx.x;
  const int head = blockIdx.y * (128 / HD) + (int)threadIdx.x / HD, d = (int)threadIdx.x % HD;
  if (head >= p.heads) return;
  const int pos = p.positions[token];
  const int first = p.window > 0 ? max(pos - p.window + 1, 0) / RUN_KEYS : 0;
  const int last = min(pos / RUN_KEYS, p.runs - 1);
  pdl_wait();
  float m_all = -INFINITY, l_all = 0.0f, all = 0.0f;
  const size_t stride = (size_t)p.tokens * p.heads * (HD + 2);
  const float* src = p.partial + (size_t)first * stride + ((size_t)token * p.heads + head) * (HD + 2);
  for (int run = first; run <= last; run += 4) {
    float m[4], l[4], a[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (run + i > last) break;
      a[i] = src[i * stride + d];
      m[i] = src[i * stride + HD];
      l[i] = src[i * stride + HD + 1];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (run + i > last) break;
      float keep, take;
      merge_run(m_all, l_all, m[i], l[i], keep, take);
      all = merge_sum(all, a[i], keep, take);
    }
    src += 4 * stride;
  }
  const float inv = l_all > 0.0f ? 1.0f / l_all : 0.0f;
  p.out[(size_t)token * p.out_stride + (size_t)head * HD + d] = __fmul_rn(all, inv);
}

// Row blocks of a step whose portions are at most max_q_len long; never fewer than there are.
int row_blocks(int tokens, int num_seqs, int max_q_len, int bq) {
  if (max_q_len <= bq) return num_seqs;                 // at most one block per request
  return (int)(((long long)tokens + (long long)num_seqs * (bq - 1)) / bq);
}

// Sixteen rows to a block where a request brings no more (single tokens bring group rows each), thirty-two where it brings no more or where
// blocks of that many still find an SM each, 64 otherwise: a block computes all its rows, in use or not, and while SMs are idle
// smaller blocks finish sooner (us, 64 / 32 rows, 28 heads over 4 of 128: three prompt tokens 6.6 / 4.6,
// seven 7.5 / 4.9, forty 11.5 / 8.1, a hundred 20.7 / 15.0; sixteen at 3,000 find no room: 47 / 66).
int rows_per_thread(int tokens, int num_seqs, int max_q_len, int max_ctx_len, int kv_heads, int group) {
  const long long rows = group * (long long)max_q_len, runs = (max_ctx_len + RUN_KEYS - 1) / RUN_KEYS;
  if (rows <= 16) return 1;
  if (rows <= 32 || (group <= 32 && row_blocks(tokens, num_seqs, max_q_len, 32 / group) * kv_heads * runs <= tge_sm_count())) return 2;
  return MAX_ROWS_PER_THREAD;
}

// Runs that are blocks of their own, 1: none.  Only where the row blocks alone leave the chip half empty, and where the
// states stay within 64 MB: a long portion deep in a long context has keys enough for every block.
constexpr long long MAX_STATE_FLOATS = 16 << 20;
int runs_of(int tokens, int num_seqs, int max_q_len, int max_ctx_len, int kv_heads, int group, int head_dim) {
  const int bq = 16 * rows_per_thread(tokens, num_seqs, max_q_len, max_ctx_len, kv_heads, group) / group;
  const long long blocks = (long long)row_blocks(tokens, num_seqs, max_q_len, bq) * kv_heads;
  const int runs = (max_ctx_len + RUN_KEYS - 1) / RUN_KEYS;
  const bool fits = (long long)runs * tokens * kv_heads * group * (head_dim + 2) <= MAX_STATE_FLOATS;
  return blocks >= 2 * tge_sm_count() || !fits ? 1 : runs;
}

template <int HD, int TR>
int launch(const F32AttnParams& p, int max_q_len, cudaStream_t stream) {
  constexpr size_t smem = f32_attn_smem<HD, TR>();
  static_assert(smem <= 227 * 1024, "a block's tiles fit its shared memory");
  cudaError_t err = cudaFuncSetAttribute(attention_f32_kernel<HD, TR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (err == cudaSuccess)
    err = tge_launch(attention_f32_kernel<HD, TR>, dim3(row_blocks(p.tokens, p.num_seqs, max_q_len, 16 * TR / p.group), p.kv_heads, p.runs),
                     dim3(THREADS), smem, stream, p);
  if (err == cudaSuccess && p.runs > 1)
    err = tge_launch(attention_f32_merge_kernel<HD>, dim3(p.tokens, (p.heads + 128 / HD - 1) / (128 / HD)), dim3(128), 0, stream, p);
  if (err != cudaSuccess) {
    tge_set_error("attention_f32: launch failed: %s", cudaGetErrorString(err));
    cudaGetLastError();
    return -2;
  }
  return tge_launched("attention_f32", p.runs > 1 ? 2 : 1);
}

template <int HD>
int launch_rows(const F32AttnParams& p, int max_q_len, int max_ctx_len, cudaStream_t stream) {
  const int rows = rows_per_thread(p.tokens, p.num_seqs, max_q_len, max_ctx_len, p.kv_heads, p.group);
  return rows == 1 ? launch<HD, 1>(p, max_q_len, stream) : rows == 2 ? launch<HD, 2>(p, max_q_len, stream) : launch<HD, MAX_ROWS_PER_THREAD>(p, max_q_len, stream);
}

bool f32_attention_takes(int heads, int kv_heads, int head_dim) {
  return kv_heads > 0 && heads > 0 && heads % kv_heads == 0 && heads / kv_heads <= 16 * MAX_ROWS_PER_THREAD && kv_heads <= 65535 &&
         (head_dim == 16 || head_dim == 32 || head_dim == 64 || head_dim == 128);
}

}  // namespace

// Floats of scratch memory the runs' states take (0: none), or a negative code for shapes the kernel does not take.
TGE_API long long tge_attention_f32_scratch_floats(int tokens, int num_seqs, int max_q_len, int max_ctx_len, int heads, int kv_heads,
                                                   int head_dim) {
  if (!f32_attention_takes(heads, kv_heads, head_dim) || tokens <= 0 || num_seqs <= 0 || max_q_len <= 0 || max_ctx_len <= 0)
    return TGE_UNSUPPORTED;
  const int runs = runs_of(tokens, num_seqs, max_q_len, max_ctx_len, kv_heads, heads / kv_heads, head_dim);
  return runs > 1 ? (long long)runs * tokens * heads * (head_dim + 2) : 0;
}

// Causal attention over pages of float32 keys and values of the same size (16, 32, 64 or 128), whole or within a window;
// what else attention_simt.cu knows (sinks, biases, gates, pooled blocks, kept first tokens) is left to it.
TGE_API int tge_attention_f32(const float* q, int q_stride, const float* k_pages, const float* v_pages, const int* block_table,
                              int max_pages, int num_pages, int page_size, const int* q_start, const int* start_pos,
                              const int* positions, int num_seqs, int max_q_len, int max_ctx_len, float* out, int out_stride,
                              int tokens, int heads, int kv_heads, int head_dim, float scale, int window, float* scratch,
                              long long scratch_floats, int* status, cudaStream_t stream) {
  if (tokens == 0) return 0;
  TGE_REQUIRE(page_size > 0 && max_pages > 0 && num_pages > 0 && window >= 0, "attention: bad page geometry or window");
  const long long need = tge_attention_f32_scratch_floats(tokens, num_seqs, max_q_len, max_ctx_len, heads, kv_heads, head_dim);
  if (need < 0 || (uintptr_t)k_pages % 16 != 0 || (uintptr_t)v_pages % 16 != 0) return TGE_UNSUPPORTED;
  TGE_REQUIRE(scratch == nullptr || scratch_floats >= need, "attention: the runs need %lld floats of scratch memory", need);
  F32AttnParams p;
  p.q = q; p.k_pages = k_pages; p.v_pages = v_pages; p.block_table = block_table; p.q_start = q_start; p.start_pos = start_pos;
  p.positions = positions; p.out = out; p.partial = scratch; p.status = status;
  p.q_stride = q_stride; p.out_stride = out_stride; p.max_pages = max_pages; p.num_pages = num_pages; p.page_size = page_size;
  p.page_shift = (page_size & (page_size - 1)) == 0 ? __builtin_ctz((unsigned)page_size) : -1;
  p.num_seqs = num_seqs; p.tokens = tokens; p.heads = heads; p.kv_heads = kv_heads; p.group = heads / kv_heads; p.window = window;
  p.scale = scale;
  // without scratch memory every block walks its runs itself, to the same bits
  p.runs = scratch != nullptr ? runs_of(tokens, num_seqs, max_q_len, max_ctx_len, kv_heads, p.group, head_dim) : 1;
  switch (head_dim) {
    case 16: return launch_rows<16>(p, max_q_len, max_ctx_len, stream);
    case 32: return launch_rows<32>(p, max_q_len, max_ctx_len, stream);
    case 64: return launch_rows<64>(p, max_q_len, max_ctx_len, stream);
    default: return launch_rows<128>(p, max_q_len, max_ctx_len, stream);
  }
}
