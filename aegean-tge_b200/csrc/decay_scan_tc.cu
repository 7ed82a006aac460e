// The decayed linear attention of long portions on the 5th-generation tensor cores: S_t = c S_(t-1) + k_t v_t^T, o_t = S_t^T q_t,
// chunks of 128 tokens, a block per (head, chunk).
//
// sequence_mix.cu's chunked kernels run the recurrence's products on the FMA pipes, and their blocks, 64 state columns each, form
// the scores of a chunk anew: 2,048 tokens of 28 heads of 128 took 337 us for the readout and 150 for the states before it,
// 45 % of the FMA pipes' rate.  The products are contractions of 64 to 128, so they belong on the tensor cores; what is float32
// (q, k, the state, the decayed scores, activated values) goes there as a sum of three bfloat16 numbers, six of the nine products of
// such sums (three where the other side is bfloat16 already, as plain values are), the smallest first, in accumulators that
// no more than 64 numbers of the contraction enter, added up in registers: the error against float64 is below that of
// the FMA chains.  Three launches:
//   1. decay_chunk_state_kernel: a chunk's own contribution to the state, sum_j c^(n-1-j) k_j v_j^T, into carry[chunk];
//   2. decay_segment_carry_kernel of sequence_mix.cu: carry[chunk] <- the state the chunk starts from, the last state to its slot;
//   3. decay_chunk_readout_kernel: o = c^(t+1) q S0 + (c^(t-j) q k^T below the diagonal) v.
// A number that is not finite, or too large for its high part, makes NaN of every product it meets: as an input its split is
// infinity - infinity, zeros above the diagonal times infinity reach earlier tokens, and so does a score that overflows.  A chunk one of
// whose results is not finite is therefore computed by the formulas themselves.
// Numbers below about 1e-33 keep fewer than 24 bits in their parts; beside anything larger in the same sum that is nothing.
// First operands lie in tensor memory (a lane per token or state row), second operands in shared memory, split on their way in.
// Measured (B200, 2,048 tokens, 28 heads of 128): states 150 -> 57 us, readout 337 -> 91 us; 14 heads of 64 with activated values of
// 128: 108 -> 33 us and 137 -> 45 us.  Error against float64 2.85e-7 -> 1.7e-7, activated 1.97e-7 -> 1.44e-7.
// One block holds an SM (all of its tensor memory), and its phases follow one another, so it is bound by their latencies: with sixteen
// warps in place of eight (in a prompt of 2,048, us a layer) states 52 -> 45, readout 84 -> 75, activated 31 -> 23 and 37 -> 33.
#include "tcgen05_ptx.cuh"

namespace {

constexpr int CHUNK = 128;               // tokens per chunk = lanes of tensor memory
constexpr int THREADS = 512;             // four warps per 32-lane quarter, a quarter of the columns each
constexpr int PARTS = THREADS / 128;
constexpr int ACC_COLS = 256;            // two accumulators of up to 128 columns
constexpr int OPERAND_BYTES = 128 * 128 * 2;   // one part of a second operand of up to 128 x 128
constexpr int TMEM_COLS = 512;

struct ScanTcParams {
  const __nv_bfloat16* rows;
  long long ld;
  const float* prepared;     // [tokens][heads][2][dim]: q and k as the recurrence takes them
  const float* decay;
  const int* q_start;
  float* carry;              // [chunks][heads][dim][vdim]
  float* out;                // [tokens][heads * vdim]
  int* status;
  int v_off, heads, num_seqs, shortest, activation, aligned;
};

__device__ __forceinline__ uint64_t mn_desc(uint32_t addr, uint32_t block_stride) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(block_stride >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// NaN from the first infinity or NaN on, else zero
template <int N>
__device__ __forceinline__ float not_finite(const float v[N]) {
  float poison = 0.0f;
#pragma unroll
  for (int i = 0; i < N; ++i) poison = fmaf(v[i], 0.0f, poison);
  return poison;
}
__device__ __forceinline__ float silu_of(float z) { return z / (1.0f + expf(-z)); }

// Which tokens block `piece` works on: chunks are counted over the step's portions of p.shortest tokens and more, 32 requests
// at a time, one to a lane (one after the other, every block of a step of many requests waited for that many loads).
__device__ __forceinline__ bool find_chunk(const ScanTcParams& p, int piece, int& first, int& count) {
  const int lane = threadIdx.x & 31;
  for (int s0 = 0; s0 < p.num_seqs; s0 += 32) {
    const int s = s0 + lane;
    const int begin = s < p.num_seqs ? p.q_start[s] : 0, length = s < p.num_seqs ? p.q_start[s + 1] - begin : 0;
    const int mine = length >= p.shortest ? (length + CHUNK - 1) / CHUNK : 0;
    int upto = mine;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
      const int other = __shfl_up_sync(0xffffffffu, upto, offset);
      if (lane >= offset) upto += other;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, piece < upto);
    if (hit != 0) {
      const int at = __ffs(hit) - 1, place = (piece - __shfl_sync(0xffffffffu, upto - mine, at)) * CHUNK;
      first = __shfl_sync(0xffffffffu, begin, at) + place;
      count = min(CHUNK, __shfl_sync(0xffffffffu, length, at) - place);
      return true;
    }
    piece -= __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}

// Eight numbers, split, as 16-byte pieces of the three parts of a second operand: row `row` of 128 bytes in the 64-number block
// `block` of `block_rows` rows, piece `piece` (of 8) in the row, swizzled.
__device__ __forceinline__ void store_parts(unsigned char* base, int block, int block_rows, int row, int piece, const float v[8], int parts) {
  uint4 h, m, l;
  split_pair(v[0], v[1], h.x, m.x, l.x);
  split_pair(v[2], v[3], h.y, m.y, l.y);
  split_pair(v[4], v[5], h.z, m.z, l.z);
  split_pair(v[6], v[7], h.w, m.w, l.w);
  unsigned char* at = base + (block * block_rows + row) * 128 + ((piece ^ (row & 7)) << 4);
  *reinterpret_cast<uint4*>(at) = h;
  if (parts == 3) {
    *reinterpret_cast<uint4*>(at + OPERAND_BYTES) = m;
    *reinterpret_cast<uint4*>(at + 2 * OPERAND_BYTES) = l;
  }
}

// The chunk's values [token][column] as a second operand whose contiguous direction is the column: blocks of 64 columns, a row of
// 128 bytes per token.  Plain values are bfloat16 (one part), activated ones float32 (three).
template <int VDIM>
__device__ __forceinline__ void load_values(const ScanTcParams& p, unsigned char* base, int first, int count, int head, int tid) {
#pragma unroll 2
  for (int e = tid; e < CHUNK * VDIM / 8; e += THREADS) {
    const int t = e / (VDIM / 8), c = (e % (VDIM / 8)) * 8;
    float v[8];
    const __nv_bfloat16* src = p.rows + (size_t)(first + t) * p.ld + p.v_off + head * VDIM + c;
    if (t >= count) {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = 0.0f;
    } else if (p.aligned) {
      const uint4 raw = *reinterpret_cast<const uint4*>(src);
      const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = __bfloat162float(src[i]);
    }
    if (p.activation) {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = silu_of(v[i]);
    }
    store_parts(base, c >> 6, CHUNK, t, (c & 63) >> 3, v, p.activation ? 3 : 1);
  }
}

// One value as the products take it.
template <int VDIM>
__device__ __forceinline__ float value_at(const ScanTcParams& p, int token, int head, int c) {
  const float v = __bfloat162float(p.rows[(size_t)token * p.ld + p.v_off + head * VDIM + c]);
  return p.activation ? silu_of(v) : v;
}

// 32 bytes, one sector, in one store: lanes write rows of their own, and 16-byte stores would fill each sector in two
__device__ __forceinline__ void store8(float* dst, const float v[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]),
               "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}

// 32 numbers of this thread's lane as columns [col, col + 16) of each part of a first operand (parts `part_cols` columns apart).
__device__ __forceinline__ void store_lane32(uint32_t taddr, int part_cols, const float v[32]) {
  uint32_t h[16], m[16], l[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) split_pair(v[2 * i], v[2 * i + 1], h[i], m[i], l[i]);
  tmem_store16(taddr, h);
  tmem_store16(taddr + part_cols, m);
  tmem_store16(taddr + 2 * part_cols, l);
}

// Products of the parts over a contraction of K numbers, 64 to an accumulator; one thread issues them.
// `a`: first operand in tensor memory (K / 2 columns per part); `b0`: descriptor of the second operand's high part; the descriptor
// moves by b_step (16-byte units) per 16 numbers and b_block more per 64 (0 where blocks follow one another).
template <int K>
__device__ __forceinline__ void issue_products(uint32_t acc, int acc_stride, uint32_t a, uint64_t b0, uint32_t idesc, uint32_t b_step,
                                               uint32_t b_half, bool b_split) {
  // (first, second operand's part) from the smallest products to the largest: 0 high, 1 middle, 2 low
  constexpr int of_a[6] = {2, 0, 1, 1, 0, 0}, of_b[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
  for (int half = 0; half < K / 64; ++half) {
    bool begun = false;
#pragma unroll
    for (int product = 0; product < 6; ++product) {
      if (!b_split && of_b[product] != 0) continue;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        mma_tmem_a(acc + half * acc_stride, a + of_a[product] * (K / 2) + half * 32 + k * 8,
                   b0 + of_b[product] * (OPERAND_BYTES >> 4) + half * b_half + k * b_step, idesc, begun ? 1u : 0u);
        begun = true;
      }
    }
  }
}

// this thread's lane of COLS accumulator columns from `col`, both halves of the contraction added
template <int COLS, int HALVES>
__device__ __forceinline__ void read_sums(uint32_t taddr, int acc_stride, float out[COLS]) {
#pragma unroll
  for (int c = 0; c < COLS; c += 16) {
    uint32_t r[16];
    tc_load16(taddr + c, r);
#pragma unroll
    for (int j = 0; j < 16; ++j) out[c + j] = __uint_as_float(r[j]);
    if (HALVES == 2) {
      tc_load16(taddr + acc_stride + c, r);
#pragma unroll
      for (int j = 0; j < 16; ++j) out[c + j] += __uint_as_float(r[j]);
    }
  }
}

__device__ __forceinline__ uint32_t product_idesc(int n, bool b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn_major ? 1u << 16 : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// What both kernels begin and end with: barrier, tensor memory, the powers of the head's decay.
struct BlockSetup {
  uint32_t tmem, base;
  unsigned char* generic;
};
__device__ __forceinline__ BlockSetup set_up(unsigned char* smem_raw, uint32_t* tmem_slot, int* abort_word, uint32_t bar, float* powers, float c,
                                             int tid, int warp) {
  BlockSetup s;
  s.base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  s.generic = smem_raw + (s.base - smem_u32(smem_raw));
  if (tid == 0) {
    mbar_init(bar, 1);
    *abort_word = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid <= CHUNK) powers[tid] = (float)pow((double)c, (double)tid);       // each power rounded once
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  s.tmem = *tmem_slot;
  pdl_trigger();                           // tensor memory is held: a block of the next kernel can at worst wait for it
  pdl_wait();
  return s;
}
__device__ __forceinline__ void tear_down(uint32_t tmem, int warp) {
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"((uint32_t)TMEM_COLS) : "memory");
  }
}
// before the products: this thread's operands in shared and tensor memory are there for the tensor core
__device__ __forceinline__ void operands_ready() {
  asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
}

// ---- a chunk's own contribution to the state: lanes are the state's rows, the contraction runs over the tokens ----
template <int DIM, int VDIM>
__global__ void __launch_bounds__(THREADS, 1) decay_chunk_state_kernel(const ScanTcParams p) {
  constexpr int COLS = VDIM / PARTS;       // result columns of a warp
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  __shared__ __align__(8) uint64_t done_bar;
  __shared__ float powers[CHUNK + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = uniform_warp_index();
  const int head = blockIdx.x, piece = blockIdx.y;
  int first = 0, count = 0;
  if (!find_chunk(p, piece, first, count)) return;
  const uint32_t bar = smem_u32(&done_bar);
  const BlockSetup s = set_up(smem_raw, &tmem_slot, &abort_word, bar, powers, p.decay[head], tid, warp);
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t a = s.tmem + ACC_COLS;
  const int part = warp >> 2, row = (warp & 3) * 32 + lane;
  // first operand: k_j[row] c^(n-1-j), this warp's 32 of the 128 tokens
  {
    const int t0 = part * (CHUNK / PARTS);
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int t = t0 + i;
      v[i] = row < DIM && t < count ? p.prepared[((size_t)(first + t) * p.heads + head) * 2 * DIM + DIM + row] : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] *= powers[max(count - 1 - (t0 + i), 0)];
    store_lane32(a + lane_base + t0 / 2, CHUNK / 2, v);
  }
  load_values<VDIM>(p, s.generic, first, count, head, tid);
  operands_ready();
  if (warp == 0) {
    if (elect_one()) {
      issue_products<CHUNK>(s.tmem, 128, a, mn_desc(s.base, CHUNK * 128), product_idesc(VDIM, true), (16 * 128) >> 4, (64 * 128) >> 4, p.activation != 0);
      tc_commit(bar);
    }
    __syncwarp();
  }
  const bool ok = mbar_wait(bar, 0, p.status, &abort_word);
  tc_fence_after();
  float* dst = p.carry + (((size_t)piece * p.heads + head) * DIM + row) * VDIM + part * COLS;
  float sums[COLS];
  read_sums<COLS, 2>(s.tmem + lane_base + part * COLS, 128, sums);
  if (__syncthreads_or(!(not_finite<COLS>(sums) == 0.0f))) {
    for (int c = 0; c < COLS && row < DIM; ++c) {
      float sum = 0.0f;
      for (int j = 0; j < count; ++j)
        sum = fmaf(p.prepared[((size_t)(first + j) * p.heads + head) * 2 * DIM + DIM + row] * powers[count - 1 - j],
                   value_at<VDIM>(p, first + j, head, part * COLS + c), sum);
      dst[c] = sum;
    }
  } else if (ok && row < DIM) {
#pragma unroll
    for (int c = 0; c < COLS; c += 8) store8(dst + c, sums + c);
  }
  tear_down(s.tmem, warp);
}

// ---- the readout of a chunk: lanes are its tokens ----
template <int DIM, int VDIM>
__global__ void __launch_bounds__(THREADS, 1) decay_chunk_readout_kernel(const ScanTcParams p) {
  constexpr int COLS = VDIM / PARTS;       // result columns of a warp
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  __shared__ __align__(8) uint64_t done_bar;
  __shared__ float powers[CHUNK + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = uniform_warp_index();
  const int head = blockIdx.x, piece = blockIdx.y;
  int first = 0, count = 0;
  if (!find_chunk(p, piece, first, count)) return;
  const uint32_t bar = smem_u32(&done_bar);
  const BlockSetup s = set_up(smem_raw, &tmem_slot, &abort_word, bar, powers, p.decay[head], tid, warp);
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t a = s.tmem + ACC_COLS;
  const int part = warp >> 2, row = (warp & 3) * 32 + lane;
  unsigned char* second = s.generic;                          // the state, then the keys
  unsigned char* values = s.generic + 3 * OPERAND_BYTES;
  const float* own = p.prepared + ((size_t)(first + min(row, count - 1)) * p.heads + head) * 2 * DIM + part * 32;
  // the token's query, 32 numbers to a warp
  if (part * 32 < DIM) {
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      const float4 q = row < count ? *reinterpret_cast<const float4*>(own + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[i] = q.x; v[i + 1] = q.y; v[i + 2] = q.z; v[i + 3] = q.w;
    }
    store_lane32(a + lane_base + part * 16, DIM / 2, v);
  }
  // the state the chunk starts from, [dim][vdim]: contiguous along vdim
  const float* state = p.carry + ((size_t)piece * p.heads + head) * DIM * VDIM;
#pragma unroll 2
  for (int e = tid; e < DIM * VDIM / 8; e += THREADS) {
    const int i = e / (VDIM / 8), c = (e % (VDIM / 8)) * 8;
    const float4 x = *reinterpret_cast<const float4*>(state + (size_t)i * VDIM + c), y = *reinterpret_cast<const float4*>(state + (size_t)i * VDIM + c + 4);
    const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
    store_parts(second, c >> 6, DIM, i, (c & 63) >> 3, v, 3);
  }
  operands_ready();
  if (warp == 0) {
    if (elect_one()) {
      issue_products<DIM>(s.tmem, 128, a, mn_desc(s.base, DIM * 128), product_idesc(VDIM, true), (16 * 128) >> 4, (64 * 128) >> 4, true);
      tc_commit(bar);
    }
    __syncwarp();
  }
  load_values<VDIM>(p, values, first, count, head, tid);      // while the products run
  bool ok = mbar_wait(bar, 0, p.status, &abort_word);
  tc_fence_after();
  float o[COLS];
  read_sums<COLS, DIM / 64>(s.tmem + lane_base + part * COLS, 128, o);
  {
    const float carried = powers[row + 1];
#pragma unroll
    for (int c = 0; c < COLS; ++c) o[c] *= carried;
  }
  // the keys [token][dim] over the state, contiguous along the contraction
#pragma unroll 2
  for (int e = tid; e < CHUNK * DIM / 8; e += THREADS) {
    const int t = e / (DIM / 8), i = (e % (DIM / 8)) * 8;
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (t < count) {
      const float* src = p.prepared + ((size_t)(first + t) * p.heads + head) * 2 * DIM + DIM + i;
      const float4 x = *reinterpret_cast<const float4*>(src), y = *reinterpret_cast<const float4*>(src + 4);
      v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
    }
    store_parts(second, i >> 6, CHUNK, t, (i & 63) >> 3, v, 3);
  }
  operands_ready();
  if (warp == 0) {
    if (elect_one()) {
      issue_products<DIM>(s.tmem, 128, a, make_smem_desc(s.base), product_idesc(CHUNK, false), 32 >> 4, (CHUNK * 128) >> 4, true);
      tc_commit(bar);
    }
    __syncwarp();
  }
  ok = mbar_wait(bar, 1, p.status, &abort_word) && ok;
  tc_fence_after();
  // decayed scores of this token with keys 32 part ... 32 part + 31, as first operand of the next product (over the query)
  {
    float v[32];
    read_sums<32, DIM / 64>(s.tmem + lane_base + part * 32, 128, v);
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int gap = row - (part * 32 + j);
      v[j] = gap >= 0 ? v[j] * powers[max(gap, 0)] : 0.0f;
    }
    store_lane32(a + lane_base + part * 16, CHUNK / 2, v);
  }
  operands_ready();
  if (warp == 0) {
    if (elect_one()) {
      issue_products<CHUNK>(s.tmem, 128, a, mn_desc(s.base + 3 * OPERAND_BYTES, CHUNK * 128), product_idesc(VDIM, true), (16 * 128) >> 4,
                            (64 * 128) >> 4, p.activation != 0);
      tc_commit(bar);
    }
    __syncwarp();
  }
  ok = mbar_wait(bar, 0, p.status, &abort_word) && ok;
  tc_fence_after();
#pragma unroll
  for (int c = 0; c < COLS; c += 16) {
    float more[16];
    read_sums<16, 2>(s.tmem + lane_base + part * COLS + c, 128, more);
#pragma unroll
    for (int j = 0; j < 16; ++j) o[c + j] += more[j];
  }
  float* dst = p.out + (size_t)(first + row) * p.heads * VDIM + (size_t)head * VDIM + part * COLS;
  if (__syncthreads_or(!(not_finite<COLS>(o) == 0.0f))) {
    const float* q = p.prepared + ((size_t)(first + row) * p.heads + head) * 2 * DIM;
    for (int c = 0; c < COLS && row < count; ++c) {
      float sum = 0.0f;
      for (int i = 0; i < DIM; ++i) sum = fmaf(q[i], state[(size_t)i * VDIM + part * COLS + c], sum);
      sum *= powers[row + 1];
      for (int j = 0; j <= row; ++j) {
        const float* k = p.prepared + ((size_t)(first + j) * p.heads + head) * 2 * DIM + DIM;
        float score = 0.0f;
        for (int i = 0; i < DIM; ++i) score = fmaf(q[i], k[i], score);
        sum = fmaf(score * powers[row - j], value_at<VDIM>(p, first + j, head, part * COLS + c), sum);
      }
      dst[c] = sum;
    }
  } else if (ok && row < count) {
#pragma unroll
    for (int c = 0; c < COLS; c += 8) store8(dst + c, o + c);
  }
  tear_down(s.tmem, warp);
}

template <int DIM, int VDIM>
int run(const ScanTcParams& p, int pieces, bool readout, cudaStream_t stream) {
  // values: one part, three when activated; the readout has the state or the keys in front of them
  const size_t smem = 1024 + (size_t)((readout ? 3 : 0) + (p.activation ? 3 : 1)) * OPERAND_BYTES;
  auto kernel = readout ? decay_chunk_readout_kernel<DIM, VDIM> : decay_chunk_state_kernel<DIM, VDIM>;
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 1024 + 6 * OPERAND_BYTES);
  if (err == cudaSuccess) {
    err = tge_launch(kernel, dim3(p.heads, pieces), dim3(THREADS), smem, stream, p);
  }
  if (err != cudaSuccess) {
    tge_set_error("decay_scan_tc: launch failed: %s", cudaGetErrorString(err));
    cudaGetLastError();
    return -2;
  }
  return 1;
}

}  // namespace

// Tokens per chunk, or 0: key and value sizes the kernels are not built for.
int decay_tc_chunk(int dim, int vdim) { return (dim == 64 || dim == 128) && (vdim == 64 || vdim == 128) ? CHUNK : 0; }

// One of the two launches around decay_segment_carry_kernel, for portions of `shortest` tokens and more; `pieces` is an upper bound of
// their chunks.  Returns 1 or an error.
int launch_decay_tc(const void* rows, long long ld, const float* prepared, int v_off, int heads, int dim, int vdim, int activation,
                    const float* decay, const int* q_start, float* carry, float* out, int num_seqs, int shortest, int pieces, bool readout,
                    int* status, cudaStream_t stream) {
  ScanTcParams p;
  p.rows = (const __nv_bfloat16*)rows; p.ld = ld; p.prepared = prepared; p.decay = decay; p.q_start = q_start; p.carry = carry; p.out = out;
  p.status = status; p.v_off = v_off; p.heads = heads; p.num_seqs = num_seqs; p.shortest = shortest; p.activation = activation;
  p.aligned = ((uintptr_t)(p.rows + v_off) % 16 == 0) && (ld * 2) % 16 == 0;
  if (dim == 64) return vdim == 64 ? run<64, 64>(p, pieces, readout, stream) : run<64, 128>(p, pieces, readout, stream);
  return vdim == 64 ? run<128, 64>(p, pieces, readout, stream) : run<128, 128>(p, pieces, readout, stream);
}
