// Causal attention over a cache of unquantised rows (T: bfloat16 or float):
//   llmopt_row_attention_{bf16,f32}
// A sequence's token p sits in pool row slots[sequence row][p]; a pool row holds, per attention layer, the
// kv_heads key vectors (size dim) and value vectors (size vdim, which may differ).  The rows of the step's
// own tokens are in the pool already.  Row t of a sequence sees keys 0 .. past + t; with a `window` only the
// last `window` of them (its own included) and the first `keep_first` of the sequence.  With `softcap` a score
// becomes softcap * tanh(score / softcap).  With `sink` the softmax denominator counts one more score of zero that
// has no value.  With `gate_stride` the read-out is multiplied by the sigmoid of the row's gate columns.
// Queries and gates are read where the projections left them: row stride, first column.
//
// Kernels behind the names:
//  * bf16, at most 16 (query head, token) rows per key/value head (decode): split over the keys;
//    the query heads of a group ride in the 16 rows of one MMA tile, four warps walk over 16-key tiles
//    with private cp.async rings.  The last CTA of a (sequence, key/value head) to arrive merges the
//    splits in split order.
//  * bf16, more rows (prompts): 64 query tokens of one head per CTA, 64- or 32-key tiles double-buffered with
//    cp.async, online softmax in fp32, P rounded to bfloat16 for P V.  Where windowed prompts leave the chip idle three groups
//    of warps share a CTA's keys.
//  * fp32, and head sizes that are no whole 16-byte vectors: one CTA per (row, head), whose warps split the keys, or, with many
//    rows, one warp.
#include <type_traits>

#include "element.cuh"

namespace llmopt {

uint32_t* context_device_error(Context* ctx);

namespace {

struct RowAttentionParams {
  uint32_t sequences, tokens, heads, kv_heads, dim, vdim;
  uint32_t token_stride, key_offset, value_offset;  // in elements
  uint32_t table_stride, table_rows, pool_rows;
  uint32_t sink, splits;
  float scale, softcap;        // 0: scores are not capped
  uint32_t window, keep_first; // 0: no window
  uint32_t query_stride, query_column, gate_stride, gate_column;  // in elements; gate_stride 0: no gate
  uint32_t weights32;  // softmax weights meet the values in 32 bits (two bfloat16 parts), not rounded to bfloat16
  bool extended() const { return weights32 || window || softcap > 0.0f || gate_stride; }
};

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLowest = -1.0e30f;
constexpr float kBoundedCap = 40.0f;  // e^40 and e^-40, and sums of many of them, are ordinary fp32 numbers

struct KeyRows {  // rows of one sequence
  const uint32_t* slots;
  uint32_t limit, pool_rows;
  // What the table says about key `position`, without waiting for it, and the pool row that this is; an index outside the table or
  // the pool reads row 0 and is reported.
  __device__ __forceinline__ uint32_t listed(uint32_t position) const { return position < limit ? slots[position] : pool_rows; }
  __device__ __forceinline__ uint32_t checked(uint32_t slot, uint32_t* error_word) const {
    if (slot < pool_rows) return slot;
    if (error_word) atomicExch(error_word, 1u);
    return 0u;
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t position, uint32_t* error_word) const {
    return checked(listed(position), error_word);
  }
};
__device__ __forceinline__ KeyRows key_rows(const RowAttentionParams& p, const uint32_t* table, uint32_t row) {
  const bool present = row < p.table_rows;
  return {table + (present ? (size_t)row * p.table_stride : 0u), present ? p.table_stride : 0u, p.pool_rows};
}

// EXTENDED kernels know windows, caps and gates, and keep the softmax weights in 32 bits; the others compile without.

// The keys a run of rows sees, positions first .. last of them: the kept ones, then those from `begin` on.
template <bool EXTENDED>
struct Visible {
  uint32_t kept, begin, end;
  __device__ __forceinline__ Visible(const RowAttentionParams& p, uint32_t first, uint32_t last) {
    end = last + 1u;
    begin = EXTENDED && p.window && first + 1u > p.window ? first + 1u - p.window : 0u;
    kept = EXTENDED && p.window ? min(p.keep_first, begin) : 0u;
  }
  __device__ __forceinline__ uint32_t count() const { return kept + end - begin; }
  __device__ __forceinline__ uint32_t position(uint32_t index) const { return index < kept ? index : index - kept + begin; }
};
template <bool EXTENDED>
__device__ __forceinline__ bool sees(const RowAttentionParams& p, uint32_t position, uint32_t key) {
  return key <= position && (!EXTENDED || !p.window || position - key < p.window || key < p.keep_first);
}

// Factor of a read-out.
template <bool EXTENDED, typename T>
__device__ __forceinline__ float gate_of(const RowAttentionParams& p, const T* gate, size_t row, uint32_t head, uint32_t column) {
  return EXTENDED && p.gate_stride ? sigmoid_f32(as_float(gate[row * p.gate_stride + p.gate_column + head * p.vdim + column])) : 1.0f;
}

// ---- one CTA per (row, head) ---------------------------------------------------------------------
// Bound by the latency of slot, key and value loads: scores of kRowKeys keys are formed side by side, eight keys of a warp in
// flight, then the weights of all of them, then a thread per column adds the values.  The arithmetic is that of a walk over
// the keys one after the other (online softmax), to the last bit: decoders that divide by nearly cancelling sums show every
// change of it.  Such a walk by one warp took 112 us for a row with 100 keys behind it (fp32, 16 heads of 128) and 66 us
// for a prompt of 100; now 46 and 34,
// launch included.
template <int SEGMENTS> __host__ __device__ constexpr int row_batch() { return SEGMENTS <= 8 ? 8 : 4; }
constexpr uint32_t kRowWarps = 4, kRowThreads = kRowWarps * 32u, kRowKeys = kRowThreads;

template <typename T, int SEGMENTS>
__global__ void __launch_bounds__(kRowThreads) attention_rows_kernel(const T* query, const T* pool, const uint32_t* table,
                                                             const uint32_t* past, const uint32_t* sequence_rows, T* out,
                                                             const T* gate, RowAttentionParams p, uint32_t* error_word) {
  grid_chain_prologue();
  constexpr int KEYS = row_batch<SEGMENTS>(), COLUMNS = (SEGMENTS * 32 + kRowThreads - 1) / kRowThreads;
  constexpr uint32_t kSpan = 32 / KEYS;  // lanes that end with the same key
  __shared__ uint32_t slots[kRowKeys];
  __shared__ float scores[kRowKeys], keeps[kRowKeys], weights[kRowKeys], warp_tops[kRowWarps];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, item = blockIdx.x;
  const uint32_t row = item / p.heads, head = item % p.heads, sequence = row / p.tokens;
  const uint32_t kv_head = head / (p.heads / p.kv_heads);
  const uint32_t position = past[sequence] + row % p.tokens;
  const Visible<true> visible(p, position, position);
  const uint32_t count = visible.count();
  const KeyRows rows = key_rows(p, table, sequence_rows[sequence]);
  float q[SEGMENTS], o[COLUMNS];
#pragma unroll
  for (int s = 0; s < SEGMENTS; ++s) {
    const uint32_t c = lane + s * 32u;
    q[s] = c < p.dim ? as_float(query[(size_t)row * p.query_stride + p.query_column + head * p.dim + c]) : 0.0f;
  }
#pragma unroll
  for (int i = 0; i < COLUMNS; ++i) o[i] = 0.0f;
  float top = p.sink ? 0.0f : kLowest, total = p.sink ? 1.0f : 0.0f;
  for (uint32_t begin = 0; begin < count; begin += kRowKeys) {
    const uint32_t present = min(kRowKeys, count - begin);
    __syncthreads();  // the keys before are read
    if (threadIdx.x < present) slots[threadIdx.x] = rows(visible.position(begin + threadIdx.x), error_word);
    __syncthreads();
    for (uint32_t first = warp * KEYS; first < present; first += kRowWarps * KEYS) {
      float k[KEYS][SEGMENTS], dots[KEYS];
#pragma unroll
      for (int j = 0; j < KEYS; ++j) {
        const T* cached = pool + (size_t)slots[min(first + j, present - 1u)] * p.token_stride + p.key_offset + kv_head * p.dim;
#pragma unroll
        for (int s = 0; s < SEGMENTS; ++s) k[j][s] = as_float(cached[min(lane + s * 32u, p.dim - 1u)]);
      }
#pragma unroll
      for (int j = 0; j < KEYS; ++j) {
        dots[j] = 0.0f;
#pragma unroll
        for (int s = 0; s < SEGMENTS; ++s)
          if (lane + s * 32u < p.dim) dots[j] = fmaf(q[s], k[j][s], dots[j]);
      }
      // the sum over lanes at distances 16, 8, ..: each exchange halves the keys that a lane keeps, lane l ends with l / kSpan
#pragma unroll
      for (int half = KEYS / 2; half > 0; half >>= 1) {
        const bool upper = (lane & (half * kSpan)) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
          const float sent = upper ? dots[i] : dots[i + half], kept = upper ? dots[i + half] : dots[i];
          dots[i] = kept + __shfl_xor_sync(0xffffffffu, sent, half * kSpan);
        }
      }
      float score = dots[0];
#pragma unroll
      for (uint32_t offset = kSpan / 2; offset > 0; offset >>= 1) score += __shfl_xor_sync(0xffffffffu, score, offset);
      score *= p.scale;
      if (p.softcap > 0.0f) score = p.softcap * tanhf(score / p.softcap);
      if (lane % kSpan == 0 && first + lane / kSpan < present) scores[first + lane / kSpan] = score;
    }
    __syncthreads();
    // the running maximum up to and with this thread's key, and ahead of it
    const float score = threadIdx.x < present ? scores[threadIdx.x] : -INFINITY;
    float highest = score;
#pragma unroll
    for (uint32_t offset = 1; offset < 32u; offset <<= 1) {
      const float earlier = __shfl_up_sync(0xffffffffu, highest, offset);
      if (lane >= offset) highest = fmaxf(earlier, highest);
    }
    if (lane == 31u) warp_tops[warp] = highest;
    float before = __shfl_up_sync(0xffffffffu, highest, 1);
    __syncthreads();
    float ahead = top;
    for (uint32_t w = 0; w < warp; ++w) ahead = fmaxf(ahead, warp_tops[w]);
    before = lane == 0 ? ahead : fmaxf(ahead, before);
    const float next = fmaxf(before, score);
    keeps[threadIdx.x] = expf(before - next);
    weights[threadIdx.x] = expf(score - next);
#pragma unroll
    for (uint32_t w = 0; w < kRowWarps; ++w) top = fmaxf(top, warp_tops[w]);
    __syncthreads();
    const T* values[COLUMNS];
#pragma unroll
    for (int i = 0; i < COLUMNS; ++i) values[i] = pool + p.value_offset + kv_head * p.vdim + min(threadIdx.x + i * kRowThreads, p.vdim - 1u);
    constexpr uint32_t kAhead = COLUMNS == 1 ? 16 : 4;
    for (uint32_t at = 0; at < present; at += kAhead) {
      float v[kAhead][COLUMNS];
#pragma unroll
      for (uint32_t j = 0; j < kAhead; ++j)
#pragma unroll
        for (int i = 0; i < COLUMNS; ++i) v[j][i] = as_float(values[i][(size_t)slots[min(at + j, present - 1u)] * p.token_stride]);
#pragma unroll
      for (uint32_t j = 0; j < kAhead; ++j) {
        if (at + j >= present) break;
        const float keep = keeps[at + j], weight = weights[at + j];
        total = total * keep + weight;
#pragma unroll
        for (int i = 0; i < COLUMNS; ++i) o[i] = o[i] * keep + weight * v[j][i];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < COLUMNS; ++i) {
    const uint32_t c = threadIdx.x + i * kRowThreads;
    if (c < p.vdim) out[(size_t)item * p.vdim + c] = from_float<T>(o[i] / total * gate_of<true>(p, gate, row, head, c));
  }
}

// ---- one warp per (row, head) --------------------------------------------------------------------
// The same arithmetic, a warp walking over the keys one after the other: with enough rows and heads to fill the chip the
// latencies hide behind other warps, and nothing is exchanged within a CTA.
template <typename T, int SEGMENTS>
__global__ void __launch_bounds__(128) attention_walk_kernel(const T* query, const T* pool, const uint32_t* table,
                                                             const uint32_t* past, const uint32_t* sequence_rows, T* out,
                                                             const T* gate, RowAttentionParams p, uint32_t* error_word) {
  grid_chain_prologue();
  const uint32_t lane = threadIdx.x & 31u, item = blockIdx.x * 4u + (threadIdx.x >> 5);
  if (item >= p.sequences * p.tokens * p.heads) return;
  const uint32_t row = item / p.heads, head = item % p.heads, sequence = row / p.tokens;
  const uint32_t kv_head = head / (p.heads / p.kv_heads);
  const uint32_t position = past[sequence] + row % p.tokens;
  const Visible<true> visible(p, position, position);
  const KeyRows rows = key_rows(p, table, sequence_rows[sequence]);
  float q[SEGMENTS], o[SEGMENTS];
#pragma unroll
  for (int s = 0; s < SEGMENTS; ++s) {
    const uint32_t c = lane + s * 32u;
    q[s] = c < p.dim ? as_float(query[(size_t)row * p.query_stride + p.query_column + head * p.dim + c]) : 0.0f;
    o[s] = 0.0f;
  }
  float top = p.sink ? 0.0f : kLowest, total = p.sink ? 1.0f : 0.0f;
  for (uint32_t index = 0; index < visible.count(); ++index) {
    const T* cached = pool + (size_t)rows(visible.position(index), error_word) * p.token_stride;
    const T* k = cached + p.key_offset + kv_head * p.dim;
    const T* v = cached + p.value_offset + kv_head * p.vdim;
    float score = 0.0f;
#pragma unroll
    for (int s = 0; s < SEGMENTS; ++s) {
      const uint32_t c = lane + s * 32u;
      if (c < p.dim) score = fmaf(q[s], as_float(k[c]), score);
    }
    score = warp_sum(score) * p.scale;
    if (p.softcap > 0.0f) score = p.softcap * tanhf(score / p.softcap);
    const float next = fmaxf(top, score), keep = expf(top - next), weight = expf(score - next);
    top = next;
    total = total * keep + weight;
#pragma unroll
    for (int s = 0; s < SEGMENTS; ++s) {
      const uint32_t c = lane + s * 32u;
      if (c < p.vdim) o[s] = o[s] * keep + weight * as_float(v[c]);
    }
  }
#pragma unroll
  for (int s = 0; s < SEGMENTS; ++s) {
    const uint32_t c = lane + s * 32u;
    if (c < p.vdim) out[(size_t)item * p.vdim + c] = from_float<T>(o[s] / total * gate_of<true>(p, gate, row, head, c));
  }
}

// ---- tensor-core pieces --------------------------------------------------------------------------
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* shared_address) {
  const uint32_t address = (uint32_t)__cvta_generic_to_shared(shared_address);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(address)
               : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* shared_address) {
  const uint32_t address = (uint32_t)__cvta_generic_to_shared(shared_address);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(address)
               : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void copy_async_16(void* shared_target, const void* source, uint32_t bytes) {
  const uint32_t address = (uint32_t)__cvta_generic_to_shared(shared_target);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(address), "l"(source), "r"(bytes) : "memory");
}
__device__ __forceinline__ float exp2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__host__ __device__ constexpr uint32_t round16(uint32_t v) { return (v + 15u) & ~15u; }

// Online softmax of one warp's 16 rows (this lane: rows r and r + 8) over KEYS keys, scores already in units
// of log2 e with invisible ones at -inf; then O += P V from the value tile at `v_tile` (row stride v_stride).
// EXTENDED: P enters the product as its bfloat16 rounding plus the bfloat16 rounding of what that leaves.
template <int KEYS, int DV, bool EXTENDED>
struct Softmax {
  float top[2], total[2], out[DV / 8][4];
  bool bounded;  // capped scores: no maximum has to be taken off
  __device__ __forceinline__ explicit Softmax(const RowAttentionParams& p)
      : bounded(EXTENDED && p.softcap > 0.0f && p.softcap <= kBoundedCap) {
    top[0] = top[1] = bounded ? 0.0f : kLowest;
    total[0] = total[1] = 0.0f;
#pragma unroll
    for (int t = 0; t < DV / 8; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) out[t][i] = 0.0f;
  }
  __device__ __forceinline__ void raise_maximum(const float (&score)[KEYS / 8][4]) {
    float next[2] = {top[0], top[1]};
#pragma unroll
    for (int j = 0; j < KEYS / 8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) next[i >> 1] = fmaxf(next[i >> 1], score[j][i]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      next[h] = fmaxf(next[h], __shfl_xor_sync(0xffffffffu, next[h], 1));
      next[h] = fmaxf(next[h], __shfl_xor_sync(0xffffffffu, next[h], 2));
      const float keep = exp2_approx(top[h] - next[h]);
      top[h] = next[h];
      total[h] *= keep;
#pragma unroll
      for (int t = 0; t < DV / 8; ++t) {
        out[t][2 * h] *= keep;
        out[t][2 * h + 1] *= keep;
      }
    }
  }
  __device__ __forceinline__ void absorb(float (&score)[KEYS / 8][4], const bf16* v_tile, uint32_t v_stride, uint32_t lane) {
    if (!bounded) raise_maximum(score);
    uint32_t weights[KEYS / 16][4], rests[EXTENDED ? KEYS / 16 : 1][4];
#pragma unroll
    for (int j = 0; j < KEYS / 8; ++j) {
      float e[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) e[i] = exp2_approx(score[j][i] - top[i >> 1]);
      total[0] += e[0] + e[1];
      total[1] += e[2] + e[3];
      const __nv_bfloat162 low = __floats2bfloat162_rn(e[0], e[1]), high = __floats2bfloat162_rn(e[2], e[3]);
      weights[j >> 1][(j & 1) * 2] = *reinterpret_cast<const uint32_t*>(&low);
      weights[j >> 1][(j & 1) * 2 + 1] = *reinterpret_cast<const uint32_t*>(&high);
      if (EXTENDED) {
        const __nv_bfloat162 low_rest = __floats2bfloat162_rn(e[0] - __low2float(low), e[1] - __high2float(low));
        const __nv_bfloat162 high_rest = __floats2bfloat162_rn(e[2] - __low2float(high), e[3] - __high2float(high));
        rests[EXTENDED ? j >> 1 : 0][(j & 1) * 2] = *reinterpret_cast<const uint32_t*>(&low_rest);
        rests[EXTENDED ? j >> 1 : 0][(j & 1) * 2 + 1] = *reinterpret_cast<const uint32_t*>(&high_rest);
      }
    }
#pragma unroll
    for (int s = 0; s < KEYS / 16; ++s)
#pragma unroll
      for (int t = 0; t < DV / 16; ++t) {
        uint32_t b[4];
        ldmatrix_x4_trans(b, v_tile + (16 * s + (lane & 7u) + ((lane >> 3) & 1u) * 8u) * v_stride + 16 * t + (lane >> 4) * 8u);
        mma_bf16(out[2 * t], weights[s], b[0], b[1]);
        mma_bf16(out[2 * t + 1], weights[s], b[2], b[3]);
        if (EXTENDED) {
          mma_bf16(out[2 * t], rests[EXTENDED ? s : 0], b[0], b[1]);
          mma_bf16(out[2 * t + 1], rests[EXTENDED ? s : 0], b[2], b[3]);
        }
      }
  }
};

// A raw score in units of log2 e; with a cap c, c tanh(s / c) = c - 2 c / (e^(2 s / c) + 1).
template <bool EXTENDED>
struct ScoreScale {
  float scale, cap;  // cap 0: none
  __device__ __forceinline__ explicit ScoreScale(const RowAttentionParams& p)
      : scale((EXTENDED && p.softcap > 0.0f ? p.scale / p.softcap * 2.0f : p.scale) * kLog2e), cap(p.softcap * kLog2e) {}
  __device__ __forceinline__ float operator()(float raw) const {
    const float score = raw * scale;
    return EXTENDED && cap > 0.0f ? fmaf(-2.0f * cap, __fdividef(1.0f, exp2_approx(score) + 1.0f), cap) : score;
  }
};

// 16 query rows (this warp's, at q_rows, row stride `stride`) against KEYS key rows.  DK > 0: the query
// fragments are in registers; DK == 0: they are read from shared memory for every 16 dimensions.
template <int KEYS, int DK>
__device__ __forceinline__ void scores(float (&score)[KEYS / 8][4], const uint32_t (*q_frag)[4], const bf16* q_rows,
                                       const bf16* k_tile, uint32_t stride, uint32_t steps, uint32_t lane) {
#pragma unroll
  for (int j = 0; j < KEYS / 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) score[j][i] = 0.0f;
  auto step = [&](const uint32_t (&a)[4], uint32_t s) {
#pragma unroll
    for (int j = 0; j < KEYS / 16; ++j) {
      uint32_t b[4];
      ldmatrix_x4(b, k_tile + (16 * j + (lane & 7u) + (lane >> 4) * 8u) * stride + 16 * s + ((lane >> 3) & 1u) * 8u);
      mma_bf16(score[2 * j], a, b[0], b[1]);
      mma_bf16(score[2 * j + 1], a, b[2], b[3]);
    }
  };
  if (DK > 0) {
#pragma unroll
    for (int s = 0; s < DK / 16; ++s) step(q_frag[s], s);
  } else {
    for (uint32_t s = 0; s < steps; ++s) {
      uint32_t a[4];
      ldmatrix_x4(a, q_rows + ((lane & 7u) + ((lane >> 3) & 1u) * 8u) * stride + 16 * s + (lane >> 4) * 8u);
      step(a, s);
    }
  }
}

// ---- prompts -------------------------------------------------------------------------------------
constexpr uint32_t kQueryTile = 64;
// Keys per tile, groups of four warps that take turns with the tiles, and CTAs per SM to compile for (0: no bound).  What bounds the
// kernel is the way from a score to its weight, which other warps hide (mma.sync alone would take a quarter of the time), and the CTAs
// that start late: the longest go first over all heads, slots are looked up a tile ahead.  2048 tokens, 16 heads of 128, before
// and now: 155 and 97 us, with windows 137 and 109.
__host__ __device__ constexpr uint32_t key_tile(int DK, bool EXTENDED) { return EXTENDED && DK == 128 ? 32u : 64u; }
constexpr int prompt_ctas(int DK, bool EXTENDED, uint32_t GROUPS) { return DK != 128 ? 0 : GROUPS > 1u ? 1 : EXTENDED ? 3 : 2; }

template <int DK, int DV, bool EXTENDED, uint32_t GROUPS>
__global__ void __launch_bounds__(128 * GROUPS, prompt_ctas(DK, EXTENDED, GROUPS)) attention_prompt_kernel(const bf16* query, const bf16* pool, const uint32_t* table,
                                                               const uint32_t* past_lengths, const uint32_t* sequence_rows,
                                                               bf16* out, const bf16* gate, RowAttentionParams p, uint32_t* error_word) {
  constexpr uint32_t kKeyTile = key_tile(DK, EXTENDED), kPerKey = 128u / kKeyTile;  // threads that fetch a key
  constexpr uint32_t kGroups = GROUPS, kThreads = 128u * kGroups;
  grid_chain_prologue();
  extern __shared__ __align__(16) unsigned char attention_shared[];
  const uint32_t padded = DK > 0 ? DK : round16(p.dim), k_stride = padded + 8u, v_stride = DV + 8u;
  bf16* q_tile = reinterpret_cast<bf16*>(attention_shared);
  const uint32_t group = kGroups > 1u ? threadIdx.x >> 7 : 0u, thread = threadIdx.x & 127u;
  bf16* k_tiles = q_tile + kQueryTile * k_stride + group * 2u * kKeyTile * (k_stride + v_stride);
  bf16* v_tiles = k_tiles + 2u * kKeyTile * k_stride;
  // the last query tiles see the most keys: they are scheduled first, over all heads
  const uint32_t q0 = (gridDim.y - 1u - blockIdx.y) * kQueryTile, head = blockIdx.x, sequence = blockIdx.z;
  const uint32_t kv_head = head / (p.heads / p.kv_heads);
  const uint32_t warp = thread >> 5, lane = threadIdx.x & 31u, r = lane >> 2, c = lane & 3u;
  const uint32_t past = past_lengths[sequence];
  const KeyRows rows = key_rows(p, table, sequence_rows[sequence]);
  const uint32_t key_end = past + min(q0 + kQueryTile, p.tokens);
  // whole key tiles: those with kept keys, then from the first row's window on
  const Visible<EXTENDED> visible(p, past + q0, key_end - 1u);
  const uint32_t kept_tiles = (visible.kept + kKeyTile - 1u) / kKeyTile;
  const uint32_t skipped = max(visible.begin / kKeyTile, kept_tiles) - kept_tiles;
  const uint32_t all_tiles = (key_end + kKeyTile - 1u) / kKeyTile - skipped;
  const uint32_t tiles = (all_tiles + kGroups - 1u - group) / kGroups;  // of this group: every kGroups-th
  auto first_key = [&](uint32_t turn) {
    const uint32_t tile = turn * kGroups + group;
    return (tile < kept_tiles ? tile : tile + skipped) * kKeyTile;
  };
  auto group_sync = [&]() {
    if (kGroups == 1u) __syncthreads();
    else asm volatile("bar.sync %0, 128;" ::"r"(1u + group) : "memory");
  };
  const uint32_t k_chunks = padded / 8u, v_chunks = DV / 8u;
  const uint32_t key = thread / kPerKey, share = thread % kPerKey;  // of the copies

  auto slot_of = [&](uint32_t tile) {
    const uint32_t position = first_key(tile) + key;
    return tile < tiles && position < key_end ? rows.listed(position) : 0u;
  };
  uint32_t slot = slot_of(0);  // of the tile that is fetched next
  auto fetch_tile = [&](uint32_t tile) {
    if (tile < tiles) {
      bf16* k_tile = k_tiles + (tile & 1u) * kKeyTile * k_stride;
      bf16* v_tile = v_tiles + (tile & 1u) * kKeyTile * v_stride;
      // a few threads per key row: one slot look-up, a share of the chunks each
      const bool present = first_key(tile) + key < key_end;
      const bf16* cached = pool + (size_t)(present ? rows.checked(slot, error_word) : 0u) * p.token_stride;
      slot = slot_of(tile + 1u);  // used a tile from now
      const bf16* k = cached + p.key_offset + kv_head * p.dim;
      const bf16* v = cached + p.value_offset + kv_head * p.vdim;
      for (uint32_t chunk = share; chunk < k_chunks; chunk += kPerKey) {
        const bool there = present && chunk * 8u < p.dim;
        copy_async_16(k_tile + key * k_stride + chunk * 8u, there ? k + chunk * 8u : pool, there ? 16u : 0u);
      }
      for (uint32_t chunk = share; chunk < v_chunks; chunk += kPerKey) {
        const bool there = present && chunk * 8u < p.vdim;
        copy_async_16(v_tile + key * v_stride + chunk * 8u, there ? v + chunk * 8u : pool, there ? 16u : 0u);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (uint32_t index = threadIdx.x; index < kQueryTile * k_chunks; index += kThreads) {
    const uint32_t row = index / k_chunks, chunk = index % k_chunks;
    const bool there = q0 + row < p.tokens && chunk * 8u < p.dim;
    copy_async_16(q_tile + row * k_stride + chunk * 8u,
                  there ? query + ((size_t)sequence * p.tokens + q0 + row) * p.query_stride + p.query_column + head * p.dim + chunk * 8u : pool,
                  there ? 16u : 0u);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  fetch_tile(0);
  asm volatile("cp.async.wait_group 1;" ::: "memory");  // the queries; their way hides behind the first look-up
  __syncthreads();
  const bf16* q_rows = q_tile + warp * 16u * k_stride;
  uint32_t q_frag[DK > 0 ? DK / 16 : 1][4];
  if (DK > 0) {
#pragma unroll
    for (int s = 0; s < DK / 16; ++s)
      ldmatrix_x4(q_frag[s], q_rows + ((lane & 7u) + ((lane >> 3) & 1u) * 8u) * k_stride + 16 * s + (lane >> 4) * 8u);
  }
  const uint32_t row_low = q0 + warp * 16u + r;  // and row_low + 8
  const ScoreScale<EXTENDED> score_of(p);
  Softmax<kKeyTile, DV, EXTENDED> state(p);

  for (uint32_t tile = 0; tile < tiles; ++tile) {
    const uint32_t k0 = first_key(tile);
    fetch_tile(tile + 1u);  // into the other buffer, which the previous iteration's last barrier released
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    group_sync();
    float score[kKeyTile / 8][4];
    scores<kKeyTile, DK>(score, q_frag, q_rows, k_tiles + (tile & 1u) * kKeyTile * k_stride, k_stride, padded / 16u, lane);
    const uint32_t first_row = past + q0 + warp * 16u;  // of this warp
    const bool all_visible = k0 + kKeyTile - 1u <= first_row &&
                             (!EXTENDED || !p.window || first_row + 15u - k0 < p.window || k0 + kKeyTile <= p.keep_first);
#pragma unroll
    for (int j = 0; j < (int)kKeyTile / 8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t token = row_low + ((i & 2) ? 8u : 0u), key = k0 + 8u * j + 2u * c + (i & 1);
        score[j][i] = all_visible || sees<EXTENDED>(p, past + token, key) ? score_of(score[j][i]) : -INFINITY;
      }
    state.absorb(score, v_tiles + (tile & 1u) * kKeyTile * v_stride, v_stride, lane);
    group_sync();  // every warp is done with this buffer before the next iteration's fetch refills it
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  // The sums of thread t of a group and its part: columns 8 t + 2 c and the one after it, row r + 8 h.  With several groups each
  // finishes its share of the t: a gate's exponential and division are a long chain.
  constexpr int kShare = (DV / 8 + (int)kGroups - 1) / (int)kGroups;
  const int first_t = kGroups > 1u ? (int)group * kShare : 0;
  auto column_of = [&](int t) { return 8u * (uint32_t)(first_t + t) + 2u * c; };
  // All gates are requested before the first is needed: a load after each store was 14 us of a prompt's attention.  With heads of 129 to 256
  // a few sums spill for it, which costs less than it saves: 16 heads of 256, 777 tokens 173 -> 97 us, 2048 457 -> 344.
  bf16 gates[EXTENDED ? 2 : 1][EXTENDED ? kShare : 1][2];
  if (EXTENDED && p.gate_stride) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const size_t row = (size_t)sequence * p.tokens + min(row_low + h * 8u, p.tokens - 1u);
      const bf16* const source = gate + row * p.gate_stride + p.gate_column + head * p.vdim;
#pragma unroll
      for (int t = 0; t < kShare; ++t)
#pragma unroll
        for (int i = 0; i < 2; ++i) gates[EXTENDED ? h : 0][EXTENDED ? t : 0][i] = source[min(column_of(t) + i, p.vdim - 1u)];
    }
  }
  float sums[kShare][4];
  if constexpr (kGroups > 1u) {  // what the groups have, added in their order; the rings are free
    constexpr uint32_t kValues = 4u + DV / 2u;  // of a thread
    float* const shared_values = reinterpret_cast<float*>(q_tile);
    auto value_of = [&](uint32_t other, uint32_t i) -> float& { return shared_values[(other * kValues + i) * 128u + thread]; };
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) value_of(group, h) = state.top[h], value_of(group, 2 + h) = state.total[h];
#pragma unroll
    for (int t = 0; t < DV / 8; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) value_of(group, 4 + 4 * t + i) = state.out[t][i];
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kShare; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) sums[t][i] = 0.0f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float top = kLowest, total = 0.0f;
#pragma unroll
      for (uint32_t other = 0; other < kGroups; ++other) top = fmaxf(top, value_of(other, h));
#pragma unroll
      for (uint32_t other = 0; other < kGroups; ++other) {
        const float weight = exp2_approx(value_of(other, h) - top);  // 1 where no maximum is taken off
        total += value_of(other, 2 + h) * weight;
#pragma unroll
        for (int t = 0; t < kShare; ++t)
          if (first_t + t < DV / 8) {
#pragma unroll
            for (int i = 0; i < 2; ++i) sums[t][2 * h + i] += value_of(other, 4 + 4 * (first_t + t) + 2 * h + i) * weight;
          }
      }
      state.top[h] = top;
      state.total[h] = total;
    }
  } else {
#pragma unroll
    for (int t = 0; t < kShare; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) sums[t][i] = state.out[t][i];
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float total = state.total[h];
    total += __shfl_xor_sync(0xffffffffu, total, 1);
    total += __shfl_xor_sync(0xffffffffu, total, 2);
    float scale = 1.0f;
    if (p.sink) {  // bring both to the larger of the two maxima
      const float top = fmaxf(state.top[h], 0.0f);
      scale = exp2f(state.top[h] - top);
      total = total * scale + exp2f(-top);
    }
    scale /= total;
    const uint32_t token = row_low + h * 8u;
    if (token >= p.tokens) continue;
    bf16* target = out + (((size_t)sequence * p.tokens + token) * p.heads + head) * p.vdim;
#pragma unroll
    for (int t = 0; t < kShare; ++t) {
      float factor[2];
#pragma unroll
      for (int i = 0; i < 2; ++i)
        factor[i] = EXTENDED && p.gate_stride ? sigmoid_f32(as_float(gates[EXTENDED ? h : 0][EXTENDED ? t : 0][i])) : 1.0f;
      if (first_t + t < DV / 8 && column_of(t) < p.vdim)  // vdim is a multiple of eight
        *reinterpret_cast<__nv_bfloat162*>(target + column_of(t)) =
            __floats2bfloat162_rn(sums[t][2 * h] * scale * factor[0], sums[t][2 * h + 1] * scale * factor[1]);
    }
  }
}

// ---- decode --------------------------------------------------------------------------------------
constexpr uint32_t kWarpKeys = 16, kDecodeWarps = 4, kMostSplits = 64;
// Record of one split: 16 maxima, 16 denominators, 16 x DV sums.
template <int DV>
__host__ __device__ constexpr uint32_t record_floats() { return 32u + 16u * DV; }

template <int DK, int DV, bool EXTENDED, uint32_t STAGES>
__global__ void __launch_bounds__(128) attention_decode_kernel(const bf16* query, const bf16* pool, const uint32_t* table,
                                                               const uint32_t* past_lengths, const uint32_t* sequence_rows,
                                                               bf16* out, const bf16* gate, uint32_t* counters, float* records,
                                                               RowAttentionParams p, uint32_t* error_word) {
  constexpr uint32_t kDecodeStages = STAGES;  // tiles in a warp's ring
  grid_chain_prologue();
  extern __shared__ __align__(16) unsigned char attention_shared[];
  const uint32_t padded = DK > 0 ? DK : round16(p.dim), k_stride = padded + 8u, v_stride = DV + 8u;
  const uint32_t stage_elements = kWarpKeys * (k_stride + v_stride);
  bf16* q_tile = reinterpret_cast<bf16*>(attention_shared);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, r = lane >> 2, c = lane & 3u;
  bf16* ring = q_tile + 16u * k_stride + warp * kDecodeStages * stage_elements;
  const uint32_t split = blockIdx.x, kv_head = blockIdx.y, sequence = blockIdx.z;
  const uint32_t group = p.heads / p.kv_heads, query_rows = p.tokens * group;
  const uint32_t past = past_lengths[sequence];
  const Visible<EXTENDED> visible(p, past, past + p.tokens - 1u);
  const uint32_t keys = visible.count();
  const KeyRows rows = key_rows(p, table, sequence_rows[sequence]);
  // whole 64-key stretches per split
  const uint32_t stretch = (kWarpKeys * kDecodeWarps);
  const uint32_t per_split = ((keys + p.splits - 1u) / p.splits + stretch - 1u) / stretch * stretch;
  const uint32_t begin = min(split * per_split, keys), end = min(begin + per_split, keys);
  const uint32_t tiles = (end - begin + stretch - 1u) / stretch;  // of this warp
  const uint32_t k_chunks = padded / 8u, v_chunks = DV / 8u;

  const uint32_t key = lane >> 1, half = lane & 1u;  // of the copies
  auto index_of = [&](uint32_t tile) { return begin + tile * stretch + warp * kWarpKeys + key; };
  auto slot_of = [&](uint32_t tile) {
    return index_of(tile) < end ? rows.listed(visible.position(index_of(tile))) : 0u;
  };
  // Of the tiles that are fetched next, so that a copy does not wait for its look-up.  us, looked up with the copy and ahead, 16 / 4 heads: 1 sequence
  // x 300 keys, dim 64 16.2, 14.4, 128 18.2, 16.5, 256 24.1, 22.7; 32 x 1300 keys 35.0, 32.5; 46.6, 46.2; 107, 103; with windows and
  // gates 34.6, 33.1; 43.7, 42.7; 103, 95.  None of 80 sizes is slower, though dim 256 has 236 registers a thread for 167.
  uint32_t slots[kDecodeStages];
#pragma unroll
  for (uint32_t s = 0; s < kDecodeStages; ++s) slots[s] = slot_of(s);
  auto fetch_tile = [&](uint32_t tile) {
    if (tile < tiles) {
      bf16* k_tile = ring + (tile % kDecodeStages) * stage_elements;
      bf16* v_tile = k_tile + kWarpKeys * k_stride;
      const bool present = index_of(tile) < end;
      const bf16* cached = pool + (size_t)(present ? rows.checked(slots[0], error_word) : 0u) * p.token_stride;
#pragma unroll
      for (uint32_t s = 0; s + 1u < kDecodeStages; ++s) slots[s] = slots[s + 1u];
      slots[kDecodeStages - 1u] = slot_of(tile + kDecodeStages);
      const bf16* k = cached + p.key_offset + kv_head * p.dim;
      const bf16* v = cached + p.value_offset + kv_head * p.vdim;
      for (uint32_t chunk = half; chunk < k_chunks; chunk += 2u) {
        const bool there = present && chunk * 8u < p.dim;
        copy_async_16(k_tile + key * k_stride + chunk * 8u, there ? k + chunk * 8u : pool, there ? 16u : 0u);
      }
      for (uint32_t chunk = half; chunk < v_chunks; chunk += 2u) {
        const bool there = present && chunk * 8u < p.vdim;
        copy_async_16(v_tile + key * v_stride + chunk * 8u, there ? v + chunk * 8u : pool, there ? 16u : 0u);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (uint32_t s = 0; s + 1u < kDecodeStages; ++s) fetch_tile(s);
  for (uint32_t index = threadIdx.x; index < 16u * k_chunks; index += 128u) {
    const uint32_t row = index / k_chunks, chunk = index % k_chunks;
    uint4 data = make_uint4(0u, 0u, 0u, 0u);
    if (row < query_rows && chunk * 8u < p.dim)
      data = *reinterpret_cast<const uint4*>(query + ((size_t)sequence * p.tokens + row / group) * p.query_stride + p.query_column +
                                             (kv_head * group + row % group) * p.dim + chunk * 8u);
    *reinterpret_cast<uint4*>(q_tile + row * k_stride + chunk * 8u) = data;
  }
  __syncthreads();
  uint32_t q_frag[DK > 0 ? DK / 16 : 1][4];
  if (DK > 0) {
#pragma unroll
    for (int s = 0; s < DK / 16; ++s)
      ldmatrix_x4(q_frag[s], q_tile + ((lane & 7u) + ((lane >> 3) & 1u) * 8u) * k_stride + 16 * s + (lane >> 4) * 8u);
  }
  const uint32_t token_low = r / group, token_high = (r + 8u) / group;
  const ScoreScale<EXTENDED> score_of(p);
  Softmax<kWarpKeys, DV, EXTENDED> state(p);
  for (uint32_t tile = 0; tile < tiles; ++tile) {
    fetch_tile(tile + kDecodeStages - 1u);
    asm volatile("cp.async.wait_group %0;" ::"n"(kDecodeStages - 1) : "memory");
    __syncwarp();  // the other lanes' copies of this tile have landed too
    const bf16* k_tile = ring + (tile % kDecodeStages) * stage_elements;
    const uint32_t k0 = begin + tile * stretch + warp * kWarpKeys;
    float score[kWarpKeys / 8][4];
    scores<kWarpKeys, DK>(score, q_frag, q_tile, k_tile, k_stride, padded / 16u, lane);
#pragma unroll
    for (int j = 0; j < (int)kWarpKeys / 8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t index = k0 + 8u * j + 2u * c + (i & 1);
        const bool seen = index < end && sees<EXTENDED>(p, past + ((i & 2) ? token_high : token_low), visible.position(index));
        score[j][i] = seen ? score_of(score[j][i]) : -INFINITY;
      }
    state.absorb(score, k_tile + kWarpKeys * k_stride, v_stride, lane);
    __syncwarp();
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    state.total[h] += __shfl_xor_sync(0xffffffffu, state.total[h], 1);
    state.total[h] += __shfl_xor_sync(0xffffffffu, state.total[h], 2);
  }
  __syncthreads();  // the rings are free: they carry the warps' results now

  constexpr uint32_t kRecord = record_floats<DV>();
  float* shared_records = reinterpret_cast<float*>(attention_shared);
  {
    float* mine = shared_records + warp * kRecord;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (c == 0) {
        mine[r + 8 * h] = state.top[h];
        mine[16 + r + 8 * h] = state.total[h];
      }
#pragma unroll
      for (int t = 0; t < DV / 8; ++t)
        *reinterpret_cast<float2*>(mine + 32 + (r + 8 * h) * DV + 8 * t + 2 * c) =
            make_float2(state.out[t][2 * h], state.out[t][2 * h + 1]);
    }
  }
  __syncthreads();
  float* record = records + (((size_t)sequence * p.kv_heads + kv_head) * p.splits + split) * kRecord;
  const bool single = p.splits == 1u;
  for (uint32_t index = threadIdx.x; index < query_rows * DV; index += 128u) {
    const uint32_t row = index / DV, column = index % DV;
    float top = kLowest;
#pragma unroll
    for (uint32_t w = 0; w < kDecodeWarps; ++w) top = fmaxf(top, shared_records[w * kRecord + row]);
    float total = 0.0f, sum = 0.0f;
#pragma unroll
    for (uint32_t w = 0; w < kDecodeWarps; ++w) {
      const float weight = exp2f(shared_records[w * kRecord + row] - top);
      total += weight * shared_records[w * kRecord + 16 + row];
      sum += weight * shared_records[w * kRecord + 32 + row * DV + column];
    }
    if (single) {
      if (p.sink) {
        const float both = fmaxf(top, 0.0f), keep = exp2f(top - both);
        sum *= keep;
        total = total * keep + exp2f(-both);
      }
      const size_t token = (size_t)sequence * p.tokens + row / group;
      const uint32_t head = kv_head * group + row % group;
      if (column < p.vdim)
        out[(token * p.heads + head) * p.vdim + column] =
            __float2bfloat16_rn(sum / total * gate_of<EXTENDED>(p, gate, token, head, column));
    } else {
      record[32 + row * DV + column] = sum;
      if (column == 0) {
        record[row] = top;
        record[16 + row] = total;
      }
    }
  }
  if (single) return;

  // the last split of this (sequence, key/value head) to get here adds all of them, in split order
  __shared__ uint32_t is_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t* counter = counters + sequence * p.kv_heads + kv_head;
    const bool last = atomicAdd(counter, 1u) + 1u == p.splits;
    if (last) *counter = 0u;  // ready for the next launch
    is_last = last ? 1u : 0u;
  }
  __syncthreads();
  if (is_last == 0u) return;
  __threadfence();
  const float* first = records + ((size_t)sequence * p.kv_heads + kv_head) * p.splits * kRecord;
  const uint32_t used = (keys + per_split - 1u) / per_split;  // the others saw no key
  // weight of every split for every row, over the row's common denominator
  float* weights = shared_records;  // [query rows][used]
  for (uint32_t row = warp; row < query_rows; row += kDecodeWarps) {
    float top = p.sink ? 0.0f : kLowest;
    for (uint32_t s = lane; s < used; s += 32u) top = fmaxf(top, __ldcg(first + (size_t)s * kRecord + row));
    top = warp_max(top);
    float total = 0.0f;
    for (uint32_t s = lane; s < used; s += 32u) {
      const float weight = exp2f(__ldcg(first + (size_t)s * kRecord + row) - top);
      total += weight * __ldcg(first + (size_t)s * kRecord + 16 + row);
      weights[row * kMostSplits + s] = weight;
    }
    total = warp_sum(total) + (p.sink ? exp2f(-top) : 0.0f);
    __syncwarp();
    for (uint32_t s = lane; s < used; s += 32u) weights[row * kMostSplits + s] /= total;
  }
  __syncthreads();
  for (uint32_t index = threadIdx.x; index < query_rows * (DV / 4); index += 128u) {
    const uint32_t row = index / (DV / 4), column = index % (DV / 4) * 4u;
    const float* source = first + 32 + row * DV + column;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t s = 0;
    for (; s + 8u <= used; s += 8u) {
      float4 part[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) part[i] = __ldcg(reinterpret_cast<const float4*>(source + (size_t)(s + i) * kRecord));
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float weight = weights[row * kMostSplits + s + i];
        sum.x = fmaf(weight, part[i].x, sum.x);
        sum.y = fmaf(weight, part[i].y, sum.y);
        sum.z = fmaf(weight, part[i].z, sum.z);
        sum.w = fmaf(weight, part[i].w, sum.w);
      }
    }
    for (; s < used; ++s) {
      const float4 part = __ldcg(reinterpret_cast<const float4*>(source + (size_t)s * kRecord));
      const float weight = weights[row * kMostSplits + s];
      sum.x = fmaf(weight, part.x, sum.x);
      sum.y = fmaf(weight, part.y, sum.y);
      sum.z = fmaf(weight, part.z, sum.z);
      sum.w = fmaf(weight, part.w, sum.w);
    }
    if (column < p.vdim) {  // vdim is a multiple of eight
      const size_t token = (size_t)sequence * p.tokens + row / group;
      const uint32_t head = kv_head * group + row % group;
      sum.x *= gate_of<EXTENDED>(p, gate, token, head, column);
      sum.y *= gate_of<EXTENDED>(p, gate, token, head, column + 1u);
      sum.z *= gate_of<EXTENDED>(p, gate, token, head, column + 2u);
      sum.w *= gate_of<EXTENDED>(p, gate, token, head, column + 3u);
      store_four(out + (token * p.heads + head) * p.vdim + column, sum);
    }
  }
}

// ---- host ----------------------------------------------------------------------------------------
template <typename T>
int run_rows(const KernelArgs& args, const RowAttentionParams& p) {
  const size_t items = (size_t)p.sequences * p.tokens * p.heads;
  const uint32_t widest = p.dim > p.vdim ? p.dim : p.vdim;
  // Rows and heads per SM up to which a CTA for each is faster than a warp for each; from there on warps hide one another's
  // latencies.  The rows of a prompt differ in length, so that the longest walks bound it and the line lies higher.  fp32, 16 heads,
  // a CTA and a warp each, us: heads of 128, 150 keys, 80 sequences 146 and 178, 200 sequences 286 and 182; a prompt of 200 tokens
  // 92 and 115, of 800 1184 and 800; heads of 256, 1000 tokens 1850 and 2100, 2048 tokens 7380 and 7030.
  const uint32_t tokens = p.tokens;
  const uint32_t per_sm = widest <= 64u    ? min(15u + tokens / 10u, 38u)
                          : widest <= 128u ? min(11u + tokens / 14u, 29u)
                                           : min(24u + tokens / 2u, 170u);
  const bool walk = items > (size_t)per_sm * (size_t)context_sm_count(args.ctx);
  auto launch = [&](auto kernel, size_t ctas) {
    launch_kernel(args, kernel, dim3((uint32_t)ctas), dim3(kRowThreads), 0, (const T*)args.buffers[0],
                  (const T*)args.buffers[1], (const uint32_t*)args.buffers[2], (const uint32_t*)args.buffers[3],
                  (const uint32_t*)args.buffers[4], (T*)args.buffers[5], (const T*)args.buffers[7], p, context_device_error(args.ctx));
  };
  auto run = [&](auto segments) {
    constexpr int SEGMENTS = decltype(segments)::value;
    if (walk) launch(attention_walk_kernel<T, SEGMENTS>, (items + kRowWarps - 1u) / kRowWarps);
    else launch(attention_rows_kernel<T, SEGMENTS>, items);
  };
  if (widest <= 64u) run(std::integral_constant<int, 2>());
  else if (widest <= 128u) run(std::integral_constant<int, 4>());
  else if (widest <= 256u) run(std::integral_constant<int, 8>());
  else if (widest <= 512u) run(std::integral_constant<int, 16>());
  else return fail(args, "head sizes above 512 are not supported");
  return check_launch(args);
}

// Head size up to which tensor cores are used.  The limit of a kernel's shared memory is set for it whatever a launch asks for:
// another thread's may be under way.
constexpr uint32_t kWidestHead = 256;

template <int DK, int DV, bool EXTENDED, uint32_t GROUPS>
int run_prompt_groups(const KernelArgs& args, const RowAttentionParams& p) {
  const uint32_t padded = DK > 0 ? DK : round16(p.dim);
  constexpr uint32_t kKeyTile = key_tile(DK, EXTENDED), kGroups = GROUPS;
  auto bytes_of = [](uint32_t width) { return (kQueryTile * (width + 8u) + kGroups * 2u * kKeyTile * (width + 8u + DV + 8u)) * 2u; };
  const uint32_t bytes = bytes_of(padded);
  static_assert(kGroups == 1u || kGroups * (4u + DV / 2u) * 512u <= (kQueryTile * (DK + 8u) + kGroups * 2u * kKeyTile * (DK + DV + 16u)) * 2u,
                "the groups' results take the tiles' place");
  auto kernel = attention_prompt_kernel<DK, DV, EXTENDED, GROUPS>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes_of(DK > 0 ? DK : kWidestHead)) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  launch_kernel(args, kernel, dim3(p.heads, (p.tokens + kQueryTile - 1u) / kQueryTile, p.sequences), dim3(128u * kGroups), bytes,
                (const bf16*)args.buffers[0], (const bf16*)args.buffers[1], (const uint32_t*)args.buffers[2],
                (const uint32_t*)args.buffers[3], (const uint32_t*)args.buffers[4], (bf16*)args.buffers[5],
                (const bf16*)args.buffers[7], p,
                context_device_error(args.ctx));
  return check_launch(args);
}

template <int DK, int DV, bool EXTENDED>
int run_prompt(const KernelArgs& args, const RowAttentionParams& p) {
  if (p.tokens > 65535u * kQueryTile) return -1;  // a grid's second dimension
  // Up to three query tiles and heads per SM, which is what fits at once with one group each, the longest of them bound the kernel,
  // and three groups walk over its keys together; beyond, CTAs that take turns hide one another's beginnings and ends.  16 heads of
  // 128, window 1024, one group and three, us: 60 tokens 13.3 and 9.8, 333 37.7 and 19.8, 777 74.8 and 36.0, 1300 107 and 74,
  // 1600 109 and 91, 2048 (512 CTAs) 109 and 120.
  if constexpr (EXTENDED && DK == 128) {
    const size_t ctas = (size_t)((p.tokens + kQueryTile - 1u) / kQueryTile) * p.heads * p.sequences;
    if (ctas <= (size_t)3u * context_sm_count(args.ctx)) return run_prompt_groups<DK, DV, EXTENDED, 3>(args, p);
  }
  return run_prompt_groups<DK, DV, EXTENDED, 1>(args, p);
}

template <int DK, int DV, bool EXTENDED, uint32_t STAGES>
int run_decode_stages(const KernelArgs& args, const RowAttentionParams& p) {
  const uint32_t padded = DK > 0 ? DK : round16(p.dim);
  auto bytes_of = [](uint32_t width) {
    const uint32_t rings = (16u * (width + 8u) + kDecodeWarps * STAGES * kWarpKeys * (width + 8u + DV + 8u)) * 2u;
    const uint32_t merge = kDecodeWarps * record_floats<DV>() * 4u;
    return rings < merge ? merge : rings;
  };
  const uint32_t bytes = bytes_of(padded);
  const size_t heads = (size_t)p.sequences * p.kv_heads, counters = (heads * 4 + 255) / 256 * 256;
  LLMOPT_REQUIRE(p.splits <= kMostSplits, "at most 64 splits");
  LLMOPT_REQUIRE(p.splits == 1u || args.lengths[6] >= counters + heads * p.splits * record_floats<DV>() * 4,
                 "split scratch is too short");
  auto kernel = attention_decode_kernel<DK, DV, EXTENDED, STAGES>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes_of(DK > 0 ? DK : kWidestHead)) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  launch_kernel(args, kernel, dim3(p.splits, p.kv_heads, p.sequences), dim3(128), bytes, (const bf16*)args.buffers[0],
                (const bf16*)args.buffers[1], (const uint32_t*)args.buffers[2], (const uint32_t*)args.buffers[3],
                (const uint32_t*)args.buffers[4], (bf16*)args.buffers[5], (const bf16*)args.buffers[7],
                (uint32_t*)args.buffers[6],
                (float*)((uint8_t*)args.buffers[6] + counters), p, context_device_error(args.ctx));
  return check_launch(args);
}

// With 128-wide heads a ring of two tiles leaves room for a third CTA on an SM, a ring of three keeps more under way.  Two where
// that saves a wave: 8 sequences x 2048 keys x 4 key heads, 416 CTAs, 19.9 us with two and 27.9 with three; 32 x 2048 x 8, 256
// CTAs, 112 and 92.
template <int DK, int DV, bool EXTENDED>
int run_decode(const KernelArgs& args, const RowAttentionParams& p) {
  if constexpr (DK == 128) {
    const size_t ctas = (size_t)p.splits * p.kv_heads * p.sequences, sms = (size_t)context_sm_count(args.ctx);
    if ((ctas + 3u * sms - 1u) / (3u * sms) < (ctas + 2u * sms - 1u) / (2u * sms)) return run_decode_stages<DK, DV, EXTENDED, 2>(args, p);
  }
  return run_decode_stages<DK, DV, EXTENDED, 3>(args, p);
}

template <int DK, int DV>
int run_tensor(const KernelArgs& args, const RowAttentionParams& p) {
  if (p.tokens * (p.heads / p.kv_heads) <= 16u)
    return p.extended() ? run_decode<DK, DV, true>(args, p) : run_decode<DK, DV, false>(args, p);
  return p.extended() ? run_prompt<DK, DV, true>(args, p) : run_prompt<DK, DV, false>(args, p);
}

int run_tensor_shapes(const KernelArgs& args, const RowAttentionParams& p) {
  if (p.dim == 128u && p.vdim == 128u) return run_tensor<128, 128>(args, p);
  if (p.dim == 64u && p.vdim == 64u) return run_tensor<64, 64>(args, p);
  if (p.vdim <= 32u) return run_tensor<0, 32>(args, p);
  if (p.vdim <= 64u) return run_tensor<0, 64>(args, p);
  if (p.vdim <= 128u) return run_tensor<0, 128>(args, p);
  return run_tensor<0, 256>(args, p);
}

// Buffers [query, pool, slot table, past, sequence rows, out, split scratch (counters zero between launches),
// gates (an absent one repeats the queries)].
template <typename T>
int launch_row_attention(const KernelArgs& args) {
  RowAttentionParams p;
  LLMOPT_REQUIRE(args.buffer_count == 8 && args.param_bytes == sizeof(p), "expects 8 buffers and 92 parameter bytes");
  memcpy(&p, args.params, sizeof(p));
  const size_t rows = (size_t)p.sequences * p.tokens, e = sizeof(T);
  LLMOPT_REQUIRE(p.heads > 0 && p.kv_heads > 0 && p.heads % p.kv_heads == 0 && p.dim > 0 && p.vdim > 0 && p.splits > 0,
                 "needs whole groups of query heads");
  LLMOPT_REQUIRE(p.key_offset + p.kv_heads * p.dim <= p.token_stride && p.value_offset + p.kv_heads * p.vdim <= p.token_stride,
                 "key or value segment lies outside the cache row");
  LLMOPT_REQUIRE(p.sequences <= 65535u && p.heads <= 65535u, "too many sequences or heads");
  LLMOPT_REQUIRE((size_t)p.query_column + p.heads * p.dim <= p.query_stride &&
                     (!p.gate_stride || (size_t)p.gate_column + p.heads * p.vdim <= p.gate_stride),
                 "query or gate columns lie outside the row");
  LLMOPT_REQUIRE(args.lengths[7] >= rows * p.gate_stride * e, "gate buffer is too short");
  LLMOPT_REQUIRE(args.lengths[0] >= rows * p.query_stride * e && args.lengths[5] >= rows * p.heads * p.vdim * e &&
                     args.lengths[1] >= (size_t)p.pool_rows * p.token_stride * e && p.pool_rows > 0 &&
                     args.lengths[2] >= (size_t)p.table_rows * p.table_stride * 4 &&
                     args.lengths[3] >= (size_t)p.sequences * 4 && args.lengths[4] >= (size_t)p.sequences * 4,
                 "buffer is too short");
  if (rows == 0) return 0;
  const bool vectors = e == 2 && p.dim % 8u == 0 && p.vdim % 8u == 0 && p.dim <= kWidestHead && p.vdim <= 256u &&
                       p.query_stride % 8u == 0 && p.query_column % 8u == 0 && p.token_stride % 8u == 0 && p.key_offset % 8u == 0 && p.value_offset % 8u == 0 &&
                       ((uintptr_t)args.buffers[0] & 15u) == 0 && ((uintptr_t)args.buffers[1] & 15u) == 0;
  if (vectors) {
    const int status = run_tensor_shapes(args, p);
    if (status >= 0) return status;
  }
  return run_rows<T>(args, p);
}

}  // namespace

const NamedLauncher* row_attention_launchers(size_t* count) {
  static const NamedLauncher table[] = {
      {"llmopt_row_attention_bf16", launch_row_attention<bf16>},
      {"llmopt_row_attention_f32", launch_row_attention<float>},
  };
  *count = sizeof(table) / sizeof(table[0]);
  return table;
}

}  // namespace llmopt
