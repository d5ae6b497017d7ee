// Dense fp16 attention of prompts on the 5th-generation tensor cores (dense_attention.cu has the contract): heads of 64 or 128,
// causal or not, without a mask.
//
// A CTA owns 128 queries of one head and walks over tiles of 128 keys.  One thread brings Q, K and V by TMA (128-byte swizzle)
// and issues tcgen05.mma: S = Q K^T into tensor memory (128 columns), later O += P V (D columns).  Warps of rows read S and write
// P = exp2(S - top) over it as fp16 pairs, the A operand of P V in tensor memory; V is the B operand as it lies in memory,
// dimensions contiguous.  O stays in tensor memory and is scaled, behind the exponentials, where a row's maximum has grown: the largest
// weight is 1 and exact in fp16.  (Left alone until a maximum has grown by 2^8 it is rounded like any other: 2 to 8 % further from 64 bits
// from 333 to 2048 tokens.)  The denominator adds what P V uses.  The first 16 of 64 keys have the remainder of their weight multiplied as
// well, which lies beside the weights: with the maxima of 128 keys instead of 64 fewer weights are exact than on mma.sync, 0.35 % more error;
// with the remainders it is 1 to 10 % less, for 2 to 10 % of the time.
//
// What bounds a tile is the chain from S to P (no pipe is busy for more than 36 % of the time), so two of them run side by side,
// in one of two forms, of which both give the same bits:
//  * ALONE: one CTA per SM, two threads per row, and the next tile's scores multiplied beside this tile's exponentials;
//  * otherwise two CTAs share an SM, a thread per row.
// Up to two CTAs per SM the first is the faster, beyond the second, with either head size.  us, causal, back to back over six sets of
// operands, CTAs and then two per SM, ALONE: heads of 64: 9 5.7, 5.1; 144 38.0, 26.4; 256 21.3, 17.9; 288 23.6, 20.6; 320 26.1, 26.9; 352
// 29.2, 31.4; 512 46.5, 59.1.  Of 128: 128 26.0, 17.0; 256 27.6, 23.9; 288 30.4, 27.3; 320 33.4, 34.4; 352 37.3, 39.4; 512 56.7, 68.4.
// K and V two tiles deep changed nothing: their way hides behind that chain.
//
// P V multiplies the weight of a masked key, zero, with its value, and zero times an infinity is no number.  Queries are left out of
// the products of 64 keys of which they see none, so a value reaches none but the queries that see it and up to 63 before, as on mma.sync.
// Rows beyond a head's keys or queries, and keys behind the last query's, are zero-filled by TMA.  Every wait on an mbarrier is bounded;
// a wait that runs out raises the context's device error word, and the CTA lets its copies land and its products end, frees its tensor
// memory and returns.
#include <cuda.h>

#include <type_traits>

#include "dense_attention.cuh"
#include "w4a16_tc_device.cuh"

namespace llmopt {
using namespace tc;

uint32_t* context_device_error(Context* ctx);

namespace {

constexpr uint32_t kTile = 128;      // queries, and keys of a tile
constexpr uint32_t kBlockBytes = kTile * 128;  // 64 dimensions of 128 rows
constexpr float kLowest = -1.0e30f;

// Keys that some query sees; beyond, memory need not hold numbers, and TMA puts zeros there.
__host__ __device__ inline uint32_t seen_by_any(const DenseParams& p) {
  return p.causal && p.k_len > p.past_length && p.k_len - p.past_length > p.q_len ? p.q_len + p.past_length : p.k_len;
}

template <int D, bool ALONE>
struct Shape {
  static constexpr uint32_t kHalves = ALONE ? 2 : 1, kRowWarps = 4 * kHalves, kThreads = (kRowWarps + 1) * 32;
  static constexpr uint32_t kKeys = kTile / kHalves;  // of a thread
  static constexpr uint32_t kScores = ALONE ? 2 : 1;  // tiles of scores in tensor memory
  static constexpr uint32_t kColumns = ALONE ? 512 : 256;
  static constexpr uint32_t kBlocks = D / 64;
  static constexpr uint32_t kTileBytes = kBlocks * kBlockBytes;
  static constexpr uint32_t kK = kTileBytes, kV = 2 * kTileBytes, kBarriers = 3 * kTileBytes;
  static constexpr uint32_t kHolder = kBarriers + 8 * 8;
  static constexpr uint32_t kExchange = kHolder + 16;  // [parity][half][row] floats
  static constexpr uint32_t kUsed = kExchange + (ALONE ? 4 * kTile * 4 : 0) + 1024;  // slack: 1024-byte alignment of the tiles
  // no more CTAs find room on an SM than there is tensor memory for
  static constexpr uint32_t kLeast = (ALONE ? 117u : 80u) * 1024u, kSharedBytes = kUsed > kLeast ? kUsed : kLeast;
};

__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tma_load_4d(uint32_t destination, const CUtensorMap* map, int32_t x, int32_t row, int32_t head,
                                            int32_t batch, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(destination), "l"(map), "r"(bar), "r"(x), "r"(row), "r"(head), "r"(batch)
      : "memory");
}
// LOWER: the first 64 rows (lanes) keep what they have.
template <bool LOWER>
__device__ __forceinline__ void mma_f16_weights(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t instruction, uint32_t accumulate) {
  if constexpr (LOWER)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %6, %6}, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(instruction), "r"(accumulate), "r"(0xffffffffu), "r"(0u)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(instruction), "r"(accumulate), "r"(0u)
        : "memory");
}
__device__ __forceinline__ void tmem_store_8(uint32_t address, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(address), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void tmem_store_16(uint32_t address, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(address), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_store_32(uint32_t address, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(address), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
        "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
        "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_load() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_store() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// B operand whose rows (k) are 128 bytes of 64 columns (n): 128-byte swizzle, eight rows 1024 bytes apart, the next 64 columns
// kBlockBytes on.
__device__ __forceinline__ uint64_t value_descriptor(uint32_t shared_address) {
  uint64_t descriptor = 0;
  descriptor |= (uint64_t)((shared_address & 0x3ffffu) >> 4);
  descriptor |= (uint64_t)(kBlockBytes >> 4) << 16;  // leading byte offset
  descriptor |= (uint64_t)(1024 >> 4) << 32;         // stride byte offset
  descriptor |= (uint64_t)1 << 46;
  descriptor |= (uint64_t)2 << 61;
  return descriptor;
}

template <int D, bool ALONE>
__global__ void __launch_bounds__(Shape<D, ALONE>::kThreads, ALONE ? 1 : 2)
dense_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                          const __grid_constant__ CUtensorMap map_v, __half* output, DenseParams p, uint32_t* error_word) {
  using S = Shape<D, ALONE>;
  extern __shared__ unsigned char shared_raw[];
  grid_chain_prologue();
  const uint32_t base = (smem_u32(shared_raw) + 1023u) & ~1023u;
  unsigned char* base_pointer = shared_raw + (base - smem_u32(shared_raw));
  const uint32_t q_full = base + S::kBarriers, k_full = q_full + 8, v_full = q_full + 16;
  const uint32_t weights_full = q_full + 24, sums_full = q_full + 32, scores_full = q_full + 40;  // scores_full: one per tile in tensor memory
  volatile uint32_t* holder = reinterpret_cast<volatile uint32_t*>(base_pointer + S::kHolder);
  volatile uint32_t* abort_flag = holder + 1;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  // the last query tiles see the most keys under a causal mask: they are scheduled first, over all heads
  const uint32_t q0 = (gridDim.y - 1u - blockIdx.y) * kTile, head = blockIdx.x, batch = blockIdx.z;
  const uint32_t key_end = p.causal ? min(p.k_len, min(q0 + kTile, p.q_len) + p.past_length) : p.k_len;
  // Tiles of keys begin so that 64 keys in line are the diagonal of 64 queries; the first may begin ahead of the first key.
  const uint32_t lead = p.causal ? (64u - p.past_length % 64u) % 64u : 0u;
  const uint32_t tiles = (key_end + lead + kTile - 1u) / kTile;

  if (threadIdx.x == 0) {
    barrier_init(q_full, 1);  // the expect_tx arrivals; complete by byte count
    barrier_init(k_full, 1);
    barrier_init(v_full, 1);
    for (uint32_t i = 0; i < S::kScores; ++i) barrier_init(scores_full + i * 8, 1);  // one tcgen05.commit
    barrier_init(weights_full, S::kRowWarps);  // one arrival per warp of rows
    barrier_init(sums_full, 1);    // one tcgen05.commit
    *abort_flag = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == S::kRowWarps) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(base + S::kHolder), "r"(S::kColumns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t scores = *holder, sums = scores + S::kScores * kTile;  // columns of tensor memory
  auto give_up = [&]() {
    *abort_flag = 1u;
    if (error_word) atomicExch(error_word, 1u);
  };

  if (warp == S::kRowWarps) {
    if (lane == 0) {
      const int32_t kv_head = (int32_t)(head / (p.heads / p.kv_heads));
      uint32_t k_issued = 0, v_issued = 0, scores_issued = 0, sums_issued = 0;
      auto load = [&](const CUtensorMap* map, uint32_t target, int32_t row, int32_t of_head, uint32_t bar) {
        barrier_expect_tx(bar, S::kTileBytes);
#pragma unroll
        for (uint32_t block = 0; block < S::kBlocks; ++block)
          tma_load_4d(base + target + block * kBlockBytes, map, (int32_t)(block * 64u), row, of_head, (int32_t)batch, bar);
      };
      auto first_key = [&](uint32_t tile) { return (int32_t)(tile * kTile) - (int32_t)lead; };
      load(&map_q, 0, (int32_t)q0, (int32_t)head, q_full);
      load(&map_k, S::kK, first_key(0), kv_head, k_full), ++k_issued;
      load(&map_v, S::kV, first_key(0), kv_head, v_full), ++v_issued;
      auto multiply = [&](uint32_t tile) {  // S = Q K^T
        if (*abort_flag || !barrier_wait(k_full, tile & 1u)) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t which = tile % S::kScores;
#pragma unroll
        for (uint32_t j = 0; j < D / 16; ++j) {
          const uint32_t at = j / 4u * kBlockBytes + j % 4u * 32u;
          mma_f16(scores + which * kTile, operand_descriptor(base + at), operand_descriptor(base + S::kK + at), j > 0 ? 1u : 0u,
                  instruction_descriptor(kTile, kTile));
        }
        mma_commit(scores_full + which * 8u), ++scores_issued;
        return true;
      };
      auto add_values = [&](uint32_t tile, uint32_t upper, auto lower) {  // O += P V of the first or last 64 keys
        const uint32_t first = scores + tile % S::kScores * kTile;
        const uint32_t instruction = instruction_descriptor(kTile, D) | (1u << 16);  // bit 16: the B operand's columns are contiguous
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
          const uint32_t j = upper * 4u + i, half = upper * 64u / S::kKeys, weights = first + half * S::kKeys;
          const uint64_t values = value_descriptor(base + S::kV + j * 2048u);
          mma_f16_weights<decltype(lower)::value>(sums, weights + (j * 16u - half * S::kKeys) / 2u, values, instruction, (tile > 0 || j > 0) ? 1u : 0u);
          if (i == 0)  // and the remainders of the weights
            mma_f16_weights<decltype(lower)::value>(sums, weights + S::kKeys / 2u + (upper - half) * 8u, values, instruction, 1u);
        }
      };
      bool ok = barrier_wait(q_full, 0) && multiply(0);
      for (uint32_t tile = 0; tile < tiles && ok; ++tile) {
        const uint32_t which = tile % S::kScores;
        ok = barrier_wait(scores_full + which * 8u, tile / S::kScores & 1u);  // K is read
        if (!ok) break;
        if (tile + 1u < tiles) {
          load(&map_k, S::kK, first_key(tile + 1u), kv_head, k_full), ++k_issued;
          if (ALONE) ok = multiply(tile + 1u);  // beside this tile's exponentials; its place was last read by P V of the tile before
        }
        ok = ok && !*abort_flag && barrier_wait(v_full, tile & 1u) && barrier_wait(weights_full, tile & 1u);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // zero times an infinity is no number: the first 64 queries leave 64 keys out of which they see none
        const bool apart = p.causal && first_key(tile) + 64 > (int32_t)(q0 + p.past_length);
        if (!apart) {
          add_values(tile, 0, std::false_type());
          add_values(tile, 1, std::false_type());
        } else if (first_key(tile) <= (int32_t)(q0 + p.past_length)) {
          add_values(tile, 0, std::false_type());
          add_values(tile, 1, std::true_type());
        } else {  // nobody sees the last ones
          add_values(tile, 0, std::true_type());
        }
        mma_commit(sums_full), ++sums_issued;
        ok = barrier_wait(sums_full, tile & 1u);  // V and the weights are read
        if (ok && tile + 1u < tiles) {
          load(&map_v, S::kV, first_key(tile + 1u), kv_head, v_full), ++v_issued;
          if (!ALONE) ok = multiply(tile + 1u);
        }
      }
      if (!ok || *abort_flag) {  // what is under way must end before shared and tensor memory are given back
        give_up();
        barrier_wait(q_full, 0);
        barrier_wait(k_full, (k_issued - 1u) & 1u);
        barrier_wait(v_full, (v_issued - 1u) & 1u);
        if (scores_issued) barrier_wait(scores_full + (scores_issued - 1u) % S::kScores * 8u, (scores_issued - 1u) / S::kScores & 1u);
        if (sums_issued) barrier_wait(sums_full, (sums_issued - 1u) & 1u);
      }
    }
  } else {
    const uint32_t row = threadIdx.x % kTile, half = threadIdx.x / kTile;  // of this thread
    const uint32_t lanes = (warp % 4u * 32u) << 16, query = q0 + row;
    float* const exchange = reinterpret_cast<float*>(base_pointer + S::kExchange);
    auto of_row = [&](uint32_t parity, uint32_t of_half) -> float& { return exchange[(parity * 2u + of_half) * kTile + row]; };
    auto halves_sync = [] { asm volatile("bar.sync 1, 256;" ::: "memory"); };
    const float scale = p.scale * 1.4426950408889634f;
    float top = kLowest;  // in units of log2 e
    float of_halves[3u - S::kHalves] = {};  // denominators; a tile's halves apart in either form, which gives both the same bits
    bool ok = true;
    for (uint32_t tile = 0; tile < tiles; ++tile) {
      const uint32_t which = tile % S::kScores, k0 = tile * kTile + half * S::kKeys;
      const uint32_t mine = scores + which * kTile + half * S::kKeys + lanes;
      ok = ok && !*abort_flag && barrier_wait(scores_full + which * 8u, tile / S::kScores & 1u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (ALONE) halves_sync();  // the other half may be waiting there
        continue;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // keys below `seen` are visible to this row; all of them to the whole warp where `whole`
      const uint32_t limit = lead + (p.causal ? min(p.k_len, query + p.past_length + 1u) : p.k_len), seen = limit > k0 ? limit - k0 : 0u;
      const bool whole = __all_sync(0xffffffffu, seen >= S::kKeys);
      uint32_t raw[S::kKeys / 32u][32];
#pragma unroll
      for (uint32_t part = 0; part < S::kKeys / 32u; ++part) tmem_load_32(mine + part * 32u, raw[part]);
      tmem_wait_load();
      if (k0 < lead) {  // what lies ahead of the first key
#pragma unroll
        for (uint32_t i = 0; i < 64u; ++i)
          if (i < lead) raw[i / 32][i % 32] = 0xff800000u;
      }
      float four[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (whole) {
#pragma unroll
        for (uint32_t i = 0; i < S::kKeys; ++i) four[i & 3] = fmaxf(four[i & 3], __uint_as_float(raw[i / 32][i % 32]));
      } else {
#pragma unroll
        for (uint32_t i = 0; i < S::kKeys; ++i)
          if (i < seen) four[i & 3] = fmaxf(four[i & 3], __uint_as_float(raw[i / 32][i % 32]));
      }
      float most = fmaxf(fmaxf(four[0], four[1]), fmaxf(four[2], four[3])) * scale;  // scale is positive
      if (ALONE) {
        of_row(tile & 1u, half) = most;
        halves_sync();
        most = fmaxf(most, of_row(tile & 1u, half ^ 1u));
      }
      const bool grown = most > top;
      const bool any = __any_sync(0xffffffffu, grown);
      const float keep = grown ? exp2_fast(top - most) : 1.0f;
      if (grown) top = most;
#pragma unroll
      for (float& part : of_halves) part *= keep;
#pragma unroll
      for (uint32_t part = 0; part < S::kKeys / 32u; ++part) {
        uint32_t weights[16], rests[8];
        float two[2] = {0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float low = exp2_fast(fmaf(__uint_as_float(raw[part][2 * i]), scale, -top));
          float high = exp2_fast(fmaf(__uint_as_float(raw[part][2 * i + 1]), scale, -top));
          if (!whole) {
            low = part * 32u + 2u * i < seen ? low : 0.0f;
            high = part * 32u + 2u * i + 1u < seen ? high : 0.0f;
          }
          const __half2 pair = __floats2half2_rn(low, high);
          weights[i] = *reinterpret_cast<const uint32_t*>(&pair);
          const float2 rounded = __half22float2(pair);
          if (part % 2u == 0 && i < 8) {
            two[0] += low;
            two[1] += high;
            const __half2 rest = __floats2half2_rn(low - rounded.x, high - rounded.y);
            rests[i] = *reinterpret_cast<const uint32_t*>(&rest);
          } else {
            two[0] += rounded.x;
            two[1] += rounded.y;
          }
        }
        of_halves[ALONE ? 0u : part / 2u] += two[0] + two[1];
        tmem_store_16(mine + part * 16u, weights);  // over scores that are in registers
        if (part % 2u == 0) tmem_store_8(mine + S::kKeys / 2u + part / 2u * 8u, rests);
      }
      // A wait names a phase by its parity, so nobody may be two phases behind: with two tiles of scores a row could be done with this
      // tile before P V of the one before has begun (V late), which would end the wait for the last P V too early, and run
      // `weights_full` past the thread that waits for it.  tests/test_barrier_order_cpu.py goes through every order.
      if (ALONE && tile > 0) ok = barrier_wait(sums_full, (tile - 1u) & 1u) && ok;
      if (any && tile > 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
        for (uint32_t part = half * (D / 32u / S::kHalves); part < (half + 1u) * (D / 32u / S::kHalves); ++part) {
          uint32_t held[32];
          tmem_load_32(sums + lanes + part * 32u, held);
          tmem_wait_load();
#pragma unroll
          for (int i = 0; i < 32; ++i) held[i] = __float_as_uint(__uint_as_float(held[i]) * keep);
          tmem_store_32(sums + lanes + part * 32u, held);
        }
      }
      tmem_wait_store();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) barrier_arrive(weights_full);
    }
    float total = of_halves[0] + of_halves[2u - S::kHalves];
    if (ALONE) {
      of_row(tiles & 1u, half) = of_halves[0];
      halves_sync();
      total = of_row(tiles & 1u, 0) + of_row(tiles & 1u, 1);
    }
    ok = ok && !*abort_flag && barrier_wait(sums_full, (tiles - 1u) & 1u);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) give_up();
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float inverse = total == 0.0f ? 0.0f : 1.0f / total;
      __half* const target = output + (p.token_first_output ? (((size_t)batch * p.q_len + query) * p.heads + head) * D
                                                            : (((size_t)batch * p.heads + head) * p.q_len + query) * D);
#pragma unroll 1
      for (uint32_t part = half * (D / 32u / S::kHalves); part < (half + 1u) * (D / 32u / S::kHalves); ++part) {
        uint32_t raw[32];
        tmem_load_32(sums + lanes + part * 32u, raw);
        tmem_wait_load();
        if (query < p.q_len) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint32_t words[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const __half2 pair = __floats2half2_rn(__uint_as_float(raw[i * 8 + j * 2]) * inverse, __uint_as_float(raw[i * 8 + j * 2 + 1]) * inverse);
              words[j] = *reinterpret_cast<const uint32_t*>(&pair);
            }
            *reinterpret_cast<uint4*>(target + part * 32u + i * 8) = make_uint4(words[0], words[1], words[2], words[3]);
          }
        }
        __syncwarp();  // tcgen05.ld needs the whole warp
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
  }

  __syncthreads();
  if (warp == S::kRowWarps) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(scores), "r"(S::kColumns) : "memory");
  }
}

// cuTensorMapEncodeTiled, resolved through the runtime so that the library does not link libcuda.
typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The first `seen` of `rows` rows of `dim` fp16 in boxes of 64 x 128: [batch][head][row], or [batch][row][head] (token first).
bool make_map(CUtensorMap* map, const void* base, uint64_t dim, uint64_t rows, uint64_t seen, uint64_t heads, uint64_t batches, bool token_first) {
  static EncodeTiled encode = []() -> EncodeTiled {
    void* pointer = nullptr;
    cudaDriverEntryPointQueryResult result;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &pointer, cudaEnableDefault, &result) != cudaSuccess ||
        result != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<EncodeTiled>(pointer);
  }();
  if (encode == nullptr) return false;
  const cuuint64_t dims[4] = {dim, seen, heads, batches};
  const cuuint64_t strides[3] = {(token_first ? heads : 1u) * dim * 2u, (token_first ? 1u : rows) * dim * 2u, rows * heads * dim * 2u};
  const cuuint32_t box[4] = {64, kTile, 1, 1}, element_strides[4] = {1, 1, 1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(base), dims, strides, box, element_strides,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int D, bool ALONE>
int run(const KernelArgs& args, const DenseParams& p) {
  using S = Shape<D, ALONE>;
  CUtensorMap map_q, map_k, map_v;
  if (!make_map(&map_q, args.buffers[0], D, p.q_len, p.q_len, p.heads, p.batches, false) ||
      !make_map(&map_k, args.buffers[1], D, p.k_len, seen_by_any(p), p.kv_heads, p.batches, false) ||
      !make_map(&map_v, args.buffers[2], D, p.k_len, seen_by_any(p), p.kv_heads, p.batches, p.token_first_value != 0))
    return -1;
  auto kernel = dense_attention_tc_kernel<D, ALONE>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSharedBytes) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  launch_kernel(args, kernel, dim3(p.heads, (p.q_len + kTile - 1u) / kTile, p.batches), dim3(S::kThreads), S::kSharedBytes, map_q, map_k,
                map_v, (__half*)args.buffers[4], p, args.ctx ? context_device_error(args.ctx) : nullptr);
  return check_launch(args);
}

}  // namespace

int launch_attention_dense_tc(const KernelArgs& args, const DenseParams& p) {
  if (!(p.scale > 0.0f)) return -1;  // the largest score is that of the largest product
  if (args.ctx == nullptr || p.mask_batches != 0 || p.batches > 65535u || p.q_len > 65535u * kTile || (p.dim != 64u && p.dim != 128u)) return -1;
  if (p.causal && (uint64_t)p.q_len + p.past_length > 0x7fffff00ull) return -1;  // TMA's coordinates
  for (int i = 0; i < 5; ++i)
    if (i != 3 && ((uintptr_t)args.buffers[i] & 15u)) return -1;
  const size_t ctas = (size_t)p.heads * ((p.q_len + kTile - 1u) / kTile) * p.batches;
  const bool alone = ctas <= 2u * (size_t)context_sm_count(args.ctx);
  if (p.dim == 64u) return alone ? run<64, true>(args, p) : run<64, false>(args, p);
  return alone ? run<128, true>(args, p) : run<128, false>(args, p);
}

}  // namespace llmopt
