// Pieces of the kernels that stream bfloat16 weight rows from HBM straight into mma.sync fragments, for few
// activation rows: a warp holds 16 weight rows against NT tiles of eight activation rows.
#pragma once
#include "dense_linear.cuh"

namespace llmopt {
namespace {

constexpr int kGemvWarps = 8;
constexpr int kGemvStages = 3;  // 64-wide k-blocks a warp keeps in flight

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint4 load_stream(const bf16* source) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(source));
  return v;
}

// A 64-wide k-block of the lane's two weight rows: low / high 32 k of each; zeros from `width` on.
__device__ __forceinline__ void stream_fetch(uint4 (&stage)[4], const bf16* w_low, const bf16* w_high, uint32_t width,
                                             uint32_t block) {
  const uint32_t t = threadIdx.x & 3u;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const uint32_t k = block * 64u + half * 32u + t * 8u;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    stage[half] = k < width ? load_stream(w_low + k) : zero;
    stage[2 + half] = k < width ? load_stream(w_high + k) : zero;
  }
}

// sum += a half (32 k) of a k-block of the weights times the same k of a tile's rows.
__device__ __forceinline__ void stream_multiply(float (&sum)[4], const uint4& low, const uint4& high, const uint4& x) {
  mma_bf16(sum, low.x, high.x, low.y, high.y, x.x, x.y);
  mma_bf16(sum, low.z, high.z, low.w, high.w, x.z, x.w);
}

// A warp's sums, [activation row][weight row].
template <int NT>
__device__ __forceinline__ void stream_collect(const float (&sum)[NT][4], float (&mine)[NT * 8][17]) {
  const uint32_t lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) mine[nt * 8 + 2 * t + (i & 1)][g + (i >> 1) * 8] = sum[nt][i];
}

template <DenseStore STORE, int N>
__device__ __forceinline__ void stream_store(const DenseTask<STORE>& p, uint32_t row, uint32_t column, const float (&value)[N]) {
  if constexpr (STORE == kStorePair) dense_store_pair<bf16>(p, row, column, value[0], value[N - 1]);
  else dense_store<bf16>(p, row, column, value[0]);
}

// Adds the warps' sums of the 16 columns from n0 on (and those of the cluster's CTAs) and stores them.
template <int NT, DenseStore STORE>
__device__ __forceinline__ void stream_finish(const DenseTask<STORE>& p, float (&partial)[kGemvWarps][NT * 8][17], uint32_t n0,
                                              uint32_t rank, uint32_t cluster) {
  const uint32_t stride = kGemvWarps * cluster;
  __syncthreads();
  constexpr uint32_t kStep = STORE == kStorePair ? 2u : 1u;  // columns a thread stores together
  for (uint32_t index = threadIdx.x * kStep; index < NT * 8u * 16u; index += kGemvWarps * 32 * kStep) {
    const uint32_t column = index & 15u, row = index >> 4;
    if (row >= p.m || n0 + column >= p.n) continue;
    float value[kStep];
#pragma unroll
    for (uint32_t i = 0; i < kStep; ++i) {
      value[i] = 0.0f;
#pragma unroll
      for (int part = 0; part < kGemvWarps; ++part) value[i] += partial[part][row][column + i];
      if (cluster > 1u) partial[0][row][column + i] = value[i];  // read and written by this thread only
    }
    if (cluster == 1u) stream_store(p, row, n0 + column, value);
  }
  if (cluster == 1u) return;
  cluster_sync();
  // the cluster's CTAs share out the outputs; sums in rank order
  for (uint32_t index = (rank * kGemvWarps * 32 + threadIdx.x) * kStep; index < NT * 8u * 16u; index += stride * 32u * kStep) {
    const uint32_t column = index & 15u, row = index >> 4;
    if (row >= p.m || n0 + column >= p.n) continue;
    float value[kStep];
#pragma unroll
    for (uint32_t i = 0; i < kStep; ++i) {
      value[i] = 0.0f;
      for (uint32_t other = 0; other < cluster; ++other) value[i] += cluster_load(&partial[0][row][column + i], other);
    }
    stream_store(p, row, n0 + column, value);
  }
  cluster_sync();  // nobody leaves while its sums may be read
}

// ---- many tiles: persistent CTAs ------------------------------------------------------------------
// A CTA walks over tiles of 16 weight rows.  Eight warps share out a tile's k-blocks as in the kernels above; the blocks come
// by cp.async into a ring of the lane that uses them (no other lane reads it, so nothing synchronises), across the ends of
// tiles.  The activation rows lie in shared memory for all tiles.  Four more warps add the eight sums of one tile and store
// it while the next is under way.
constexpr uint32_t kRingDepth = 4, kFinishWarps = 4, kWideThreads = (kGemvWarps + kFinishWarps) * 32;
constexpr uint32_t kWideMost = 232448;  // bytes of shared memory a CTA can have

__device__ __forceinline__ void ring_copy(uint4* target, const bf16* source, bool present) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(target)), "l"(source),
               "r"(present ? 16u : 0u)
               : "memory");
}
__device__ __forceinline__ void wide_barrier_sync(uint32_t id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kWideThreads) : "memory");
}
__device__ __forceinline__ void wide_barrier_arrive(uint32_t id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(kWideThreads) : "memory");
}

// Shared memory: rings, two tiles' sums, activation rows of whole k-blocks.
template <int NT>
struct WideShape {
  static constexpr uint32_t kRingBytes = kGemvWarps * kRingDepth * 4u * 32u * 16u;
  static constexpr uint32_t kMostPerSm = NT == 1 ? 2u : 1u;  // CTAs, by registers
  typedef float Sums[kGemvWarps][NT * 8][17];
  static constexpr uint32_t kRowsAt = kRingBytes + 2u * sizeof(Sums);
  __host__ __device__ static constexpr uint32_t bytes(uint32_t k) { return kRowsAt + NT * 8u * ((k + 63u) / 64u * 128u); }
};
// Sixteen-byte chunk `chunk` of a row; odd rows swap the halves of a k-block, so that two rows fill the banks.
__device__ __forceinline__ uint32_t wide_chunk(uint32_t row, uint32_t blocks, uint32_t chunk) {
  return row * blocks * 8u + (chunk ^ ((row & 1u) * 4u));
}

// Rows of k elements to shared memory, zeros behind row `m` up to `count` and behind k.  Eight pieces of a thread are under way
// together: one at a time, 8 rows of k 4096 took 5 us.
__device__ __forceinline__ void wide_stage_rows(uint4* rows, const bf16* x, uint32_t count, uint32_t m, uint32_t k, uint32_t blocks) {
  constexpr int kAhead = 8;
  const uint32_t chunks = blocks * 8u, all = count * chunks;
  for (uint32_t begin = threadIdx.x; begin < all; begin += kAhead * kWideThreads) {
    uint4 value[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const uint32_t index = begin + i * kWideThreads, row = index / chunks, chunk = index - row * chunks;
      value[i] = make_uint4(0u, 0u, 0u, 0u);
      if (index < all && row < m && chunk * 8u < k) value[i] = *reinterpret_cast<const uint4*>(x + (size_t)row * k + chunk * 8u);
    }
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const uint32_t index = begin + i * kWideThreads, row = index / chunks, chunk = index - row * chunks;
      if (index < all) rows[wide_chunk(row, blocks, chunk)] = value[i];
    }
  }
}

// The ring of one lane.  tile_of(index, low, high) says where the lane's two weight rows of the CTA's tile number `index`
// begin.
template <typename Tile>
struct WideRing {
  uint4* slots;  // of the lane: piece i of stage s at (4 s + i) * 32
  const Tile& tile_of;
  const bf16 *low, *high;
  uint32_t k, blocks, warp, t, tiles, tile, block, fill, drain;
  __device__ __forceinline__ WideRing(unsigned char* shared, const Tile& tile_of, uint32_t k, uint32_t tiles)
      : slots(reinterpret_cast<uint4*>(shared) + (threadIdx.x >> 5) * kRingDepth * 128u + (threadIdx.x & 31u)), tile_of(tile_of), k(k),
        blocks((k + 63u) / 64u), warp(threadIdx.x >> 5), t(threadIdx.x & 3u), tiles(warp < blocks ? tiles : 0u), tile(0), block(warp),
        fill(0), drain(0) {
    if (tile < this->tiles) tile_of(tile, low, high);
#pragma unroll
    for (uint32_t i = 0; i + 1u < kRingDepth; ++i) fetch();
  }
  __device__ __forceinline__ void fetch() {
    if (tile < tiles) {
#pragma unroll
      for (uint32_t half = 0; half < 2u; ++half) {
        const uint32_t at = block * 64u + half * 32u + t * 8u;
        const bool present = at < k;
        ring_copy(slots + (fill * 4u + half) * 32u, present ? low + at : low, present);
        ring_copy(slots + (fill * 4u + 2u + half) * 32u, present ? high + at : high, present);
      }
      block += kGemvWarps;
      if (block >= blocks) {
        block = warp;
        if (++tile < tiles) tile_of(tile, low, high);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    fill = (fill + 1u) % kRingDepth;
  }
  // The next block's pieces: low / high 32 k of the row g, then of row g + 8.
  __device__ __forceinline__ void next(uint4 (&pieces)[4]) {
    fetch();  // into the slot that the block before was read from
    asm volatile("cp.async.wait_group %0;" ::"n"(kRingDepth - 1) : "memory");
#pragma unroll
    for (uint32_t i = 0; i < 4u; ++i) pieces[i] = slots[(drain * 4u + i) * 32u];
    drain = (drain + 1u) % kRingDepth;
  }
};

// A tile's eight sums in warp order, stored by the finishing warps' thread number `thread`.
template <int NT, DenseStore STORE>
__device__ __forceinline__ void wide_finish(const DenseTask<STORE>& p, const float (&sums)[kGemvWarps][NT * 8][17], uint32_t n0, uint32_t thread) {
  constexpr uint32_t kStep = STORE == kStorePair ? 2u : 1u;  // columns a thread stores together
#pragma unroll 2
  for (uint32_t index = thread * kStep; index < NT * 8u * 16u; index += kFinishWarps * 32u * kStep) {
    const uint32_t column = index & 15u, row = index >> 4;
    if (row >= p.m || n0 + column >= p.n) continue;
    float value[kStep];
#pragma unroll
    for (uint32_t i = 0; i < kStep; ++i) {
      value[i] = 0.0f;
#pragma unroll
      for (int part = 0; part < kGemvWarps; ++part) value[i] += sums[part][row][column + i];
    }
    stream_store(p, row, n0 + column, value);
  }
}

// CTAs for `tiles` tiles: whole rounds of as many as fit, shared out evenly.  `bytes` of shared memory, at most `most` per SM by
// registers.
inline uint32_t wide_ctas(const KernelArgs& args, uint32_t tiles, uint32_t bytes, uint32_t most) {
  const uint32_t per_sm = most >= 2u && kWideMost / (bytes + 1024u) >= 2u ? 2u : 1u;
  const uint32_t together = per_sm * (uint32_t)context_sm_count(args.ctx), rounds = (tiles + together - 1u) / together;
  return (tiles + rounds - 1u) / rounds;
}

// CTAs per cluster that share out the k-blocks of `tiles` 16-row tiles: at least one CTA per SM, and a warp of a
// split keeps at least one of the `blocks`.
inline uint32_t stream_cluster(const KernelArgs& args, uint32_t tiles, uint32_t blocks) {
  const uint32_t wanted = (uint32_t)context_sm_count(args.ctx);
  uint32_t cluster = 1;
  while (cluster < 8u && tiles * cluster < wanted && blocks >= 2u * cluster * kGemvWarps) cluster *= 2u;
  return cluster;
}

}  // namespace
}  // namespace llmopt
