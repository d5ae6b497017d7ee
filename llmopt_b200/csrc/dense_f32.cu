// Dense linear layer in fp32 (CUDA cores, no TF32) where weight and activation rows are whole 16-byte vectors:
//  * up to 8 rows: dense_f32_stream_kernel, bound by the weight stream.  A warp takes four columns, so that an activation
//    vector serves four weight vectors, and four warps share out a column's k.
//  * more rows: dense_f32_tile_kernel, bound by the multiply-adds (128 per cycle and SM).  Operands go through shared memory
//    by cp.async in k-major rows as they lie in memory; a thread reads four k of a row at once and feeds packed
//    multiply-adds (fma.rn.f32x2) whose two halves are the even and the odd k, which needs no rearrangement.  Few rows make
//    few tiles: a cluster of up to eight CTAs shares out a tile's k and adds its sums in rank order through distributed
//    shared memory.
// Measured against one warp per column with 4-byte loads and 64 x 64 tiles over all of k (dense_linear.cu), 100 rows:
// 2048 x 7168 1076 -> 99 us, 7168 x 2048 438 -> 106, 2048 x 2048 313 -> 32, 256 x 2048 183 -> 20 (28 TFLOP/s at the first,
// of 74 that the multiply-adds could do; 128 rows are computed for 100).
#include "dense_linear.cuh"

namespace llmopt {
namespace {

constexpr uint32_t kColumns = 128;  // of a tile
constexpr uint32_t kDepth = 32;    // k of a stage: a row is one 128-byte line
constexpr uint32_t kPitch = kDepth + 4;  // floats; eight consecutive rows start in eight different groups of four banks
constexpr uint32_t kStages = 3;
constexpr uint32_t kThreads = 128;

__device__ __forceinline__ void multiply_add_two(unsigned long long& sum, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum) : "l"(a), "l"(b));
}
__device__ __forceinline__ float both(unsigned long long sum) {
  return __uint_as_float((uint32_t)sum) + __uint_as_float((uint32_t)(sum >> 32));
}
// 16 bytes to shared memory, zeros where absent.
__device__ __forceinline__ void copy_vector(float* to, const float* from, bool present) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from),
               "r"(present ? 16u : 0u)
               : "memory");
}
__device__ __forceinline__ float4 cluster_load_four(const float* local, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(remote)
               : "memory");
  return v;
}

// A tile of 8 TM rows x 128 columns; thread (mi, ni) of 8 x 16 owns rows mi + 8 i and columns ni + 16 j.  With 8 x 8 sums a
// thread reads sixteen vectors for 128 packed multiply-adds, so that the reads (four cycles of the shared memory per warp) and
// the arithmetic take the same time; with 8 x 4 the reads bound it (7168 x 2048: 121 us).
template <int TM, DenseStore STORE>
__global__ void __launch_bounds__(kThreads, TM == 8 ? 2 : 3) dense_f32_tile_kernel(const DenseTask<STORE> p, const DensePlan plan) {
  constexpr uint32_t kRows = 8 * TM;
  constexpr uint32_t kStageFloats = (kRows + kColumns) * kPitch;
  constexpr uint32_t kSumPitch = kColumns + 4;
  static_assert(kRows * kSumPitch <= kStages * kStageFloats, "the sums take the stages' place");
  extern __shared__ __align__(16) float stages[];
  const uint32_t cluster = p.cluster, rank = blockIdx.x % cluster, n0 = blockIdx.x / cluster * kColumns;
  const float* x = reinterpret_cast<const float*>(p.x);
  const float* w = reinterpret_cast<const float*>(p.w);
  uint32_t m0 = blockIdx.y * kRows, row_end = p.m;
  grid_launch_dependents();
  if (plan.tiles) {  // rows sorted by expert; a tile of the plan is cut into tiles of this kernel
    grid_dependency_wait();
    constexpr uint32_t kParts = kExpertTile / kRows;
    const uint32_t index = blockIdx.y / kParts;
    if (index >= plan.tiles[0]) return;  // all CTAs of a cluster have the same rows
    const DenseTile tile = dense_tile(plan, index);
    m0 = tile.first + blockIdx.y % kParts * kRows;
    row_end = min(tile.end, p.m);
    if (m0 >= row_end || tile.expert >= plan.experts) return;
    w += (size_t)tile.expert * p.n * p.k;
  }
  const uint32_t blocks = (p.k + kDepth - 1u) / kDepth;
  const uint32_t first = (uint32_t)((unsigned long long)blocks * rank / cluster);
  const uint32_t end = (uint32_t)((unsigned long long)blocks * (rank + 1u) / cluster);
  const uint32_t lane_k = (threadIdx.x & 7u) * 4u, lane_row = threadIdx.x >> 3;  // of the copies
  auto copy_x = [&](uint32_t block) {
    float* const to = stages + block % kStages * kStageFloats;
    const uint32_t k = block * kDepth + lane_k;
#pragma unroll
    for (uint32_t row = lane_row; row < kRows; row += 16u) {
      const bool present = k < p.k && m0 + row < row_end;
      copy_vector(to + row * kPitch + lane_k, present ? x + (size_t)(m0 + row) * p.k + k : x, present);
    }
  };
  auto copy_w = [&](uint32_t block) {
    float* const to = stages + block % kStages * kStageFloats + kRows * kPitch;
    const uint32_t k = block * kDepth + lane_k;
#pragma unroll
    for (uint32_t row = lane_row; row < kColumns; row += 16u) {
      const bool present = k < p.k && n0 + row < p.n;
      copy_vector(to + row * kPitch + lane_k, present ? w + (size_t)(n0 + row) * p.k + k : w, present);
    }
  };
  // the weights are nobody's output: their first stages may be requested before the predecessor ends
#pragma unroll
  for (uint32_t s = 0; s + 1u < kStages; ++s)
    if (first + s < end) copy_w(first + s);
  grid_dependency_wait();
#pragma unroll
  for (uint32_t s = 0; s + 1u < kStages; ++s) {
    if (first + s < end) copy_x(first + s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t mi = (lane >> 3) + 4u * (warp & 1u), ni = (lane & 7u) + 8u * (warp >> 1);
  unsigned long long sum[TM][8];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) sum[i][j] = 0ull;
  for (uint32_t block = first; block < end; ++block) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();  // this stage has arrived, and the one before it is read
    if (block + kStages - 1u < end) {
      copy_w(block + kStages - 1u);
      copy_x(block + kStages - 1u);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* const xs = stages + block % kStages * kStageFloats + mi * kPitch;
    const float* const ws = stages + block % kStages * kStageFloats + (kRows + ni) * kPitch;
#pragma unroll
    for (uint32_t k = 0; k < kDepth; k += 4u) {
      ulonglong2 b[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(ws + j * 16 * kPitch + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(xs + i * 8 * kPitch + k);
#pragma unroll
        for (int j = 0; j < 8; ++j) multiply_add_two(sum[i][j], a.x, b[j].x);
#pragma unroll
        for (int j = 0; j < 8; ++j) multiply_add_two(sum[i][j], a.y, b[j].y);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* const sums = stages;
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) sums[(mi + 8u * i) * kSumPitch + ni + 16u * j] = both(sum[i][j]);
  if (cluster > 1u) cluster_sync();
  else __syncthreads();
  // the cluster's CTAs share out the rows
  for (uint32_t index = rank * kThreads + threadIdx.x; index < kRows * kColumns / 4u; index += cluster * kThreads) {
    const uint32_t row = index / (kColumns / 4u), column = index % (kColumns / 4u) * 4u;
    if (m0 + row >= row_end || n0 + column >= p.n) continue;
    const float* const at = sums + row * kSumPitch + column;
    float4 total = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (uint32_t other = 0; other < cluster; ++other) {
      const float4 part = cluster > 1u ? cluster_load_four(at, other) : *reinterpret_cast<const float4*>(at);
      total.x += part.x, total.y += part.y, total.z += part.z, total.w += part.w;
    }
    const float value[4] = {total.x, total.y, total.z, total.w};
#pragma unroll
    for (uint32_t c = 0; c < 4u; ++c) {
      if (n0 + column + c >= p.n) continue;
      if constexpr (STORE == kStorePair) {
        if (c % 2u == 0u) dense_store_pair<float>(p, m0 + row, n0 + column + c, value[c], value[(c + 1u) % 4u]);
      } else {
        dense_store<float>(p, m0 + row, n0 + column + c, value[c]);
      }
    }
  }
  if (cluster > 1u) cluster_sync();  // nobody leaves while its sums may be read
}

// Four columns and up to ROWS rows per group of four warps, which share out k; two groups per CTA.
template <int ROWS, DenseStore STORE>
__global__ void __launch_bounds__(256, 2) dense_f32_stream_kernel(const DenseTask<STORE> p) {
  grid_launch_dependents();
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, group = warp >> 2, part = warp & 3u;
  const uint32_t n0 = (blockIdx.x * 2u + group) * 4u, vectors = p.k / 4u;
  const float* w[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) w[c] = reinterpret_cast<const float*>(p.w) + (size_t)min(n0 + c, p.n - 1u) * p.k;
  auto stream = [](const float* source) {
    ulonglong2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u64 {%0,%1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(source));
    return v;
  };
  constexpr int kAhead = ROWS > 4 ? 1 : 2;  // vectors of each column in flight beside those in use
  const uint32_t stride = 4u * 32u;
  uint32_t at = part * 32u + lane;
  ulonglong2 next[kAhead][4];
  auto fetch = [&](ulonglong2 (&stage)[4], uint32_t vector) {
#pragma unroll
    for (int c = 0; c < 4; ++c) stage[c] = vector < vectors ? stream(w[c] + 4u * (size_t)vector) : make_ulonglong2(0ull, 0ull);
  };
  // the weights are nobody's output: their first vectors may be requested before the predecessor ends
#pragma unroll
  for (int s = 0; s < kAhead; ++s) fetch(next[s], at + s * stride);
  grid_dependency_wait();
  const float* x = reinterpret_cast<const float*>(p.x);
  unsigned long long sum[4][ROWS];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int r = 0; r < ROWS; ++r) sum[c][r] = 0ull;
  for (; at < vectors; at += kAhead * stride) {
#pragma unroll
    for (int s = 0; s < kAhead; ++s) {
      const uint32_t vector = at + s * stride;
      ulonglong2 now[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) now[c] = next[s][c];
      fetch(next[s], vector + kAhead * stride);
      if (vector >= vectors) continue;
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        if (ROWS > 1 && r >= p.m) break;
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(x + (size_t)r * p.k + 4u * (size_t)vector);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          multiply_add_two(sum[c][r], a.x, now[c].x);
          multiply_add_two(sum[c][r], a.y, now[c].y);
        }
      }
    }
  }
  __shared__ float partial[2][4][ROWS][4];  // group, part, row, column
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const float total = warp_sum(both(sum[c][r]));
      if (lane == 0) partial[group][part][r][c] = total;
    }
  __syncthreads();
  constexpr uint32_t kStep = STORE == kStorePair ? 2u : 1u;
  for (uint32_t index = threadIdx.x * kStep; index < 2u * ROWS * 4u; index += 256u * kStep) {
    const uint32_t c = index & 3u, r = index / 4u % ROWS, g = index / (4u * ROWS);
    const uint32_t column = (blockIdx.x * 2u + g) * 4u + c;
    if (r >= p.m || column >= p.n) continue;
    float value[kStep];
#pragma unroll
    for (uint32_t i = 0; i < kStep; ++i)
      value[i] = (partial[g][0][r][c + i] + partial[g][1][r][c + i]) + (partial[g][2][r][c + i] + partial[g][3][r][c + i]);
    if constexpr (STORE == kStorePair) dense_store_pair<float>(p, r, column, value[0], value[kStep - 1]);
    else dense_store<float>(p, r, column, value[0]);
  }
}

template <DenseStore STORE>
int run(const KernelArgs& args, DenseProblem p, uint32_t tiles) {
  // 8 rows: more would hold their sums at the price of vectors in flight, and the tiles are full enough from there on
  if (!p.plan.tiles && p.m <= 8u) {
    const DenseTask<STORE> task(p);
    const dim3 grid((p.n + 7u) / 8u);
    if (p.m == 1u) launch_kernel(args, dense_f32_stream_kernel<1, STORE>, grid, dim3(256), 0, task);
    else if (p.m <= 4u) launch_kernel(args, dense_f32_stream_kernel<4, STORE>, grid, dim3(256), 0, task);
    else launch_kernel(args, dense_f32_stream_kernel<8, STORE>, grid, dim3(256), 0, task);
    return check_launch(args);
  }
  // the plan's tiles are 128 rows at most and hold m / tiles on average, the experts' tails among them
  const uint32_t rows = p.plan.tiles ? p.m / (tiles ? tiles : 1u) : p.m;
  const uint32_t high = rows <= 32u ? 32u : 64u;
  const uint32_t columns = (p.n + kColumns - 1u) / kColumns;
  const uint32_t down = p.plan.tiles ? tiles * (kExpertTile / high) : (p.m + high - 1u) / high;
  LLMOPT_REQUIRE(down <= 65535u, "too many rows");
  // The split of k for which the fullest SM has the least to do, a share being four stages or more.  An SM takes its CTAs two at
  // a time; one alone (four warps) runs at half the rate: 2048 x 7168 as 128 CTAs of one per SM 191 us, as 256 104 us.
  const uint32_t tiles_in_use = columns * (p.plan.tiles ? tiles : down), sms = (uint32_t)context_sm_count(args.ctx);
  const uint32_t blocks = (p.k + kDepth - 1u) / kDepth;
  auto fullest = [&](uint32_t cluster) {
    const uint32_t most = (tiles_in_use * cluster + sms - 1u) / sms;
    return (float)(most < 2u ? 2u : most) / (float)cluster;
  };
  p.cluster = 1u;
  for (uint32_t cluster = 2u; cluster <= 8u && blocks >= 4u * cluster; ++cluster)
    if (fullest(cluster) < 0.9f * fullest(p.cluster)) p.cluster = cluster;
  const DenseTask<STORE> task(p);
  const size_t shared = (size_t)kStages * (high + kColumns) * kPitch * sizeof(float);
  auto launch = [&](auto kernel) {
    // per device and kernel; cheap beside the launch, and remembered nowhere
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared) != cudaSuccess)
      return fail(args, "shared memory could not be raised");
    const dim3 grid(columns * p.cluster, down);
    if (p.cluster == 1u) launch_kernel(args, kernel, grid, dim3(kThreads), shared, task, p.plan);
    else launch_cluster_kernel(args, kernel, grid, dim3(kThreads), shared, p.cluster, task, p.plan);
    return check_launch(args);
  };
  return high == 32u ? launch(dense_f32_tile_kernel<4, STORE>) : launch(dense_f32_tile_kernel<8, STORE>);
}

}  // namespace

int launch_dense_f32(const KernelArgs& args, const DenseProblem& p, DenseStore store, uint32_t tiles) {
  if (p.k % 4u != 0 || ((uintptr_t)p.x & 15u) != 0 || ((uintptr_t)p.w & 15u) != 0) return -1;
  switch (store) {
    case kStoreCached: return run<kStoreCached>(args, p, tiles);
    case kStorePair: return run<kStorePair>(args, p, tiles);
    case kStoreResidual: return run<kStoreResidual>(args, p, tiles);
    default: return run<kStorePlain>(args, p, tiles);
  }
}

}  // namespace llmopt
