// Dense linear layer in fp32 (CUDA cores, no TF32) where weight and activation rows are whole 16-byte vectors:
//  * up to 32 rows: dense_f32_stream_kernel, bound by the weight stream.  A warp takes two columns and up to eight rows and
//    keeps up to 32 loads of weights in flight.
//  * more rows: dense_f32_tile_kernel, bound by reads of shared memory.  Operands come by cp.async in k-major rows as they lie
//    in memory; a thread reads four k of a row at once.
// Both add the products of an output in the order of the general kernels (dense_linear.cu: lanes 32 apart, and k one after
// the other), to the last bit: fp32 is what checkpoints are checked with, and decoders that divide by nearly cancelling sums
// show every change of it.  k shared out over a cluster, with even and odd k as the halves of packed multiply-adds, was faster (2048 x
// 2048 x 100 rows 32 us) but moved logits by 2.9e-5.  Now, 100 rows back to back over cold operands, with the time of 64 x 64
// tiles and 4-byte loads: n 2048, k 2048 66 us, 305 before; n 2048, k 7168 227, 1075 before; n 7168, k 2048 123, 337 before.
#include "dense_linear.cuh"

namespace llmopt {
namespace {

constexpr uint32_t kDepth = 32;    // k of a stage: a row is one 128-byte line
constexpr uint32_t kPitch = kDepth + 4;  // floats; eight consecutive rows start in eight different groups of four banks
constexpr uint32_t kThreads = 128;
constexpr uint32_t kMostDown = 65535;  // tiles of rows: a grid's second dimension

// 16 bytes to shared memory, zeros where absent.
__device__ __forceinline__ void copy_vector(float* to, const float* from, bool present) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from),
               "r"(present ? 16u : 0u)
               : "memory");
}
// Stages of 32 k: what two CTAs of an SM have room for.  A sum is not split, so a CTA walks over all of k and a stage takes as
// long as its way from memory unless many are under way.
__host__ __device__ constexpr uint32_t tile_stages(int TM, int TN) { return TM * TN <= 16 ? 8u : TM * TN <= 32 ? 6u : 4u; }

// A tile of 8 TM rows x 16 TN columns; thread (mi, ni) of 8 x 16 owns rows mi + 8 i and columns ni + 16 j.  Every sum walks
// over all of k in order; four k of an operand are one read.
template <int TM, int TN, DenseStore STORE>
__global__ void __launch_bounds__(kThreads, 2) dense_f32_tile_kernel(const DenseTask<STORE> p, const DensePlan plan) {
  constexpr uint32_t kRows = 8 * TM, kColumns = 16 * TN, kStages = tile_stages(TM, TN);
  constexpr uint32_t kStageFloats = (kRows + kColumns) * kPitch;
  constexpr uint32_t kSumPitch = kColumns + 4;
  static_assert(kRows * kSumPitch <= kStages * kStageFloats, "the sums take the stages' place");
  extern __shared__ __align__(16) float stages[];
  const uint32_t n0 = blockIdx.x * kColumns;
  const float* x = reinterpret_cast<const float*>(p.x);
  const float* w = reinterpret_cast<const float*>(p.w);
  uint32_t m0 = blockIdx.y * kRows, row_end = p.m;
  grid_launch_dependents();
  if (plan.tiles) {  // rows sorted by expert; a tile of the plan is cut into tiles of this kernel
    grid_dependency_wait();
    constexpr uint32_t kParts = kExpertTile / kRows;
    const uint32_t index = blockIdx.y / kParts;
    if (index >= plan.tiles[0]) return;
    const DenseTile tile = dense_tile(plan, index);
    m0 = tile.first + blockIdx.y % kParts * kRows;
    row_end = min(tile.end, p.m);
    if (m0 >= row_end || tile.expert >= plan.experts) return;
    w += (size_t)tile.expert * p.n * p.k;
  }
  const uint32_t blocks = (p.k + kDepth - 1u) / kDepth;
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
    if (s < blocks) copy_w(s);
  grid_dependency_wait();
#pragma unroll
  for (uint32_t s = 0; s + 1u < kStages; ++s) {
    if (s < blocks) copy_x(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t mi = (lane >> 3) + 4u * (warp & 1u), ni = (lane & 7u) + 8u * (warp >> 1);
  float sum[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) sum[i][j] = 0.0f;
  for (uint32_t block = 0; block < blocks; ++block) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();  // this stage has arrived, and the one before it is read
    if (block + kStages - 1u < blocks) {
      copy_w(block + kStages - 1u);
      copy_x(block + kStages - 1u);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* const xs = stages + block % kStages * kStageFloats + mi * kPitch;
    const float* const ws = stages + block % kStages * kStageFloats + (kRows + ni) * kPitch;
#pragma unroll
    for (uint32_t k = 0; k < kDepth; k += 4u) {
      float4 a[TM], b[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(ws + j * 16 * kPitch + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(xs + i * 8 * kPitch + k);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) sum[i][j] = fmaf(a[i].x, b[j].x, sum[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) sum[i][j] = fmaf(a[i].y, b[j].y, sum[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) sum[i][j] = fmaf(a[i].z, b[j].z, sum[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) sum[i][j] = fmaf(a[i].w, b[j].w, sum[i][j]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* const sums = stages;
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) sums[(mi + 8u * i) * kSumPitch + ni + 16u * j] = sum[i][j];
  __syncthreads();
  for (uint32_t index = threadIdx.x; index < kRows * kColumns / 2u; index += kThreads) {
    const uint32_t row = index / (kColumns / 2u), column = index % (kColumns / 2u) * 2u;
    if (m0 + row >= row_end || n0 + column >= p.n) continue;
    const float2 value = *reinterpret_cast<const float2*>(sums + row * kSumPitch + column);
    if constexpr (STORE == kStorePair) {
      dense_store_pair<float>(p, m0 + row, n0 + column, value.x, value.y);
    } else {
      dense_store<float>(p, m0 + row, n0 + column, value.x);
      if (n0 + column + 1u < p.n) dense_store<float>(p, m0 + row, n0 + column + 1u, value.y);
    }
  }
}

// Two columns and up to ROWS rows per warp: lane l adds k = l, l + 32, .. in order, then the lanes' sums are added.
template <int ROWS, DenseStore STORE>
__global__ void __launch_bounds__(256) dense_f32_stream_kernel(const DenseTask<STORE> p) {
  grid_launch_dependents();
  constexpr int kAhead = ROWS == 1 ? 16 : ROWS <= 4 ? 8 : 4;  // k of a lane in flight
  const uint32_t lane = threadIdx.x & 31u, column = (blockIdx.x * 8u + (threadIdx.x >> 5)) * 2u, row0 = blockIdx.y * ROWS;
  const float* first = reinterpret_cast<const float*>(p.w) + (size_t)min(column, p.n - 1u) * p.k;
  const float* second = reinterpret_cast<const float*>(p.w) + (size_t)min(column + 1u, p.n - 1u) * p.k;
  float next[kAhead][2];
  auto stream = [](const float* source) {
    float v;
    asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(source));
    return v;
  };
  auto fetch = [&](uint32_t k0) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const uint32_t k = k0 + i * 32u + lane;
      next[i][0] = k < p.k ? stream(first + k) : 0.0f;
      next[i][1] = k < p.k ? stream(second + k) : 0.0f;
    }
  };
  // the weights are nobody's output: the first may be requested before the predecessor ends
  fetch(0);
  grid_dependency_wait();
  if (column >= p.n) return;
  const float* x = reinterpret_cast<const float*>(p.x) + (size_t)row0 * p.k;
  const uint32_t rows = min(p.m - row0, (uint32_t)ROWS);
  float sum[2][ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) sum[0][r] = sum[1][r] = 0.0f;
  for (uint32_t k0 = 0; k0 < p.k; k0 += kAhead * 32u) {
    float now[kAhead][2], a[kAhead][ROWS];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      now[i][0] = next[i][0], now[i][1] = next[i][1];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const uint32_t k = k0 + i * 32u + lane;
        a[i][r] = k < p.k && r < rows ? x[(size_t)r * p.k + k] : 0.0f;
      }
    }
    if (k0 + kAhead * 32u < p.k) fetch(k0 + kAhead * 32u);
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        sum[0][r] = fmaf(now[i][0], a[i][r], sum[0][r]);
        sum[1][r] = fmaf(now[i][1], a[i][r], sum[1][r]);
      }
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const float one = warp_sum(sum[0][r]), two = warp_sum(sum[1][r]);
    if (r >= rows || lane != 0) continue;
    if constexpr (STORE == kStorePair) {
      dense_store_pair<float>(p, row0 + r, column, one, two);
    } else {
      dense_store<float>(p, row0 + r, column, one);
      if (column + 1u < p.n) dense_store<float>(p, row0 + r, column + 1u, two);
    }
  }
}

template <DenseStore STORE>
int run(const KernelArgs& args, DenseProblem p, uint32_t tiles) {
  const DenseTask<STORE> task(p);
  // up to 32 rows the weights are what is read; beyond, tiles
  if (!p.plan.tiles && p.m <= 32u) {
    const uint32_t columns = (p.n + 15u) / 16u;
    if (p.m == 1u) launch_kernel(args, dense_f32_stream_kernel<1, STORE>, dim3(columns), dim3(256), 0, task);
    else if (p.m <= 4u) launch_kernel(args, dense_f32_stream_kernel<4, STORE>, dim3(columns), dim3(256), 0, task);
    else launch_kernel(args, dense_f32_stream_kernel<8, STORE>, dim3(columns, (p.m + 7u) / 8u), dim3(256), 0, task);
    return check_launch(args);
  }
  // The tile for which the fullest SM has the least to read from shared memory, which bounds all of them: 16 (TM + TN) cycles per
  // four k and CTA.  One CTA alone on an SM runs at about half the rate.
  const uint32_t sms = (uint32_t)context_sm_count(args.ctx);
  auto down = [&](uint32_t high) { return p.plan.tiles ? tiles * (kExpertTile / high) : p.m / high + (p.m % high ? 1u : 0u); };
  if (down(64u) > kMostDown) return -1;
  auto cost = [&](uint32_t high, uint32_t wide) {
    // the plan's tiles are 128 rows at most and hold m / tiles on average; those without rows end at once
    const uint32_t rows = p.plan.tiles ? p.m / (tiles ? tiles : 1u) : p.m;
    const uint32_t full = p.plan.tiles ? tiles * ((rows + high - 1u) / high) : down(high);
    const uint32_t most = ((p.n + wide - 1u) / wide * full + sms - 1u) / sms;
    return (most < 2u ? 2u : most) * (high / 8u + wide / 16u);
  };
  auto launch = [&](auto kernel, uint32_t high, uint32_t wide) {
    const size_t shared = (size_t)tile_stages((int)high / 8, (int)wide / 16) * (high + wide) * kPitch * sizeof(float);
    // per device and kernel; cheap beside the launch, and remembered nowhere
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared) != cudaSuccess)
      return fail(args, "shared memory could not be raised");
    launch_kernel(args, kernel, dim3((p.n + wide - 1u) / wide, down(high)), dim3(kThreads), shared, task, p.plan);
    return check_launch(args);
  };
  const uint32_t large = cost(64u, 128u), middle = cost(64u, 64u), small = cost(32u, 64u);
  if (down(32u) <= kMostDown && small <= middle && small <= large) return launch(dense_f32_tile_kernel<4, 4, STORE>, 32u, 64u);
  if (middle <= large) return launch(dense_f32_tile_kernel<8, 4, STORE>, 64u, 64u);
  return launch(dense_f32_tile_kernel<8, 8, STORE>, 64u, 128u);
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
