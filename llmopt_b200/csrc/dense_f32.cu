// Dense linear layer in fp32 (CUDA cores, no TF32) where weight and activation rows are whole 16-byte vectors:
//  * up to 32 rows: dense_f32_stream_kernel, bound by the weight stream.  A warp takes two columns and up to eight rows and
//    keeps up to 32 loads of weights in flight.
//  * more rows: dense_f32_tile_kernel, bound by the multiply-adds and the reads of shared memory side by side (0.55 to 0.6 of the fp32
//    rate where all SMs are busy).  Operands come by cp.async.
// Both add the products of an output in the order of the general kernels (dense_linear.cu: lanes 32 apart, and k one after
// the other), to the last bit: fp32 is what checkpoints are checked with, and decoders that divide by nearly cancelling sums
// show every change of it.  k shared out over a cluster, with even and odd k as the halves of packed multiply-adds, was faster (2048 x
// 2048 x 100 rows 32 us) but moved logits by 2.9e-5.  Pairs of rows keep the order.  Back to back over cold operands, before (scalar
// multiply-adds, 16 bytes of either operand in four cycles a read, two CTAs on one SM while others idle) and now, us: 100 rows n 2048 k
// 2048 66, 41; n 2048 k 7168 226, 133; n 7168 k 2048 123, 111; n 9248 k 2048 123, 110; 333 rows n 7168 k 2048 445, 290.
#include "dense_linear.cuh"

namespace llmopt {
namespace {

constexpr uint32_t kDepth = 32;    // k of a stage: a row is one 128-byte line
constexpr uint32_t kPitch = kDepth + 4;  // floats; eight consecutive rows start in eight different groups of four banks
constexpr uint32_t kOnePerSm = 117u * 1024u;  // bytes of shared memory of which an SM has no two
constexpr uint32_t kMostDown = 65535;  // tiles of rows: a grid's second dimension

// 16 or 4 bytes to shared memory, zeros where absent.
__device__ __forceinline__ void copy_vector(float* to, const float* from, bool present) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from),
               "r"(present ? 16u : 0u)
               : "memory");
}
__device__ __forceinline__ void copy_one(float* to, const float* from, bool present) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from),
               "r"(present ? 4u : 0u)
               : "memory");
}
// Two sums at once: the halves are rounded one by one, as fmaf does.
__device__ __forceinline__ void multiply_add_pair(unsigned long long& sum, unsigned long long two, float one) {
  asm("{.reg .b64 both;\n\tmov.b64 both, {%2, %2};\n\tfma.rn.f32x2 %0, %1, both, %0;}" : "+l"(sum) : "l"(two), "f"(one));
}

// DOWN x ACROSS threads; thread (mi, ni) owns rows TM mi .. TM mi + TM - 1 and columns ni + j ACROSS.  Every sum walks over all
// of k in order.  Weights lie as in memory, four k of a column are one read; rows are transposed on their way in, so that one read
// holds two pairs of them: packed multiply-adds take half the issue slots, and the copies of a weight to both halves go
// where those are free.
template <int TM, int TN, int DOWN, int ACROSS>
struct Tile {
  static constexpr uint32_t kThreads = DOWN * ACROSS, kRows = TM * DOWN, kColumns = TN * ACROSS;
  static constexpr uint32_t kRowPitch = kRows + 4, kStageFloats = kDepth * kRowPitch + kColumns * kPitch;
  // A sum is not split, so a CTA walks over all of k and a stage takes as long as its way from memory unless many are under way:
  // what two CTAs of an SM have room for, one of the largest tiles.
  static constexpr uint32_t kStages = kRows == 32u ? 8u : kColumns == 64u ? 6u : 8u;
  static constexpr uint32_t kBytes = kStages * kStageFloats * sizeof(float);
  static constexpr uint32_t kPerSm = kBytes <= 114u * 1024u ? 2u : 1u;
};

template <int TM, int TN, int DOWN, int ACROSS, DenseStore STORE>
__global__ void __launch_bounds__(Tile<TM, TN, DOWN, ACROSS>::kThreads, Tile<TM, TN, DOWN, ACROSS>::kPerSm)
    dense_f32_tile_kernel(const DenseTask<STORE> p, const DensePlan plan) {
  typedef Tile<TM, TN, DOWN, ACROSS> Shape;
  constexpr uint32_t kThreads = Shape::kThreads, kWarps = kThreads / 32u;
  constexpr uint32_t kRows = Shape::kRows, kColumns = Shape::kColumns, kStages = Shape::kStages, kRowPitch = Shape::kRowPitch;
  constexpr uint32_t kSumPitch = kColumns + 4;
  static_assert(kRows * kSumPitch * sizeof(float) <= Shape::kBytes, "the sums take the stages' place");
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
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  auto copy_x = [&](uint32_t block) {  // a warp's copy: four rows, eight k of each, to 32 banks
    float* const to = stages + block % kStages * Shape::kStageFloats;
#pragma unroll
    for (uint32_t part = 0; part < kRows / kWarps; ++part) {
      const uint32_t row = (warp + part * kWarps) / 4u * 4u + (lane >> 3), k = warp % 4u * 8u + (lane & 7u);
      const bool present = block * kDepth + k < p.k && m0 + row < row_end;
      copy_one(to + k * kRowPitch + row, present ? x + (size_t)(m0 + row) * p.k + block * kDepth + k : x, present);
    }
  };
  auto copy_w = [&](uint32_t block) {
    float* const to = stages + block % kStages * Shape::kStageFloats + kDepth * kRowPitch;
    const uint32_t lane_k = (threadIdx.x & 7u) * 4u, k = block * kDepth + lane_k;
#pragma unroll
    for (uint32_t row = threadIdx.x >> 3; row < kColumns; row += kThreads / 8u) {
      const bool present = k < p.k && n0 + row < p.n;
      copy_vector(to + row * kPitch + lane_k, present ? w + (size_t)(n0 + row) * p.k + k : w, present);
    }
  };
  // the weights are nobody's output: their first stages may be requested before the predecessor ends
#pragma unroll
  for (uint32_t s = 0; s < kStages; ++s)
    if (s < blocks) copy_w(s);
  grid_dependency_wait();
#pragma unroll
  for (uint32_t s = 0; s < kStages; ++s) {
    if (s < blocks) copy_x(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // A read of 16 bytes a lane takes two cycles instead of four where lanes one apart, or lanes two apart, read the same: bit 0 of
  // the lane only chooses among rows, bit 1 only among columns.
  constexpr uint32_t kWarpsDown = DOWN / 4u;
  const uint32_t mi = (lane & 1u) + (lane >> 1 & 2u) + warp % kWarpsDown * 4u;
  const uint32_t ni = (lane >> 1 & 1u) + (lane >> 2 & 6u) + warp / kWarpsDown * 8u;
  unsigned long long sum[TM / 2][TN];  // rows 2 i and 2 i + 1
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) sum[i][j] = 0ull;
  float4 b[2][TN];  // four k each: those that are multiplied, and the next ones on their way
  ulonglong2 a[2][4][TM / 4];
  auto read = [&](int side, uint32_t block, uint32_t k) {
    const float* const xs = stages + block % kStages * Shape::kStageFloats + k * kRowPitch + mi * TM;
    const float* const ws = stages + block % kStages * Shape::kStageFloats + kDepth * kRowPitch + ni * kPitch + k;
#pragma unroll
    for (int j = 0; j < TN; ++j) b[side][j] = *reinterpret_cast<const float4*>(ws + j * ACROSS * kPitch);
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int i = 0; i < TM / 4; ++i) a[side][q][i] = *reinterpret_cast<const ulonglong2*>(xs + q * kRowPitch + i * 4);
  };
  asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
  __syncthreads();
  read(0, 0, 0);
  for (uint32_t block = 0; block < blocks; ++block) {
#pragma unroll
    for (uint32_t k = 0; k < kDepth; k += 4u) {
      const int side = k / 4u & 1u;
      if (k + 4u < kDepth) {
        read(side ^ 1, block, k + 4u);
      } else {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();  // the next stage has arrived, and this one is read
        if (block + kStages < blocks) {
          copy_w(block + kStages);
          copy_x(block + kStages);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        read(side ^ 1, block + 1u, 0);  // past the last block: what an earlier one left, multiplied by nobody
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          const float4& four = b[side][j];
          const float weight = q == 0 ? four.x : q == 1 ? four.y : q == 2 ? four.z : four.w;
#pragma unroll
          for (int i = 0; i < TM / 4; ++i) {
            multiply_add_pair(sum[2 * i][j], a[side][q][i].x, weight);
            multiply_add_pair(sum[2 * i + 1][j], a[side][q][i].y, weight);
          }
        }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* const sums = stages;
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j)
      sums[(mi * TM + i) * kSumPitch + ni + j * ACROSS] =
          __uint_as_float(i & 1 ? (uint32_t)(sum[i / 2][j] >> 32) : (uint32_t)sum[i / 2][j]);
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
  // The tile with which the fullest SM is done first.  Measured per 2048 k: a tile of 32 x 64 alone on its SM 40 us, two side by side 60;
  // 64 x 64 68 and 128; 64 x 128, which has an SM to itself, 107.
  const uint32_t sms = (uint32_t)context_sm_count(args.ctx);
  auto down = [&](uint32_t high) { return p.plan.tiles ? tiles * (kExpertTile / high) : p.m / high + (p.m % high ? 1u : 0u); };
  if (down(64u) > kMostDown) return -1;
  auto cost = [&](uint32_t high, uint32_t wide, uint32_t alone, uint32_t beside) {
    // the plan's tiles are 128 rows at most and hold m / tiles on average; those without rows end at once
    const uint32_t rows = p.plan.tiles ? p.m / (tiles ? tiles : 1u) : p.m;
    const uint32_t full = p.plan.tiles ? tiles * ((rows + high - 1u) / high) : down(high);
    const uint32_t most = ((p.n + wide - 1u) / wide * full + sms - 1u) / sms;
    return (size_t)(most / 2u) * beside + (most % 2u) * alone;
  };
  auto launch = [&](auto kernel, auto shape) {
    typedef decltype(shape) Shape;
    const dim3 grid((p.n + Shape::kColumns - 1u) / Shape::kColumns, down(Shape::kRows));
    // Where every CTA finds an SM of its own none shares one: CTAs that start beside the last ones of the launch before double up
    // (2048 x 2048 x 100 rows 59 us, 41 this way).
    constexpr uint32_t kMostBytes = Shape::kBytes > kOnePerSm ? Shape::kBytes : kOnePerSm;
    const uint32_t bytes = (size_t)grid.x * grid.y <= sms ? kMostBytes : Shape::kBytes;
    // Per device and kernel; cheap beside the launch, and remembered nowhere.  Always the most: another thread may be between this call
    // and its launch.
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostBytes) != cudaSuccess)
      return fail(args, "shared memory could not be raised");
    launch_kernel(args, kernel, grid, dim3(Shape::kThreads), bytes, task, p.plan);
    return check_launch(args);
  };
  // Narrow products and few rows: tiles of 32 x 16 or 32 x 32 where each has an SM to itself; a thread's sums are what a step over k
  // takes time for.  k 2048, 100 rows n 256 45 -> 28 us; 40 rows n 2048 41 -> 30.  (Two of 32 x 32 beside one another are slower than
  // one of 32 x 64: 98 for 59 with 100 rows.)
  const size_t tall = down(32u);
  if (tall <= kMostDown && (p.n + 15u) / 16u * tall <= sms) return launch(dense_f32_tile_kernel<4, 1, 8, 16, STORE>, Tile<4, 1, 8, 16>());
  if (tall <= kMostDown && (p.n + 31u) / 32u * tall <= sms) return launch(dense_f32_tile_kernel<4, 2, 8, 16, STORE>, Tile<4, 2, 8, 16>());
  const size_t large = cost(64u, 128u, 107u, 214u), middle = cost(64u, 64u, 68u, 128u), small = cost(32u, 64u, 40u, 60u);
  if (down(32u) <= kMostDown && small <= middle && small <= large)
    return launch(dense_f32_tile_kernel<4, 4, 8, 16, STORE>, Tile<4, 4, 8, 16>());
  if (middle <= large) return launch(dense_f32_tile_kernel<4, 4, 16, 16, STORE>, Tile<4, 4, 16, 16>());
  return launch(dense_f32_tile_kernel<8, 4, 8, 32, STORE>, Tile<8, 4, 8, 32>());
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
