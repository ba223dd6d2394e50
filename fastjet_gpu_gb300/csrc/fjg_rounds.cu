// The rounds kernel (fjg_cluster_rounds.cuh) and its launcher.
#include "fjg_kernels.cuh"

namespace fjg {

// SM: the event's slots in shared memory.
template <int T, int MINB, bool SM>
__global__ void __launch_bounds__(T, MINB) k_cluster_rounds(BatchArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RoundShared& S = *reinterpret_cast<RoundShared*>(smem_raw);
  if (threadIdx.x == 0) {
    S.tiles = A.round_tiles;
    S.cells = A.round_cells;
    S.slots = A.round_slots;
  }
  const int count = *A.n_order;
  for (;;) {
    if (threadIdx.x == 0) S.event = next_event(A, count, true);
    __syncthreads();
    const int e = S.event;
    if (e < 0) break;
    if (refused_event(A, e)) continue;  // ends with a barrier
    const bool done = cluster_event_rounds<T, SM>(S, A, e);
    __syncthreads();
    if (threadIdx.x == 0) {
      if (done)
        signal_done(A, e);
      else
        A.retry[atomicAdd(A.n_retry, 1)] = e;
    }
  }
}

namespace {

using Kernel = void (*)(BatchArgs);

// Per list: kernel, threads, tiles (at most 1.5 per particle), tiles with their
// frame, and slots in shared memory.
struct RoundConfig {
  Kernel kernel;
  int threads, tiles, cells, slots;
};

//
// An event with an SM to itself (kRoundsFew, kRoundsOne) has the widest: one event, anti-kt R
// = 0.4, 128 / 256 -> 512 threads: 300 particles 0.90 -> 0.71 ms, 500 1.27 -> 0.87,
// 1000 1.61 -> 1.44, 2000 3.41 -> 2.91.
constexpr int kWidest = 4;

RoundConfig config_of(int q) {
  switch (q) {
    case 0: return {k_cluster_rounds<128, 4, true>, 128, 384, 1024, 256};
    case 1: return {k_cluster_rounds<128, 4, true>, 128, 768, 1536, 512};
    case 2: return {k_cluster_rounds<256, 2, true>, 256, 1024, 1792, 1024};
    case 3: return {k_cluster_rounds<256, 2, true>, 256, 1024, 1792, 2048};
    case 4: return {k_cluster_rounds<512, 1, true>, 512, 1024, 1792, 4096};
    default: return {k_cluster_rounds<kRoundThreadsWs, 1, false>, kRoundThreadsWs, kRoundMaxTiles, kRoundMaxCells, 0};
  }
}

size_t bytes_of(const RoundConfig& c) {
  return c.slots ? round_smem_bytes<true>(c.tiles, c.cells, c.slots) : round_smem_bytes<false>(c.tiles, c.cells, 0);
}

static_assert(round_smem_bytes<true>(1024, 1792, 2048) + 1024 <= 233472 / 2, "2048 slots: two CTAs per SM");
static_assert(round_smem_bytes<true>(1024, 1792, 4096) <= 232448, "4096 slots: one CTA per SM");

}  // namespace

int rounds_occupancy(int q) {
  static int cache[64][kNumQueues] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  int* slot = (dev >= 0 && dev < 64) ? &cache[dev][q] : nullptr;
  if (slot && *slot) return *slot;
  const RoundConfig c = config_of(q);
  int nb = 0;
  // the attribute belongs to the kernel: the largest any list asks for
  size_t most = 0;
  for (int p = 0; p < kNumQueues; ++p)
    if (config_of(p).kernel == c.kernel && bytes_of(config_of(p)) > most) most = bytes_of(config_of(p));
  if (cudaFuncSetAttribute(c.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, c.kernel, c.threads, bytes_of(c)) != cudaSuccess || nb < 1)
    nb = 1;
  if (slot) *slot = nb;
  return nb;
}

cudaError_t launch_rounds(int q, BatchArgs A, int grid, cudaStream_t s) {
  const bool alone = A.rounds_mode == kRoundsFew || A.rounds_mode == kRoundsOne;
  const int shape = alone && q != kLargeQueue ? kWidest : q;
  rounds_occupancy(shape);  // sets the shared-memory attribute
  const RoundConfig c = config_of(shape);
  A.round_tiles = c.tiles;
  A.round_cells = c.cells;
  A.round_slots = c.slots;
  const int level = q == kLargeQueue ? tiled_priority_level(A.serve_order) : bucket_priority_level(q, A.serve_order);
  return launch_with_priority(c.kernel, grid, c.threads, bytes_of(c), s, level, A);
}

}  // namespace fjg
