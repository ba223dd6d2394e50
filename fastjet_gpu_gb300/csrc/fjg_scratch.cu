// Device scratch of a launch sequence (ScratchSet, fjg_context.h): what each call
// needs is kept and grows with the largest call.
#include "fjg_context.h"

namespace fjg {

cudaError_t ScratchSet::grow(DeviceBuffer& b, size_t bytes) {
  cudaError_t err = b.reserve(bytes);
  if (err != cudaErrorMemoryAllocation || !rounds.ptr) return err;
  cudaGetLastError();
  cudaDeviceSynchronize();  // queued work may use it
  rounds.release();
  if (sc.round_ws_particles < no_room) no_room = sc.round_ws_particles;
  sc.round_ws = nullptr;
  sc.round_ws_particles = 0;
  return b.reserve(bytes);
}

cudaError_t ScratchSet::reserve_lists(int n_events) {
  if (n_events < 1) n_events = 1;
  if (sc.order && sc.cap_events >= n_events) return cudaSuccess;
  int cap = n_events + n_events / 4 + 64;
  const size_t hist_bytes = (sizeof(int32_t) * kHistBins + 255) & ~size_t(255);
  size_t bytes = sizeof(int32_t) * (size_t)kNumLists * cap + 512 + hist_bytes;
  sc.order = nullptr;
  cudaError_t err = grow(lists, bytes);
  if (err != cudaSuccess) return err;
  char* p = static_cast<char*>(lists.ptr);
  sc.offsets1 = reinterpret_cast<int64_t*>(p);
  sc.counts = reinterpret_cast<int32_t*>(p + 64);
  sc.queues = reinterpret_cast<int*>(p + 128);
  static_assert(sizeof(int32_t) * kNumLists <= 64 && sizeof(int) * (kNumLists + kNumQueues) <= 128, "their room");
  sc.status = reinterpret_cast<int*>(p + 256);
  sc.hist = reinterpret_cast<int32_t*>(p + 512);
  sc.order = reinterpret_cast<int32_t*>(p + 512 + hist_bytes);
  sc.cap_events = cap;
  err = cudaMemset(sc.status, 0, sizeof(int));
  if (err == cudaSuccess) err = cudaDeviceSynchronize();
  return err;
}

cudaError_t ScratchSet::reserve_ws(int64_t particles) {
  if (particles < 1) particles = 1;
  if (sc.ws && sc.ws_stride >= particles) return cudaSuccess;
  const int64_t stride = particles + particles / 4 + 1024;
  sc.ws = nullptr;
  cudaError_t err = grow(ws, sizeof(double) * kWsFields * (size_t)stride);
  if (err != cudaSuccess) return err;
  sc.ws = static_cast<double*>(ws.ptr);
  sc.ws_stride = (int64_t)(ws.cap / (sizeof(double) * kWsFields));
  return cudaSuccess;
}

cudaError_t ScratchSet::reserve_large(int64_t particles) {
  if (particles <= kSmemMaxN) return cudaSuccess;
  if (sc.large_ws && sc.large_ws_particles >= particles) return cudaSuccess;
  sc.large_ws = nullptr;
  cudaError_t err = grow(large, (size_t)kLargeWsBytesPerParticle * (size_t)particles + 256);
  if (err != cudaSuccess) return err;
  sc.large_ws = static_cast<unsigned char*>(large.ptr);
  sc.large_ws_particles = (int64_t)((large.cap - 256) / kLargeWsBytesPerParticle);
  return cudaSuccess;
}

// (A refusal is remembered: trying again at each call would synchronise the
// device each time.)
void ScratchSet::reserve_rounds(int64_t particles) {
  if ((sc.round_ws && sc.round_ws_particles >= particles) || particles >= no_room) return;
  sc.round_ws = nullptr;
  sc.round_ws_particles = 0;
  if (rounds.reserve((size_t)kRoundBytesPerParticle * (size_t)particles + 256) != cudaSuccess) {
    cudaGetLastError();
    no_room = particles;
    return;
  }
  sc.round_ws = static_cast<unsigned char*>(rounds.ptr);
  sc.round_ws_particles = (int64_t)((rounds.cap - 256) / kRoundBytesPerParticle);
}

cudaError_t ScratchSet::reserve(int n_events, int64_t particles, bool with_rounds) {
  cudaError_t err = reserve_lists(n_events);
  if (err == cudaSuccess) err = reserve_ws(particles);
  if (err == cudaSuccess) err = reserve_large(particles);
  if (err == cudaSuccess && with_rounds) reserve_rounds(particles);
  return err;
}

}  // namespace fjg
