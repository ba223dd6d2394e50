// Host check of the scratch's growth (fjg_scratch.cu) on a device of limited memory,
// played by the functions below; built with nvcc and run on the CPU by
// tests/test_scratch.py.  The rounds kernel's workspace is optional: it is taken
// where asked for and where there is room, a refusal is not asked for again, and it
// is given up where something that a call needs does not fit beside it.  Prints "ok".
#include <cstdio>
#include <cstdlib>
#include <map>

#include <cuda_runtime.h>

namespace {

std::map<void*, size_t> blocks;
size_t room = 0, used = 0;
int asked = 0;

cudaError_t fake_malloc(void** p, size_t n) {
  ++asked;
  *p = nullptr;
  if (used + n > room) return cudaErrorMemoryAllocation;
  *p = std::malloc(1);
  blocks[*p] = n;
  used += n;
  return cudaSuccess;
}

cudaError_t fake_free(void* p) {
  used -= blocks.at(p);
  blocks.erase(p);
  std::free(p);
  return cudaSuccess;
}

cudaError_t fake_ok() { return cudaSuccess; }

}  // namespace

#define cudaMalloc(p, n) fake_malloc(reinterpret_cast<void**>(p), n)
#define cudaFree(p) fake_free(p)
#define cudaMemset(p, v, n) fake_ok()
#define cudaDeviceSynchronize() fake_ok()
#define cudaGetLastError() fake_ok()
#include "fjg_scratch.cu"

#define CHECK(x)                                   \
  do {                                             \
    if (!(x)) {                                    \
      std::printf("line %d: %s\n", __LINE__, #x);  \
      return 1;                                    \
    }                                              \
  } while (0)

int main() {
  const int64_t n = 100000;
  const size_t per_rounds = fjg::kRoundBytesPerParticle, per_ws = sizeof(double) * fjg::kWsFields;
  {  // not asked for: not taken
    fjg::ScratchSet s;
    room = size_t(1) << 40;
    CHECK(s.reserve(10, n, false) == cudaSuccess && !s.sc.round_ws && used < n * (per_ws * 2 + 200));
    CHECK(s.reserve(10, n, true) == cudaSuccess && s.sc.round_ws && s.sc.round_ws_particles >= n);
    s.release();
    CHECK(used == 0);
  }
  {  // no room for it: the call goes on, and it is not asked for each time
    fjg::ScratchSet s;
    CHECK(s.reserve(10, n, false) == cudaSuccess);
    room = used + n * per_rounds / 2;
    CHECK(s.reserve(10, n, true) == cudaSuccess && !s.sc.round_ws && s.sc.ws);
    const int before = asked;
    for (int k = 0; k < 5; ++k) CHECK(s.reserve(10, n, true) == cudaSuccess && !s.sc.round_ws);
    CHECK(asked == before);
    CHECK(s.reserve(10, n / 8, true) == cudaSuccess && s.sc.round_ws && s.sc.round_ws_particles < n);
    s.release();
    CHECK(used == 0);
  }
  {  // what a call needs does not fit beside it
    fjg::ScratchSet s;
    room = size_t(1) << 40;
    CHECK(s.reserve(10, n, true) == cudaSuccess && s.sc.round_ws);
    room = used + 300 * n;
    CHECK(s.reserve(10, 4 * n, false) == cudaSuccess && s.sc.ws_stride >= 4 * n && !s.sc.round_ws);
    s.release();
    CHECK(used == 0);
  }
  {  // nothing fits: an error, and no pointer to what was freed
    fjg::ScratchSet s;
    room = size_t(1) << 40;
    CHECK(s.reserve(10, n, true) == cudaSuccess);
    room = used;
    CHECK(s.reserve(10, 1000 * n, true) == cudaErrorMemoryAllocation && !s.sc.ws && !s.sc.round_ws);
    room = size_t(1) << 40;
    CHECK(s.reserve(10, n, true) == cudaSuccess && s.sc.ws && s.sc.ws_stride >= n);
    s.release();
    CHECK(used == 0);
  }
  std::printf("ok\n");
  return 0;
}
