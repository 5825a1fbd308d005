// The shared-memory opt-in of a kernel (hss_optin.h) against fakes of the runtime
// calls: once per device and kernel, and again after a failure.  Prints one line per
// failure.
#include <cstdio>
#include <map>
#include <utility>

#include "hss_optin.h"

namespace {
int device = 0, calls = 0;
cudaError_t answer = cudaSuccess;
std::map<std::pair<int, const void*>, int> limit;
}  // namespace

extern "C" cudaError_t cudaGetDevice(int* d) {
  *d = device;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  ++calls;
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize && answer == cudaSuccess) limit[{device, f}] = v;
  return answer;
}

#define EXPECT(c) \
  if (!(c)) std::printf("failed: %s (line %d)\n", #c, __LINE__)

int main() {
  hss::SmemOptIn a, b;
  const int ka = 0, kb = 0;
  for (int turn = 0; turn < 2; ++turn)
    for (device = 0; device < 3; ++device) {
      EXPECT(a(&ka, 100000) == cudaSuccess);
      EXPECT((limit[{device, &ka}] == 100000));
    }
  EXPECT(calls == 3);
  device = 1;
  EXPECT(b(&kb, 200000) == cudaSuccess && (limit[{1, &kb}] == 200000) && calls == 4);
  device = 2;
  answer = cudaErrorInvalidValue;
  EXPECT(b(&kb, 200000) == cudaErrorInvalidValue);
  EXPECT(b(&kb, 200000) == cudaErrorInvalidValue);
  answer = cudaSuccess;
  EXPECT(b(&kb, 200000) == cudaSuccess && (limit[{2, &kb}] == 200000) && calls == 7);
  device = 70;   // beyond the table: set every time
  EXPECT(b(&kb, 200000) == cudaSuccess && b(&kb, 200000) == cudaSuccess && calls == 9);
  return 0;
}
