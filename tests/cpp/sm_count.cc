// sm_count (csrc/sm_count.h) against a device table of the test's own.
#include "sm_count.h"

#include <cstdio>
#include <initializer_list>

static int current = 0, asked = 0;
static bool answers = true;
extern "C" cudaError_t cudaGetDevice(int* d) {
  *d = current;
  return cudaSuccess;
}
extern "C" cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int d) {
  ++asked;
  if (!answers || a != cudaDevAttrMultiProcessorCount) return cudaErrorInvalidValue;
  *v = 100 + d;
  return cudaSuccess;
}

int main() {
  answers = false;
  if (hlbg::sm_count() != hlbg::kMeasuredSms) return 1;
  answers = true;
  for (int again = 0; again < 3; ++again)
    for (int d : {0, 1, 63, 70}) {
      current = d;
      if (hlbg::sm_count() != 100 + d) return std::fprintf(stderr, "device %d: %d\n", d, hlbg::sm_count()), 1;
    }
  return asked == 1 + 3 + 3 ? 0 : 2;  // once for each device of the table, every time beyond it
}
