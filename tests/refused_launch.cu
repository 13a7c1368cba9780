// The host side of the three-term product with a launch that is refused, without a GPU: its launches are replaced by ones that count, of
// which the n-th fails.  Prints, for n = 0 (none), 1, 2: what the entry point returned, and how many launches it made.
#include <cstdio>
#include "common.cuh"
#include "tcgen05.cuh"

static int made, refused;
template <typename... Args> cudaError_t counted_launch(Args&&...) { return ++made == refused ? cudaErrorLaunchOutOfResources : cudaSuccess; }
static cudaError_t device_zero(int* device) { *device = 0; return cudaSuccess; }
#define fmx_launch counted_launch
#define fmx_launch_cluster counted_launch
#define make_map_k128(...) 0
#define cudaFuncSetAttribute(...) cudaSuccess
#define cudaGetDevice device_zero
#include "gemm_three.cu"

int main() {
  alignas(16) static float a[64], c[64];
  alignas(16) static bf16 w[64];
  alignas(16) static char ws[1024];
  for (refused = 0; refused <= 2; ++refused) {
    made = 0;
    const int rc = fmx_gemm_three(a, 8, w, 8, nullptr, c, 8, 4, 8, 8, 8, ws, 148, nullptr, nullptr);
    printf("%d %d\n", rc, made);
  }
  return 0;
}
