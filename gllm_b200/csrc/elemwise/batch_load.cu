// The arrays of a step, copied to the device as one block of 32-bit words, put into their own buffers. A small step has eight to
// fourteen arrays of a few words: a copy each costs some 2.5 us on the device and 4 on the host.
#include "../common/host_utils.h"

namespace b200 {

static constexpr int kMaxArrays = 16;

struct BatchArrays {
  struct {
    uint32_t* dst;
    int64_t pitch;        // words between rows of dst
    int from, rows, cols; // words of src
  } a[kMaxArrays];
};

// one grid column per array; rows are contiguous in src
__global__ void __launch_bounds__(256) batch_load_kernel(const uint32_t* __restrict__ src, const BatchArrays p) {
  const auto& a = p.a[blockIdx.x];
  const int n = a.rows * a.cols;
  for (int i = blockIdx.y * 256 + threadIdx.x; i < n; i += gridDim.y * 256) {
    const int r = i / a.cols;
    a.dst[r * a.pitch + (i - r * a.cols)] = src[a.from + i];
  }
}

}  // namespace b200

using namespace b200;

// arrays: n x (device pointer, row pitch in words, first word in src, rows, columns), on the host. `words`: of the largest array.
GLLM_EXPORT int gllm_batch_load(const void* src, const int64_t* arrays, int n, int64_t words, void* stream) {
  if (n <= 0) return 0;
  if (n > kMaxArrays) return 1;
  BatchArrays p;
  for (int i = 0; i < n; ++i) {
    const int64_t* v = arrays + 5 * i;
    p.a[i] = {reinterpret_cast<uint32_t*>(v[0]), v[1], static_cast<int>(v[2]), static_cast<int>(v[3]), static_cast<int>(v[4])};
  }
  const int64_t blocks = (words + 1023) / 1024;
  batch_load_kernel<<<dim3(n, static_cast<unsigned>(blocks < 1 ? 1 : blocks > 64 ? 64 : blocks)), 256, 0,
                      reinterpret_cast<cudaStream_t>(stream)>>>(reinterpret_cast<const uint32_t*>(src), p);
  CUDA_CHECK_RET(cudaGetLastError());
  return 0;
}
