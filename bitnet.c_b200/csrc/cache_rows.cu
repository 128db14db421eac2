// The state of a new sequence set to zero: its row of every state tensor of a cache, in one launch.
//
// A cache keeps one tensor per state (recurrent matrices, convolution histories: 11 in a four-layer model), each [slots, ...].
// One fill per tensor and sequence took the host 9 us each, 1.1 ms for the 16 sequences of a batch, before its first step could begin;
// the kernel itself is bound by the bytes it writes.
#include "common.cuh"

#define CR_THREADS 256
#define CR_BLOCKS 16  // blocks per tensor: a row of a megabyte is 16 stores of 16 bytes per thread

// rows[i]: the address of tensor i and the bytes of one slot of it.
__global__ void __launch_bounds__(CR_THREADS) zero_slot_kernel(const long long* __restrict__ rows, int slot) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t bytes = (size_t)rows[2 * blockIdx.y + 1];
  unsigned char* p = (unsigned char*)rows[2 * blockIdx.y] + (size_t)slot * bytes;
  const size_t first = (size_t)blockIdx.x * CR_THREADS + threadIdx.x, step = (size_t)gridDim.x * CR_THREADS;
  if ((((uintptr_t)p | bytes) & 15) == 0) {
    for (size_t i = first; i < bytes / 16; i += step) reinterpret_cast<uint4*>(p)[i] = make_uint4(0u, 0u, 0u, 0u);
  } else {
    for (size_t i = first; i < bytes; i += step) p[i] = 0;
  }
}

// rows: [n][2] on the device, as above.
extern "C" int bn_zero_slot(const long long* rows, int n, int slot, cudaStream_t stream) {
  if (n <= 0) return BN_OK;
  if (!rows || slot < 0 || n > 65535) return BN_ERR_BAD_ARG;
  BN_LAUNCH(zero_slot_kernel, dim3(CR_BLOCKS, n), CR_THREADS, 0, stream, rows, slot);
  BN_CHECK_LAUNCH();
  return BN_OK;
}
