// Blocks of information bits to rate-matched codewords (cb_encode): a CTA per block, the
// encoder of nr_encode.cuh on packed columns, then the sent bits (BitSelection::select,
// crates/com-fec/src/puncture.rs:144-148) as bytes.
//
// Bound: the copies between the caller's host memory and the device, K' + E bytes a block;
// the call takes 0.14 ms for 128 blocks of BG1 Z = 384 (1.1 + 3.2 MB of pageable host
// memory), 40 ms with the host loop over bytes, 317 us a block.
#include <cuda_runtime.h>

#include "kernels.h"
#include "nr_encode.cuh"

namespace cbk {
namespace {

constexpr int kEncodeThreads = 256;

__global__ void __launch_bounds__(kEncodeThreads) nr_encode_kernel(const __grid_constant__ NrEncodeArgs a) {
  extern __shared__ uint32_t s_cols[];
  const cbd::DevCode& c = a.code;
  const int z = c.z, wz = (z + 31) >> 5, ws = wz + 1, ncol = c.n_full / z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* cwp = s_cols;
  uint32_t* synp = cwp + ncol * ws;
  for (int64_t f = blockIdx.x; f < a.n_frames; f += gridDim.x) {
    const uint8_t* info = a.info + f * c.k_info;
    uint8_t* out = a.out + f * c.e;
    // the systematic columns, filler bits 0
    for (int task = warp; task < c.cols_k * wz; task += kEncodeThreads / 32) {
      const int j = task / wz, w = task - j * wz, b = w * 32 + lane, i = j * z + b;
      const uint32_t word = __ballot_sync(0xffffffffu, b < z && i < c.k_info && (info[i] & 1));
      if (lane == 0) {
        cwp[j * ws + w] = word;
        if (w == wz - 1) cwp[j * ws + wz] = 0u;
      }
    }
    __syncthreads();
    encode_packed_columns(c, cwp, synp, tid, kEncodeThreads);
    auto bit = [&](int t) -> uint32_t {
      const int v = c.map_is_offset ? 2 * z + t : c.map[t], j = v / z, b = v - j * z;
      return (cwp[j * ws + (b >> 5)] >> (b & 31)) & 1u;
    };
    if ((c.e & 3) == 0) {  // every block's row of a.out (device memory) is then 4-byte aligned
      for (int q = tid; q < (c.e >> 2); q += kEncodeThreads)
        reinterpret_cast<uint32_t*>(out)[q] =
            bit(4 * q) | bit(4 * q + 1) << 8 | bit(4 * q + 2) << 16 | bit(4 * q + 3) << 24;
    } else {
      for (int t = tid; t < c.e; t += kEncodeThreads) out[t] = (uint8_t)bit(t);
    }
    __syncthreads();
  }
}

}  // namespace

cudaError_t launch_nr_encode(const NrEncodeArgs& a, cudaStream_t stream) {
  if (a.n_frames <= 0) return cudaSuccess;
  const int ws = (a.code.z + 31) / 32 + 1;
  const size_t smem = (size_t)(a.code.n_full / a.code.z + 4) * ws * 4;  // at most 3.8 KB
  void* args[] = {(void*)&a};
  return cudaLaunchKernel((void*)nr_encode_kernel, dim3((unsigned)(a.n_frames < 4096 ? a.n_frames : 4096)),
                          dim3(kEncodeThreads), args, smem, stream);
}

}  // namespace cbk
