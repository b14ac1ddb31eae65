// Host <-> device state transfer: packed (x, y, z) triples on the host side, float4
// arrays (w = charge or inverse mass) on the device side.  The triples cross the bus as
// one contiguous copy into a device buffer and are spread over the float4 array there:
// a strided 2-D copy of 12-byte rows moves one row at a time (230,400 atoms, positions
// and velocities in: 5.3 ms as 2-D copies, 0.13 ms this way; out: 0.65 -> 0.13 ms).
#include "common.cuh"
#include "kernels.h"

namespace fzk {

// out[i].xyz = in[3 i ...], w kept; flag (may be null) is raised: the lists follow
__global__ void __launch_bounds__(256) k_unpack3(const float* __restrict__ in, float4* out, int n, int* flag) {
  griddep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && flag) *flag = 1;
  if (i >= n) return;
  out[i] = make_float4(in[3 * i], in[3 * i + 1], in[3 * i + 2], out[i].w);
}

__global__ void __launch_bounds__(256) k_pack3(const float4* __restrict__ in, float* out, int n) {
  griddep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 v = in[i];
  out[3 * i] = v.x;
  out[3 * i + 1] = v.y;
  out[3 * i + 2] = v.z;
}

// fixed-point forces (x[n] y[n] z[n]) to doubles (x, y, z per atom); the scale is a
// power of two, so every value is the host division's
__global__ void __launch_bounds__(256) k_forces_out(const long long* __restrict__ facc, double* out, int n) {
  griddep_wait();
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= 3 * n) return;
  const int i = j / 3, c = j - 3 * i;
  out[j] = (double)facc[(size_t)c * n + i] * (1.0 / kFixFd);
}

void launch_unpack3(const float* in, float4* out, int n, int* flag, cudaStream_t st) {
  launch_pdl(k_unpack3, dim3((n + 255) / 256), dim3(256), 0, st, in, out, n, flag);
}
void launch_pack3(const float4* in, float* out, int n, cudaStream_t st) {
  launch_pdl(k_pack3, dim3((n + 255) / 256), dim3(256), 0, st, in, out, n);
}
void launch_forces_out(const long long* facc, double* out, int n, cudaStream_t st) {
  launch_pdl(k_forces_out, dim3((3 * n + 255) / 256), dim3(256), 0, st, facc, out, n);
}

}  // namespace fzk
