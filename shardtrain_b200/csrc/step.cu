// The bookkeeping of a training step: shifted targets, the number of labels, the loss of a micro-step
// and the values the host reads at the end.  Chains of scalar torch operators did this (14 launches
// per micro-step, 24 per step); a small step, bound by the host, spent 0.3 of its 3.3 ms on launching
// them.  Compiled without fast math: the divisions are the operators' divisions.
#include <algorithm>

#include "api.h"
#include "common.cuh"

namespace stb {

namespace {

constexpr int kIgnored = -100;

// target[b, s] = labels[b, s + 1], nothing after the last token; optionally the number of targets that count
__global__ void __launch_bounds__(256)
shift_targets_kernel(const int64_t* __restrict__ labels, int64_t row_stride, int64_t col_stride, int64_t n,
                     int64_t seq, int64_t* __restrict__ target, unsigned long long* __restrict__ count) {
  int mine = 0;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t b = i / seq, s = i - b * seq;
    const int64_t t = s + 1 < seq ? labels[b * row_stride + (s + 1) * col_stride] : kIgnored;
    if (target != nullptr) target[i] = t;
    mine += t != kIgnored;
  }
  if (count == nullptr) return;
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if ((threadIdx.x & 31) == 0 && mine != 0) atomicAdd(count, static_cast<unsigned long long>(mine));
}

// loss = total * degree / labels, factor = degree / labels (what the gradient of a row's loss is scaled by)
__global__ void loss_kernel(const float* __restrict__ total, const int64_t* __restrict__ labels, float degree,
                            float* __restrict__ loss, float* __restrict__ factor) {
  const float n = static_cast<float>(*labels);
  *loss = __fdiv_rn(__fmul_rn(*total, degree), n);
  *factor = __fmul_rn(__frcp_rn(n), degree);
}

// out = {finite, loss, labels, padding, status}: what a step's host read needs; clears the check flags
__global__ void step_metrics_kernel(int* __restrict__ flags, const float* __restrict__ total,
                                    const int64_t* __restrict__ labels, const int64_t* __restrict__ count,
                                    const int* __restrict__ status, double* __restrict__ out) {
  const float loss = __fdiv_rn(*total, static_cast<float>(*labels));
  out[0] = flags[0] == 0 && isfinite(loss) ? 1.0 : 0.0;
  out[1] = loss;
  out[2] = static_cast<double>(*count);
  out[3] = flags[1];
  out[4] = *status;
  flags[0] = 0;
  flags[1] = 0;
}

}  // namespace

cudaError_t launch_shift_targets(const int64_t* labels, int64_t row_stride, int64_t col_stride, int64_t batch,
                                 int64_t seq, int64_t* target, int64_t* count, cudaStream_t s) {
  if (count != nullptr) {
    const cudaError_t e = cudaMemsetAsync(count, 0, 8, s);
    if (e != cudaSuccess) return e;
  }
  const int64_t n = batch * seq;
  if (n == 0) return cudaSuccess;
  shift_targets_kernel<<<static_cast<int>(std::min<int64_t>((n + 255) / 256, sm_count() * 4)), 256, 0, s>>>(
      labels, row_stride, col_stride, n, seq, target, reinterpret_cast<unsigned long long*>(count));
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_loss(const float* total, const int64_t* labels, float degree, float* loss, float* factor,
                        cudaStream_t s) {
  loss_kernel<<<1, 1, 0, s>>>(total, labels, degree, loss, factor);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_step_metrics(int* flags, const float* total, const int64_t* labels, const int64_t* count,
                                const int* status, double* out, cudaStream_t s) {
  step_metrics_kernel<<<1, 1, 0, s>>>(flags, total, labels, count, status, out);
  count_launch();
  return cudaGetLastError();
}

}  // namespace stb
