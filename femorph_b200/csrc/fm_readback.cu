// Read-back kernels of fm_problem_get_state: a problem's state from the
// batch's columns (batch order) into the caller's rows (problem order), a piece
// at a time.  The host used to copy each column and permute it on one thread
// (96^3 cavity, velocity and pressure: 10.9 ms; 41x27x33 with subscales 16.0
// ms); the gathers take tens of microseconds here.
#include <cuda_runtime.h>

#include <algorithm>

#include "fm_device.cuh"

namespace fm {

static int blocks_for(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 16)); }

// u: n x 3 velocities (components in the mask `fixed` zero), p: n pressures;
// either may be null.  slot: each node's place in the problem's node range,
// which starts at nb.
__global__ void read_nodes_kernel(DevBatch B, int64_t nb, const int32_t* slot, int64_t n, int fixed, double* u,
                                  double* p) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t g = nb + slot[i];
    if (u) {
      u[3 * i] = (fixed & FM_FIX_X) ? 0.0 : B.su[g];
      u[3 * i + 1] = (fixed & FM_FIX_Y) ? 0.0 : B.sv[g];
      u[3 * i + 2] = (fixed & FM_FIX_Z) ? 0.0 : B.sw[g];
    }
    if (p) p[i] = B.sp[g];
  }
}

// out: n x 12 subscales, or with CENTROID n x 3 their quarter-weighted sums
// over the Gauss points (eval_centroid_subgrid,
// femVMSExplicitFluidSolver.cpp:713-724).
template <bool CENTROID>
__global__ void read_subscales_kernel(DevBatch B, int64_t eb, const int32_t* slot, int64_t n, double* out) {
  constexpr int W = CENTROID ? 3 : 12;
  const int64_t E = B.E;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n * W; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = i / W;
    const int q = (int)(i - e * W);
    const int64_t k = eb + slot[e];
    auto at = [&](int row) -> double {
      return B.sdus32 ? (double)B.sdus32[(int64_t)row * E + k] : B.sdus[(int64_t)row * E + k];
    };
    double v;
    if (CENTROID) {
      v = 0.0;
#pragma unroll
      for (int g = 0; g < 4; ++g) v += at(g * 3 + q) * 0.25;
    } else {
      v = at(q);
    }
    out[i] = v;
  }
}

// out: n values of a, or n x 2 of (a, c).
__global__ void read_pair_kernel(const double* a, const double* c, const int32_t* slot, int64_t n, double* out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = slot[i];
    if (c) {
      out[2 * i] = a[k];
      out[2 * i + 1] = c[k];
    } else {
      out[i] = a[k];
    }
  }
}

cudaError_t launch_read_nodes(const DevBatch& B, int64_t nb, const int32_t* slot, int64_t n, int fixed, double* u,
                              double* p, cudaStream_t s) {
  read_nodes_kernel<<<blocks_for(n), 256, 0, s>>>(B, nb, slot, n, fixed, u, p);
  return cudaGetLastError();
}

cudaError_t launch_read_subscales(const DevBatch& B, int64_t eb, const int32_t* slot, int64_t n, bool centroid,
                                  double* out, cudaStream_t s) {
  if (centroid)
    read_subscales_kernel<true><<<blocks_for(n * 3), 256, 0, s>>>(B, eb, slot, n, out);
  else
    read_subscales_kernel<false><<<blocks_for(n * 12), 256, 0, s>>>(B, eb, slot, n, out);
  return cudaGetLastError();
}

cudaError_t launch_read_pair(const double* a, const double* c, const int32_t* slot, int64_t n, double* out,
                             cudaStream_t s) {
  read_pair_kernel<<<blocks_for(n), 256, 0, s>>>(a, c, slot, n, out);
  return cudaGetLastError();
}

}  // namespace fm
