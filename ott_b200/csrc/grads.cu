// Gradient of reg_ot_cost with the potentials held fixed, assembled from
// the two plan applications in one pass over the points (declared in
// include/ott_b200.h).
//
// Bound by launches, not by bytes: the same arithmetic written with tensor
// operations takes about fifty small kernels (0.5 ms of host time a term at
// n = m = 4096, d = 64, where the bytes take 1 us); here it takes one launch
// for the points and two for the weights.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/ott_b200.h"

namespace ottb {
namespace {

constexpr int kTile = 32;

template <class T>
struct PointArgs {
  const float* pts;  // [cnt, d]
  const float* vec;  // [1 + d, cnt]: the plan applied to a column of ones and the coordinates
  int64_t cnt;
  T* out;            // [cnt, d]
};

// out_ik = scale 2 inv (vec_0i pts_ik - vec_(1+k)i), FP64; tiles of 32 points
// x 32 coordinates, vec read along the points and turned in shared memory.
// blockIdx.z = side.
template <class T>
__global__ void point_grads_kernel(PointArgs<T> sx, PointArgs<T> sy, int d, double inv,
                                   const double* scale) {
  __shared__ float tile[kTile][kTile + 1];
  const PointArgs<T> s = blockIdx.z ? sy : sx;
  if (!s.out) return;
  const int64_t i0 = (int64_t)blockIdx.x * kTile;
  const int k0 = blockIdx.y * kTile;
  if (i0 >= s.cnt) return;
  for (int r = threadIdx.y; r < kTile; r += blockDim.y) {
    const int64_t i = i0 + threadIdx.x;
    if (k0 + r < d && i < s.cnt) tile[r][threadIdx.x] = s.vec[(int64_t)(1 + k0 + r) * s.cnt + i];
  }
  __syncthreads();
  const double c = 2.0 * inv;
  const double sc = scale ? *scale : 1.0;
  for (int r = threadIdx.y; r < kTile; r += blockDim.y) {
    const int64_t i = i0 + r;
    const int k = k0 + threadIdx.x;
    if (k < d && i < s.cnt) {
      const double v = c * ((double)s.vec[i] * (double)s.pts[i * d + k] - (double)tile[threadIdx.x][r]);
      s.out[i * d + k] = (T)(sc * v);
    }
  }
}

// sums[0] = sum a, sums[1] = sum b; one CTA a side, a fixed order.
__global__ void weight_sums_kernel(const float* a, int64_t n, const float* b, int64_t m,
                                   double* sums) {
  __shared__ double red[32];
  const float* w = blockIdx.x ? b : a;
  const int64_t cnt = blockIdx.x ? m : n;
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < cnt; i += blockDim.x) s += (double)w[i];
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += red[k];
    sums[blockIdx.x] = t;
  }
}

template <class T>
struct WeightArgs {
  const float* w;
  const float* pot;
  int64_t cnt;
  T* out;
};

// out_i = scale ([w_i > 0] (pot_i - eps log w_i - eps) + eps sum of the other
// side's weights). blockIdx.y = side.
template <class T>
__global__ void weight_grads_kernel(WeightArgs<T> sa, WeightArgs<T> sb, double eps,
                                    const double* sums, const double* scale) {
  const WeightArgs<T> s = blockIdx.y ? sb : sa;
  if (!s.out) return;
  const double other = eps * sums[1 - blockIdx.y];
  const double sc = scale ? *scale : 1.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < s.cnt;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double w = (double)s.w[i];
    const double v = w > 0.0 ? (double)s.pot[i] - eps * log(w) - eps : 0.0;
    s.out[i] = (T)(sc * (v + other));
  }
}

template <class T>
int grads(const float* x, const float* y, const float* a, const float* b, const float* f,
          const float* g, const float* rv, const float* cv, int64_t n, int64_t m, int d, double eps,
          double inv, const double* scale, T* gx, T* gy, T* ga, T* gb, double* sums,
          cudaStream_t stream) {
  const int64_t most = std::max(gx ? n : 0, gy ? m : 0);
  const int64_t tiles = (most + kTile - 1) / kTile;
  if (tiles > 0x7fffffff) return OTTB_ERR_UNSUPPORTED;
  if (most > 0) {
    const dim3 grid((unsigned)tiles, (unsigned)((d + kTile - 1) / kTile), 2);
    point_grads_kernel<T><<<grid, dim3(kTile, 8), 0, stream>>>(
        PointArgs<T>{x, rv, n, gx}, PointArgs<T>{y, cv, m, gy}, d, inv, scale);
  }
  if (ga || gb) {
    weight_sums_kernel<<<2, 1024, 0, stream>>>(a, n, b, m, sums);
    const int64_t w = std::max(ga ? n : 0, gb ? m : 0);
    const dim3 grid((unsigned)std::min<int64_t>((w + 255) / 256, 1024), 2);
    weight_grads_kernel<T><<<grid, 256, 0, stream>>>(WeightArgs<T>{a, f, n, ga},
                                                     WeightArgs<T>{b, g, m, gb}, eps, sums, scale);
  }
  return cudaGetLastError() == cudaSuccess ? OTTB_OK : OTTB_ERR_CUDA;
}

}  // namespace
}  // namespace ottb

extern "C" int32_t ottb_reg_ot_cost_grads(const float* x, const float* y, const float* a,
                                          const float* b, const float* f, const float* g,
                                          const float* row_vec, const float* col_vec, int64_t n,
                                          int64_t m, int32_t d, double epsilon,
                                          double inv_scale_cost, const double* scale,
                                          int32_t out_f32, void* gx, void* gy, void* ga, void* gb,
                                          double* sums, void* stream) {
  if (n < 1 || m < 1 || d < 1 || (gx && (!x || !row_vec)) || (gy && (!y || !col_vec)) ||
      ((ga || gb) && (!a || !b || !sums)) || (ga && !f) || (gb && !g) || (d + 31) / 32 > 65535)
    return OTTB_ERR_INVALID;
  const cudaStream_t st = (cudaStream_t)stream;
  if (out_f32)
    return ottb::grads<float>(x, y, a, b, f, g, row_vec, col_vec, n, m, d, epsilon, inv_scale_cost,
                              scale, (float*)gx, (float*)gy, (float*)ga, (float*)gb, sums, st);
  return ottb::grads<double>(x, y, a, b, f, g, row_vec, col_vec, n, m, d, epsilon, inv_scale_cost,
                             scale, (double*)gx, (double*)gy, (double*)ga, (double*)gb, sums, st);
}
