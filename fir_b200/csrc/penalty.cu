// The quadratic smoothness penalty of the differentiable projector and its
// gradient, in one pass over the image each.
//
// As separate tensor operations over the 13 offsets of half the neighbourhood
// the penalty took about 70 launches forward and 80 backward, each reading
// shifted views of the image: 2.2 ms of host time per gradient at any size.
// One kernel reads each voxel's neighbours, which neighbouring threads share
// through L1, and is bound by the launch on small images and by L1 on large
// ones.
#include "internal.h"

namespace fir
{
namespace
{
constexpr int kBlock = 256;

// 1 / distance of a neighbour with n non-zero offsets.
__device__ __forceinline__ double inverse_distance(int n)
{
  return n == 1 ? 1.0 : (n == 2 ? 0.70710678118654752 : 0.57735026918962576);
}

// Blocks stride over the voxels of all frames; block b's share of the value
// goes to partials[b], summed in a fixed order.
template<typename T, bool kValue, bool kGrad>
__global__ void __launch_bounds__(kBlock) k_penalty(int nx, int ny, int nz, long long n, const T* __restrict__ img,
                                                    double scale, double* __restrict__ partials,
                                                    T* __restrict__ grad)
{
  const long long nxy = (long long)nx * ny, nvox = nxy * nz;
  double sum = 0.0;
  for (long long i = blockIdx.x * (long long)kBlock + threadIdx.x; i < n; i += (long long)gridDim.x * kBlock)
  {
    const long long j = i % nvox;
    const int z = (int)(j / nxy);
    const int r = (int)(j - z * nxy);
    const int y = r / nx, x = r - y * nx;
    const double v = (double)__ldg(img + i);
    double g = 0.0;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
    {
#pragma unroll
      for (int dy = -1; dy <= 1; ++dy)
      {
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx)
        {
          // the value counts each pair once, from its later voxel's side
          const bool later = dz > 0 || (dz == 0 && (dy > 0 || (dy == 0 && dx > 0)));
          if (!(later || (kGrad && (dz != 0 || dy != 0 || dx != 0))))
          {
            continue;
          }
          const int zz = z + dz, yy = y + dy, xx = x + dx;
          if (zz >= 0 && zz < nz && yy >= 0 && yy < ny && xx >= 0 && xx < nx)
          {
            const double w = inverse_distance((dz != 0) + (dy != 0) + (dx != 0));
            const double d = v - (double)__ldg(img + i + dz * nxy + (long long)dy * nx + dx);
            g += w * d;
            if (kValue && later)
            {
              sum += w * d * d;
            }
          }
        }
      }
    }
    if (kGrad)
    {
      grad[i] = (T)(2.0 * scale * g);
    }
  }
  if (kValue)
  {
    __shared__ double part[kBlock];
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int h = kBlock / 2; h > 0; h /= 2)
    {
      if ((int)threadIdx.x < h)
      {
        part[threadIdx.x] += part[threadIdx.x + h];
      }
      __syncthreads();
    }
    if (threadIdx.x == 0)
    {
      partials[blockIdx.x] = scale * part[0];
    }
  }
}

template<typename T>
void penalty(int nx, int ny, int nz, long long n, const void* img, double scale, double* partials, int n_partials,
             void* grad, cudaStream_t stream)
{
  const T* in = static_cast<const T*>(img);
  T* out = static_cast<T*>(grad);
  if (partials != nullptr && grad != nullptr)
  {
    k_penalty<T, true, true><<<n_partials, kBlock, 0, stream>>>(nx, ny, nz, n, in, scale, partials, out);
  }
  else if (partials != nullptr)
  {
    k_penalty<T, true, false><<<n_partials, kBlock, 0, stream>>>(nx, ny, nz, n, in, scale, partials, nullptr);
  }
  else if (grad != nullptr)
  {
    const long long blocks = (n + kBlock - 1) / kBlock;
    k_penalty<T, false, true><<<(unsigned)(blocks < 0x7fffffff ? blocks : 0x7fffffff), kBlock, 0, stream>>>(
      nx, ny, nz, n, in, scale, nullptr, out);
  }
}
}  // namespace

void launch_quadratic_penalty(int nx, int ny, int nz, int nf, const void* img, bool f64, double scale,
                              double* partials, int n_partials, void* grad, cudaStream_t stream)
{
  const long long n = (long long)nx * ny * nz * nf;
  if (n <= 0)
  {
    return;
  }
  if (f64)
    penalty<double>(nx, ny, nz, n, img, scale, partials, n_partials, grad, stream);
  else
    penalty<float>(nx, ny, nz, n, img, scale, partials, n_partials, grad, stream);
}
}  // namespace fir
