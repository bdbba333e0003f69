// ela3d_media.cu -- earth models generated on the GPU straight into a
// shot's padded model arrays (no host arrays, no upload).
//  - homogeneous: constant cp, cs, rho (simpelmodel.cpp:45-59);
//  - layered dome: interfaces z_i(x, y) = depth_i - A exp(-r^2 / (2 s^2))
//    (cells); layer L = number of interfaces at or above the cell, capped at
//    nlayers-1; cs = cp / ratio_L, rho = coef * cp^pow; then cp and rho get
//    independent uniform relative noise of +-perturb from a counter-based
//    hash of (seed, cell) (SplitMix64), so any cell's value is reproducible
//    without a sequential generator;
//  - the five-medium anticline of generate_3d_model_anticline.m: dome
//    Z = ((sin X + sin Y)/2 - 0.5)/0.5 clipped at 0 on X, Y in [0, pi]
//    (:2-13), interfaces h - 100 Z with h = 121/161/201 (:17-30), the k < 80
//    pocket inside medium 3 (:50-55) and the media table (:71-76); depths
//    scale with nz / 201 (exactly the MATLAB model at 201 cells).
// Values are computed in double and rounded to float32, the precision the
// model is defined in, before being stored in the plan's type.
#include <limits.h>
#include <math.h>
#include <stdint.h>

#include "ela3d_internal.h"

namespace ela3d {

// the 53 bits of the noise's uniform fraction
__device__ __forceinline__ uint64_t hash_bits(uint64_t seed, uint64_t cell, uint64_t stream) {
  uint64_t z = seed + 0x9E3779B97F4A7C15ull * (cell * 2 + stream + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return z >> 11;
}

// The noise's factor in [-1, 1): 2 u - 1 of the fraction u = m 2^-53, built
// from the bits of m (exact) without a 64-bit integer conversion.
__device__ __forceinline__ double hash_symmetric(uint64_t seed, uint64_t cell, uint64_t stream) {
  const uint64_t m = hash_bits(seed, cell, stream);
  const double v = __longlong_as_double((long long)(0x3ff0000000000000ull | (m >> 1)));   // 1 + (m >> 1) 2^-52
  return __fma_rn(2.0, v, -3.0) + ((m & 1) ? 0x1p-52 : 0.0);
}

// Each thread fills kModelPlanes planes of one column.  FP64 arithmetic
// bounds the generator (two lanes a cycle on each SM), so what a column's
// cells share is computed once for them: the dome's height and with it the
// first plane of each layer, and in each block the layers' cs and rho.  A
// cell's own FP64 work is its noise, five operations for each of cp and rho.
// With one exp and one pow per cell a plan of 640x512x384 cells took 36.9 ms
// to create, now 7.9 (256^3: 5.6, now 1.5); the models are the same bits.
constexpr int kModelPlanes = 32;
constexpr int kModelThreads = 128;

// the first integer k with k >= t (none for NaN)
__device__ __forceinline__ int first_plane(double t) {
  if (isnan(t)) return INT_MAX;
  return (int)fmin(fmax(ceil(t), -1073741824.0), 1073741824.0);
}

template <typename T>
__global__ void __launch_bounds__(kModelThreads)
    model_kernel(ModelSpec s, int nx, int ny, int nz, int px, long long columns, int run0, T *cp, T *cs, T *rho) {
  __shared__ double layer_vp[kMaxLayers], layer_vs[kMaxLayers], layer_rho[kMaxLayers];
  if (s.kind == MODEL_LAYERED_DOME) {
    const int L = threadIdx.x;
    if (L < kMaxLayers) {
      layer_vp[L] = s.cp[L];
      layer_vs[L] = s.cp[L] / s.cs_ratio[L];
      layer_rho[L] = s.rho_coef * pow(s.cp[L], s.rho_pow);
    }
    __syncthreads();
  }
  const long long c = blockIdx.x * (long long)kModelThreads + threadIdx.x;   // column: y * px + x
  if (c >= columns) return;
  const int y = (int)(c / px), x = (int)(c - (long long)y * px);
  const int k0 = (run0 + blockIdx.y) * kModelPlanes, k1 = min(k0 + kModelPlanes, nz);
  long long q = k0 * columns + c;
  if (x >= nx) {
    for (int k = k0; k < k1; ++k, q += columns) cp[q] = cs[q] = rho[q] = T(0);
    return;
  }
  if (s.kind == MODEL_HOMOGENEOUS) {
    const T a = (T)(float)s.cp0, b = (T)(float)s.cs0, r = (T)(float)s.rho0;
    for (int k = k0; k < k1; ++k, q += columns) {
      cp[q] = a;
      cs[q] = b;
      rho[q] = r;
    }
  } else if (s.kind == MODEL_LAYERED_DOME) {
    const double dx = x - s.dome_xc, dy = y - s.dome_yc;
    const double dome = s.dome_amp * exp(-(dx * dx + dy * dy) / (2.0 * s.dome_sigma * s.dome_sigma));
    int top[kMaxLayers];   // interface i lies above plane k where k >= top[i]
#pragma unroll
    for (int i = 0; i < kMaxLayers; ++i) top[i] = i < s.nlayers ? first_plane(s.depth[i] - dome) : INT_MAX;
    uint64_t cell = ((uint64_t)k0 * ny + y) * nx + x;
    for (int k = k0; k < k1; ++k, q += columns, cell += (uint64_t)nx * ny) {
      int L = 0;
#pragma unroll
      for (int i = 0; i < kMaxLayers; ++i) L += k >= top[i] ? 1 : 0;
      L = max(0, min(L, min(s.nlayers, kMaxLayers) - 1));
      double vp = layer_vp[L], dn = layer_rho[L];
      if (s.perturb > 0) {
        vp *= 1.0 + s.perturb * hash_symmetric(s.seed, cell, 0);
        dn *= 1.0 + s.perturb * hash_symmetric(s.seed, cell, 1);
      }
      cp[q] = (T)(float)vp;
      cs[q] = (T)(float)layer_vs[L];
      rho[q] = (T)(float)dn;
    }
  } else {  // MODEL_MATLAB_ANTICLINE
    const double PI = 3.141592653589793238462643;
    const double X = PI * x / (nx - 1), Y = PI * y / (ny - 1);
    double Z = ((sin(X) + sin(Y)) / 2.0 - 0.5) / 0.5;
    if (Z < 0) Z = 0;
    const double sc = nz / 201.0;
    const double s1 = 121 * sc - 100 * sc * Z, s2 = 161 * sc - 100 * sc * Z, s3 = 201 * sc - 100 * sc * Z;
    const float media[6][3] = {{0, 0, 0}, {3000, 1700, 2800}, {3600, 1400, 2300}, {3000, 1700, 2800},
                               {3600, 1700, 2800}, {3650, 1500, 2450}};
    for (int k = k0; k < k1; ++k, q += columns) {
      const double kk = k + 1;   // 1-based depth index of the MATLAB loop
      int m = 1;
      if (kk > s1) m = 2;
      if (kk > s2) { m = 3; if (kk < 80 * sc) m = 4; }
      if (kk > s3) m = 5;
      cp[q] = (T)media[m][0];
      cs[q] = (T)media[m][1];
      rho[q] = (T)media[m][2];
    }
  }
}

template <typename T>
static cudaError_t launch_model(const ModelSpec &s, int nx, int ny, int nz, int px, T *cp, T *cs, T *rho,
                                cudaStream_t st) {
  const long long columns = (long long)px * ny;
  const long long blocks = (columns + kModelThreads - 1) / kModelThreads;
  const int runs = (nz + kModelPlanes - 1) / kModelPlanes;
  for (int r = 0; r < runs; r += 65535) {   // (the most a launch's y dimension takes)
    const dim3 grid((unsigned)blocks, (unsigned)(runs - r < 65535 ? runs - r : 65535));
    model_kernel<T><<<grid, kModelThreads, 0, st>>>(s, nx, ny, nz, px, columns, r, cp, cs, rho);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
cudaError_t launch_model_f32(const ModelSpec &s, int nx, int ny, int nz, int px, float *cp, float *cs, float *rho,
                             cudaStream_t st) {
  return launch_model(s, nx, ny, nz, px, cp, cs, rho, st);
}
cudaError_t launch_model_f64(const ModelSpec &s, int nx, int ny, int nz, int px, double *cp, double *cs, double *rho,
                             cudaStream_t st) {
  return launch_model(s, nx, ny, nz, px, cp, cs, rho, st);
}

}  // namespace ela3d
