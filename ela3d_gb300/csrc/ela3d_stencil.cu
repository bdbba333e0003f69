// ela3d_stencil.cu -- compiled instances of the stress and velocity kernels.
// Each instance fixes the real type, the x-y tile (TX x TY cells) and the
// number of shared-memory stages NS; the engine's autotuner picks one per
// grid size.
#include "ela3d_internal.h"
#include "ela3d_stencil.cuh"

namespace ela3d {

// NSV: places of the velocity kernel's rings (its planes are smaller than the
// stress kernel's, so it can hold more of them); the dataflow kernel runs
// both half-steps in rings of NS places.
template <typename T, int TX, int TY, int NS, int CPT = Vec<T>::N, int MB = 0, int LOAD = LOAD_TMA, int NSV = NS>
static Variant make_variant() {
  using G = Geo<T, TX, TY, NS, CPT, MB>;
  using GV = Geo<T, TX, TY, NSV, CPT, MB>;
  Variant v;
  v.fp64 = sizeof(T) == 8;
  v.tx = TX;
  v.ty = TY;
  v.ns = NS;
  v.ns_vel = NSV;
  v.threads = G::THREADS;
  v.stress_smem = kKernelSmem<G, StressRing<G>>;
  v.vel_smem = kKernelSmem<GV, VelocityRing<GV>>;
  v.halo = G::H;
  v.loads = LOAD;
  v.stress = reinterpret_cast<const void *>(&stress_kernel<T, TX, TY, NS, CPT, MB, LOAD>);
  v.velocity = reinterpret_cast<const void *>(&velocity_kernel<T, TX, TY, NSV, CPT, MB, LOAD>);
  v.flow = nullptr;
  v.flow_smem = 0;
  v.flow_once = nullptr;
  v.flow_coef = nullptr;
  v.flow_coef_smem = 0;
  if constexpr (LOAD == LOAD_TMA) {
    v.flow = reinterpret_cast<const void *>(&flow_kernel<T, TX, TY, NS, CPT, MB, false, false>);
    v.flow_smem = Flow<G, T, NS>::SMEM;
    // FP32 tiles of seven or eight warps: also with the L2 hints
    if constexpr (sizeof(T) == 4 && G::NCW >= 7)
      v.flow_once = reinterpret_cast<const void *>(&flow_kernel<T, TX, TY, NS, CPT, MB, false, true>);
    // FP64 with one cell per thread and one block per SM: also with coefficients from arrays
    if constexpr (sizeof(T) == 8 && CPT == 1 && MB == 0) {
      v.flow_coef = reinterpret_cast<const void *>(&flow_kernel<T, TX, TY, NS, CPT, MB, true, false>);
      v.flow_coef_smem = Flow<Geo<T, TX, TY, NS, CPT, MB, true>, T, NS>::SMEM;
    }
  }
  return v;
}

static const Variant kVariants[] = {
    // velocity rings of 5 places: more bytes in flight per SM, 1.2% less
    // velocity time at 256^3
    make_variant<float, 128, 7, 4, 4, 0, LOAD_TMA, 5>(),
    make_variant<float, 128, 6, 5>(),
    make_variant<float, 128, 5, 6>(),
    make_variant<float, 64, 14, 4>(),
    make_variant<float, 128, 3, 4>(),
    make_variant<float, 64, 6, 4>(),
    // 28 threads per row, so a warp spans two rows: covers rows of ~100
    // cells with less waste than the 128-wide tile (101: 90% against 79%)
    make_variant<float, 112, 8, 4>(),
    // the 128x7 tile with its stages filled by cp.async instead of TMA (the
    // measured alternative to the tensor-memory-accelerator loads)
    make_variant<float, 128, 7, 4, 4, 0, LOAD_CP_ASYNC>(),
    // FP64 (the accuracy build; its rate on GB300 makes it compute-bound):
    // one cell per thread keeps it free of register spills
    make_variant<double, 32, 7, 4, 1>(),
    make_variant<double, 32, 3, 4, 1, 2>(),
    make_variant<double, 32, 6, 3>(),
    make_variant<double, 64, 3, 4>(),
    // narrow FP32 tiles for rows that fill the wide ones badly (150: 94% of
    // five 32-wide tiles, 67% of two 112-wide ones)
    make_variant<float, 56, 16, 4>(),
    make_variant<float, 32, 28, 4>(),
    // FP32 tiles of eight consumer warps (their launch splits its registers
    // unevenly): grids are often multiples of 8 or 16 rows, and near the L2
    // size the warps are what limits the kernel (128^3 43.6 -> 46.2
    // Gcell-updates/s, 192^3 46.6 -> 47.7).  At 168 registers a thread seven of
    // their dataflow instances spill 24 bytes (112x9 and 56x18, and all five
    // with the L2 hints)
    make_variant<float, 128, 8, 4>(),
    make_variant<float, 64, 16, 4>(),
    make_variant<float, 32, 32, 4>(),
    make_variant<float, 112, 9, 4>(),
    make_variant<float, 56, 18, 4>(),
    // and narrow FP64 tiles: its arithmetic bounds FP64, idle lanes included
    make_variant<double, 16, 14, 4, 1>(),
    make_variant<double, 8, 28, 4, 1>(),
    make_variant<double, 32, 8, 4, 1>(),
    make_variant<double, 16, 16, 4, 1>(),
};

cudaError_t launch_coef_f64(const ShotDesc<double> &shot, double *out, cudaStream_t s) {
  const long long cells = (long long)shot.nz * shot.ny * shot.px;
  const long long blocks = (cells + 255) / 256;
  coef_kernel<double><<<(unsigned)(blocks < 4864 ? blocks : 4864), 256, 0, s>>>(shot, out, cells);
  return cudaGetLastError();
}

const Variant *variants(int *count) {
  *count = (int)(sizeof(kVariants) / sizeof(kVariants[0]));
  return kVariants;
}

}  // namespace ela3d
