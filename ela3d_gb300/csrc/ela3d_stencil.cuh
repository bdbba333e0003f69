// ela3d_stencil.cuh -- the time-loop kernels, templated on the real type and
// the x-y tile: the stress and the velocity half-step (stress_item,
// velocity_item), as a kernel each and as items of one persistent dataflow
// kernel (flow_kernel).
//
// Scheme (2.5-D z-march):
//  - a block owns a list of work items (shot, x-y tile, z-run [k0, k1));
//  - one producer warp walks the block's planes and, for each, issues TMA
//    tiled loads of every input array's x-y tile (with the one-cell halos
//    the stencil needs) into two rings of shared-memory places (what the
//    plane below reads too, and the rest); each place has a "full" mbarrier
//    (TMA bytes landed) and an "empty" mbarrier (all consumer warps done), so
//    refills start as soon as a place is released;
//  - out-of-grid halo cells arrive as zeros (the TMA fill), which is also
//    the zero plane above k = nz-1 that the reference's sigma_xz/sigma_yz
//    loop reads (simpelmodel.cpp:450,477);
//  - consumer warps compute plane k from places k and k+1 (the z+1
//    neighbours) and keep the z-1 neighbours in registers; each thread owns
//    16 bytes of consecutive x cells of one row (float4 / double2);
//  - C-PML memory variables are read and written only in the PML slabs, each
//    thread copying its own cells' one plane ahead (PsiSlots);
//  - cells outside the update ranges of the reference's loops keep their
//    value (the Dirichlet edges); receivers are sampled after the velocity
//    update and the force source is added after that (simpelmodel.cpp:592-622).
// Every wait is bounded: on expiry the kernel ORs DEV_ERR_TIMEOUT into the
// error word, the producer waits (bounded) for its issued copies, and the
// threads return.
#pragma once

#include <limits.h>

#include <type_traits>

#include "ela3d_device.cuh"

namespace ela3d {

// COEF: the update coefficients (dt lambda and so on) come from arrays
// computed once per plan instead of from the model (FP64 dataflow kernels).
// ONCE: the model and the C-PML memory variables, which a step reads (and
// writes) once or twice, are the first lines that L2 gives up, so that the
// fields, which pass from half-step to half-step and to the neighbouring tiles,
// stay there (FP32 dataflow kernels of shots whose arrays about fill the L2).
template <typename T, int TX_, int TY_, int NS_, int CPT_ = Vec<T>::N, int MINB_ = 0, bool COEF_ = false,
          bool ONCE_ = false>
struct Geo {
  static constexpr bool COEF = COEF_, ONCE = ONCE_;
  static constexpr int VEC = CPT_;       // cells per thread (consecutive in x)
  static constexpr int H = Vec<T>::N;    // halo width in x (16 bytes, the TMA x alignment)
  static constexpr int TX = TX_, TY = TY_, NS = NS_;
  static constexpr int NTX = TX / VEC;
  static constexpr int NCW = (NTX * TY + 31) / 32;   // consumer warps
  static constexpr int NT = 32 * NCW;      // consumer threads (a last few may have no cells)
  // Seven consumer warps and the loading warp fill the register file at up to
  // 255 registers a thread.  Eight consumer warps cannot: the loading warp would
  // be a ninth, a sub-partition's third.  They are launched as three warpgroups
  // of 168 registers a thread, and the loading warp's group hands registers over
  // to the consumers (setmaxnreg; 8 x 216 + 4 x 72 = 12 x 168).
  static constexpr bool SPLIT = NCW == 8;
  static constexpr int CONSUMER_REGS = 216, LOADER_REGS = 72;
  static_assert(8 * CONSUMER_REGS + 4 * LOADER_REGS <= 12 * 168, "registers of the launch");
  static constexpr int THREADS = SPLIT ? 384 : NT + 32;  // + the loading warp (or its group)
  // blocks per SM the register budget is sized for (64K registers per SM):
  // two blocks of four warps keep 255 registers per thread; fewer cells per
  // thread trade registers for resident warps
  static constexpr int MINB = MINB_ ? MINB_ : (THREADS <= 128 ? 2 : 1);
  static constexpr int WW = TX + H;
  static_assert(H % VEC == 0 && TX % H == 0 && TX + H <= 256 && TY + 1 <= 256, "tile shape");
  __host__ __device__ static constexpr int al(int b) { return (b + 127) & ~127; }
  static constexpr int C = TX * TY;          // center box
  static constexpr int W1 = WW * (TY + 1);   // wide box with one extra row
  static constexpr int W0 = WW * TY;         // wide box
  static constexpr int Y1 = TX * (TY + 1);   // narrow box with one extra row
  __host__ __device__ static constexpr int sz(int e) { return al(e * (int)sizeof(T)); }
  static constexpr int SC = (C * (int)sizeof(T) + 127) & ~127;  // bytes of a centre box
  // A plane is held in two parts, each in a ring of its own: the first part is
  // what the plane below reads too (as its z+1 neighbours), the second the
  // rest.  The first ring has NS places; the second does with one place less
  // where shared memory is short.
  // stress: vx vy cs rho (W1) | vz (W1), cp and the six stresses (C); with
  // COEF: vx vy | vz, the five coefficients in cp's place, the stresses
  static constexpr int S_VX = 0;
  static constexpr int S_VY = S_VX + sz(W1);
  static constexpr int S_CS = S_VY + sz(W1);
  static constexpr int S_RHO = S_CS + sz(W1);
  static constexpr int S_A = COEF ? S_CS : S_RHO + sz(W1);
  static constexpr int S_CENTRE = COEF ? 5 : 1;   // centre boxes before the stresses
  static constexpr int S_VZ = 0;
  static constexpr int S_CP = S_VZ + sz(W1);
  static constexpr int S_SIG = S_CP + S_CENTRE * sz(C);  // six centre boxes follow
  static constexpr int S_B = S_SIG + 6 * sz(C);
  static constexpr int S_TXA = (int)sizeof(T) * (COEF ? 2 : 4) * W1;   // bytes loaded
  static constexpr int S_TXB = (int)sizeof(T) * (W1 + (S_CENTRE + 6) * C);
  // velocity: szz (C), rho (W1) | sxx syy sxy sxz syz with their halos, vx vy
  // vz (C); with COEF: szz | the same and three coefficients (C)
  static constexpr int V_SZZ = 0;
  static constexpr int V_RHO = V_SZZ + sz(C);
  static constexpr int V_A = COEF ? V_RHO : V_RHO + sz(W1);
  static constexpr int V_SXX = 0;                 // W0
  static constexpr int V_SYY = V_SXX + sz(W0);    // Y1
  static constexpr int V_SXY = V_SYY + sz(Y1);    // W1
  static constexpr int V_SXZ = V_SXY + sz(W1);    // W0
  static constexpr int V_SYZ = V_SXZ + sz(W0);    // Y1
  static constexpr int V_V = V_SYZ + sz(Y1);      // vx vy vz (C)
  static constexpr int V_COEF = V_V + 3 * sz(C);
  static constexpr int V_B = COEF ? V_COEF + 3 * sz(C) : V_COEF;
  static constexpr int V_TXA = (int)sizeof(T) * (COEF ? C : C + W1);
  static constexpr int V_TXB = (int)sizeof(T) * (2 * W0 + 2 * Y1 + (COEF ? 6 : 3) * C + W1);
  // memory-variable slots (PsiSlots): one 16-byte (or smaller) vector per
  // consumer thread for each of the three variables of each axis
  static constexpr int PSI_BYTES = 9 * NT * VEC * (int)sizeof(T);
  static constexpr int MAX_SMEM = 232448;   // of one block
  // places of the second ring for parts of a and b bytes, with `other` bytes
  // of shared memory beside the rings
  __host__ __device__ static constexpr int places_b(int a, int b, int other) {
    return NS * (a + b) + 32 * NS + PSI_BYTES + other <= MAX_SMEM / MINB ? NS : NS - 1;
  }
};

// The two rings of a kernel's planes, at the (aligned) base of dynamic shared
// memory, and their mbarriers behind them: full (TMA bytes landed) and empty
// (all consumer warps done) for every place.
template <int NA_, int NB_, int A_, int B_>
struct Ring {
  static constexpr int NA = NA_, NB = NB_, A = A_, B = B_;
  static constexpr int BARRIERS = NA * A + NB * B;
  static constexpr int BYTES = BARRIERS + 16 * (NA + NB);
  unsigned char *base;
  __device__ __forceinline__ unsigned char *a(int s) const { return base + s * A; }
  __device__ __forceinline__ unsigned char *b(int s) const { return base + NA * A + s * B; }
  __device__ __forceinline__ uint64_t *bars() const { return reinterpret_cast<uint64_t *>(base + BARRIERS); }
  __device__ __forceinline__ uint64_t *full_a(int s) const { return bars() + s; }
  __device__ __forceinline__ uint64_t *full_b(int s) const { return bars() + NA + s; }
  __device__ __forceinline__ uint64_t *empty_a(int s) const { return bars() + NA + NB + s; }
  __device__ __forceinline__ uint64_t *empty_b(int s) const { return bars() + 2 * NA + NB + s; }
};

// A place in a ring of N, and the parity of the pass over it.
template <int N>
struct Place {
  int s = 0;
  uint32_t parity = 0;
  __device__ __forceinline__ void next() {
    if (++s == N) {
      s = 0;
      parity ^= 1;
    }
  }
};

template <int REGS> __device__ __forceinline__ void more_registers() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS));
}
template <int REGS> __device__ __forceinline__ void fewer_registers() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS));
}

template <typename T>
__device__ __forceinline__ int tiles_x_of(const ShotDesc<T> &s, int TX) {
  return (s.nx + TX - 1) / TX;
}

// Arithmetic with the rounding written out: these are never fused with a
// neighbouring operation.
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }

// The same over the V cells of a thread; operands are arrays (a value per
// cell) or one value for all.  FP32 cells go two at a time through the packed
// f32x2 instructions, with the same roundings: half the instructions.
template <typename T, int V> constexpr bool kPacked = sizeof(T) == 4 && V % 2 == 0;
struct Pair { unsigned long long v; };
__device__ __forceinline__ Pair pair_of(float a, float b) {
  Pair p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "f"(a), "f"(b));
  return p;
}
template <int V> __device__ __forceinline__ Pair pair_at(const float (&a)[V], int e) { return pair_of(a[e], a[e + 1]); }
__device__ __forceinline__ Pair pair_at(const float &a, int) { return pair_of(a, a); }
template <typename T, int V> __device__ __forceinline__ T cell_at(const T (&a)[V], int e) { return a[e]; }
template <typename T> __device__ __forceinline__ T cell_at(const T &a, int) { return a; }
template <int V> __device__ __forceinline__ void put_pair(float (&d)[V], int e, Pair p) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d[e]), "=f"(d[e + 1]) : "l"(p.v));
}
// d = a b + c
template <typename T, int V, typename A, typename B, typename C>
__device__ __forceinline__ void fma_v(T (&d)[V], const A &a, const B &b, const C &c) {
#pragma unroll
  for (int e = 0; e < V; e += kPacked<T, V> ? 2 : 1) {
    if constexpr (kPacked<T, V>) {
      Pair p;
      asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p.v) : "l"(pair_at(a, e).v), "l"(pair_at(b, e).v), "l"(pair_at(c, e).v));
      put_pair(d, e, p);
    } else {
      d[e] = fma_rn(cell_at(a, e), cell_at(b, e), cell_at(c, e));
    }
  }
}
template <typename T, int V, typename A, typename B>
__device__ __forceinline__ void mul_v(T (&d)[V], const A &a, const B &b) {
#pragma unroll
  for (int e = 0; e < V; e += kPacked<T, V> ? 2 : 1) {
    if constexpr (kPacked<T, V>) {
      Pair p;
      asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p.v) : "l"(pair_at(a, e).v), "l"(pair_at(b, e).v));
      put_pair(d, e, p);
    } else {
      d[e] = mul_rn(cell_at(a, e), cell_at(b, e));
    }
  }
}
template <typename T, int V, typename A, typename B>
__device__ __forceinline__ void add_v(T (&d)[V], const A &a, const B &b) {
#pragma unroll
  for (int e = 0; e < V; e += kPacked<T, V> ? 2 : 1) {
    if constexpr (kPacked<T, V>) {
      Pair p;
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(p.v) : "l"(pair_at(a, e).v), "l"(pair_at(b, e).v));
      put_pair(d, e, p);
    } else {
      d[e] = add_rn(cell_at(a, e), cell_at(b, e));
    }
  }
}
// d = a - b (FP32: a + (-1) b in one rounding, the same value)
template <typename T, int V, typename A, typename B>
__device__ __forceinline__ void sub_v(T (&d)[V], const A &a, const B &b) {
  if constexpr (kPacked<T, V>) {
    fma_v(d, b, T(-1), a);
  } else {
#pragma unroll
    for (int e = 0; e < V; ++e) d[e] = sub_rn(cell_at(a, e), cell_at(b, e));
  }
}
// the cells' west neighbours (first: the value west of cell 0) and east ones
template <typename T, int V>
__device__ __forceinline__ void west_of(T (&d)[V], const T (&a)[V], T first) {
#pragma unroll
  for (int e = 0; e < V; ++e) d[e] = e > 0 ? a[e > 0 ? e - 1 : 0] : first;
}
template <typename T, int V>
__device__ __forceinline__ void east_of(T (&d)[V], const T (&a)[V], T last) {
#pragma unroll
  for (int e = 0; e < V; ++e) d[e] = e < V - 1 ? a[e < V - 1 ? e + 1 : e] : last;
}
// s <- n for the cells whose bit is set in m (selects: a branch for warps
// without a masked cell costs more than it saves, 101^3 36.3 against 37.1
// Gcell-updates/s)
template <typename T, int V>
__device__ __forceinline__ void keep_masked(T (&s)[V], const T (&n)[V], unsigned m) {
#pragma unroll
  for (int e = 0; e < V; ++e) s[e] = ((m >> e) & 1u) ? n[e] : s[e];
}

// dt / (R / 2), R the sum of two densities: FP32 uses the hardware
// reciprocal-based divide (<= 2 ulp from the IEEE quotient).
__device__ __forceinline__ float dt_over_rho(float dt, float R) { return __fdividef(dt, mul_rn(R, 0.5f)); }
// FP64: the IEEE quotient dt / (R / 2) = 2 dt / R, with fewer FP64
// operations than a general division: the FP64 pipe (two lanes a cycle on
// each SM) bounds the FP64 kernels.  R is a sum of two float32 model values.
// Its reciprocal is found in pairs of float32 numbers on the FP32 unit (R = rh
// + rl; y = yf + yl from the hardware reciprocal yf of rh and one cubic Newton
// step, e = 1 - R yf, yl = yf (e + e^2); relative error below 2^-45), and the
// quotient takes one Markstein correction (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990): q + (2
// dt - q R) y, whose remainder is exact for an R of 33 bits, is off by 2^-90
// before its rounding, while a quotient by such an R stays 2^-87 away from the
// midpoints between doubles, so it rounds to the IEEE quotient.  Floats are
// widened by integer operations.  Sums of more bits (densities about 512 times
// apart or more) and sums outside [2^-60, 2^60) divide as usual.
__device__ __forceinline__ double widen_signed(float f) {   // (0 becomes 2^-127)
  const unsigned b = __float_as_uint(f);
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}
__device__ __forceinline__ double dt_over_rho(double dt, double R) {
  const double a = 2.0 * dt;
  const int hi = __double2hiint(R);
  const unsigned lo = (unsigned)__double2loint(R);
  if ((unsigned)(hi - 0x3c300000) >= 0x07800000u || (lo & 0xfffffu) != 0) return a / R;
  const unsigned hb = ((unsigned)(hi - 0x38000000) << 3) | (lo >> 29);   // rh: the first 24 bits
  const float rh = __uint_as_float(hb);
  const float rl = (float)(lo & 0x1fffffffu) * __uint_as_float((hb & 0x7f800000u) - (52u << 23));
  float yf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(rh));
  const float e = __fmaf_rn(-rl, yf, __fmaf_rn(-rh, yf, 1.0f));
  const float yl = __fmul_rn(__fmaf_rn(e, e, e), yf);
  const double y = add_rn(widen_signed(yf), widen_signed(yl));
  const double q = mul_rn(a, y);
  return fma_rn(fma_rn(-q, R, a), y, q);
}

// dt mu of the averaged shear velocity S / 2 and density R / 2:
// dt ((R/2 S/2) S/2), the halves taken out as one factor 1/8 (exact: the
// products only change their exponents).
template <typename T, int V>
__device__ __forceinline__ void dt_mu(T (&mu)[V], T dt8, const T (&c0)[V], const T (&c1)[V], const T (&r0)[V],
                                      const T (&r1)[V]) {
  T S[V];
  add_v(S, c0, c1);
  add_v(mu, r0, r1);
  mul_v(mu, mu, S);
  mul_v(mu, mu, S);
  mul_v(mu, mu, dt8);
}

// dt (lambda + 2 mu) and dt lambda: lambda = rho (vp^2 - 2 vs^2).  FP64: the
// model's values are float32 numbers, so the squares are exact and
// rho (vp vp) rounds to what (rho vp) vp does.
template <typename T, int V>
__device__ __forceinline__ void dt_moduli(T dt, const T (&vp)[V], const T (&vs)[V], const T (&rho)[V], T (&l2m)[V],
                                          T (&lam)[V]) {
  if constexpr (sizeof(T) == 4) {
    mul_v(l2m, rho, vp);
    mul_v(l2m, l2m, vp);
    mul_v(lam, vs, T(-2));
    mul_v(lam, lam, vs);
    fma_v(lam, vp, vp, lam);
  } else {
    T vp2[V];
    mul_v(vp2, vp, vp);
    mul_v(l2m, rho, vp2);
    mul_v(lam, vs, vs);
    fma_v(lam, lam, T(-2), vp2);
  }
  mul_v(l2m, l2m, dt);
  mul_v(lam, lam, rho);
  mul_v(lam, lam, dt);
}

// b = dt / rho_avg of the densities r0 and r1.  (FP32 divides for every cell: a
// branch around it costs more.  FP64 leaves out the cells outside the mask,
// whose density may be 0.)
template <typename T, int V>
__device__ __forceinline__ void dt_over_rho(T (&b)[V], T dt, const T (&r0)[V], const T (&r1)[V], unsigned m) {
  add_v(b, r0, r1);
#pragma unroll
  for (int e = 0; e < V; ++e)
    if (sizeof(T) == 4 || ((m >> e) & 1u)) b[e] = dt_over_rho(dt, b[e]);
}

// v + b (d1 + d2 sy + d3 sz) for the cells of the mask.
template <typename T, int V>
__device__ __forceinline__ void velocity_update(T sy, T sz, const T (&b)[V], const T (&d1)[V], const T (&d2)[V],
                                                const T (&d3)[V], T (&v)[V], unsigned m) {
  T t[V];
  fma_v(t, d2, sy, d1);
  fma_v(t, d3, sz, t);
  fma_v(t, b, t, v);
  keep_masked(v, t, m);
}

// sig + (l2m d + lam (t0 + t1)) for the cells of the mask; OWN: the product
// with the component's own derivative d is the fused one, the other is
// rounded first.
template <bool OWN, typename T, int V>
__device__ __forceinline__ void normal_stress(const T (&l2m)[V], const T (&lam)[V], const T (&d)[V], const T (&t0)[V],
                                              const T (&t1)[V], T (&sig)[V], unsigned m) {
  T t[V], u[V];
  add_v(t, t0, t1);
  if constexpr (OWN) {
    mul_v(u, lam, t);
    fma_v(t, l2m, d, u);
  } else {
    mul_v(u, l2m, d);
    fma_v(t, lam, t, u);
  }
  add_v(t, t, sig);
  keep_masked(sig, t, m);
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// L2 prefetch of every 128-byte line of [p, p + bytes).
__device__ __forceinline__ void prefetch_l2(const void *p, int bytes) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  for (uintptr_t q = a & ~uintptr_t(127); q < a + (uintptr_t)bytes; q += 128)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(q));
}

// L2 prefetch of the C-PML memory variables var0 .. var0+2 that the
// consumers of a tile will copy into their slots (PsiSlots, which reach one
// plane ahead and read through L2): issued by the producer warp's lanes (one
// (variable, row) pair per lane) when a plane's stage is requested, NS-2
// planes ahead of the consumers.  A hint: no result depends on it.  A lane has
// one pair, so of a tile with more than 32 of them (three variables of more
// than ten rows) only the first 32 are prefetched: all of the 7- to 9-row
// tiles' pairs, 32 of 64x16's 48, of 32x32's 96 one variable's (pick_tile's
// weights for grids that stream were measured so).  The x slab's row ends are
// short and unaligned (CTL_PF_X, line by line); the rows of the y and z slabs
// are whole (CTL_PF_YZ, bulk prefetches).
__device__ __forceinline__ void prefetch_l2_bulk(const void *p, int bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

template <typename T, int TX, int TY>
struct PsiPrefetch {
  const T *left = nullptr, *right = nullptr;  // this lane's x-slab segments at plane 0
  const T *yrow = nullptr, *zrow = nullptr;   // this lane's y-slab row at plane 0, z-slab row at slab plane 0
  int lbytes = 0, rbytes = 0, wbytes = 0;
  long long pstride = 0, ystride = 0, zstride = 0;  // elements per plane of the x, y and z slabs
  int nz = 0, zl = 0, zr = 0;
  __device__ __forceinline__ void begin(const ShotDesc<T> &sd, int x0, int y0, int var0, int lane, int ctl) {
    const int rows = min(TY, sd.ny - y0);
    lbytes = rbytes = wbytes = 0;
    yrow = zrow = nullptr;
    nz = sd.nz;
    zl = sd.zl;
    zr = sd.zr;
    pstride = (long long)sd.ny * sd.xw;
    ystride = (long long)sd.yw * sd.px;
    zstride = (long long)sd.ny * sd.px;
    if (lane >= 3 * rows) return;
    const int var = var0 + lane / rows, y = y0 + lane % rows;
    if (ctl & CTL_PF_X) {
      const T *row = sd.psi_x + var * sd.psx + (long long)y * sd.xw;
      const int xb = min(x0 + TX, sd.xl);
      const int xc = max(x0, sd.xr), xd = min(x0 + TX, sd.px);
      if (x0 < xb) { left = row + x0; lbytes = (xb - x0) * (int)sizeof(T); }
      if (xc < xd) { right = row + sd.xl + (xc - sd.xr); rbytes = (xd - xc) * (int)sizeof(T); }
    }
    if (ctl & CTL_PF_YZ) {
      wbytes = min(TX, sd.px - x0) * (int)sizeof(T);
      if (y < sd.yl || y >= sd.yr) {
        const int ys = y < sd.yl ? y : sd.yl + (y - sd.yr);
        yrow = sd.psi_y + var * sd.psy + (long long)ys * sd.px + x0;
      }
      zrow = sd.psi_z + var * sd.psz + (long long)y * sd.px + x0;
    }
  }
  __device__ __forceinline__ void plane(int k) const {
    if (k < 0 || k >= nz) return;
    if (lbytes) prefetch_l2(left + k * pstride, lbytes);
    if (rbytes) prefetch_l2(right + k * pstride, rbytes);
    if (yrow) prefetch_l2_bulk(yrow + k * ystride, wbytes);
    if (zrow && (k < zl || k >= zr)) prefetch_l2_bulk(zrow + (k < zl ? k : zl + (k - zr)) * zstride, wbytes);
  }
};

// cp.async counterpart of one TMA box load: the BW x BH box of plane k of
// `base` with origin (x, y), stored densely row by row like the TMA box;
// cells outside [0, nx) x [0, ny) x [0, nz) read as zeros.  Each lane copies
// every 32nd 16-byte chunk.
template <typename T, int BW, int BH>
__device__ __forceinline__ void copy_box_async(unsigned char *dst, const T *base, const ShotDesc<T> &sd, int x, int y,
                                               int k, int lane) {
  constexpr int E = 16 / (int)sizeof(T);  // elements per chunk
  constexpr int CPR = BW / E, N = CPR * BH;
  static_assert(BW % E == 0, "box rows are whole chunks");
  const bool kin = k >= 0 && k < sd.nz;
  for (int c = lane; c < N; c += 32) {
    const int r = c / CPR, xx = x + (c - r * CPR) * E, yy = y + r;
    uint32_t bytes = 0;
    const T *src = base;
    if (kin && yy >= 0 && yy < sd.ny && xx >= 0 && xx < sd.nx) {
      bytes = (uint32_t)(min(E, sd.nx - xx) * (int)sizeof(T));
      src = base + ((long long)k * sd.ny + yy) * sd.px + xx;
    }
    cp_async_16(dst + (size_t)c * 16, src, bytes);
  }
}


// Producer warp: walks the block's items and issues every plane's loads
// (lane 0) and the plane's memory-variable prefetches (all lanes).  An item's
// planes k0 .. k1 - 1 take a place in both rings, its look-ahead plane k1
// (possibly nz, which the TMA fills with zeros) one in the first ring only.
// The consumers of plane k need both parts of k and the first part of k + 1,
// so the first parts run one plane ahead of the second.  Before a place is
// filled again lane 0 waits for the consumers' release of what it held.  (A
// fresh barrier counts as having completed a phase of parity 1.)
// With ASYNC every lane copies a share of each plane's boxes (cp.async)
// instead of lane 0 issuing TMA loads.
template <typename R>
struct Loads {
  Place<R::NA> a;
  Place<R::NB> b;
  unsigned na = 0, nb = 0;   // parts loaded so far
};

template <bool ASYNC, typename R, typename IssueA, typename IssueB, typename Prefetch>
__device__ __forceinline__ bool produce_item(const Item &it, const R &ring, Loads<R> &ld, IssueA issue_a,
                                             IssueB issue_b, Prefetch &prefetch, int lane) {
  for (int k = it.k0 - 1; k < it.k1; ++k) {
    const bool both = k >= it.k0;
    int good = 1;
    if (lane == 0) {
      good = mbar_wait_bounded(ring.empty_a(ld.a.s), ld.a.parity ^ 1);
      if (both) good = good && mbar_wait_bounded(ring.empty_b(ld.b.s), ld.b.parity ^ 1);
    }
    if (!__shfl_sync(0xffffffffu, good, 0)) return false;
    if (ASYNC || lane == 0) {
      issue_a(k + 1, ring.a(ld.a.s), ring.full_a(ld.a.s));
      if (both) issue_b(k, ring.b(ld.b.s), ring.full_b(ld.b.s));
    }
    ld.a.next();
    ++ld.na;
    if (both) {
      ld.b.next();
      ++ld.nb;
    }
    prefetch.plane(k + 1);
  }
  return true;
}

// The block must not exit with copies in flight: waits (bounded) for the
// last loads of each ring, and reports a timeout seen earlier.
template <bool ASYNC, typename R>
__device__ __forceinline__ void produce_drain(const R &ring, const Loads<R> &ld, bool ok, unsigned *__restrict__ err,
                                              int lane) {
  if (ASYNC) cp_async_wait_all();
  if (lane != 0) return;
  if (!ok) atomicOr(err, DEV_ERR_TIMEOUT);
  for (unsigned q = ld.na > R::NA ? ld.na - R::NA : 0; q < ld.na; ++q)
    mbar_wait_bounded(ring.full_a(q % R::NA), (uint32_t)((q / R::NA) & 1), 200000000ull);
  for (unsigned q = ld.nb > R::NB ? ld.nb - R::NB : 0; q < ld.nb; ++q)
    mbar_wait_bounded(ring.full_b(q % R::NB), (uint32_t)((q / R::NB) & 1), 200000000ull);
}

// The producer lanes' memory-variable prefetcher for one half-step (var0 =
// PSI_S0 for the stress half-step, PSI_V0 for the velocity half-step).
template <typename T, int TX, int TY>
struct ItemPrefetch {
  PsiPrefetch<T, TX, TY> pf;
  const ShotDesc<T> *shots;
  int lane, ctl, var0;
  __device__ __forceinline__ void begin(const Item &it) { begin(it, shots[it.shot]); }
  __device__ __forceinline__ void begin(const Item &it, const ShotDesc<T> &sd) {
    const int txs = tiles_x_of(sd, TX);
    pf.begin(sd, (it.tile % txs) * TX, (it.tile / txs) * TY, var0, lane, ctl);
  }
  __device__ __forceinline__ void plane(int k) const { pf.plane(k); }
};

// ------------------------------------------------------- stage loads ----
template <bool ONCE>
__device__ __forceinline__ void load_model(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
  if constexpr (ONCE) tma_load_3d_first(dst, map, x, y, z, bar);
  else tma_load_3d(dst, map, x, y, z, bar);
}

// The two parts of one stress plane (box shapes in ela3d_device.cuh, ShotMaps):
// vx vy cs rho with their halos | vz with its halo, cp and the six stresses.
template <typename G, int LOAD, typename T>
__device__ __forceinline__ void stress_issue_a(const ShotDesc<T> &sd, const ShotMaps &maps, const Item &it, int k,
                                         unsigned char *st, uint64_t *bar, int lane) {
  constexpr int H = G::H, TX = G::TX, TY = G::TY;
  const int txs = tiles_x_of(sd, TX);
  const int x0 = (it.tile % txs) * TX, y0 = (it.tile / txs) * TY;
  if constexpr (LOAD == LOAD_CP_ASYNC) {
    copy_box_async<T, TX + H, TY + 1>(st + G::S_VX, sd.f[0], sd, x0, y0, k, lane);
    copy_box_async<T, TX + H, TY + 1>(st + G::S_VY, sd.f[1], sd, x0 - H, y0 - 1, k, lane);
    copy_box_async<T, TX + H, TY + 1>(st + G::S_CS, sd.cs, sd, x0 - H, y0, k, lane);
    copy_box_async<T, TX + H, TY + 1>(st + G::S_RHO, sd.rho, sd, x0 - H, y0, k, lane);
    cp_async_arrive_noinc(bar);
  } else {
    const CUtensorMap *m = maps.stress;
    mbar_arrive_expect_tx(bar, G::S_TXA);
    tma_load_3d(st + G::S_VX, &m[0], x0, y0, k, bar);
    tma_load_3d(st + G::S_VY, &m[1], x0 - H, y0 - 1, k, bar);
    if constexpr (!G::COEF) {
      load_model<G::ONCE>(st + G::S_CS, &m[3], x0 - H, y0, k, bar);
      load_model<G::ONCE>(st + G::S_RHO, &m[4], x0 - H, y0, k, bar);
    }
  }
}

template <typename G, int LOAD, typename T>
__device__ __forceinline__ void stress_issue_b(const ShotDesc<T> &sd, const ShotMaps &maps, const Item &it, int k,
                                         unsigned char *st, uint64_t *bar, int lane) {
  constexpr int H = G::H, TX = G::TX, TY = G::TY;
  const int txs = tiles_x_of(sd, TX);
  const int x0 = (it.tile % txs) * TX, y0 = (it.tile / txs) * TY;
  if constexpr (LOAD == LOAD_CP_ASYNC) {
    copy_box_async<T, TX + H, TY + 1>(st + G::S_VZ, sd.f[2], sd, x0 - H, y0, k, lane);
    copy_box_async<T, TX, TY>(st + G::S_CP, sd.cp, sd, x0, y0, k, lane);
#pragma unroll
    for (int c = 0; c < 6; ++c) copy_box_async<T, TX, TY>(st + G::S_SIG + c * G::SC, sd.f[3 + c], sd, x0, y0, k, lane);
    cp_async_arrive_noinc(bar);
  } else {
    const CUtensorMap *m = maps.stress;
    mbar_arrive_expect_tx(bar, G::S_TXB);
    tma_load_3d(st + G::S_VZ, &m[2], x0 - H, y0, k, bar);
    if constexpr (G::COEF) {
#pragma unroll
      for (int c = 0; c < 5; ++c) tma_load_3d(st + G::S_CP + c * G::SC, &maps.coef[c], x0, y0, k, bar);
    } else {
      load_model<G::ONCE>(st + G::S_CP, &m[5], x0, y0, k, bar);
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) tma_load_3d(st + G::S_SIG + c * G::SC, &m[6 + c], x0, y0, k, bar);
  }
}

// The two parts of one velocity plane: szz, rho with its halo | the other
// stresses with the halos the divergence needs, and vx vy vz of the tile.
template <typename G, int LOAD, typename T>
__device__ __forceinline__ void velocity_issue_a(const ShotDesc<T> &sd, const ShotMaps &maps, const Item &it, int k,
                                         unsigned char *st, uint64_t *bar, int lane) {
  constexpr int H = G::H, TX = G::TX, TY = G::TY;
  const int txs = tiles_x_of(sd, TX);
  const int x0 = (it.tile % txs) * TX, y0 = (it.tile / txs) * TY;
  if constexpr (LOAD == LOAD_CP_ASYNC) {
    copy_box_async<T, TX, TY>(st + G::V_SZZ, sd.f[5], sd, x0, y0, k, lane);
    copy_box_async<T, TX + H, TY + 1>(st + G::V_RHO, sd.rho, sd, x0 - H, y0, k, lane);
    cp_async_arrive_noinc(bar);
  } else {
    const CUtensorMap *m = maps.vel;
    mbar_arrive_expect_tx(bar, G::V_TXA);
    tma_load_3d(st + G::V_SZZ, &m[2], x0, y0, k, bar);
    if constexpr (!G::COEF) load_model<G::ONCE>(st + G::V_RHO, &m[6], x0 - H, y0, k, bar);
  }
}

template <typename G, int LOAD, typename T>
__device__ __forceinline__ void velocity_issue_b(const ShotDesc<T> &sd, const ShotMaps &maps, const Item &it, int k,
                                         unsigned char *st, uint64_t *bar, int lane) {
  constexpr int H = G::H, TX = G::TX, TY = G::TY;
  const int txs = tiles_x_of(sd, TX);
  const int x0 = (it.tile % txs) * TX, y0 = (it.tile / txs) * TY;
  if constexpr (LOAD == LOAD_CP_ASYNC) {
    copy_box_async<T, TX + H, TY>(st + G::V_SXX, sd.f[3], sd, x0 - H, y0, k, lane);
    copy_box_async<T, TX, TY + 1>(st + G::V_SYY, sd.f[4], sd, x0, y0, k, lane);
    copy_box_async<T, TX + H, TY + 1>(st + G::V_SXY, sd.f[6], sd, x0, y0 - 1, k, lane);
    copy_box_async<T, TX + H, TY>(st + G::V_SXZ, sd.f[7], sd, x0, y0, k, lane);
    copy_box_async<T, TX, TY + 1>(st + G::V_SYZ, sd.f[8], sd, x0, y0 - 1, k, lane);
#pragma unroll
    for (int c = 0; c < 3; ++c) copy_box_async<T, TX, TY>(st + G::V_V + c * G::SC, sd.f[0 + c], sd, x0, y0, k, lane);
    cp_async_arrive_noinc(bar);
  } else {
    const CUtensorMap *m = maps.vel;
    mbar_arrive_expect_tx(bar, G::V_TXB);
    tma_load_3d(st + G::V_SXX, &m[0], x0 - H, y0, k, bar);
    tma_load_3d(st + G::V_SYY, &m[1], x0, y0, k, bar);
    tma_load_3d(st + G::V_SXY, &m[3], x0, y0 - 1, k, bar);
    tma_load_3d(st + G::V_SXZ, &m[4], x0, y0, k, bar);
    tma_load_3d(st + G::V_SYZ, &m[5], x0, y0 - 1, k, bar);
#pragma unroll
    for (int c = 0; c < 3; ++c) tma_load_3d(st + G::V_V + c * G::SC, &m[7 + c], x0, y0, k, bar);
    if constexpr (G::COEF) {
#pragma unroll
      for (int c = 0; c < 3; ++c) tma_load_3d(st + G::V_COEF + c * G::SC, &maps.coef[5 + c], x0, y0, k, bar);
    }
  }
}

// Waits for both parts of plane k (places a, b) and the first part of plane
// k + 1 (place ahead); a was already waited for as the previous plane's ahead
// unless k is the first plane of its work item.  False when a wait passed its
// limit; the caller returns.
template <typename R>
__device__ __forceinline__ bool wait_planes(const R &ring, const Place<R::NA> &a, const Place<R::NB> &b,
                                            const Place<R::NA> &ahead, bool first, unsigned long long wait_ns,
                                            unsigned *err, int lane) {
  // all three have usually completed: one vote
  bool ok = !first || mbar_try_wait(ring.full_a(a.s), a.parity);
  ok &= mbar_try_wait(ring.full_b(b.s), b.parity);
  ok &= mbar_try_wait(ring.full_a(ahead.s), ahead.parity);
  if (__all_sync(0xffffffffu, ok)) return true;
  ok = !first || mbar_wait_bounded(ring.full_a(a.s), a.parity, wait_ns);
  ok = ok && mbar_wait_bounded(ring.full_b(b.s), b.parity, wait_ns);
  ok = ok && mbar_wait_bounded(ring.full_a(ahead.s), ahead.parity, wait_ns);
  if (__any_sync(0xffffffffu, !ok)) {
    if (lane == 0) atomicOr(err, DEV_ERR_TIMEOUT);
    return false;
  }
  return true;
}

// Load that bypasses L1, for values another block wrote during this launch
// (the dataflow kernel's z-1 planes at the start of an item).
template <typename T, int N>
__device__ __forceinline__ void ld_vec_l2(const T *p, T (&o)[N]) {
  unpack<T, N>(__ldcg(reinterpret_cast<const typename VType<T, N>::V *>(p)), o);
}

// Consumers of the dataflow kernel: waits (bounded) until the producer has
// acquired the item's dependencies and arrived on its ready barrier.
__device__ __forceinline__ bool flow_ready(uint64_t *ready, uint32_t parity, unsigned long long wait_ns,
                                           unsigned *err, int lane) {
  const bool ok = mbar_wait_bounded(ready, parity, wait_ns);
  if (__any_sync(0xffffffffu, !ok)) {
    if (lane == 0) atomicOr(err, DEV_ERR_TIMEOUT);
    return false;
  }
  return true;
}

// C-PML memory variables of one thread's cells, one plane ahead.  A thread
// reads the variables of its own V cells only, so it copies them with
// cp.async into slots of shared memory that no other thread touches: no
// barrier is needed, only its own wait.  The copies of plane k+1 are issued
// once plane k's variables are used (their stores precede the copies in
// program order, so a slot is never refilled before it was read), and land
// while plane k's update, stores and the next stage wait run.  Loaded into
// registers at the top of the plane instead, their latency was exposed in
// every plane of every warp that crosses a layer (grids near the L2 size ran
// at 0.7-0.8 of their rate without layers), and 36 of them stayed live across
// the plane's update.  Built-in choices, 10 layer cells, Gcell-updates/s:
// 101^3 33.2 -> 36.5, 128^3 36.0 -> 40.7, 192^3 41.1 -> 42.2, 256^3 47.5 ->
// 48.7; the two kernels at 128^3 29.8 -> 33.5.
template <typename T, int NT, int V, bool ONCE>
struct PsiSlots {
  unsigned char *base;   // this thread's slot of variable 0
  static constexpr int B = V * (int)sizeof(T);
  static_assert(!ONCE || B == 16, "accesses with an L2 policy are 16 bytes");
  __device__ __forceinline__ PsiSlots(unsigned char *psi, int tid) : base(psi + tid * B) {}
  // variables 0..2 of `axis` from p, p + stride, p + 2 stride
  __device__ __forceinline__ void fetch(int axis, const T *p, long long stride) const {
#pragma unroll
    for (int v = 0; v < 3; ++v)
      if constexpr (ONCE) cp_async_16_first(base + (axis * 3 + v) * NT * B, p + v * stride);
      else cp_async_vec<B>(base + (axis * 3 + v) * NT * B, p + v * stride);
  }
  // d <- d / K + psi with psi <- b psi + a d, written back to p.  RAW: d
  // holds plain differences, to be multiplied by 1/h first.  AFIRST: which
  // of the two products is rounded before the fused add.
  template <bool RAW, bool AFIRST, typename A>
  __device__ __forceinline__ void apply(int axis, int v, T *p, const A &a, const A &b, const A &ik, T h,
                                        T (&d)[V]) const {
    T q[V], x[V], t[V];
    ld_vec(reinterpret_cast<const T *>(base + (axis * 3 + v) * NT * B), q);
    if constexpr (RAW) {
      mul_v(x, d, h);
    } else {
#pragma unroll
      for (int e = 0; e < V; ++e) x[e] = d[e];
    }
    if constexpr (AFIRST) {
      mul_v(t, b, q);
      fma_v(q, a, x, t);
    } else {
      mul_v(t, a, x);
      fma_v(q, b, q, t);
    }
    fma_v(d, x, ik, q);
    if constexpr (ONCE) st_first(p, q);
    else st_vec(p, q);
  }
};

// ----------------------------------------------------------- stress ----
// The stress half-step over one work item (the block's consumer warps).
// a, b: the places of the item's first plane in the rings.  FLOW (the dataflow
// kernel): the item's inputs were written by other blocks of the same
// launch; the caller has waited for the item's ready barrier, on which the
// producer arrives once it has acquired the item's dependencies, and the z-1
// plane, written during this launch, bypasses L1.  inject_tick (FLOW): the
// tick of the step before, whose explosive source is still to be added to
// the source cell's stresses (INT_MIN: none).
template <typename G, bool FLOW, typename T, typename R>
__device__ __forceinline__ bool stress_item(const ShotDesc<T> &sd, const Item &item, const R &ring, Place<R::NA> &a,
                                            Place<R::NB> &b, unsigned char *psi, unsigned *__restrict__ err,
                                            unsigned long long wait_ns, int tid, int inject_tick = INT_MIN) {
  constexpr int TX = G::TX, TY = G::TY;
  constexpr int V = G::VEC, H = G::H, WW = G::WW;
  const int lane = tid & 31;
  const int tx = tid % G::NTX;
  // (a thread without cells reads the last row's and has its row outside any grid)
  const bool spare = G::NT != G::NTX * TY && tid >= G::NTX * TY;
  const int ty = spare ? TY - 1 : tid / G::NTX;
  const int nx = sd.nx, ny = sd.ny, nz = sd.nz, px = sd.px;
  const int txs = (nx + TX - 1) / TX;
  const int x0 = (item.tile % txs) * TX, y0 = (item.tile / txs) * TY;
  const int xg = x0 + tx * V, y = spare ? INT_MAX / 2 : y0 + ty;
  const bool live = (xg < nx) && (y < ny);
  const T dt = sd.dt, idx = sd.idx, idy = sd.idy, idz = sd.idz;
  const long long plane = (long long)ny * px;
  const long long rowoff = (long long)y * px + xg;
  T *const f3 = sd.f[3], *const f4 = sd.f[4], *const f5 = sd.f[5];
  T *const f6 = sd.f[6], *const f7 = sd.f[7], *const f8 = sd.f[8];
  const int zl = sd.zl, zr = sd.zr;
  const T *const prof_z = sd.prof_z;
  T *const psi_x = sd.psi_x, *const psi_y = sd.psi_y, *const psi_z = sd.psi_z;
  const long long psx = sd.psx, psy = sd.psy, psz = sd.psz;
  const int xw = sd.xw, yw = sd.yw;
  // the thread whose cells hold an explosive source, in a step that follows
  // one with an injection
  const int inject = inject_tick == INT_MIN ? 0 : inject_tick - sd.tick0;
  const bool src_row = FLOW && inject >= 1 && inject <= sd.nstep && sd.src_kind == 1 && y == sd.src_j &&
                       sd.src_i >= xg && sd.src_i < xg + V;

  // z-1 neighbour of vz for the first plane of the run
  T vz_zm[V];
#pragma unroll
  for (int e = 0; e < V; ++e) vz_zm[e] = T(0);
  if (live && item.k0 > 0) {
    if constexpr (FLOW) ld_vec_l2(sd.f[2] + (long long)(item.k0 - 1) * plane + rowoff, vz_zm);
    else ld_vec_rw(sd.f[2] + (long long)(item.k0 - 1) * plane + rowoff, vz_zm);
  }

  // x-slab profile and placement (fixed over the run)
  const bool in_x = live && (xg < sd.xl || xg >= sd.xr);
  const int xs = xg < sd.xl ? xg : sd.xl + (xg - sd.xr);
  T ax[V], bx[V], ikx[V], axh[V], bxh[V], ikxh[V];
  if (in_x) {
    ld_vec_global(sd.prof_x + PR_A * px + xg, ax);
    ld_vec_global(sd.prof_x + PR_B * px + xg, bx);
    ld_vec_global(sd.prof_x + PR_IK * px + xg, ikx);
    ld_vec_global(sd.prof_x + PR_AH * px + xg, axh);
    ld_vec_global(sd.prof_x + PR_BH * px + xg, bxh);
    ld_vec_global(sd.prof_x + PR_IKH * px + xg, ikxh);
  } else {
#pragma unroll
    for (int e = 0; e < V; ++e) { ax[e] = axh[e] = T(0); bx[e] = bxh[e] = ikx[e] = ikxh[e] = T(1); }
  }
  const bool row_y = y < sd.yl || y >= sd.yr;   // the row lies in the y slab
  const bool in_y = live && row_y;
  const int ys = y < sd.yl ? y : sd.yl + (y - sd.yr);
  T ay = 0, by = 1, iky = 1, ayh = 0, byh = 1, ikyh = 1;
  if (in_y) {
    ay = sd.prof_y[PR_A * ny + y]; by = sd.prof_y[PR_B * ny + y]; iky = sd.prof_y[PR_IK * ny + y];
    ayh = sd.prof_y[PR_AH * ny + y]; byh = sd.prof_y[PR_BH * ny + y]; ikyh = sd.prof_y[PR_IKH * ny + y];
  }
  const int sb = (ty * WW + tx * V);       // vx box (origin x0, y0)
  const int sl = (ty * WW + H + tx * V);   // vz/cs/rho boxes (origin x0-H, y0)
  const int syl = sl + WW;                 // vy box (origin x0-H, y0-1): own row is ty+1
  const int sc = ty * TX + tx * V;         // centre boxes

  // the update ranges (simpelmodel.cpp:378-498) as per-cell bits, set once
  // per work item; the normal stresses also need k >= 1 (applied per plane)
  unsigned mbits = 0;
#pragma unroll
  for (int e = 0; e < V; ++e) {
    const int x = xg + e;
    mbits |= ((y >= 1) && (x <= nx - 2) ? 1u : 0u) << e;                   // normal: j >= 2, i <= NX-1
    mbits |= ((y <= ny - 2) && (x >= 1) && (x <= nx - 1) ? 1u : 0u) << (8 + e);   // sigma_xy
    mbits |= ((x >= 1) && (x <= nx - 1) ? 1u : 0u) << (16 + e);            // sigma_xz
    mbits |= ((y <= ny - 2) && (x <= nx - 1) ? 1u : 0u) << (24 + e);       // sigma_yz
  }
  const T dt8 = T(0.125) * dt;
  T *gx = psi_x + ((long long)item.k0 * ny + y) * xw + xs;
  T *gy = psi_y + ((long long)item.k0 * yw + ys) * px + xg;
  const long long dgx = (long long)ny * xw, dgy = (long long)yw * px;
  long long g = (long long)item.k0 * plane + rowoff;
  // the memory variables of the first plane; each plane then copies the next
  // one's as it has used its own
  const PsiSlots<T, G::NT, V, G::ONCE> slots(psi, tid);
  auto fetch_z = [&](int k) {
    if (live && (k < zl || k >= zr)) {
      const int zs = k < zl ? k : zl + (k - zr);
      slots.fetch(2, psi_z + PSI_S0 * psz + ((long long)zs * ny + y) * px + xg, psz);
    }
  };
  if (in_x) slots.fetch(0, gx + PSI_S0 * psx, psx);
  if (in_y) slots.fetch(1, gy + PSI_S0 * psy, psy);
  fetch_z(item.k0);
  for (int k = item.k0; k < item.k1; ++k, gx += dgx, gy += dgy, g += plane) {
    // z profile first: its latency overlaps the wait
    const bool plane_z = k < zl || k >= zr;       // the plane lies in the z slab
    const bool in_z = live && plane_z;
    T az = 0, bz = 1, ikz = 1, azh = 0, bzh = 1, ikzh = 1;
    if (in_z) {
      az = prof_z[PR_A * nz + k]; bz = prof_z[PR_B * nz + k]; ikz = prof_z[PR_IK * nz + k];
      azh = prof_z[PR_AH * nz + k]; bzh = prof_z[PR_BH * nz + k]; ikzh = prof_z[PR_IKH * nz + k];
    }

    Place<R::NA> ahead = a;
    ahead.next();
    if (!wait_planes(ring, a, b, ahead, k == item.k0, wait_ns, err, lane)) {
      cp_async_wait_all();   // (no copy outlives its thread)
      return false;
    }
    const unsigned char *cur = ring.a(a.s), *rest = ring.b(b.s), *nxt = ring.a(ahead.s);
    const T *bvx = reinterpret_cast<const T *>(cur + G::S_VX);
    const T *bvy = reinterpret_cast<const T *>(cur + G::S_VY);
    const T *bvz = reinterpret_cast<const T *>(rest + G::S_VZ);
    const T *bcs = reinterpret_cast<const T *>(cur + G::S_CS);
    const T *brho = reinterpret_cast<const T *>(cur + G::S_RHO);
    const T *bcp = reinterpret_cast<const T *>(rest + G::S_CP);
    const T *bsig = reinterpret_cast<const T *>(rest + G::S_SIG);
    constexpr int CS = G::SC / (int)sizeof(T);

    T vx_c[V], vx_yp[V], vx_zp[V], vy_c[V], vy_ym[V], vy_zp[V], vz_c[V], vz_yp[V];
    T cs_c[V], cs_yp[V], cs_zp[V], rho_c[V], rho_yp[V], rho_zp[V], cp_c[V];
    ld_vec(bvx + sb, vx_c);
    ld_vec(bvx + sb + WW, vx_yp);
    const T vx_e = bvx[sb + V];
    ld_vec(reinterpret_cast<const T *>(nxt + G::S_VX) + sb, vx_zp);
    ld_vec(bvy + syl, vy_c);
    ld_vec(bvy + syl - WW, vy_ym);
    const T vy_w = bvy[syl - 1];
    ld_vec(reinterpret_cast<const T *>(nxt + G::S_VY) + syl, vy_zp);
    ld_vec(bvz + sl, vz_c);
    ld_vec(bvz + sl + WW, vz_yp);
    const T vz_w = bvz[sl - 1];
    T cs_w = T(0), rho_w = T(0);
    T DT_l2m[V], DT_l[V], mu_xy[V], mu_xz[V], mu_yz[V];
    if constexpr (G::COEF) {
      ld_vec(bcp + 0 * CS + sc, DT_l2m);
      ld_vec(bcp + 1 * CS + sc, DT_l);
      ld_vec(bcp + 2 * CS + sc, mu_xy);
      ld_vec(bcp + 3 * CS + sc, mu_xz);
      ld_vec(bcp + 4 * CS + sc, mu_yz);
    } else {
      ld_vec(bcs + sl, cs_c);
      ld_vec(bcs + sl + WW, cs_yp);
      cs_w = bcs[sl - 1];
      ld_vec(reinterpret_cast<const T *>(nxt + G::S_CS) + sl, cs_zp);
      ld_vec(brho + sl, rho_c);
      ld_vec(brho + sl + WW, rho_yp);
      rho_w = brho[sl - 1];
      ld_vec(reinterpret_cast<const T *>(nxt + G::S_RHO) + sl, rho_zp);
      ld_vec(bcp + sc, cp_c);
    }
    T sxx[V], syy[V], szz[V], sxy[V], sxz[V], syz[V];
    ld_vec(bsig + 0 * CS + sc, sxx);
    ld_vec(bsig + 1 * CS + sc, syy);
    ld_vec(bsig + 2 * CS + sc, szz);
    ld_vec(bsig + 3 * CS + sc, sxy);
    ld_vec(bsig + 4 * CS + sc, sxz);
    ld_vec(bsig + 5 * CS + sc, syz);

    // explosive source of the step before, simpelmodel.cpp:607-622, as
    // explosive_kernel adds it: this item is the first to read the cell since
    if (FLOW && src_row && k == sd.src_k) {
      const T s = sd.stf[inject - 1];
      const int ns = sd.nstep + 1;
#pragma unroll
      for (int e = 0; e < V; ++e)
        if (xg + e == sd.src_i) {
          const long long gs = (long long)k * plane + rowoff + e;
          const T l2m = mul_rn(mul_rn(sd.rho[gs], sd.cp[gs]), sd.cp[gs]);
          sxx[e] = fma_rn(mul_rn(mul_rn(sd.expl_w[0], s), dt), l2m, sxx[e]);
          syy[e] = fma_rn(mul_rn(mul_rn(sd.expl_w[1], s), dt), l2m, syy[e]);
          szz[e] = fma_rn(mul_rn(mul_rn(sd.expl_w[2], s), dt), l2m, szz[e]);
          sd.src_trace[inject] = sxx[e];
          sd.src_trace[ns + inject] = syy[e];
          sd.src_trace[2 * ns + inject] = szz[e];
        }
    }

    // this warp no longer reads the plane's places (ahead still is, as the next plane)
    const bool last = (k == item.k1 - 1);
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(ring.empty_a(a.s));
      mbar_arrive(ring.empty_b(b.s));
      if (last) mbar_arrive(ring.empty_a(ahead.s));
    }

    // this plane's update masks: bit e of byte c = component c of cell e
    const unsigned mk = k >= 1 ? mbits : (mbits & 0xffffff00u);
    // The nine velocity derivatives.  Those along y and z that only enter a
    // sum stay plain differences D with a factor S (1/h, or 1 once the C-PML
    // term has been applied), so the sum is one fma either way.  Every
    // rounding is written out (fma_rn, mul_rn, add_rn), operand order
    // included: results are the same bits whatever the compiler contracts,
    // in every tile variant and schedule.
    T exx[V], eyx[V], ezx[V], eyy[V], exy[V], ezy[V], ezz[V], exz[V], eyz[V];
    {
      T n[V];
      east_of(n, vx_c, vx_e);
      sub_v(exx, n, vx_c);
      mul_v(exx, exx, idx);
      west_of(n, vy_c, vy_w);
      sub_v(eyx, vy_c, n);
      mul_v(eyx, eyx, idx);
      west_of(n, vz_c, vz_w);
      sub_v(ezx, vz_c, n);
      mul_v(ezx, ezx, idx);
      sub_v(eyy, vy_c, vy_ym);
      mul_v(eyy, eyy, idy);
      sub_v(exy, vx_yp, vx_c);   // D
      sub_v(ezy, vz_yp, vz_c);   // D
      sub_v(ezz, vz_c, vz_zm);
      mul_v(ezz, ezz, idz);
      sub_v(exz, vx_zp, vx_c);   // D
      sub_v(eyz, vy_zp, vy_c);   // D
#pragma unroll
      for (int e = 0; e < V; ++e) vz_zm[e] = vz_c[e];
    }
    // C-PML terms, only for the cells inside a slab (elsewhere a = 0 and
    // 1/K = 1 and the terms are exact no-ops).  Memory variables are updated
    // whether or not the cell's stress is: a cell outside the update ranges
    // never uses them.
    constexpr bool F32 = sizeof(T) == 4;
    T sy = idy, sz = idz;
    cp_async_wait_all();
    if (in_x) {
      slots.template apply<false, false>(0, 0, gx + PSI_S0 * psx, axh, bxh, ikxh, idx, exx);
      slots.template apply<false, false>(0, 1, gx + PSI_S1 * psx, ax, bx, ikx, idx, eyx);
      slots.template apply<false, false>(0, 2, gx + PSI_S2 * psx, ax, bx, ikx, idx, ezx);
      if (!last) slots.fetch(0, gx + PSI_S0 * psx + dgx, psx);
    }
    if (in_y) {
      slots.template apply<false, F32>(1, 0, gy + PSI_S0 * psy, ay, by, iky, idy, eyy);
      slots.template apply<true, F32>(1, 1, gy + PSI_S1 * psy, ayh, byh, ikyh, idy, exy);
      slots.template apply<true, F32>(1, 2, gy + PSI_S2 * psy, ayh, byh, ikyh, idy, ezy);
      if (!last) slots.fetch(1, gy + PSI_S0 * psy + dgy, psy);
      sy = T(1);
    }
    if (in_z) {
      const int zs = k < zl ? k : zl + (k - zr);
      T *gz = psi_z + ((long long)zs * ny + y) * px + xg;
      slots.template apply<false, F32>(2, 0, gz + PSI_S0 * psz, az, bz, ikz, idz, ezz);
      slots.template apply<true, F32>(2, 1, gz + PSI_S1 * psz, azh, bzh, ikzh, idz, exz);
      if (F32 && row_y) slots.template apply<true, true>(2, 2, gz + PSI_S2 * psz, azh, bzh, ikzh, idz, eyz);
      else slots.template apply<true, false>(2, 2, gz + PSI_S2 * psz, azh, bzh, ikzh, idz, eyz);
      sz = T(1);
    }
    if (!last) fetch_z(k + 1);

    // normal stresses, simpelmodel.cpp:378-413
    if constexpr (!G::COEF) dt_moduli(dt, cp_c, cs_c, rho_c, DT_l2m, DT_l);
    if (!F32) {
      normal_stress<true>(DT_l2m, DT_l, exx, eyy, ezz, sxx, mk);
      normal_stress<true>(DT_l2m, DT_l, eyy, exx, ezz, syy, mk);
      normal_stress<true>(DT_l2m, DT_l, ezz, exx, eyy, szz, mk);
    } else if (plane_z) {
      normal_stress<true>(DT_l2m, DT_l, exx, eyy, ezz, sxx, mk);
      normal_stress<true>(DT_l2m, DT_l, eyy, exx, ezz, syy, mk);
      normal_stress<false>(DT_l2m, DT_l, ezz, exx, eyy, szz, mk);
    } else if (row_y) {
      normal_stress<true>(DT_l2m, DT_l, exx, eyy, ezz, sxx, mk);
      normal_stress<false>(DT_l2m, DT_l, eyy, exx, ezz, syy, mk);
      normal_stress<true>(DT_l2m, DT_l, ezz, exx, eyy, szz, mk);
    } else {
      normal_stress<false>(DT_l2m, DT_l, exx, eyy, ezz, sxx, mk);
      normal_stress<true>(DT_l2m, DT_l, eyy, exx, ezz, syy, mk);
      normal_stress<true>(DT_l2m, DT_l, ezz, exx, eyy, szz, mk);
    }

    // the shear stresses: sigma_xy :416-442, sigma_xz :445-471 (z+1 of plane
    // nz-1 is the zero plane), sigma_yz :473-498
    {
      T cw[V], rw[V], t[V];
      if constexpr (!G::COEF) {
        west_of(cw, cs_c, cs_w);
        west_of(rw, rho_c, rho_w);
        dt_mu(mu_xy, dt8, cw, cs_yp, rw, rho_yp);
      }
      fma_v(t, exy, sy, eyx);
      fma_v(t, mu_xy, t, sxy);
      keep_masked(sxy, t, mk >> 8);
      if constexpr (!G::COEF) dt_mu(mu_xz, dt8, cw, cs_zp, rw, rho_zp);
      fma_v(t, exz, sz, ezx);
      fma_v(t, mu_xz, t, sxz);
      keep_masked(sxz, t, mk >> 16);
      if constexpr (!G::COEF) dt_mu(mu_yz, dt8, cs_yp, cs_zp, rho_yp, rho_zp);
      // (a derivative whose C-PML term was applied has S = 1, and its
      // product with S is exact)
      if (F32 ? row_y : !plane_z) {
        mul_v(t, ezy, sy);
        fma_v(t, eyz, sz, t);
      } else {
        mul_v(t, eyz, sz);
        fma_v(t, ezy, sy, t);
      }
      fma_v(t, mu_yz, t, syz);
      keep_masked(syz, t, mk >> 24);
    }

    if (live) {
      st_vec(f3 + g, sxx);
      st_vec(f4 + g, syy);
      st_vec(f5 + g, szz);
      st_vec(f6 + g, sxy);
      st_vec(f7 + g, sxz);
      st_vec(f8 + g, syz);
    }
    a = ahead;
    if (last) a.next();
    b.next();
  }
  return true;
}

// --------------------------------------------------------- velocity ----
// Writes the velocities of one plane's receivers rec[lo, end) (sorted by
// row, then column) that lie in this warp's cells.  The whole warp looks them
// up together: a 32-way search for the first receiver of its rows, then 32
// receivers a step, each lane taking its receiver's velocity from the lane
// that holds the cell.  (Every thread searching for its own cells' receivers
// costs a chain of dependent loads, one per halving and one per receiver, in
// every warp of the plane's tiles: 64^3 with 64 receivers 22.1 us a step
// that way, 20.6 this way and without receivers; 101^3 with 11, 29.6 and
// 28.7.)
template <int NTX, int TY, typename T, int V>
__device__ __forceinline__ void sample_receivers(const int4 *__restrict__ rec, int lo, int end, int x0, int y0,
                                                 int tid, const T (&vx)[V], const T (&vy)[V], const T (&vz)[V],
                                                 T *out, int nsamp) {
  const int lane = tid & 31, t0 = tid - lane;                // the warp's first thread
  const int ya = y0 + t0 / NTX, yb = y0 + min((t0 + 31) / NTX, TY - 1);   // its first and last row
  // the first receiver at or after (ya, x0) lies in [lo, hi]
  for (int hi = end; hi - lo > 32;) {
    const int step = (hi - lo + 31) / 32, q = lo + lane * step;
    bool before = false;
    if (q < hi) {
      const int4 r = rec[q];
      before = r.y < ya || (r.y == ya && r.x < x0);
    }
    const int c = __popc(__ballot_sync(0xffffffffu, before));   // (true on a prefix of the lanes)
    if (c == 0) break;
    hi = min(hi, lo + c * step);
    lo += (c - 1) * step + 1;
  }
  for (; lo < end; lo += 32) {
    int4 r = make_int4(x0, yb + 1, 0, 0);
    if (lo + lane < end) r = rec[lo + lane];
    const int col = r.x - x0, t = (r.y - y0) * NTX + col / V - t0;
    const bool mine = r.y >= ya && r.y <= yb && col >= 0 && col < NTX * V && t >= 0 && t < 32;
    if (__any_sync(0xffffffffu, mine)) {
      const int src = mine ? t : 0, e = mine ? col % V : 0;
      T rx = T(0), ry = T(0), rz = T(0);
#pragma unroll
      for (int c = 0; c < V; ++c) {
        const T a = __shfl_sync(0xffffffffu, vx[c], src), b = __shfl_sync(0xffffffffu, vy[c], src),
                d = __shfl_sync(0xffffffffu, vz[c], src);
        if (c == e) { rx = a; ry = b; rz = d; }
      }
      if (mine) {
        T *o = out + (long long)r.w * 3 * nsamp;
        o[0] = rx;
        o[nsamp] = ry;
        o[2 * nsamp] = rz;
      }
    }
    if (__any_sync(0xffffffffu, r.y > yb)) break;
  }
}

// The velocity half-step over one work item at step `tick` (see
// stress_item for a, b and FLOW), with the receivers and the force source.
template <typename G, bool FLOW, typename T, typename R>
__device__ __forceinline__ bool velocity_item(const ShotDesc<T> &sd, const Item &item, int tick, const R &ring,
                                              Place<R::NA> &a, Place<R::NB> &b, unsigned char *psi,
                                              unsigned *__restrict__ err, unsigned long long wait_ns, int tid) {
  constexpr int TX = G::TX, TY = G::TY;
  constexpr int V = G::VEC, H = G::H, WW = G::WW;
  constexpr int CS = G::SC / (int)sizeof(T);
  const int lane = tid & 31;
  const int tx = tid % G::NTX;
  // (a thread without cells reads the last row's and has its row outside any grid)
  const bool spare = G::NT != G::NTX * TY && tid >= G::NTX * TY;
  const int ty = spare ? TY - 1 : tid / G::NTX;
  const int nx = sd.nx, ny = sd.ny, nz = sd.nz, px = sd.px;
  const int txs = (nx + TX - 1) / TX;
  const int x0 = (item.tile % txs) * TX, y0 = (item.tile / txs) * TY;
  const int xg = x0 + tx * V, y = spare ? INT_MAX / 2 : y0 + ty;
  const bool live = (xg < nx) && (y < ny);
  const T dt = sd.dt, idx = sd.idx, idy = sd.idy, idz = sd.idz;
  const long long plane = (long long)ny * px;
  const long long rowoff = (long long)y * px + xg;
  T *const f0 = sd.f[0], *const f1 = sd.f[1], *const f2 = sd.f[2];
  const int zl = sd.zl, zr = sd.zr;
  const T *const prof_z = sd.prof_z;
  T *const psi_x = sd.psi_x, *const psi_y = sd.psi_y, *const psi_z = sd.psi_z;
  const long long psx = sd.psx, psy = sd.psy, psz = sd.psz;
  const int xw = sd.xw, yw = sd.yw;
  const int it_step = tick - sd.tick0;
  const bool sample = (it_step % sd.sampgat == 0) && (it_step / sd.sampgat <= sd.nsamp) && it_step > 0;
  const int samp = it_step / sd.sampgat - 1;
  const int *const rec_plane = sd.rec_plane;
  // receivers exist in this item's planes at all (most items have none)
  const bool item_rec = sample && rec_plane[item.k1] > rec_plane[item.k0];
  const bool src_row = sd.src_kind == 0 && y == sd.src_j && sd.src_i >= xg && sd.src_i < xg + V &&
                       it_step >= 1 && it_step <= sd.nstep;

  T sxz_zm[V], syz_zm[V];
#pragma unroll
  for (int e = 0; e < V; ++e) sxz_zm[e] = syz_zm[e] = T(0);
  if (live && item.k0 > 0) {
    const long long g = (long long)(item.k0 - 1) * plane + rowoff;
    if constexpr (FLOW) {
      ld_vec_l2(sd.f[7] + g, sxz_zm);
      ld_vec_l2(sd.f[8] + g, syz_zm);
    } else {
      ld_vec_rw(sd.f[7] + g, sxz_zm);
      ld_vec_rw(sd.f[8] + g, syz_zm);
    }
  }

  const bool in_x = live && (xg < sd.xl || xg >= sd.xr);
  const int xs = xg < sd.xl ? xg : sd.xl + (xg - sd.xr);
  T ax[V], bx[V], ikx[V], axh[V], bxh[V], ikxh[V];
  if (in_x) {
    ld_vec_global(sd.prof_x + PR_A * px + xg, ax);
    ld_vec_global(sd.prof_x + PR_B * px + xg, bx);
    ld_vec_global(sd.prof_x + PR_IK * px + xg, ikx);
    ld_vec_global(sd.prof_x + PR_AH * px + xg, axh);
    ld_vec_global(sd.prof_x + PR_BH * px + xg, bxh);
    ld_vec_global(sd.prof_x + PR_IKH * px + xg, ikxh);
  } else {
#pragma unroll
    for (int e = 0; e < V; ++e) { ax[e] = axh[e] = T(0); bx[e] = bxh[e] = ikx[e] = ikxh[e] = T(1); }
  }
  const bool row_y = y < sd.yl || y >= sd.yr;   // the row lies in the y slab
  const bool in_y = live && row_y;
  const int ys = y < sd.yl ? y : sd.yl + (y - sd.yr);
  T ay = 0, by = 1, iky = 1, ayh = 0, byh = 1, ikyh = 1;
  if (in_y) {
    ay = sd.prof_y[PR_A * ny + y]; by = sd.prof_y[PR_B * ny + y]; iky = sd.prof_y[PR_IK * ny + y];
    ayh = sd.prof_y[PR_AH * ny + y]; byh = sd.prof_y[PR_BH * ny + y]; ikyh = sd.prof_y[PR_IKH * ny + y];
  }
  const int sl0 = ty * WW + H + tx * V;     // sxx box (origin x0-H, y0)
  const int sr0 = ty * WW + tx * V;         // sxz box (origin x0, y0)
  const int sr1 = (ty + 1) * WW + tx * V;   // sxy box (origin x0, y0-1): own row ty+1
  const int sc = ty * TX + tx * V;          // syy box (origin x0, y0) / centre boxes
  const int sc1 = (ty + 1) * TX + tx * V;   // syz box (origin x0, y0-1)

  // the update ranges (simpelmodel.cpp:502-590) as per-cell bits, set once
  // per work item; the plane conditions are applied per plane
  unsigned mbits = 0;
#pragma unroll
  for (int e = 0; e < V; ++e) {
    const int x = xg + e;
    mbits |= ((y >= 1) && (x >= 1) && (x <= nx - 1) ? 1u : 0u) << e;        // vx (with k >= 1)
    mbits |= ((y <= ny - 2) && (x <= nx - 2) ? 1u : 0u) << (8 + e);         // vy (with k >= 1)
    mbits |= ((y >= 1) && (x <= nx - 2) ? 1u : 0u) << (16 + e);             // vz (with k <= nz-2)
  }
  T *gx = psi_x + ((long long)item.k0 * ny + y) * xw + xs;
  T *gy = psi_y + ((long long)item.k0 * yw + ys) * px + xg;
  const long long dgx = (long long)ny * xw, dgy = (long long)yw * px;
  long long g = (long long)item.k0 * plane + rowoff;
  // the memory variables of the first plane; each plane then copies the next
  // one's as it has used its own
  const PsiSlots<T, G::NT, V, G::ONCE> slots(psi, tid);
  auto fetch_z = [&](int k) {
    if (live && (k < zl || k >= zr)) {
      const int zs = k < zl ? k : zl + (k - zr);
      slots.fetch(2, psi_z + PSI_V0 * psz + ((long long)zs * ny + y) * px + xg, psz);
    }
  };
  if (in_x) slots.fetch(0, gx + PSI_V0 * psx, psx);
  if (in_y) slots.fetch(1, gy + PSI_V0 * psy, psy);
  fetch_z(item.k0);
  for (int k = item.k0; k < item.k1; ++k, gx += dgx, gy += dgy, g += plane) {
    const bool plane_z = k < zl || k >= zr;       // the plane lies in the z slab
    const bool in_z = live && plane_z;
    T az = 0, bz = 1, ikz = 1, azh = 0, bzh = 1, ikzh = 1;
    if (in_z) {
      az = prof_z[PR_A * nz + k]; bz = prof_z[PR_B * nz + k]; ikz = prof_z[PR_IK * nz + k];
      azh = prof_z[PR_AH * nz + k]; bzh = prof_z[PR_BH * nz + k]; ikzh = prof_z[PR_IKH * nz + k];
    }

    int rlo = 0, rhi = 0;   // receivers of this plane
    if (item_rec) {
      rlo = rec_plane[k];
      rhi = rec_plane[k + 1];
    }

    Place<R::NA> ahead = a;
    ahead.next();
    if (!wait_planes(ring, a, b, ahead, k == item.k0, wait_ns, err, lane)) {
      cp_async_wait_all();   // (no copy outlives its thread)
      return false;
    }
    const unsigned char *cur = ring.a(a.s), *rest = ring.b(b.s), *nxt = ring.a(ahead.s);
    const T *bsxx = reinterpret_cast<const T *>(rest + G::V_SXX);
    const T *bsyy = reinterpret_cast<const T *>(rest + G::V_SYY);
    const T *bszz = reinterpret_cast<const T *>(cur + G::V_SZZ);
    const T *bsxy = reinterpret_cast<const T *>(rest + G::V_SXY);
    const T *bsxz = reinterpret_cast<const T *>(rest + G::V_SXZ);
    const T *bsyz = reinterpret_cast<const T *>(rest + G::V_SYZ);
    const T *brho = reinterpret_cast<const T *>(cur + G::V_RHO);
    const T *bv = reinterpret_cast<const T *>(rest + G::V_V);

    T sxx_c[V], syy_c[V], syy_yp[V], szz_c[V], szz_zp[V], sxy_c[V], sxy_ym[V], sxz_c[V];
    T syz_c[V], syz_ym[V], rho_c[V], rho_yp[V], rho_zp[V], vx[V], vy[V], vz[V];
    ld_vec(bsxx + sl0, sxx_c);
    const T sxx_w = bsxx[sl0 - 1];
    ld_vec(bsyy + sc, syy_c);
    ld_vec(bsyy + sc + TX, syy_yp);
    ld_vec(bszz + sc, szz_c);
    ld_vec(reinterpret_cast<const T *>(nxt + G::V_SZZ) + sc, szz_zp);
    ld_vec(bsxy + sr1, sxy_c);
    ld_vec(bsxy + sr1 - WW, sxy_ym);
    const T sxy_e = bsxy[sr1 + V];
    ld_vec(bsxz + sr0, sxz_c);
    const T sxz_e = bsxz[sr0 + V];
    ld_vec(bsyz + sc1, syz_c);
    ld_vec(bsyz + sc1 - TX, syz_ym);
    T rho_w = T(0);
    T bx_[V], by_[V], bz_[V];   // dt / rho of the three components
    if constexpr (G::COEF) {
      const T *bco = reinterpret_cast<const T *>(rest + G::V_COEF);
      ld_vec(bco + 0 * CS + sc, bx_);
      ld_vec(bco + 1 * CS + sc, by_);
      ld_vec(bco + 2 * CS + sc, bz_);
    } else {
      ld_vec(brho + sl0, rho_c);
      ld_vec(brho + sl0 + WW, rho_yp);
      rho_w = brho[sl0 - 1];
      ld_vec(reinterpret_cast<const T *>(nxt + G::V_RHO) + sl0, rho_zp);
    }
    ld_vec(bv + 0 * CS + sc, vx);
    ld_vec(bv + 1 * CS + sc, vy);
    ld_vec(bv + 2 * CS + sc, vz);

    const bool last = (k == item.k1 - 1);
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(ring.empty_a(a.s));
      mbar_arrive(ring.empty_b(b.s));
      if (last) mbar_arrive(ring.empty_a(ahead.s));
    }

    // this plane's update masks: bit e of byte c = component c of cell e
    const unsigned mk = (k >= 1 ? (mbits & 0x00ffffu) : 0u) | (k <= nz - 2 ? (mbits & 0xff0000u) : 0u);
    // the nine stress derivatives (x1: of vx's update along x, and so on);
    // y and z as plain differences with a factor, roundings written out (as
    // in the stress half-step)
    T x1[V], x2[V], x3[V], y1[V], y2[V], y3[V], z1[V], z2[V], z3[V];
    {
      T n[V];
      west_of(n, sxx_c, sxx_w);
      sub_v(x1, sxx_c, n);
      mul_v(x1, x1, idx);
      sub_v(x2, sxy_c, sxy_ym);
      sub_v(x3, sxz_c, sxz_zm);
      east_of(n, sxy_c, sxy_e);
      sub_v(y1, n, sxy_c);
      mul_v(y1, y1, idx);
      sub_v(y2, syy_yp, syy_c);
      sub_v(y3, syz_c, syz_zm);
      east_of(n, sxz_c, sxz_e);
      sub_v(z1, n, sxz_c);
      mul_v(z1, z1, idx);
      sub_v(z2, syz_c, syz_ym);
      sub_v(z3, szz_zp, szz_c);
#pragma unroll
      for (int e = 0; e < V; ++e) {
        sxz_zm[e] = sxz_c[e];
        syz_zm[e] = syz_c[e];
      }
    }
    // C-PML terms only inside the slabs; memory variables updated whether or
    // not the cell's velocity is (as in the stress half-step)
    constexpr bool F32 = sizeof(T) == 4;
    T sy = idy, sz = idz;
    cp_async_wait_all();
    if (in_x) {
      slots.template apply<false, false>(0, 0, gx + PSI_V0 * psx, ax, bx, ikx, idx, x1);
      slots.template apply<false, false>(0, 1, gx + PSI_V1 * psx, axh, bxh, ikxh, idx, y1);
      slots.template apply<false, false>(0, 2, gx + PSI_V2 * psx, axh, bxh, ikxh, idx, z1);
      if (!last) slots.fetch(0, gx + PSI_V0 * psx + dgx, psx);
    }
    if (in_y) {
      slots.template apply<true, F32>(1, 0, gy + PSI_V0 * psy, ay, by, iky, idy, x2);
      slots.template apply<true, F32>(1, 1, gy + PSI_V1 * psy, ayh, byh, ikyh, idy, y2);
      slots.template apply<true, F32>(1, 2, gy + PSI_V2 * psy, ay, by, iky, idy, z2);
      if (!last) slots.fetch(1, gy + PSI_V0 * psy + dgy, psy);
      sy = T(1);
    }
    if (in_z) {
      const int zs = k < zl ? k : zl + (k - zr);
      T *gz = psi_z + ((long long)zs * ny + y) * px + xg;
      slots.template apply<true, F32>(2, 0, gz + PSI_V0 * psz, az, bz, ikz, idz, x3);
      slots.template apply<true, F32>(2, 1, gz + PSI_V1 * psz, az, bz, ikz, idz, y3);
      slots.template apply<true, F32>(2, 2, gz + PSI_V2 * psz, azh, bzh, ikzh, idz, z3);
      sz = T(1);
    }
    if (!last) fetch_z(k + 1);

    // simpelmodel.cpp:502-530, :532-559, :563-590
    T rw[V];
    if constexpr (!G::COEF) {
      west_of(rw, rho_c, rho_w);
      dt_over_rho(bx_, dt, rho_c, rw, mk);
    }
    velocity_update(sy, sz, bx_, x1, x2, x3, vx, mk);
    if constexpr (!G::COEF) dt_over_rho(by_, dt, rho_c, rho_yp, mk >> 8);
    velocity_update(sy, sz, by_, y1, y2, y3, vy, mk >> 8);
    if constexpr (!G::COEF) dt_over_rho(bz_, dt, rho_c, rho_zp, mk >> 16);
    velocity_update(sy, sz, bz_, z1, z2, z3, vz, mk >> 16);

    // receivers in this warp's cells (velocity after the update, :593-602)
    if (rlo < rhi)
      sample_receivers<G::NTX, TY>(sd.rec_sorted, rlo, rhi, x0, y0, tid, vx, vy, vz, sd.seis + samp, sd.nsamp);
    if (live) {
      // force source after the update (cudazerocopy.cu:451-453)
      if (src_row && k == sd.src_k) {
        const T s = sd.stf[it_step - 1];
        const int se = sd.src_i - xg;
        // the averaged densities at the source cell, from the model itself
        // (out-of-grid neighbours are zero, as in the stage boxes)
        const long long gs = (long long)k * plane + rowoff + se;
        const T r0 = sd.rho[gs];
        const T rxs = (r0 + (sd.src_i >= 1 ? sd.rho[gs - 1] : T(0))) / T(2);
        const T rys = (r0 + (y + 1 < ny ? sd.rho[gs + px] : T(0))) / T(2);
        const T rzs = (r0 + (k + 1 < nz ? sd.rho[gs + plane] : T(0))) / T(2);
        const bool wx = sd.src_w[0] != T(0), wy = sd.src_w[1] != T(0), wz = sd.src_w[2] != T(0);
        const T fx = sd.src_w[0] * s, fy = sd.src_w[1] * s, fz = sd.src_w[2] * s;
        T tvx = vx[0], tvy = vy[0], tvz = vz[0];
#pragma unroll
        for (int c = 0; c < V; ++c) {
          const bool hit = (c == se);
          vx[c] = (hit && wx) ? vx[c] + fx * dt / rxs : vx[c];
          vy[c] = (hit && wy) ? vy[c] + fy * dt / rys : vy[c];
          vz[c] = (hit && wz) ? vz[c] + fz * dt / rzs : vz[c];
          tvx = hit ? vx[c] : tvx;
          tvy = hit ? vy[c] : tvy;
          tvz = hit ? vz[c] : tvz;
        }
        // source-point trace: the velocity after the injection
        const int ns = sd.nstep + 1;
        sd.src_trace[it_step] = tvx;
        sd.src_trace[ns + it_step] = tvy;
        sd.src_trace[2 * ns + it_step] = tvz;
      }
      st_vec(f0 + g, vx);
      st_vec(f1 + g, vy);
      st_vec(f2 + g, vz);
    }
    a = ahead;
    if (last) a.next();
    b.next();
  }
  return true;
}

// ------------------------------------------------- half-step kernels ----
// Barrier set-up shared by the kernels: full expects the producer's one
// arrival plus the part's bytes (TMA) or one arrival per lane (cp.async);
// empty one arrival per consumer warp.
template <int NCW, int LOAD, typename R>
__device__ __forceinline__ void init_ring(const R &ring) {
  if (threadIdx.x == 0) {
    for (int s = 0; s < R::NA + R::NB; ++s) {
      mbar_init(ring.bars() + s, LOAD == LOAD_TMA ? 1 : 32);
      mbar_init(ring.bars() + R::NA + R::NB + s, NCW);
    }
    fence_mbar_init();
  }
  __syncthreads();
}

// The loading warp of the half-step kernels: the block's items in turn.
template <bool ASYNC, typename R, typename IssueA, typename IssueB, typename Prefetch>
__device__ __forceinline__ void produce(const Item *__restrict__ items, int2 range, const R &ring, IssueA issue_a,
                                        IssueB issue_b, Prefetch &prefetch, unsigned *__restrict__ err, int ctl,
                                        int lane) {
  if (ctl & CTL_WITHHOLD_LOADS) return;  // test mode: no place is ever filled
  Loads<R> ld;
  bool ok = true;
  for (int ii = range.x; ii < range.y && ok; ++ii) {
    const Item it = items[ii];
    prefetch.begin(it);
    ok = produce_item<ASYNC>(
        it, ring, ld, [&](int k, unsigned char *st, uint64_t *bar) { issue_a(it, k, st, bar, lane); },
        [&](int k, unsigned char *st, uint64_t *bar) { issue_b(it, k, st, bar, lane); }, prefetch, lane);
  }
  produce_drain<ASYNC>(ring, ld, ok, err, lane);
}

// Rings of the half-step kernels, and their shared memory: the rings, the
// memory-variable slots behind them.
template <typename G> using StressRing = Ring<G::NS, G::places_b(G::S_A, G::S_B, 128), G::S_A, G::S_B>;
template <typename G> using VelocityRing = Ring<G::NS, G::places_b(G::V_A, G::V_B, 128), G::V_A, G::V_B>;
template <typename G, typename R> constexpr int kPsiOffset = (R::BYTES + 127) & ~127;
template <typename G, typename R> constexpr int kKernelSmem = kPsiOffset<G, R> + G::PSI_BYTES;

// (tick and dtick are unused by the stress half-step; the parameter list is
// shared with the velocity kernel so both launch from one argument array)
template <typename T, int TX, int TY, int NS, int CPT, int MB, int LOAD>
__global__ void __launch_bounds__(Geo<T, TX, TY, NS, CPT, MB>::THREADS, Geo<T, TX, TY, NS, CPT, MB>::MINB)
    stress_kernel(const ShotDesc<T> *__restrict__ shots, const ShotMaps *__restrict__ maps,
                  const Item *__restrict__ items, const int2 *__restrict__ ranges, int tick,
                  const int *__restrict__ dtick, unsigned *__restrict__ err, int ctl) {
  using G = Geo<T, TX, TY, NS, CPT, MB>;
  using R = StressRing<G>;
  extern __shared__ __align__(1024) unsigned char smem[];
  const R ring{smem};

  const int tid = threadIdx.x;
  const int2 range = ranges[blockIdx.x];
  if (range.x >= range.y) return;
  init_ring<G::NCW, LOAD>(ring);

  if (tid >= G::NT) {  // producer warp
    if constexpr (G::SPLIT) fewer_registers<G::LOADER_REGS>();
    const int lane = tid - G::NT;
    if (lane >= 32) return;   // (the rest of its group)
    auto issue_a = [&](const Item &it, int k, unsigned char *st, uint64_t *bar, int l) {
      stress_issue_a<G, LOAD>(shots[it.shot], maps[it.shot], it, k, st, bar, l);
    };
    auto issue_b = [&](const Item &it, int k, unsigned char *st, uint64_t *bar, int l) {
      stress_issue_b<G, LOAD>(shots[it.shot], maps[it.shot], it, k, st, bar, l);
    };
    ItemPrefetch<T, TX, TY> prefetch{{}, shots, lane, ctl, PSI_S0};
    produce<LOAD == LOAD_CP_ASYNC>(items, range, ring, issue_a, issue_b, prefetch, err, ctl, lane);
    return;
  }
  if constexpr (G::SPLIT) more_registers<G::CONSUMER_REGS>();

  const unsigned long long wait_ns = (ctl & CTL_WITHHOLD_LOADS) ? kTestWaitLimitNs : kWaitLimitNs;
  Place<R::NA> a;
  Place<R::NB> b;
  for (int ii = range.x; ii < range.y; ++ii) {
    const Item item = items[ii];
    if (!stress_item<G, false>(shots[item.shot], item, ring, a, b, smem + kPsiOffset<G, R>, err, wait_ns, tid))
      return;
  }
}

template <typename T, int TX, int TY, int NS, int CPT, int MB, int LOAD>
__global__ void __launch_bounds__(Geo<T, TX, TY, NS, CPT, MB>::THREADS, Geo<T, TX, TY, NS, CPT, MB>::MINB)
    velocity_kernel(const ShotDesc<T> *__restrict__ shots, const ShotMaps *__restrict__ maps,
                    const Item *__restrict__ items, const int2 *__restrict__ ranges, int tick,
                    const int *__restrict__ dtick, unsigned *__restrict__ err, int ctl) {
  using G = Geo<T, TX, TY, NS, CPT, MB>;
  using R = VelocityRing<G>;
  extern __shared__ __align__(1024) unsigned char smem[];
  const R ring{smem};

  const int tid = threadIdx.x;
  const int2 range = ranges[blockIdx.x];
  if (range.x >= range.y) return;
  init_ring<G::NCW, LOAD>(ring);

  if (tid >= G::NT) {  // producer warp
    if constexpr (G::SPLIT) fewer_registers<G::LOADER_REGS>();
    const int lane = tid - G::NT;
    if (lane >= 32) return;   // (the rest of its group)
    auto issue_a = [&](const Item &it, int k, unsigned char *st, uint64_t *bar, int l) {
      velocity_issue_a<G, LOAD>(shots[it.shot], maps[it.shot], it, k, st, bar, l);
    };
    auto issue_b = [&](const Item &it, int k, unsigned char *st, uint64_t *bar, int l) {
      velocity_issue_b<G, LOAD>(shots[it.shot], maps[it.shot], it, k, st, bar, l);
    };
    ItemPrefetch<T, TX, TY> prefetch{{}, shots, lane, ctl, PSI_V0};
    produce<LOAD == LOAD_CP_ASYNC>(items, range, ring, issue_a, issue_b, prefetch, err, ctl, lane);
    return;
  }
  if constexpr (G::SPLIT) more_registers<G::CONSUMER_REGS>();

  const unsigned long long wait_ns = (ctl & CTL_WITHHOLD_LOADS) ? kTestWaitLimitNs : kWaitLimitNs;
  // step counter: an argument for direct launches, device memory plus an
  // offset inside a replayable CUDA graph
  if (dtick) tick += *dtick;
  Place<R::NA> a;
  Place<R::NB> b;
  for (int ii = range.x; ii < range.y; ++ii) {
    const Item item = items[ii];
    if (!velocity_item<G, false>(shots[item.shot], item, tick, ring, a, b, smem + kPsiOffset<G, R>, err, wait_ns,
                                 tid))
      return;
  }
}

// ------------------------------------------------- dataflow kernel ----
// Many time steps in one persistent launch.  The work is a list of items,
// each the stress or the velocity half-step of one (shot, x-y tile,
// z-chunk) at one of list_steps steps; a launch of nsteps steps walks the
// list again for every further list_steps steps (the item of list step s
// in pass p runs step p * list_steps + s; items of steps >= nsteps are
// skipped, so one list serves shorter launches).  A block takes the next
// place whenever its loading warp is done with an item (an atomic counter,
// read one item ahead), or, without a counter, places b, b + G, ... (G
// blocks, all resident: the launch is cooperative); either way a block's
// places ascend and every earlier place is taken.  The loading warp passes
// the item and a copy of its shot's descriptor to the consumers in shared
// memory: read from global memory, both miss L1 at every item, since each
// acquire of the counters empties it.  An explosive source acts on the
// stresses after a step: the next step's stress item adds it as it reads the
// cell, and explosive_kernel adds the last step's after the launch.  Chunk j
// of a shot
// covers planes [jC, (j+1)C) for stress and the same range shifted down by
// one plane for velocity, so that
//   stress (j, tile, step r)   reads v written by velocity (j and j+1) of
//                              step r-1 on the tile and its four
//                              neighbours, and overwrites the stresses
//                              those items read;
//   velocity (j, tile, step r) reads the stresses of stress (j-1 and j) of
//                              step r on the tile and its neighbours.
// Each item, before its loads, waits for those items' completion counters
// (flags[kind][chunk][tile], NCW added once an item is written: NCW (r + 1)
// once step r is done); the host orders the list so that every dependency
// comes earlier (checked there), so the waits always end.  The host places
// each item soon after the items it waits for (and, with overlapping
// steps, lets a step start where the previous one is done): a velocity
// chunk runs right after the stresses it reads were
// written, while they are still in L2.  Results are bit-identical to the
// two half-step kernels.  Memory ordering: consumer warps write, fence the
// async proxy (the TMA of the reading block), __syncwarp, and arrive (CTA
// scope) on a shared per-item count; the last warp releases the item's
// counter at gpu scope; the producer's lanes acquire the counters, fence
// the async proxy and meet (__syncwarp); lane 0 arrives on the item's
// ready barrier and then issues its loads; consumers read global
// memory for the item only after that barrier.  Every wait is bounded: a wait that passes its limit
// sets DEV_ERR_TIMEOUT and the block stops.
// RB ready barriers: the producer is at most NA loads ahead of the slowest
// consumer warp and every item takes at least two of them, so it never gets
// RB items ahead (a barrier is re-armed only after every warp passed it).
template <typename G_, typename T, int NS>
struct Flow {
  using G = G_;
  static constexpr int A = G::S_A > G::V_A ? G::S_A : G::V_A, B = G::S_B > G::V_B ? G::S_B : G::V_B;
  static constexpr int RB = 8;
  static_assert(RB >= NS / 2 + 2, "ready barriers for the items in flight");
  // per item in flight: the item (kind < 0: the list is done) and a copy of
  // its shot's descriptor
  struct alignas(16) Slot {
    FlowItem fi;
    ShotDesc<T> sd;
  };
  static_assert(sizeof(ShotDesc<T>) % 16 == 0 && sizeof(FlowItem) % 16 == 0, "descriptors are copied 16 bytes at a time");
  using R = Ring<NS, G::places_b(A, B, RB * ((int)sizeof(Slot) + 12) + 128), A, B>;
  static constexpr int READY = R::BYTES;
  static constexpr int SLOTS = (READY + 8 * RB + 4 * RB + 15) & ~15;
  static constexpr int PSI = (SLOTS + RB * (int)sizeof(Slot) + 15) & ~15;   // memory-variable slots
  static constexpr int SMEM = PSI + G::PSI_BYTES;
  static_assert(SMEM <= G::MAX_SMEM, "shared memory of one block");
};

__device__ __forceinline__ int ld_acquire_gpu(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void red_release_gpu_add(int *p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// CTA-scope acquire-release add on a shared-memory counter; returns the old value.
__device__ __forceinline__ int atom_acq_rel_cta_add(int *p, int v) {
  int old;
  asm volatile("atom.acq_rel.cta.shared::cta.add.s32 %0, [%1], %2;" : "=r"(old) : "r"(smem_u32(p)), "r"(v) : "memory");
  return old;
}

// The producer warp: waits until every counter this item depends on has
// reached its target.  Each of the (up to ten) counters is read by a lane of
// its own, so a satisfied item costs one L2 round trip.  (Acquiring loads;
// relaxed ones with a gpu-scope fence behind them ran 64^3 at 19.5 against
// 20.3 Gcell-updates/s, 101^3 at 37.8 against 38.3.)
template <typename T>
__device__ __forceinline__ bool flow_wait_deps(const ShotDesc<T> &sd, const FlowItem &fi, int txs, int tys, int ncw,
                                               unsigned long long wait_ns, int lane) {
  const int ntiles = txs * tys;
  const int tile = fi.it.tile, tx = tile % txs, ty = tile / txs;
  // stress: velocity of the previous step, chunks j and j+1; velocity: stress
  // of this step, chunks j and j-1
  const int target = ncw * (fi.kind == 0 ? fi.step : fi.step + 1);
  if (target <= 0) return true;
  const int q = lane >> 1;   // 0: the tile itself, 1..4: its neighbours
  const int x = tx + (q == 2) - (q == 1), y = ty + (q == 4) - (q == 3);
  const int c = fi.chunk + ((lane & 1) ? (fi.kind == 0 ? 1 : -1) : 0);
  const bool mine = lane < 10 && x >= 0 && x < txs && y >= 0 && y < tys && c >= 0 && c < sd.flow_chunks;
  const int *p = sd.flow_flags + ((fi.kind == 0 ? (size_t)sd.flow_chunks : 0) + (mine ? c : 0)) * ntiles +
                 (mine ? y * txs + x : 0);
  unsigned long long t0 = 0;
  while (!__all_sync(0xffffffffu, !mine || ld_acquire_gpu(p) >= target)) {
    const unsigned long long t = globaltimer_ns();
    if (t0 == 0) t0 = t;
    else if (__any_sync(0xffffffffu, t - t0 > wait_ns)) return false;
  }
  fence_proxy_async_global();
  __syncwarp();
  return true;
}

template <typename T, int TX, int TY, int NS, int CPT, int MB, bool COEF, bool ONCE>
__global__ void __launch_bounds__(Geo<T, TX, TY, NS, CPT, MB>::THREADS, Geo<T, TX, TY, NS, CPT, MB>::MINB)
    flow_kernel(const ShotDesc<T> *__restrict__ shots, const ShotMaps *__restrict__ maps,
                const FlowItem *__restrict__ items, int nitems, int list_steps, int nsteps, int tick,
                const int *__restrict__ dtick, unsigned *__restrict__ err, int ctl, int *__restrict__ claim) {
  using G = Geo<T, TX, TY, NS, CPT, MB, COEF, ONCE>;
  using F = Flow<G, T, NS>;
  extern __shared__ __align__(1024) unsigned char smem[];
  using R = typename F::R;
  const R ring{smem};
  uint64_t *ready = reinterpret_cast<uint64_t *>(smem + F::READY);   // F::RB barriers, one per item in flight
  int *arrived = reinterpret_cast<int *>(ready + F::RB);   // F::RB consumer-warp counters
  typename F::Slot *slots = reinterpret_cast<typename F::Slot *>(smem + F::SLOTS);
  const int tid = threadIdx.x;
  if (tid == 0)
    for (int r = 0; r < F::RB; ++r) {
      mbar_init(&ready[r], 1);
      arrived[r] = 0;
    }
  init_ring<G::NCW, LOAD_TMA>(ring);
  const unsigned long long wait_ns = (ctl & CTL_WITHHOLD_LOADS) ? kTestWaitLimitNs : kWaitLimitNs;

  if (tid >= G::NT) {  // producer warp
    if constexpr (G::SPLIT) fewer_registers<G::LOADER_REGS>();
    const int lane = tid - G::NT;
    if (lane >= 32) return;   // (the rest of its group)
    if (ctl & CTL_WITHHOLD_LOADS) return;  // test mode: no place is ever filled
    ItemPrefetch<T, TX, TY> pf_s{{}, shots, lane, ctl, PSI_S0};
    ItemPrefetch<T, TX, TY> pf_v{{}, shots, lane, ctl, PSI_V0};
    const int pass_steps = list_steps > 0 ? list_steps : nsteps;   // (one pass if the list's length is unset)
    const int total = nitems * ((nsteps + pass_steps - 1) / pass_steps);
    Loads<R> ld;
    unsigned idx = 0;
    bool ok = true;
    if (dtick) tick += *dtick;
    int next = 0;   // lane 0: the place claimed next
    if (lane == 0) next = claim ? atomicAdd(claim, 1) : (int)blockIdx.x;
    while (true) {
      const int q = __shfl_sync(0xffffffffu, next, 0);
      const bool end = q >= total;
      FlowItem fi{{0, 0, 0, 0}, -1, 0, 0, 0};
      if (!end) {
        // (the next claim is in flight while this item's loads are issued)
        if (lane == 0) next = claim ? atomicAdd(claim, 1) : q + (int)gridDim.x;
        fi = items[q % nitems];
        fi.step += q / nitems * pass_steps;
        if (fi.step >= nsteps) continue;   // a list of more steps than this launch runs
      }
      // the item and its shot's descriptor for the consumers (their slot's
      // last item, RB items ago, is done: see RB)
      typename F::Slot &slot = slots[idx % F::RB];
      if (!end) {
        const uint4 *src = reinterpret_cast<const uint4 *>(shots + fi.it.shot);
        uint4 *dst = reinterpret_cast<uint4 *>(&slot.sd);
        for (int c = lane; c < (int)(sizeof(ShotDesc<T>) / 16); c += 32) dst[c] = __ldg(src + c);
      }
      if (lane == 0) slot.fi = fi;
      __syncwarp();
      if (!end && (ctl & CTL_RETIRE) && tick + fi.step - slot.sd.tick0 > slot.sd.nstep) {
        __syncwarp();   // (the slot is filled again next)
        continue;
      }
      if (!end) {
        const int txs = (slot.sd.nx + TX - 1) / TX, tys = (slot.sd.ny + TY - 1) / TY;
        ok = flow_wait_deps(slot.sd, fi, txs, tys, G::NCW, wait_ns, lane);
      }
      if (ok && lane == 0) mbar_arrive(&ready[idx % F::RB]);   // release the consumers' reads
      ++idx;
      if (!ok || end) break;
      const ShotMaps &sm = maps[fi.it.shot];
      if (fi.kind == 0) {
        pf_s.begin(fi.it, slot.sd);
        ok = produce_item<false>(
            fi.it, ring, ld,
            [&](int k, unsigned char *st, uint64_t *bar) { stress_issue_a<G, LOAD_TMA>(slot.sd, sm, fi.it, k, st, bar, lane); },
            [&](int k, unsigned char *st, uint64_t *bar) { stress_issue_b<G, LOAD_TMA>(slot.sd, sm, fi.it, k, st, bar, lane); },
            pf_s, lane);
      } else {
        pf_v.begin(fi.it, slot.sd);
        ok = produce_item<false>(
            fi.it, ring, ld,
            [&](int k, unsigned char *st, uint64_t *bar) { velocity_issue_a<G, LOAD_TMA>(slot.sd, sm, fi.it, k, st, bar, lane); },
            [&](int k, unsigned char *st, uint64_t *bar) { velocity_issue_b<G, LOAD_TMA>(slot.sd, sm, fi.it, k, st, bar, lane); },
            pf_v, lane);
      }
      if (!ok) break;
    }
    produce_drain<false>(ring, ld, ok, err, lane);
    return;
  }
  if constexpr (G::SPLIT) more_registers<G::CONSUMER_REGS>();

  const int lane = tid & 31;
  if (dtick) tick += *dtick;
  Place<R::NA> a;
  Place<R::NB> b;
  for (unsigned idx = 0;; ++idx) {
    if (!flow_ready(&ready[idx % F::RB], (idx / F::RB) & 1, wait_ns, err, lane)) return;
    const typename F::Slot &slot = slots[idx % F::RB];
    const FlowItem fi = slot.fi;
    if (fi.kind < 0) return;   // the list is done
    const ShotDesc<T> &sd = slot.sd;
    bool ok;
    if (fi.kind == 0)
      ok = stress_item<G, true>(sd, fi.it, ring, a, b, smem + F::PSI, err, wait_ns, tid,
                                fi.step > 0 ? tick + fi.step - 1 : INT_MIN);
    else
      ok = velocity_item<G, true>(sd, fi.it, tick + fi.step, ring, a, b, smem + F::PSI, err, wait_ns, tid);
    if (!ok) return;
    // this warp's share of the item is written: it arrives (CTA scope) on
    // the item's counter, and the last warp to arrive releases the whole
    // item at gpu scope -- cumulative over the other warps' writes it has
    // acquired -- so one gpu-scope fence per item instead of one per warp
    fence_proxy_async_global();
    __syncwarp();
    if (lane == 0 && atom_acq_rel_cta_add(&arrived[idx % F::RB], 1) == G::NCW - 1) {
      arrived[idx % F::RB] = 0;   // re-armed for item idx + RB (no warp is that far ahead)
      const int txs = (sd.nx + TX - 1) / TX, tys = (sd.ny + TY - 1) / TY;
      int *flag = sd.flow_flags + ((size_t)fi.kind * sd.flow_chunks + fi.chunk) * (txs * tys) + fi.it.tile;
      red_release_gpu_add(flag, G::NCW);
    }
  }
}

// The update coefficients of every cell, eight arrays of `cells` values each:
// dt (lambda + 2 mu), dt lambda, dt mu of sigma_xy, sigma_xz and sigma_yz, and
// dt / rho of vx, vy and vz -- by the functions that the kernels without them
// use, so results are the same bits.  Neighbours outside the grid are zero, as
// in the kernels' boxes.
template <typename T>
__global__ void __launch_bounds__(256) coef_kernel(const ShotDesc<T> sd, T *out, long long cells) {
  const T dt = sd.dt;
  const long long plane = (long long)sd.ny * sd.px;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < cells; i += gridDim.x * 256ll) {
    const int k = (int)(i / plane);
    const long long r = i - k * plane;
    const int y = (int)(r / sd.px), x = (int)(r - (long long)y * sd.px);
    T v[8] = {};
    if (x < sd.nx) {
      const bool w = x > 0, s = y + 1 < sd.ny, u = k + 1 < sd.nz;
      const T cp[1] = {sd.cp[i]}, cs[1] = {sd.cs[i]}, rho[1] = {sd.rho[i]};
      const T cw[1] = {w ? sd.cs[i - 1] : T(0)}, rw[1] = {w ? sd.rho[i - 1] : T(0)};
      const T cy[1] = {s ? sd.cs[i + sd.px] : T(0)}, ry[1] = {s ? sd.rho[i + sd.px] : T(0)};
      const T cz[1] = {u ? sd.cs[i + plane] : T(0)}, rz[1] = {u ? sd.rho[i + plane] : T(0)};
      T a[1], b[1];
      dt_moduli(dt, cp, cs, rho, a, b);
      v[0] = a[0];
      v[1] = b[0];
      dt_mu(a, T(0.125) * dt, cw, cy, rw, ry);
      v[2] = a[0];
      dt_mu(a, T(0.125) * dt, cw, cz, rw, rz);
      v[3] = a[0];
      dt_mu(a, T(0.125) * dt, cy, cz, ry, rz);
      v[4] = a[0];
      dt_over_rho(a, dt, rho, rw, 1u);
      v[5] = a[0];
      dt_over_rho(a, dt, rho, ry, 1u);
      v[6] = a[0];
      dt_over_rho(a, dt, rho, rz, 1u);
      v[7] = a[0];
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) out[c * cells + i] = v[c];
  }
}

}  // namespace ela3d
