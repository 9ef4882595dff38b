// step_ops.cu -- single-step drop-in operators of the reference's custom-op
// library: AcousticOneStep forward/backward, ScatterAddOps, GatherOps,
// AddSource and GetReceive.
//
// This translation unit is compiled with --fmad=false and the forward keeps the
// reference's expression order, so the FP64 acoustic forward reproduces
// AcousticOneStepCpuForward (deps/CustomOps/AcousticOneStepCpu/
// AcousticOneStepCpu.h:1-48) bit for bit.  Threads map x -> j (the contiguous
// depth axis), so every warp access is coalesced (the reference GPU kernel maps
// threadIdx.x to the strided axis, AcousticOneStep.cu:28-34).
#include <algorithm>

#include "ads_internal.h"

namespace ads {

// Device-side record of rejected indices (out-of-range source / receiver /
// scatter indices are skipped, never dereferenced).
__device__ int g_bad_index = 0;

namespace {

constexpr int BJ = 32, BI = 8;

// The scalar factors of one step, each formed on the host by the operations, in
// the order, that the reference writes them, so they carry its rounding bit for
// bit.  Forming them in the kernels cost each cell about ten divisions, and an
// FP64 division is some twenty instructions on a pipe that issues a warp's
// instruction in 64 cycles: 1001 x 1001 FP64, variant W, one GB300: forward
// 322 us, gradient 793 us with the factors formed per cell.
template <typename T>
struct StepK {
  T dt, dt2, hx, hy, hx2, hy2;  // hx2 = 2 hx, hy2 = 2 hy
  T k1, k2;  // 2 dt^2 / hx^2, 2 dt^2 / hy^2 (each variant in its own order)
  T ax, ay;  // dt / hx, dt / hy
  T cx, cy;  // their squares
  T fx, fy;  // dt^2 / (2 hx), dt^2 / (2 hy)
  int plain;  // dt, hx, hy in the range where the undamped short forms hold
};

template <typename T>
StepK<T> make_k(double dt_, double hx_, double hy_, int variant) {
  const T dt = T(dt_), hx = T(hx_), hy = T(hy_), two = 2;
  StepK<T> K;
  K.dt = dt;
  K.dt2 = dt * dt;
  K.hx = hx;
  K.hy = hy;
  K.hx2 = two * hx;
  K.hy2 = two * hy;
  K.k1 = variant == 0 ? two * dt * dt / hx / hx : two * K.dt2 / (hx * hx);
  K.k2 = variant == 0 ? two * dt * dt / hy / hy : two * K.dt2 / (hy * hy);
  K.ax = dt / hx;
  K.ay = dt / hy;
  K.cx = K.ax * K.ax;
  K.cy = K.ay * K.ay;
  K.fx = K.dt2 / K.hx2;
  K.fy = K.dt2 / K.hy2;
  auto ok = [](T x) { return x >= T(1e-15) && x <= T(1e15); };
  K.plain = ok(dt) && ok(hx) && ok(hy);
  return K;
}

// |x| < 2^1023 (2^127): finite, and so is the difference of two of them.  Integer
// tests: they cost nothing on the FP64 pipe.
__device__ __forceinline__ bool tame(double x) {
  return (__double2hiint(x) & 0x7ff00000) < 0x7fe00000;
}
__device__ __forceinline__ bool tame(float x) {
  return (__float_as_int(x) & 0x7f800000) < 0x7f000000;
}
// |x| < 2^512 (2^64): its product with a step factor stays finite
__device__ __forceinline__ bool small(double x) {
  return (__double2hiint(x) & 0x7ff00000) < 0x5ff00000;
}
__device__ __forceinline__ bool small(float x) {
  return (__float_as_int(x) & 0x7f800000) < 0x5f800000;
}
__device__ __forceinline__ bool neg_zero(double x) {
  return __double2hiint(x) == (int)0x80000000 && __double2loint(x) == 0;
}
__device__ __forceinline__ bool neg_zero(float x) {
  return __float_as_int(x) == (int)0x80000000;
}
// x == 0 (either sign) as an integer test
__device__ __forceinline__ bool is_zero(double x) {
  return ((__double2hiint(x) << 1) | __double2loint(x)) == 0;
}
__device__ __forceinline__ bool is_zero(float x) { return x == 0.f; }
__device__ __forceinline__ bool zero_bits(double x) {
  return (__double2hiint(x) | __double2loint(x)) == 0;
}
__device__ __forceinline__ bool zero_bits(float x) { return __float_as_int(x) == 0; }

// A cell without damping (sigma = tau = 0): the factors 1 - (sigma + tau) dt/2,
// 1 + (sigma + tau) dt/2, 1 - dt sigma, 1 - dt tau are exactly 1 and sigma tau
// dt^2 and dt c (tau - sigma) exactly 0, so their products drop out and the
// division is by 1; what is left is the same value bit for bit.
template <typename T>
__device__ __forceinline__ bool undamped(const StepK<T>& K, T sg, T ta, T c) {
  return K.plain && is_zero(sg) && is_zero(ta) && small(c);
}

// phi' = (1 - 0) phi + 0 (difference): phi itself where the difference is
// finite (0 times it is a zero) and phi is not -0 (which a +0 would turn).
template <typename T>
__device__ __forceinline__ bool kept(T phi, T a, T b) {
  return tame(a) && tame(b) && !neg_zero(phi);
}

// The field update of one interior cell, in the reference's order (variant W
// AcousticOneStepCpu.h:18-46; U src/Core.jl:528-549).  Undamped cells take 22
// FP64 operations of 34 and no division.
template <typename T, int VARIANT>
__device__ __forceinline__ T new_u(const StepK<T>& K, int64_t k, int64_t S, T sg, T ta, T ck,
                                   bool plain, const T* __restrict__ w,
                                   const T* __restrict__ wold, const T* __restrict__ phi,
                                   const T* __restrict__ psi) {
  const T two = 2, one = 1;
  const T wn = w[k + S], ws = w[k - S], we = w[k + 1], ww = w[k - 1];
  T a = two;
  if (!plain) {
    if (VARIANT == 0) a = two - sg * ta * K.dt * K.dt;
    else a = two - sg * ta * K.dt2;
  }
  T v;
  if (VARIANT == 0)
    v = (a - K.k1 * ck - K.k2 * ck) * w[k] + ck * K.ax * K.ax * (wn + ws) +
        ck * K.ay * K.ay * (we + ww);
  else
    v = (a - K.k1 * ck - K.k2 * ck) * w[k] + ck * K.cx * (wn + ws) + ck * K.cy * (we + ww);
  v = v + K.fx * (phi[k + S] - phi[k - S]) + K.fy * (psi[k + 1] - psi[k - 1]);
  if (plain) return v - wold[k];
  v = v - (one - (sg + ta) * K.dt / two) * wold[k];
  return v / (one + (sg + ta) / two * K.dt);
}

// One thread per cell.  FP64 issue bounds it (82% of the pipe's active cycles):
// 22 operations an undamped cell, 28 a cell at 1001 x 1001 with a PML of 12, whose cells
// divide five times.  75 us there in FP64, 322 us with the factors and the division
// formed in every cell.
template <typename T>
__global__ void __launch_bounds__(BJ* BI)
k_acoustic_fwd_w(const T* __restrict__ w, const T* __restrict__ wold,
                 const T* __restrict__ phi, const T* __restrict__ psi,
                 const T* __restrict__ sigma, const T* __restrict__ tau,
                 const T* __restrict__ c, StepK<T> K, int NX, int NY, T* __restrict__ u,
                 T* __restrict__ phiout, T* __restrict__ psiout) {
  const int j = blockIdx.x * BJ + threadIdx.x;
  const int i = blockIdx.y * BI + threadIdx.y;
  if (i > NX + 1 || j > NY + 1) return;
  const int64_t S = NY + 2;
  const int64_t k = (int64_t)i * S + j;
  if (i == 0 || i == NX + 1 || j == 0 || j == NY + 1) {
    u[k] = 0;
    phiout[k] = 0;
    psiout[k] = 0;
    return;
  }
  const T sg = sigma[k], ta = tau[k], ck = c[k], one = 1;
  const bool plain = undamped<T>(K, sg, ta, ck);
  u[k] = new_u<T, 0>(K, k, S, sg, ta, ck, plain, w, wold, phi, psi);
  const T pk = phi[k], qk = psi[k];
  const T wn = w[k + S], ws = w[k - S], we = w[k + 1], ww = w[k - 1];
  if (plain && kept(pk, wn, ws) && kept(qk, we, ww)) {
    phiout[k] = pk;
    psiout[k] = qk;
  } else {
    phiout[k] = (one - K.dt * sg) * pk + K.dt * ck * (ta - sg) / T(2.0) / K.hx * (wn - ws);
    psiout[k] = (one - K.dt * ta) * qk + K.dt * ck * (sg - ta) / T(2.0) / K.hy * (we - ww);
  }
}

// Variant U: u over a tile and the ring of cells around it, then phi / psi of
// the tile from the new u: one launch and one read of the fields where two
// kernels passed u through memory.  Tiles of BI = 8 rows: the ring's second
// computation is a third of the tile's, but 16- and 32-row tiles leave the last
// wave emptier (1001 x 1001 FP64: 87.8 us with 8 rows, 88.3 with 16, 98.0 with 32;
// 1001 x 641: 66.6, 70.6, 79.7).
template <typename T>
__global__ void __launch_bounds__(BJ* BI)
k_acoustic_fwd_u(const T* __restrict__ w, const T* __restrict__ wold,
                 const T* __restrict__ phi, const T* __restrict__ psi,
                 const T* __restrict__ sigma, const T* __restrict__ tau,
                 const T* __restrict__ c, StepK<T> K, int NX, int NY, T* __restrict__ u,
                 T* __restrict__ phiout, T* __restrict__ psiout) {
  constexpr int W = BJ + 2, H = BI + 2, RING = 2 * W + 2 * BI;
  __shared__ T su[H][W];
  const int j0 = blockIdx.x * BJ, i0 = blockIdx.y * BI;
  const int r = threadIdx.y, q = threadIdx.x, i = i0 + r, j = j0 + q;
  const int64_t S = NY + 2;
  const T one = 1;
  auto cell = [&](int a, int b) -> T {  // u of cell (a, b)
    if (a < 1 || a > NX || b < 1 || b > NY) return T(0);
    const int64_t k = (int64_t)a * S + b;
    const T sg = sigma[k], ta = tau[k], ck = c[k];
    return new_u<T, 1>(K, k, S, sg, ta, ck, undamped<T>(K, sg, ta, ck), w, wold, phi, psi);
  };
  const T v = cell(i, j);
  su[r + 1][q + 1] = v;
  const int e = r * BJ + q;
  if (e < RING) {  // the ring: top and bottom rows, then the two columns
    const int f = e - 2 * W;
    const int a = e < W ? -1 : e < 2 * W ? BI : f >> 1;
    const int b = e < W ? e - 1 : e < 2 * W ? e - W - 1 : (f & 1) ? BJ : -1;
    su[a + 1][b + 1] = cell(i0 + a, j0 + b);
  }
  __syncthreads();
  if (i > NX + 1 || j > NY + 1) return;
  const int64_t k = (int64_t)i * S + j;
  u[k] = v;
  if (i == 0 || i == NX + 1 || j == 0 || j == NY + 1) {
    phiout[k] = 0;
    psiout[k] = 0;
    return;
  }
  const T sg = sigma[k], ta = tau[k], ck = c[k], pk = phi[k], qk = psi[k];
  const T un = su[r + 2][q + 1], us = su[r][q + 1], ue = su[r + 1][q + 2], uw = su[r + 1][q];
  if (undamped<T>(K, sg, ta, ck) && kept(pk, un, us) && kept(qk, ue, uw)) {
    phiout[k] = pk;
    psiout[k] = qk;
  } else {
    phiout[k] = (one - K.dt * sg) * pk + K.dt * ck * (ta - sg) / K.hx2 * (un - us);
    psiout[k] = (one - K.dt * ta) * qk + K.dt * ck * (sg - ta) / K.hy2 * (ue - uw);
  }
}

__device__ __forceinline__ double fm(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fm(float a, float b, float c) { return fmaf(a, b, c); }

// Gather-form transpose of one step (both variants).  Each output cell sums
// the contributions the reference's scatter loop (AcousticOneStepCpu.h:76-124)
// sends it; frame cells receive them too.
//
// What a cell y sends is formed once, in shared memory, over a tile and the
// ring around it: g / den (den = 1 where undamped: no division), c g / den, and
// in damped cells the phi / psi terms PX = dt c (tau - sigma) / (2 hx) gphi and
// PY likewise.  Variant U first adds what phi' / psi' send back through their u
// differences to g, so PX and PY reach one ring further.  An undamped cell takes
// 17 FP64 operations.  Forming each neighbour's terms again, with its division,
// took 793 us at 1001 x 1001 FP64 for variant W; this takes 84 us (92 with
// 16-row tiles, 109 with 32-row ones, whose last wave is nearly empty).
template <typename T, int VARIANT>
__global__ void __launch_bounds__(BJ* BI)
k_acoustic_bwd(T* __restrict__ grad_w, T* __restrict__ grad_wold, T* __restrict__ grad_phi,
               T* __restrict__ grad_psi, T* __restrict__ grad_c,
               const T* __restrict__ grad_u, const T* __restrict__ grad_phiout,
               const T* __restrict__ grad_psiout, const T* __restrict__ w,
               const T* __restrict__ sigma, const T* __restrict__ tau,
               const T* __restrict__ c, StepK<T> K, T kxy, int NX, int NY,
               const T* __restrict__ u) {
  constexpr int HP = VARIANT == 0 ? 1 : 2;  // ring of PX, PY
  constexpr int WP = BJ + 2 * HP, HPR = BI + 2 * HP, W = BJ + 2, H = BI + 2;
  __shared__ T sx[HPR][WP], sy[HPR][WP], sg_[H][W], sc[H][W];
  const int j0 = blockIdx.x * BJ, i0 = blockIdx.y * BI;
  const int64_t S = NY + 2;
  const T one = 1, two = 2;
  const int tid = threadIdx.y * BJ + threadIdx.x;
  auto inside = [&](int i, int j) { return i >= 1 && i <= NX && j >= 1 && j <= NY; };
  for (int e = tid; e < HPR * WP; e += BJ * BI) {
    const int r = e / WP, q = e - r * WP;
    const int i = i0 + r - HP, j = j0 + q - HP;
    T px = 0, py = 0;
    if (inside(i, j)) {
      const int64_t k = (int64_t)i * S + j;
      const T s = sigma[k], t = tau[k], gp = grad_phiout[k], gq = grad_psiout[k], ck = c[k];
      // (0 times a gradient that is not finite is kept as the NaN it is)
      if (!undamped<T>(K, s, t, ck) || !tame(gp) || !tame(gq)) {
        const T d = K.dt * ck * (t - s);
        px = d / K.hx2 * gp;
        py = -d / K.hy2 * gq;
      }
    }
    sx[r][q] = px;
    sy[r][q] = py;
  }
  if (VARIANT != 0) __syncthreads();
  for (int e = tid; e < H * W; e += BJ * BI) {
    const int r = e / W, q = e - r * W;
    const int i = i0 + r - 1, j = j0 + q - 1;
    T g = 0, cg = 0;
    if (inside(i, j)) {
      const int64_t k = (int64_t)i * S + j;
      const T s = sigma[k], t = tau[k], ck = c[k];
      g = grad_u[k];
      if (VARIANT != 0) {
        // PX, PY are zero on the frame and outside the grid
        const T a = sx[r][q + 1], b = sx[r + 2][q + 1], d = sy[r + 1][q], f = sy[r + 1][q + 2];
        if (!(zero_bits(a) && zero_bits(b) && zero_bits(d) && zero_bits(f)))
          g += (a - b) + (d - f);
      }
      if (!undamped<T>(K, s, t, ck)) g = g / (one + (s + t) / two * K.dt);
      cg = ck * g;
    }
    sg_[r][q] = g;
    sc[r][q] = cg;
  }
  __syncthreads();
  const int r = threadIdx.y, q = threadIdx.x, i = i0 + r, j = j0 + q;
  if (i > NX + 1 || j > NY + 1) return;
  const int64_t k = (int64_t)i * S + j;
  // from the neighbours (zero outside the interior)
  T gw = K.cx * (sc[r][q + 1] + sc[r + 2][q + 1]);
  gw = fm(K.cy, sc[r + 1][q] + sc[r + 1][q + 2], gw);
  T gph = K.fx * (sg_[r][q + 1] - sg_[r + 2][q + 1]);
  T gps = K.fy * (sg_[r + 1][q] - sg_[r + 1][q + 2]);
  if (VARIANT == 0) {
    const T a = sx[r][q + 1], b = sx[r + 2][q + 1], d = sy[r + 1][q], f = sy[r + 1][q + 2];
    if (!(zero_bits(a) && zero_bits(b) && zero_bits(d) && zero_bits(f)))
      gw += (a - b) + (d - f);
  }
  T gwo = 0, gc = 0;
  if (inside(i, j)) {
    const T s = sigma[k], t = tau[k], ck = c[k], g = sg_[r + 1][q + 1];
    const T wn = w[k + S], ws = w[k - S], we = w[k + 1], ww = w[k - 1];
    const T gp = grad_phiout[k], gq = grad_psiout[k];
    const bool plain = undamped<T>(K, s, t, ck);
    T lap = K.cx * (wn + ws);
    lap = fm(K.cy, we + ww, lap);
    lap = fm(-kxy, w[k], lap);
    gc = lap * g;
    T un, us, ue, uw;  // the field phi' and psi' difference
    if (VARIANT == 0) {
      un = wn;
      us = ws;
      ue = we;
      uw = ww;
    } else {
      un = u[k + S];
      us = u[k - S];
      ue = u[k + 1];
      uw = u[k - 1];
    }
    if (plain) {
      gw = fm(fm(-kxy, ck, two), g, gw);
      gwo = -g;
      gph += gp;
      gps += gq;
    } else {
      gw = fm(fm(-kxy, ck, two - s * t * K.dt2), g, gw);
      gwo = -(one - (s + t) * K.dt / two) * g;
      gph = fm(one - K.dt * s, gp, gph);
      gps = fm(one - K.dt * t, gq, gps);
    }
    if (!plain || !(tame(un) && tame(us) && tame(ue) && tame(uw) && tame(gp) && tame(gq))) {
      const T d = K.dt * (t - s);
      gc = fm(d / K.hx2 * (un - us), gp, gc);
      gc = fm(-d / K.hy2 * (ue - uw), gq, gc);
    }
  }
  grad_w[k] = gw;
  grad_wold[k] = gwo;
  grad_phi[k] = gph;
  grad_psi[k] = gps;
  grad_c[k] = gc;
}

template <typename T>
int acoustic_fwd(const T* w, const T* wold, const T* phi, const T* psi, const T* sigma,
                 const T* tau, const T* c, double dt, double hx, double hy, int64_t NX,
                 int64_t NY, T* u, T* phiout, T* psiout, int variant, cudaStream_t st) {
  if (int e = require_device()) return e;
  ADS_REQUIRE(NX >= 1 && NY >= 1 && NX < (1 << 30) && NY < (1 << 30),
              "NX, NY out of range (%lld, %lld)", (long long)NX, (long long)NY);
  ADS_REQUIRE(w && wold && phi && psi && sigma && tau && c && u && phiout && psiout,
              "null pointer argument");
  ADS_REQUIRE(variant == 0 || variant == 1, "variant must be 0 (w) or 1 (u)");
  const StepK<T> K = make_k<T>(dt, hx, hy, variant);
  const dim3 blk(BJ, BI), grd((unsigned)div_up(NY + 2, BJ), (unsigned)div_up(NX + 2, BI));
  if (variant == 0)
    k_acoustic_fwd_w<T><<<grd, blk, 0, st>>>(w, wold, phi, psi, sigma, tau, c, K, (int)NX,
                                             (int)NY, u, phiout, psiout);
  else
    k_acoustic_fwd_u<T><<<grd, blk, 0, st>>>(w, wold, phi, psi, sigma, tau, c, K, (int)NX,
                                             (int)NY, u, phiout, psiout);
  ADS_LAUNCHED(1);
  return ADS_OK;
}

template <typename T>
int acoustic_bwd(T* grad_w, T* grad_wold, T* grad_phi, T* grad_psi, T* grad_c,
                 const T* grad_u, const T* grad_phiout, const T* grad_psiout, const T* w,
                 const T* sigma, const T* tau, const T* c, double dt, double hx, double hy,
                 int64_t NX, int64_t NY, const T* u, int variant, cudaStream_t st) {
  if (int e = require_device()) return e;
  ADS_REQUIRE(NX >= 1 && NY >= 1 && NX < (1 << 30) && NY < (1 << 30),
              "NX, NY out of range");
  ADS_REQUIRE(grad_w && grad_wold && grad_phi && grad_psi && grad_c && grad_u &&
                  grad_phiout && grad_psiout && w && sigma && tau && c,
              "null pointer argument");
  ADS_REQUIRE(variant == 0 || (variant == 1 && u), "variant must be 0, or 1 with u given");
  const StepK<T> K = make_k<T>(dt, hx, hy, 0);  // (the transposes of both sum k1, k2 alike)
  const T kxy = K.k1 + K.k2;
  const dim3 blk(BJ, BI), grd((unsigned)div_up(NY + 2, BJ), (unsigned)div_up(NX + 2, BI));
  auto launch = [&](auto kernel) {
    kernel<<<grd, blk, 0, st>>>(grad_w, grad_wold, grad_phi, grad_psi, grad_c, grad_u,
                                grad_phiout, grad_psiout, w, sigma, tau, c, K, kxy, (int)NX,
                                (int)NY, u);
  };
  if (variant == 0) launch(k_acoustic_bwd<T, 0>);
  else launch(k_acoustic_bwd<T, 1>);
  ADS_LAUNCHED(1);
  return ADS_OK;
}

// ---------------------------------------------------------------- index ops

__global__ void k_copy(double* __restrict__ out, const double* __restrict__ in, int64_t n) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x)
    out[t] = in[t];
}

__global__ void k_zero(double* __restrict__ out, int64_t n) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x)
    out[t] = 0.0;
}

__global__ void k_scatter_add(double* out, const int64_t* __restrict__ ii,
                              const double* __restrict__ upd, int64_t d, int64_t n) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int64_t x = ii[t] - 1;
  if (x < 0 || x >= d) {
    atomicOr(&g_bad_index, 1);
    return;
  }
  atomicAdd(out + x, upd[t]);
}

__global__ void k_gather(double* __restrict__ out, const double* __restrict__ v,
                         const int64_t* __restrict__ ii, int64_t n, int64_t dlen) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int64_t x = ii[t] - 1;
  if (x < 0 || x >= dlen) {
    atomicOr(&g_bad_index, 1);
    out[t] = 0.0;
    return;
  }
  out[t] = v[x];
}

struct Five {
  double* p[5];
};
struct CFive {
  const double* p[5];
};

// AddSource field order (sxx, syy, sxy, vx, vy); srctype 0 vx, 1 vy, 2 sxx,
// 3 syy, 4 sxy -> positions 3, 4, 0, 1, 2.
__device__ __forceinline__ int type_slot(int64_t t) {
  return t == 0 ? 3 : t == 1 ? 4 : t == 2 ? 0 : t == 3 ? 1 : t == 4 ? 2 : -1;
}

__global__ void k_add_source(Five out, const int64_t* __restrict__ si,
                             const int64_t* __restrict__ sj, const int64_t* __restrict__ st,
                             const double* __restrict__ sv, int64_t nsrc, int64_t NX,
                             int64_t NY) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nsrc) return;
  const int slot = type_slot(st[t]);
  if (slot < 0) return;
  const int64_t a = si[t] - 1, b = sj[t] - 1;
  if (a < 0 || a > NX + 1 || b < 0 || b > NY + 1) {
    atomicOr(&g_bad_index, 2);
    return;
  }
  atomicAdd(out.p[slot] + a * (NY + 2) + b, sv[t]);
}

__global__ void k_add_source_grad(CFive g, double* __restrict__ gs,
                                  const int64_t* __restrict__ si,
                                  const int64_t* __restrict__ sj,
                                  const int64_t* __restrict__ st, int64_t nsrc, int64_t NX,
                                  int64_t NY) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nsrc) return;
  const int slot = type_slot(st[t]);
  const int64_t a = si[t] - 1, b = sj[t] - 1;
  if (slot < 0 || a < 0 || a > NX + 1 || b < 0 || b > NY + 1) {
    if (slot >= 0) atomicOr(&g_bad_index, 2);
    gs[t] = 0.0;
    return;
  }
  gs[t] = g.p[slot][a * (NY + 2) + b];
}

// GetReceive field order (vx, vy, sxx, syy, sxy) = srctype order.
__global__ void k_get_receive(double* __restrict__ out, CFive f, int64_t nt,
                              const int64_t* __restrict__ ri, const int64_t* __restrict__ rj,
                              const int64_t* __restrict__ rt, int64_t nrcv, int64_t NX,
                              int64_t NY) {
  const int64_t r = blockIdx.y;
  const int64_t N = (NX + 2) * (NY + 2);
  if (r >= nrcv) return;
  const int64_t type = rt[r], a = ri[r] - 1, b = rj[r] - 1;
  const bool ok = type >= 0 && type <= 4 && a >= 0 && a <= NX + 1 && b >= 0 && b <= NY + 1;
  if (!ok && threadIdx.x == 0 && blockIdx.x == 0) atomicOr(&g_bad_index, 4);
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nt;
       k += (int64_t)gridDim.x * blockDim.x)
    out[nt * r + k] = ok ? f.p[type][k * N + a * (NY + 2) + b] : 0.0;
}

__global__ void k_get_receive_grad(Five g, const double* __restrict__ gout, int64_t nt,
                                   const int64_t* __restrict__ ri,
                                   const int64_t* __restrict__ rj,
                                   const int64_t* __restrict__ rt, int64_t nrcv, int64_t NX,
                                   int64_t NY) {
  const int64_t r = blockIdx.y;
  const int64_t N = (NX + 2) * (NY + 2);
  if (r >= nrcv) return;
  const int64_t type = rt[r], a = ri[r] - 1, b = rj[r] - 1;
  if (!(type >= 0 && type <= 4 && a >= 0 && a <= NX + 1 && b >= 0 && b <= NY + 1)) return;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nt;
       k += (int64_t)gridDim.x * blockDim.x)
    atomicAdd(g.p[type] + k * N + a * (NY + 2) + b, gout[nt * r + k]);
}

int copy_if_needed(double* out, const double* in, int64_t n, cudaStream_t st) {
  if (out == in || n == 0) return ADS_OK;
  k_copy<<<(unsigned)std::min<int64_t>(div_up(n, 256), 4096), 256, 0, st>>>(out, in, n);
  ADS_LAUNCHED(1);
  return ADS_OK;
}

}  // namespace
}  // namespace ads

using namespace ads;

extern "C" {

int ads_acoustic_step_fwd_f64(const double* w, const double* wold, const double* phi,
                              const double* psi, const double* sigma, const double* tau,
                              const double* c, double dt, double hx, double hy, int64_t NX,
                              int64_t NY, double* u, double* phiout, double* psiout,
                              int variant, ads_stream_t stream) {
  return acoustic_fwd<double>(w, wold, phi, psi, sigma, tau, c, dt, hx, hy, NX, NY, u,
                              phiout, psiout, variant, (cudaStream_t)stream);
}

int ads_acoustic_step_fwd_f32(const float* w, const float* wold, const float* phi,
                              const float* psi, const float* sigma, const float* tau,
                              const float* c, double dt, double hx, double hy, int64_t NX,
                              int64_t NY, float* u, float* phiout, float* psiout,
                              int variant, ads_stream_t stream) {
  return acoustic_fwd<float>(w, wold, phi, psi, sigma, tau, c, dt, hx, hy, NX, NY, u, phiout,
                             psiout, variant, (cudaStream_t)stream);
}

int ads_acoustic_step_bwd_f64(double* grad_w, double* grad_wold, double* grad_phi,
                              double* grad_psi, double* grad_c, const double* grad_u,
                              const double* grad_phiout, const double* grad_psiout,
                              const double* w, const double* wold, const double* phi,
                              const double* psi, const double* sigma, const double* tau,
                              const double* c, double dt, double hx, double hy, int64_t NX,
                              int64_t NY, const double* u, const double* phiout,
                              const double* psiout, int variant, ads_stream_t stream) {
  (void)wold; (void)phi; (void)psi; (void)phiout; (void)psiout;
  return acoustic_bwd<double>(grad_w, grad_wold, grad_phi, grad_psi, grad_c, grad_u,
                              grad_phiout, grad_psiout, w, sigma, tau, c, dt, hx, hy, NX, NY,
                              u, variant, (cudaStream_t)stream);
}

int ads_acoustic_step_bwd_f32(float* grad_w, float* grad_wold, float* grad_phi,
                              float* grad_psi, float* grad_c, const float* grad_u,
                              const float* grad_phiout, const float* grad_psiout,
                              const float* w, const float* wold, const float* phi,
                              const float* psi, const float* sigma, const float* tau,
                              const float* c, double dt, double hx, double hy, int64_t NX,
                              int64_t NY, const float* u, const float* phiout,
                              const float* psiout, int variant, ads_stream_t stream) {
  (void)wold; (void)phi; (void)psi; (void)phiout; (void)psiout;
  return acoustic_bwd<float>(grad_w, grad_wold, grad_phi, grad_psi, grad_c, grad_u,
                             grad_phiout, grad_psiout, w, sigma, tau, c, dt, hx, hy, NX, NY, u,
                             variant, (cudaStream_t)stream);
}

int ads_scatter_add_f64(double* out, const double* ipt, const int64_t* ii,
                        const double* update, int64_t d, int64_t n, ads_stream_t stream) {
  if (int e = require_device()) return e;
  ADS_REQUIRE(d >= 0 && n >= 0, "negative size");
  ADS_REQUIRE(out && ipt && (n == 0 || (ii && update)), "null pointer argument");
  cudaStream_t st = (cudaStream_t)stream;
  if (int e = copy_if_needed(out, ipt, d, st)) return e;
  if (n == 0) return ADS_OK;
  k_scatter_add<<<(unsigned)div_up(n, 256), 256, 0, st>>>(out, ii, update, d, n);
  ADS_LAUNCHED(1);
  return ADS_OK;
}

int ads_gather_f64(double* out, const double* v, const int64_t* ii, int64_t n,
                   ads_stream_t stream) {
  if (int e = require_device()) return e;
  ADS_REQUIRE(n >= 0, "negative size");
  if (n == 0) return ADS_OK;
  ADS_REQUIRE(out && v && ii, "null pointer argument");
  // GatherOps carries no length for v: only indices below 1 can be rejected.
  k_gather<<<(unsigned)div_up(n, 256), 256, 0, (cudaStream_t)stream>>>(out, v, ii, n,
                                                                        INT64_MAX);
  ADS_LAUNCHED(1);
  return ADS_OK;
}

int ads_add_source_f64(double* out_sxx, double* out_syy, double* out_sxy, double* out_vx,
                       double* out_vy, const double* sxx, const double* syy,
                       const double* sxy, const double* vx, const double* vy,
                       const int64_t* srci, const int64_t* srcj, const int64_t* srctype,
                       int64_t nsrc, int64_t NX, int64_t NY, const double* srcv,
                       ads_stream_t stream) {
  if (int e = require_device()) return e;
  ADS_REQUIRE(NX >= 1 && NY >= 1 && nsrc >= 0, "invalid sizes");
  ADS_REQUIRE(out_sxx && out_syy && out_sxy && out_vx && out_vy && sxx && syy && sxy && vx &&
                  vy && (nsrc == 0 || (srci && srcj && srctype && srcv)),
              "null pointer argument");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t N = (NX + 2) * (NY + 2);
  double* o[5] = {out_sxx, out_syy, out_sxy, out_vx, out_vy};
  const double* in[5] = {sxx, syy, sxy, vx, vy};
  for (int f = 0; f < 5; f++)
    if (int e = copy_if_needed(o[f], in[f], N, st)) return e;
  if (nsrc == 0) return ADS_OK;
  Five F{{out_sxx, out_syy, out_sxy, out_vx, out_vy}};
  k_add_source<<<(unsigned)div_up(nsrc, 128), 128, 0, st>>>(F, srci, srcj, srctype, srcv,
                                                             nsrc, NX, NY);
  ADS_LAUNCHED(1);
  return ADS_OK;
}

int ads_add_source_bwd_f64(double* g_sxx, double* g_syy, double* g_sxy, double* g_vx,
                           double* g_vy, double* grad_srcv, const double* gout_sxx,
                           const double* gout_syy, const double* gout_sxy,
                           const double* gout_vx, const double* gout_vy,
                           const int64_t* srci, const int64_t* srcj,
                           const int64_t* srctype, int64_t nsrc, int64_t NX, int64_t NY,
                           ads_stream_t stream) {
  if (int e = require_device()) return e;
  ADS_REQUIRE(NX >= 1 && NY >= 1 && nsrc >= 0, "invalid sizes");
  ADS_REQUIRE(g_sxx && g_syy && g_sxy && g_vx && g_vy && gout_sxx && gout_syy && gout_sxy &&
                  gout_vx && gout_vy && (nsrc == 0 || (srci && srcj && srctype && grad_srcv)),
              "null pointer argument");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t N = (NX + 2) * (NY + 2);
  double* o[5] = {g_sxx, g_syy, g_sxy, g_vx, g_vy};
  const double* in[5] = {gout_sxx, gout_syy, gout_sxy, gout_vx, gout_vy};
  for (int f = 0; f < 5; f++)
    if (int e = copy_if_needed(o[f], in[f], N, st)) return e;
  if (nsrc == 0) return ADS_OK;
  CFive G{{gout_sxx, gout_syy, gout_sxy, gout_vx, gout_vy}};
  k_add_source_grad<<<(unsigned)div_up(nsrc, 128), 128, 0, st>>>(G, grad_srcv, srci, srcj,
                                                                  srctype, nsrc, NX, NY);
  ADS_LAUNCHED(1);
  return ADS_OK;
}

int ads_get_receive_f64(double* out, const double* vx, const double* vy, const double* sxx,
                        const double* syy, const double* sxy, int64_t nt,
                        const int64_t* rcvi, const int64_t* rcvj, const int64_t* rcvtype,
                        int64_t nrcv, int64_t NX, int64_t NY, ads_stream_t stream) {
  if (int e = require_device()) return e;
  ADS_REQUIRE(NX >= 1 && NY >= 1 && nt >= 0 && nrcv >= 0 && nrcv < 65536,
              "invalid sizes (nrcv must be < 65536)");
  if (nt == 0 || nrcv == 0) return ADS_OK;
  ADS_REQUIRE(out && vx && vy && sxx && syy && sxy && rcvi && rcvj && rcvtype,
              "null pointer argument");
  CFive F{{vx, vy, sxx, syy, sxy}};
  dim3 grd((unsigned)std::min<int64_t>(div_up(nt, 128), 64), (unsigned)nrcv);
  k_get_receive<<<grd, 128, 0, (cudaStream_t)stream>>>(out, F, nt, rcvi, rcvj, rcvtype, nrcv,
                                                       NX, NY);
  ADS_LAUNCHED(1);
  return ADS_OK;
}

int ads_get_receive_bwd_f64(double* g_vx, double* g_vy, double* g_sxx, double* g_syy,
                            double* g_sxy, const double* gout, int64_t nt,
                            const int64_t* rcvi, const int64_t* rcvj,
                            const int64_t* rcvtype, int64_t nrcv, int64_t NX, int64_t NY,
                            ads_stream_t stream) {
  if (int e = require_device()) return e;
  ADS_REQUIRE(NX >= 1 && NY >= 1 && nt >= 0 && nrcv >= 0 && nrcv < 65536, "invalid sizes");
  ADS_REQUIRE(g_vx && g_vy && g_sxx && g_syy && g_sxy, "null pointer argument");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t n = nt * (NX + 2) * (NY + 2);
  double* g[5] = {g_vx, g_vy, g_sxx, g_syy, g_sxy};
  for (int f = 0; f < 5; f++) {
    if (n == 0) break;
    k_zero<<<(unsigned)std::min<int64_t>(div_up(n, 256), 8192), 256, 0, st>>>(g[f], n);
    ADS_LAUNCHED(1);
  }
  if (nt == 0 || nrcv == 0) return ADS_OK;
  ADS_REQUIRE(gout && rcvi && rcvj && rcvtype, "null pointer argument");
  Five G{{g_vx, g_vy, g_sxx, g_syy, g_sxy}};
  dim3 grd((unsigned)std::min<int64_t>(div_up(nt, 128), 64), (unsigned)nrcv);
  k_get_receive_grad<<<grd, 128, 0, st>>>(G, gout, nt, rcvi, rcvj, rcvtype, nrcv, NX, NY);
  ADS_LAUNCHED(1);
  return ADS_OK;
}

// Reads (and optionally clears) the device-side flags of rejected indices
// (bit 0 scatter, bit 1 source, bit 2 receiver).  Synchronises the device.
int ads_device_index_errors(int clear, int* flags) {
  if (int e = require_device()) return e;
  ADS_REQUIRE(flags, "null output");
  ADS_CUDA(cudaDeviceSynchronize());
  ADS_CUDA(cudaMemcpyFromSymbol(flags, g_bad_index, sizeof(int)));
  if (clear) {
    int z = 0;
    ADS_CUDA(cudaMemcpyToSymbol(g_bad_index, &z, sizeof(int)));
  }
  return ADS_OK;
}

}  // extern "C"
