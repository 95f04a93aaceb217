// GB300 (sm_103a) FDTD engine, adjoint (gradient) form.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "iris_engine.h"

using namespace iris;

// ---------------------------------------------------------------------------
// Adjoint (gradient) form: the exact discrete adjoint of the time loop of
// code/driver.f90:338-451 as the engine runs it.
//
// One forward step maps the interior state (E, D, H, B; ghosts are Bloch
// images of interior cells) linearly, plus a TF/SF source that does not
// depend on the state:
//   E pass  D' = a D + b_e C,  E' = al E + g_e D + be_e C,   C  = curl_b H
//   H pass  B' = a B + b_h C', H' = al H + g_h B + be_h C',  C' = curl_f E'
// with, outside the UPML slabs, E' = E + m C (m = eps_inv, or 1/eps1, 1/eps3)
// and H' = H - dtcq2 C'.  Its conjugate transpose, applied in reverse order,
// uses curl_b^H = curl_f and curl_f^H = curl_b, whose Bloch ghosts carry the
// conjugated phase of the opposite side:
//   adjoint H pass  Ebar += curl_b(V),  V = b_h Bbar + be_h Hbar,
//                   then Hbar <- al Hbar, Bbar <- a Bbar + g_h Hbar
//   adjoint E pass  Hbar += curl_f(W),  W = b_e Dbar + be_e Ebar,
//                   then Ebar <- al Ebar, Dbar <- a Dbar + g_e Ebar
// Each "then" part touches one cell of a field whose neighbours the same
// kernel still reads, so it is deferred to the next kernel, which reads only
// its own cell of that field: both kernels update in place.  In FP32 the planes
// outside the slabs take both passes in one (iris_march.cuh), into second
// buffers of E and H; the kernels here then do the slabs and the plane next to
// each, from the old buffers into the new.
// dL/d eps_inv(c) = sum_n Re <Ebar'_n(c), C_n(c)>, Ebar'_n the adjoint of the
// E pass output of step n, C_n the forward curl of H that pass used.

namespace iris {

unsigned long long bc_take_adjoint() { return bc_take_module(); }

namespace {

// adjoint UPML rows, 24 per UPML plane (+k: component)
enum { AJ_A = 0, AJ_AL = 3, AJ_GE = 6, AJ_BE = 9, AJ_DE = 12, AJ_GH = 15, AJ_BH = 18, AJ_DH = 21 };

struct Design {
  int x0, y0, z0, nx, ny, nz;
  long n;
};

template <typename T> struct AdjArgs {
  FieldArgs<T> f;                // adjoint state; coef = adjoint rows, eps_r = forward material
  int z0, z1;                    // planes of the launch (blockIdx.z counts from z0): z0 .. z1,
  int z2, z3;                    // then z2 .. z3 (none when z3 < z2)
  typename V2<T>::t* eo;         // where the new E and H go (in place: f.e, f.h)
  typename V2<T>::t* ho;
  int images;                    // also store H's images at x = 0 and y = 0 (the march reads them)
  Design d;
  const typename V2<T>::t* rec;  // forward curl of H at the design cells for this step, [3][n]
  double* grad;                  // dL/d eps_inv accumulators [n], or null
  int first;                     // no deferred E transform pending
};

struct AdjFace {
  long b[6];  // first sample index per component (Ex, Ey, Ez, Hx, Hy, Hz)
  long n;
  int nu, x0, y0, z;
};

template <typename T> __device__ __forceinline__ bool in_pml(const FieldArgs<T>& a, int z) {
  return z <= a.pmlzi || z >= a.pmlzf;
}

// UPML row and auxiliary index of interior cell (x, y, z) inside a slab.
template <typename T>
__device__ __forceinline__ void pml_at(const FieldArgs<T>& a, int x, int y, int z, int& slab, int& row, long& pi) {
  slab = z <= a.pmlzi ? 0 : 1;
  const int zr = slab == 0 ? z - 1 : z - a.pmlzf;
  row = slab == 0 ? z - 1 : a.pmlzi + z - a.pmlzf;
  pi = ((long)zr * a.g.ny + (y - 1)) * (long)a.g.nx + (x - 1);
}

// V_k = b_h Bbar_k + be_h Hbar_k (UPML) or -dtcq2 Hbar_k at interior cell
// (x, y, z); UPML = false: the caller knows z is outside the slabs.
template <typename T, bool UPML>
__device__ __forceinline__ cx<T> adj_v(const FieldArgs<T>& a, int x, int y, int z, int k) {
  const cx<T> hb = ld<T>(a.h + k * a.g.comp + a.g.at(x, y, z));
  if (UPML && in_pml(a, z)) {
    int slab, row;
    long pi;
    pml_at(a, x, y, z, slab, row, pi);
    const T* cf = a.coef + NCOEF * row;
    const cx<T> bb = ld<T>(a.pml_b[slab] + k * a.pcomp[slab] + pi);
    return cadd(rmul(cf[AJ_DH + k], bb), rmul(cf[AJ_BH + k], hb));
  }
  return rmul(-a.dtcq2, hb);
}

// W_k = b_e Dbar_k + be_e Ebar_k (UPML) or m Ebar_k at interior cell
// (x, y, z); UPML = false: the caller knows z is outside the slabs.
template <typename T, bool UPML>
__device__ __forceinline__ cx<T> adj_w(const FieldArgs<T>& a, int x, int y, int z, int k) {
  const Geo& g = a.g;
  const cx<T> eb = ld<T>(a.e + k * g.comp + g.at(x, y, z));
  if (UPML && in_pml(a, z)) {
    int slab, row;
    long pi;
    pml_at(a, x, y, z, slab, row, pi);
    const T* cf = a.coef + NCOEF * row;
    const cx<T> dd = ld<T>(a.pml_d[slab] + k * a.pcomp[slab] + pi);
    return cadd(rmul(cf[AJ_DE + k], dd), rmul(cf[AJ_BE + k], eb));
  }
  if (z >= a.hi && z <= a.hf) return rmul(a.eps_r[(long)(z - a.hi) * g.plane + (long)y * g.pitch + (x + g.xo)], eb);
  return rmul(z < a.hi ? a.m1 : a.m3, eb);
}

// The images at x = 0 and y = 0 of the new H of cell (x, y, z).
template <typename T> __device__ __forceinline__ void adj_images(const AdjArgs<T>& A, int x, int y, int z, const cx<T> h[3]) {
  const FieldArgs<T>& a = A.f;
  const Geo& g = a.g;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (x == g.nx) st<T>(A.ho + k * g.comp + g.at(0, y, z), cmul(a.pxm, h[k]));
    if (y == g.ny) st<T>(A.ho + k * g.comp + g.at(x, 0, z), cmul(a.pym, h[k]));
  }
}

// Adjoint of the H pass (plus the E pass transform deferred from the step
// after it): Ebar += curl_b(V); the gradient term of the design cells.
// Planes z0 .. z1 of the launch; UPML = false: neither they nor the planes
// below them lie in a UPML slab.
template <typename T, bool CURL, bool UPML> __global__ void __launch_bounds__(256) k_adj_h(AdjArgs<T> A) {
  const FieldArgs<T>& a = A.f;
  const Geo& g = a.g;
  const int x = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int y = blockIdx.y * blockDim.y + threadIdx.y + 1;
  int z = A.z0 + blockIdx.z * blockDim.z + threadIdx.z;
  if (z > A.z1) {
    z += A.z2 - A.z1 - 1;
    if (z > A.z3) return;
  }
  if (x > g.nx || y > g.ny) return;
  const long i = g.at(x, y, z);
  cx<T> e[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) e[k] = ld<T>(a.e + k * g.comp + i);
  if (UPML && !A.first && in_pml(a, z)) {
    int slab, row;
    long pi;
    pml_at(a, x, y, z, slab, row, pi);
    const T* cf = a.coef + NCOEF * row;
    auto* D = a.pml_d[slab];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const long j = k * a.pcomp[slab] + pi;
      st<T>(D + j, cadd(rmul(cf[AJ_A + k], ld<T>(D + j)), rmul(cf[AJ_GE + k], e[k])));
      e[k] = rmul(cf[AJ_AL + k], e[k]);
    }
  }
  if (CURL) {
    cx<T> v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = adj_v<T, UPML>(a, x, y, z, k);
    const int xm = x == 1 ? g.nx : x - 1, ym = y == 1 ? g.ny : y - 1, zm = z == 1 ? g.nz : z - 1;
    cx<T> v1x = adj_v<T, UPML>(a, xm, y, z, 1), v2x = adj_v<T, UPML>(a, xm, y, z, 2);
    cx<T> v0y = adj_v<T, UPML>(a, x, ym, z, 0), v2y = adj_v<T, UPML>(a, x, ym, z, 2);
    cx<T> v0z = adj_v<T, UPML>(a, x, y, zm, 0), v1z = adj_v<T, UPML>(a, x, y, zm, 1);
    if (x == 1) { v1x = cmul(a.pxm, v1x); v2x = cmul(a.pxm, v2x); }
    if (y == 1) { v0y = cmul(a.pym, v0y); v2y = cmul(a.pym, v2y); }
    if (z == 1) { v0z = cmul(a.pzm, v0z); v1z = cmul(a.pzm, v1z); }
    e[0] = cadd(e[0], cadd(csub(csub(v[2], v2y), v[1]), v1z));
    e[1] = cadd(e[1], cadd(csub(csub(v[0], v0z), v[2]), v2x));
    e[2] = cadd(e[2], cadd(csub(csub(v[1], v1x), v[0]), v0y));
    const Design& d = A.d;
    if (A.grad && x >= d.x0 && x < d.x0 + d.nx && y >= d.y0 && y < d.y0 + d.ny && z >= d.z0 && z < d.z0 + d.nz) {
      const long q = ((long)(z - d.z0) * d.ny + (y - d.y0)) * d.nx + (x - d.x0);
      T s = 0;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const cx<T> c = ld<T>(A.rec + k * d.n + q);
        s = add_(s, add_(mul_(e[k].re, c.re), mul_(e[k].im, c.im)));
      }
      A.grad[q] += (double)s;
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) st<T>(A.eo + k * g.comp + i, e[k]);
}

// Adjoint of the E pass (plus the H pass transform of the same step):
// Hbar <- al Hbar + curl_f(W), Bbar <- a Bbar + g_h Hbar.  Planes z0 .. z1;
// UPML = false: neither they nor the planes above them lie in a UPML slab.
template <typename T, bool UPML> __global__ void __launch_bounds__(256) k_adj_e(AdjArgs<T> A) {
  const FieldArgs<T>& a = A.f;
  const Geo& g = a.g;
  const int x = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int y = blockIdx.y * blockDim.y + threadIdx.y + 1;
  int z = A.z0 + blockIdx.z * blockDim.z + threadIdx.z;
  if (z > A.z1) {
    z += A.z2 - A.z1 - 1;
    if (z > A.z3) return;
  }
  if (x > g.nx || y > g.ny) return;
  const long i = g.at(x, y, z);
  cx<T> h[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) h[k] = ld<T>(a.h + k * g.comp + i);
  if (UPML && in_pml(a, z)) {
    int slab, row;
    long pi;
    pml_at(a, x, y, z, slab, row, pi);
    const T* cf = a.coef + NCOEF * row;
    auto* B = a.pml_b[slab];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const long j = k * a.pcomp[slab] + pi;
      st<T>(B + j, cadd(rmul(cf[AJ_A + k], ld<T>(B + j)), rmul(cf[AJ_GH + k], h[k])));
      h[k] = rmul(cf[AJ_AL + k], h[k]);
    }
  }
  cx<T> w[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) w[k] = adj_w<T, UPML>(a, x, y, z, k);
  const int xp = x == g.nx ? 1 : x + 1, yp = y == g.ny ? 1 : y + 1, zp = z == g.nz ? 1 : z + 1;
  cx<T> w1x = adj_w<T, UPML>(a, xp, y, z, 1), w2x = adj_w<T, UPML>(a, xp, y, z, 2);
  cx<T> w0y = adj_w<T, UPML>(a, x, yp, z, 0), w2y = adj_w<T, UPML>(a, x, yp, z, 2);
  cx<T> w0z = adj_w<T, UPML>(a, x, y, zp, 0), w1z = adj_w<T, UPML>(a, x, y, zp, 1);
  if (x == g.nx) { w1x = cmul(a.pxp, w1x); w2x = cmul(a.pxp, w2x); }
  if (y == g.ny) { w0y = cmul(a.pyp, w0y); w2y = cmul(a.pyp, w2y); }
  if (z == g.nz) { w0z = cmul(a.pzp, w0z); w1z = cmul(a.pzp, w1z); }
  h[0] = cadd(h[0], cadd(csub(csub(w2y, w[2]), w1z), w[1]));
  h[1] = cadd(h[1], cadd(csub(csub(w0z, w[0]), w2x), w[2]));
  h[2] = cadd(h[2], cadd(csub(csub(w1x, w[1]), w0y), w[0]));
#pragma unroll
  for (int k = 0; k < 3; ++k) st<T>(A.ho + k * g.comp + i, h[k]);
  if (A.images) adj_images<T>(A, x, y, z, h);
}

// H's images of every plane, from the interior (ho = f.h).
template <typename T> __global__ void __launch_bounds__(256) k_adj_images(AdjArgs<T> A) {
  const Geo& g = A.f.g;
  const int x = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int y = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int z = blockIdx.z * blockDim.z + threadIdx.z + 1;
  if (x > g.nx || y > g.ny || z > g.nz || (x < g.nx && y < g.ny)) return;
  cx<T> h[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) h[k] = ld<T>(A.f.h + k * g.comp + g.at(x, y, z));
  adj_images<T>(A, x, y, z, h);
}

// The planes outside the slabs in one pass (FP32): E, H read and written once, 96
// bytes a cell instead of 144.  160x160x352 on GB300: 148 us for 325 planes,
// the two passes 201; with the slabs and the source 240 us a step, before 314.
template <typename TL>
__global__ void __launch_bounds__(MR_T, 2) k_adj_march(MarchArgs A, const __grid_constant__ MarchGrad J, int za, int zb,
                                                       int zc) {
  extern __shared__ __align__(128) unsigned char mr_dyn[];
  const int z0 = za + zc * (int)blockIdx.z, z1 = min(z0 + zc - 1, zb);
  march_tile<TL, false, true>(A, mr_dyn, blockIdx.x, blockIdx.y, z0, z1, nullptr, &J);
}
using AdjMarchFn = void (*)(MarchArgs, const MarchGrad, int, int, int);
AdjMarchFn adj_march_kernel(int id) {
#define IRIS_MARCH_K(ID, W, R) \
  if (id == ID) return (AdjMarchFn)k_adj_march<MarchTile<W, R>>;
  IRIS_MARCH_SHAPES(IRIS_MARCH_K)
#undef IRIS_MARCH_K
  return nullptr;
}

// Forward curl_b H of the E pass at the design cells (the H the next E pass
// reads, ghosts included), as e_update forms it.
template <typename T>
__global__ void __launch_bounds__(256) k_adj_record(FieldArgs<T> a, Design d, typename V2<T>::t* __restrict__ rec) {
  const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= d.n) return;
  const int x = d.x0 + (int)(q % d.nx), y = d.y0 + (int)((q / d.nx) % d.ny), z = d.z0 + (int)(q / ((long)d.nx * d.ny));
  const Geo& g = a.g;
  const long i = g.at(x, y, z);
  const auto* H1 = a.h;
  const auto* H2 = a.h + g.comp;
  const auto* H3 = a.h + 2 * g.comp;
  const cx<T> h0 = ld<T>(H1 + i), h1 = ld<T>(H2 + i), h2 = ld<T>(H3 + i);
  st<T>(rec + q, cadd(csub(csub(h2, ld<T>(H3 + i - g.pitch)), h1), ld<T>(H2 + i - g.plane)));
  st<T>(rec + d.n + q, cadd(csub(csub(h0, ld<T>(H1 + i - g.plane)), h2), ld<T>(H3 + i - 1)));
  st<T>(rec + 2 * d.n + q, cadd(csub(csub(h1, ld<T>(H2 + i - 1)), h0), ld<T>(H1 + i - g.pitch)));
}

// Adjoint DFT source of one sampled step on one z face:
//   Ebar_x += c Y_Hy, Ebar_y -= c Y_Hx, Hbar_x -= c Y_Ey, Hbar_y += c Y_Ex
// summed over frequencies, c = w * exp(-i fw t), Y the final DFT values.
// FP64 mode: one step a launch, in FP64.
__global__ void __launch_bounds__(256) k_adj_source(double2* __restrict__ ae, double2* __restrict__ ah, Geo g,
                                                    const double2* __restrict__ fd, long P, AdjFace f,
                                                    const double* __restrict__ w, const double* __restrict__ fw,
                                                    int nof, int t) {
  extern __shared__ double2 tw[];
  for (int iw = threadIdx.x; iw < nof; iw += blockDim.x) {
    double s, c;
    sincos(fw[iw] * (double)t, &s, &c);
    tw[iw] = make_double2(w[iw] * c, -w[iw] * s);
  }
  __syncthreads();
  const long L = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (L >= f.n) return;
  double2 gex = {0, 0}, gey = {0, 0}, ghx = {0, 0}, ghy = {0, 0};
  for (int iw = 0; iw < nof; ++iw) {
    const double2* row = fd + (long)iw * P + L;
    const double2 xe = row[f.b[0]], ye = row[f.b[1]], xh = row[f.b[3]], yh = row[f.b[4]];
    const double2 c = tw[iw];
    gex.x += c.x * yh.x - c.y * yh.y; gex.y += c.x * yh.y + c.y * yh.x;
    ghy.x += c.x * xe.x - c.y * xe.y; ghy.y += c.x * xe.y + c.y * xe.x;
    gey.x -= c.x * xh.x - c.y * xh.y; gey.y -= c.x * xh.y + c.y * xh.x;
    ghx.x -= c.x * ye.x - c.y * ye.y; ghx.y -= c.x * ye.y + c.y * ye.x;
  }
  const long i = g.at(f.x0 + (int)(L % f.nu), f.y0 + (int)(L / f.nu), f.z);
  auto addv = [](double2* p, double2 v) {
    double2 o = *p;
    o.x += v.x;
    o.y += v.y;
    *p = o;
  };
  addv(ae + i, gex);
  addv(ae + g.comp + i, gey);
  addv(ah + i, ghx);
  addv(ah + g.comp + i, ghy);
}

// FP32 mode forms the same sums for a block of sampled steps at a time, in
// integers.  A step's sum over 64 frequencies of 25600 points is 26 million
// FP64 multiply-adds, and half as many conversions of the double-float
// accumulators: at two FP64 lanes a cycle an SM, 231 us a step, half of a
// backward pass on 160x160x352.  Here the accumulators of a point (a component
// of a face point) are scaled by one power of two to 56-bit fixed point, as
// the twiddles are, both as two limbs of 28 bits: three 32 x 32 -> 64 bit
// integer multiply-adds a product, exact; the product of the two low limbs is
// left out (2^-58 of the point's largest term).  24 us a step.
// Error of a sum against long double, relative to the sum, rms over random
// spectra of 1, 8, 64 and 128 frequencies whose amplitudes spread over e^+-3:
// 7e-17, 7e-17, 1.1e-16 and 1.5e-16; of FP64 multiply-adds 8e-17, 1.1e-16,
// 2.1e-16 and 4.7e-16.
constexpr int SRC_M = 8;                // steps of a thread
constexpr int SRC_CHUNK = 64;           // frequencies an integer sum holds: terms below 2^56.5
constexpr size_t SRC_BYTES = 32 << 20;  // bound on a block's sums
constexpr int SRC_MAX = 64;             // and on its steps

// The frequencies' weights as g[iw] c, |c| <= 1, g = 2^k relative to the
// largest: g[iw] and, per step j of the block (sampled DFT index t0 - j dt),
// the limbs of c exp(-i fw t): (re 1, re 2, im 1, im 2).
__device__ __forceinline__ int2 limbs56(double v) {
  const long long q = llrint(v * 0x1p56), h = (q + (1ll << 27)) >> 28;
  return make_int2((int)h, (int)(q - (h << 28)));
}
__global__ void __launch_bounds__(128) k_adj_twiddle(int4* __restrict__ tw, float* __restrict__ gw,
                                                     const double* __restrict__ w, int kmax,
                                                     const double* __restrict__ fw, int nof, int t0, int dt, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * nof) return;
  const int j = i / nof, iw = i - j * nof;
  int k;
  const double m = frexp(w[iw], &k);
  double s, c;
  sincos(fw[iw] * (double)(t0 - j * dt), &s, &c);
  const int2 re = limbs56(m * c), im = limbs56(-m * s);
  tw[i] = make_int4(re.x, re.y, im.x, im.y);
  if (j == 0) gw[iw] = m == 0.0 ? 0.f : isfinite(m) ? ldexpf(1.f, k - kmax) : __int_as_float(0x7fc00000);
}

// Component q of the source reads component 4 - q (q = 0), 3, 1, 0 of the DFT.
__device__ __forceinline__ long adj_from(const AdjFace& f, int q) { return q == 0 ? f.b[4] : q == 1 ? f.b[3] : q == 2 ? f.b[1] : f.b[0]; }

// Per component and point: the exponent of the largest g |Y| (all terms below
// 2^sx), NaN if some Y or weight is not finite.
__global__ void __launch_bounds__(128) k_adj_scale(float* __restrict__ sx, const float4* __restrict__ fd, long P,
                                                   AdjFace f, const float* __restrict__ gw, int nof) {
  const long L = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (L >= f.n) return;
  const float4* y = fd + adj_from(f, blockIdx.y) + L;
  float m = 0.f;
  bool ok = true;
  for (int iw = 0; iw < nof; ++iw) {
    const float4 v = y[(long)iw * P];
    const float a = fmaxf(fabsf(v.x), fabsf(v.y));
    ok = ok && isfinite(gw[iw]) && isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w);
    m = fmaxf(m, gw[iw] * a);
  }
  int e;
  frexpf(m, &e);
  sx[blockIdx.y * f.n + L] = !ok ? __int_as_float(0x7fc00000) : m == 0.f ? 0.f : (float)max(e, -126);
}

// h + l (|h| <= 1, |l| at most half an ulp of h) in units of 2^-56, as limbs:
// h 2^28 and l 2^28 round to integers, their remainders 2^28 to others.
__device__ __forceinline__ int2 limbs_df(float h, float l) {
  h *= 0x1p28f;
  l *= 0x1p28f;
  const float q = rintf(h), p = rintf(l);
  const int lo = __float2int_rn((h - q) * 0x1p28f) + __float2int_rn((l - p) * 0x1p28f), c = (lo + (1 << 27)) >> 28;
  return make_int2(__float2int_rn(q) + __float2int_rn(p) + c, lo - (c << 28));
}

// a + b 2^-28, rounded once.
__device__ __forceinline__ double limbs_sum(long long a, long long b) {
  const long long h = a + (b >> 28);
  const double d = (double)h;
  return d + ((double)(h - (long long)d) + (double)(int)(b & 0xfffffff) * 0x1p-28);
}

// The sums of a block of n steps at the face's points, src[step][4][f.n] of
// Hy, Hx, Ey, Ex (the CTAs of a run of points, SRC_M steps each, are
// neighbours: their accumulators hit L2).
__global__ void __launch_bounds__(128) k_adj_sums(double2* __restrict__ src, const float4* __restrict__ fd, long P,
                                                  AdjFace f, const int4* __restrict__ tw, const float* __restrict__ gw,
                                                  const float* __restrict__ sx, int nof, int n, int kmax) {
  const unsigned groups = (n + SRC_M - 1) / SRC_M;
  const long L = (long)(blockIdx.x / groups) * blockDim.x + threadIdx.x;
  if (L >= f.n) return;
  const int j0 = blockIdx.x % groups * SRC_M, q = blockIdx.y;
  const float ex = sx[q * f.n + L], sc = ldexpf(1.f, isfinite(ex) ? -(int)ex : 0);
  const double back = isfinite(ex) ? ldexp(1.0, (int)ex + kmax - 56) : (double)ex;
  const float4* y = fd + adj_from(f, q) + L;
  for (int i0 = 0; i0 < nof; i0 += SRC_CHUNK) {
    long long a1r[SRC_M], a1i[SRC_M], a2r[SRC_M], a2i[SRC_M];
#pragma unroll
    for (int j = 0; j < SRC_M; ++j) a1r[j] = a1i[j] = a2r[j] = a2i[j] = 0;
    for (int iw = i0; iw < min(nof, i0 + SRC_CHUNK); ++iw) {
      const float4 v = y[(long)iw * P];
      const float g = gw[iw] * sc;
      const int2 re = limbs_df(v.x * g, v.z * g), im = limbs_df(v.y * g, v.w * g);
#pragma unroll
      for (int j = 0; j < SRC_M; ++j) {
        const int4 c = tw[(long)min(j0 + j, n - 1) * nof + iw];
        a1r[j] += (long long)c.x * re.x;
        a1r[j] += (long long)c.z * -im.x;
        a2r[j] += (long long)c.x * re.y;
        a2r[j] += (long long)c.y * re.x;
        a2r[j] += (long long)c.z * -im.y;
        a2r[j] += (long long)c.w * -im.x;
        a1i[j] += (long long)c.x * im.x;
        a1i[j] += (long long)c.z * re.x;
        a2i[j] += (long long)c.x * im.y;
        a2i[j] += (long long)c.y * im.x;
        a2i[j] += (long long)c.z * re.y;
        a2i[j] += (long long)c.w * re.x;
      }
    }
#pragma unroll
    for (int j = 0; j < SRC_M; ++j)
      if (j0 + j < n) {
        double2& o = src[((long)(j0 + j) * 4 + q) * f.n + L];
        double2 v = make_double2(limbs_sum(a1r[j], a2r[j]) * back, limbs_sum(a1i[j], a2i[j]) * back);
        if (i0) v = make_double2(o.x + v.x, o.y + v.y);
        o = v;
      }
  }
}

// One step's sums onto the adjoint fields, H's images included.
__global__ void __launch_bounds__(128) k_adj_add(float2* __restrict__ ae, float2* __restrict__ ah, Geo g, AdjFace f,
                                                 const double2* __restrict__ src, cx<float> pxm, cx<float> pym) {
  const long L = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (L >= f.n) return;
  const int x = f.x0 + (int)(L % f.nu), y = f.y0 + (int)(L / f.nu);
  const long i = g.at(x, y, f.z);
  float2* const dst[4] = {ae + i, ae + g.comp + i, ah + i, ah + g.comp + i};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const double2 v = src[q * f.n + L];
    float2 o = *dst[q];
    o.x = (float)(q == 1 || q == 2 ? (double)o.x - v.x : (double)o.x + v.x);
    o.y = (float)(q == 1 || q == 2 ? (double)o.y - v.y : (double)o.y + v.y);
    *dst[q] = o;
    if (q >= 2 && x == g.nx) st<float>(dst[q] - g.nx, cmul(pxm, cx<float>{o.x, o.y}));
    if (q >= 2 && y == g.ny) st<float>(dst[q] - g.ny * g.pitch, cmul(pym, cx<float>{o.x, o.y}));
  }
}

template <typename T> __global__ void k_adj_scatter(T* __restrict__ eps, Geo g, int hi, Design d, const T* __restrict__ v) {
  const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= d.n) return;
  const int x = d.x0 + (int)(q % d.nx), y = d.y0 + (int)((q / d.nx) % d.ny), z = d.z0 + (int)(q / ((long)d.nx * d.ny));
  eps[(long)(z - hi) * g.plane + (long)y * g.pitch + (x + g.xo)] = v[q];
}

}  // namespace
}  // namespace iris

struct iris_adjoint {
  iris_engine* F = nullptr;  // forward engine (z-face DFT of box 1)
  iris_engine* A = nullptr;  // adjoint state: e, h, pml_d, pml_b
  void* acoef = nullptr;     // adjoint UPML rows
  Design d{};
  int K = 256;                 // checkpoint interval
  std::vector<double> w;       // [2][nof] objective weights
  double* d_w = nullptr;       // [2][nof] weight * sign * flux scale * dt
  bool side_on[2] = {false, false};
  double* d_grad = nullptr;    // [n]
  void* rec = nullptr;         // [K][3][n]
  int rec_seg = -1;            // segment whose curls rec holds
  void* d_design = nullptr;    // [n] staging for set_design
  // FP32: the DFT sources of a block of src_n sampled steps (src_cap at most)
  // from step src_it down, and their twiddles, per side
  double2* d_src[2] = {nullptr, nullptr};
  int4* d_stw[2] = {nullptr, nullptr};
  float* d_sgw[2] = {nullptr, nullptr};  // the weights' powers of two, the points' exponents
  float* d_ssx[2] = {nullptr, nullptr};
  int kmax[2] = {0, 0};                  // the largest weight's exponent
  bool src_scaled = false;               // d_ssx holds the forward pass's
  int src_cap = 1, src_it = 0, src_n = 0;
  // FP32: the step's march, its slab kernels on st2 beside it
  bool marched = false;
  cudaStream_t st2 = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  std::vector<void*> ckpt;     // per segment: e, h, d0, d1, b0, b1
  size_t fbytes = 0, sbytes[2] = {0, 0};
  int nsteps = 0;
  double ms[3] = {0, 0, 0};
  cudaEvent_t ev[2] = {nullptr, nullptr};
};

namespace {

template <typename T> AdjArgs<T> adj_args(const iris_adjoint* J, bool first, int slot, bool grad) {
  AdjArgs<T> A{};
  A.f = field_args<T>(J->A);
  const FieldArgs<T> f = field_args<T>(J->F);
  A.f.coef = (const T*)J->acoef;
  A.f.eps_r = f.eps_r;
  A.f.eps_c = nullptr;
  auto conj = [](cx<T> c) { return cx<T>{c.re, -c.im}; };
  A.f.pxm = conj(f.pxp);
  A.f.pym = conj(f.pyp);
  A.f.pzm = conj(f.pzp);
  A.f.pxp = conj(f.pxm);
  A.f.pyp = conj(f.pym);
  A.f.pzp = conj(f.pzm);
  A.d = J->d;
  A.eo = A.f.e;
  A.ho = A.f.h;
  A.z2 = 0;
  A.z3 = -1;
  A.first = first ? 1 : 0;
  if (grad) {
    A.grad = J->d_grad;
    A.rec = (const typename V2<T>::t*)J->rec + (long)slot * 3 * J->d.n;
  }
  return A;
}

template <typename T> void adj_record(iris_adjoint* J, int slot) {
  iris_engine* F = J->F;
  using V = typename V2<T>::t;
  V* r = (V*)J->rec + (long)slot * 3 * J->d.n;
  k_adj_record<T><<<(unsigned)((J->d.n + 255) / 256), 256, 0, F->st>>>(field_args<T>(F), J->d, r);
}

// The DFT source of forward step it, a sampled one.
template <typename T> void adj_source(iris_adjoint* J, int it) {
  iris_engine* F = J->F;
  const FaceMap& M = F->fm[0][2];
  const iris_params& p = F->p;
  const int t = it + 1 - p.to_fourier, sf = p.sample_fourier;
  const bool refill = F->prec == IRIS_FP32 && (J->src_n == 0 || it > J->src_it || it <= J->src_it - J->src_n * sf);
  if (refill) {
    J->src_it = it;
    J->src_n = std::min(J->src_cap, (it - std::max(p.to_fourier, 1)) / sf + 1);
  }
  const AdjArgs<float> ph = adj_args<float>(J, false, -1, false);
  for (int side = 0; side < 2; ++side) {
    if (!J->side_on[side]) continue;
    AdjFace f{};
    for (int c = 0; c < 6; ++c) f.b[c] = M.base[side][c];
    f.n = M.nloc;
    f.nu = M.nu;
    f.x0 = p.box1[0];
    f.y0 = p.box1[2];
    f.z = side == 0 ? p.box1[4] : p.box1[5];
    if (F->prec == IRIS_FP64) {
      k_adj_source<<<(unsigned)((f.n + 255) / 256), 256, sizeof(double2) * p.nof, F->st>>>(
          (double2*)J->A->e, (double2*)J->A->h, F->g, (const double2*)F->fd, F->P, f, J->d_w + side * p.nof, F->d_fw,
          p.nof, t);
      continue;
    }
    const unsigned nb = (unsigned)((f.n + 127) / 128);
    if (refill) {
      k_adj_twiddle<<<(unsigned)((J->src_n * p.nof + 127) / 128), 128, 0, F->st>>>(
          J->d_stw[side], J->d_sgw[side], J->d_w + side * p.nof, J->kmax[side], F->d_fw, p.nof, t, sf, J->src_n);
      if (!J->src_scaled)
        k_adj_scale<<<dim3(nb, 4), 128, 0, F->st>>>(J->d_ssx[side], (const float4*)F->fd, F->P, f, J->d_sgw[side], p.nof);
      k_adj_sums<<<dim3(nb * ((J->src_n + SRC_M - 1) / SRC_M), 4), 128, 0, F->st>>>(
          J->d_src[side], (const float4*)F->fd, F->P, f, J->d_stw[side], J->d_sgw[side], J->d_ssx[side], p.nof, J->src_n,
          J->kmax[side]);
    }
    k_adj_add<<<nb, 128, 0, F->st>>>((float2*)J->A->e, (float2*)J->A->h, F->g, f,
                                     J->d_src[side] + (long)((J->src_it - it) / sf) * 4 * f.n, ph.f.pxm, ph.f.pym);
  }
  if (refill) J->src_scaled = true;
}

// Back to stepping in place.
void adj_drop_march(iris_adjoint* J) {
  cudaStreamSynchronize(J->F->st);
  cudaGetLastError();
  J->marched = false;
  if (J->A->e2) cudaFree(J->A->e2);
  if (J->A->h2) cudaFree(J->A->h2);
  J->A->e2 = J->A->h2 = nullptr;
}

// Launch shape of planes z0 .. z1 (none when z1 < z0).
dim3 adj_grid(const iris_engine* F, int z0, int z1) {
  return dim3(F->grd.x, F->grd.y, z1 < z0 ? 0u : (unsigned)((z1 - z0 + F->blk.z) / F->blk.z));
}

// One step with the planes pmlzi+2 .. pmlzf-2 marched: K1 of the planes below
// and above (on the forward engine's second stream) beside them, then K2 of
// the same planes, which reads W of both.
void adj_step_march(iris_adjoint* J, bool first, int slot) {
  iris_engine *F = J->F, *S = J->A;
  const iris_params& p = F->p;
  AdjArgs<float> a = adj_args<float>(J, first, slot, slot >= 0);
  a.eo = (float2*)S->e2;
  a.ho = (float2*)S->h2;
  a.z0 = 1;
  a.z1 = p.pmlzi + 1;
  a.z2 = p.pmlzf - 1;
  a.z3 = p.nz;
  a.images = 1;
  const int planes = a.z1 + a.z3 - a.z2 + 1;
  const dim3 gr(F->grd.x, F->grd.y, (unsigned)((planes + F->blk.z - 1) / F->blk.z));
  MarchArgs m{};
  m.f = a.f;
  m.e_new = a.eo;
  m.h_new = a.ho;
  m.tx = S->mshape.tx;
  m.ty = S->mshape.ty;
  const MarchGrad G{a.d.x0, a.d.y0, a.d.z0, a.d.nx, a.d.ny, a.d.nz, a.d.n, a.rec, a.grad};
  const int za = p.pmlzi + 2, zb = p.pmlzf - 2, zc = march_chunk(zb - za + 1);
  cudaEventRecord(J->fork, F->st);
  cudaStreamWaitEvent(J->st2, J->fork, 0);
  k_adj_h<float, true, true><<<gr, F->blk, 0, J->st2>>>(a);
  adj_march_kernel(S->mshape.id)<<<dim3(m.tx, m.ty, (zb - za + zc) / zc), MR_T, S->mshape.smem, F->st>>>(m, G, za, zb, zc);
  cudaEventRecord(J->join, J->st2);
  cudaStreamWaitEvent(F->st, J->join, 0);
  a.f.e = a.eo;  // K2 reads the new E
  k_adj_e<float, true><<<gr, F->blk, 0, F->st>>>(a);
  std::swap(S->e, S->e2);
  std::swap(S->h, S->h2);
}

// One adjoint step (K1 then K2) for forward step it; rec slot or -1.  Each
// kernel runs as the planes whose stencil stays outside the UPML slabs,
// compiled without slab code, and the rest (the slabs and their neighbours).
template <typename T> void adj_step(iris_adjoint* J, bool first, int slot) {
  iris_engine* F = J->F;
  const iris_params& p = F->p;
  const bool grad = slot >= 0;
  if (J->marched) return adj_step_march(J, first, slot);
  AdjArgs<T> a = adj_args<T>(J, first, slot, grad);
  auto k1 = [&](int z0, int z1, bool upml) {
    a.z0 = z0;
    a.z1 = z1;
    const dim3 gr = adj_grid(F, z0, z1);
    if (gr.z == 0) return;
    if (upml) k_adj_h<T, true, true><<<gr, F->blk, 0, F->st>>>(a);
    else k_adj_h<T, true, false><<<gr, F->blk, 0, F->st>>>(a);
  };
  // K1 reads planes z and z-1: free of slab code for z in [pmlzi+2, pmlzf-1]
  const int a1 = std::min(p.pmlzi + 1, p.pmlzf - 1);
  k1(1, a1, true);
  k1(a1 + 1, p.pmlzf - 1, false);
  k1(p.pmlzf, p.nz, true);
  AdjArgs<T> b = adj_args<T>(J, first, -1, false);
  auto k2 = [&](int z0, int z1, bool upml) {
    b.z0 = z0;
    b.z1 = z1;
    const dim3 gr = adj_grid(F, z0, z1);
    if (gr.z == 0) return;
    if (upml) k_adj_e<T, true><<<gr, F->blk, 0, F->st>>>(b);
    else k_adj_e<T, false><<<gr, F->blk, 0, F->st>>>(b);
  };
  // K2 reads planes z and z+1: free of slab code for z in [pmlzi+1, pmlzf-2]
  const int b2 = std::max(p.pmlzf - 2, p.pmlzi);
  k2(1, p.pmlzi, true);
  k2(p.pmlzi + 1, b2, false);
  k2(b2 + 1, p.nz, true);
}

template <typename T> void adj_finalize(iris_adjoint* J) {
  iris_engine* F = J->F;
  AdjArgs<T> a = adj_args<T>(J, false, -1, false);
  a.z0 = 1;
  a.z1 = F->p.nz;
  k_adj_h<T, false, true><<<adj_grid(F, 1, F->p.nz), F->blk, 0, F->st>>>(a);
}

int ckpt_io(iris_adjoint* J, int seg, bool save) {
  iris_engine* F = J->F;
  unsigned char* c = (unsigned char*)J->ckpt[seg];
  void* parts[6] = {F->e, F->h, F->pml_d[0], F->pml_d[1], F->pml_b[0], F->pml_b[1]};
  const size_t sz[6] = {J->fbytes, J->fbytes, J->sbytes[0], J->sbytes[1], J->sbytes[0], J->sbytes[1]};
  size_t off = 0;
  for (int k = 0; k < 6; ++k) {
    if (save) CK(cudaMemcpyAsync(c + off, parts[k], sz[k], cudaMemcpyDeviceToDevice, F->st));
    else CK(cudaMemcpyAsync(parts[k], c + off, sz[k], cudaMemcpyDeviceToDevice, F->st));
    off += sz[k];
  }
  return IRIS_OK;
}

int zero_state(iris_engine* E, size_t fbytes, const size_t* sbytes) {
  CK(cudaMemsetAsync(E->e, 0, fbytes, E->st));
  CK(cudaMemsetAsync(E->h, 0, fbytes, E->st));
  for (int s = 0; s < 2; ++s) {
    CK(cudaMemsetAsync(E->pml_d[s], 0, sbytes[s], E->st));
    CK(cudaMemsetAsync(E->pml_b[s], 0, sbytes[s], E->st));
  }
  return IRIS_OK;
}

// Second buffers and launch of the march, where its offsets reach, there are
// planes to march and memory allows.
void adj_setup_march(iris_adjoint* J) {
  iris_engine* S = J->A;
  const iris_params& p = J->F->p;
  if (J->F->prec != IRIS_FP32 || 3 * S->g.comp >= (1L << 31) || p.pmlzf - 2 < p.pmlzi + 2) return;
  const MarchShape ms = march_shape(p.nx, p.ny);
  if (ms.ty > MR_MAX_ROWS) return;
  S->mshape = ms;
  int lo = 0, hi = 0;
  cudaDeviceGetStreamPriorityRange(&lo, &hi);
  J->marched = cudaMalloc(&S->e2, J->fbytes) == cudaSuccess && cudaMalloc(&S->h2, J->fbytes) == cudaSuccess &&
               cudaMemsetAsync(S->e2, 0, J->fbytes, J->F->st) == cudaSuccess &&
               cudaMemsetAsync(S->h2, 0, J->fbytes, J->F->st) == cudaSuccess &&
               cudaStreamCreateWithPriority(&J->st2, cudaStreamNonBlocking, hi) == cudaSuccess &&
               cudaEventCreateWithFlags(&J->fork, cudaEventDisableTiming) == cudaSuccess &&
               cudaEventCreateWithFlags(&J->join, cudaEventDisableTiming) == cudaSuccess &&
               cudaFuncSetAttribute((const void*)adj_march_kernel(S->mshape.id),
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S->mshape.smem) == cudaSuccess;
  if (!J->marched) adj_drop_march(J);
}

template <typename T> int adj_forward(iris_adjoint* J, int nsteps) {
  iris_engine* F = J->F;
  const int S = (nsteps + J->K - 1) / J->K;
  const size_t cbytes = 2 * J->fbytes + 2 * (J->sbytes[0] + J->sbytes[1]);
  while ((int)J->ckpt.size() < S) {
    void* q = nullptr;
    cudaError_t e = cudaMalloc(&q, cbytes);
    if (e != cudaSuccess && J->marched) {
      // the checkpoints come first: step in place, without the second buffers
      cudaGetLastError();
      adj_drop_march(J);
      e = cudaMalloc(&q, cbytes);
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(IRIS_ENOMEM, "checkpoint allocation failed (" + std::to_string(S) + " checkpoints of " +
                                   std::to_string(cbytes) + " bytes)");
    }
    J->ckpt.push_back(q);
  }
  int rc = zero_state(F, J->fbytes, J->sbytes);
  if (rc) return rc;
  CK(cudaMemsetAsync(F->fd, 0, (size_t)F->P * F->p.nof * 16, F->st));
  F->fd_zero = false;
  F->nslot = 0;
  F->tf_end = 0;
  CK(cudaEventRecord(J->ev[0], F->st));
  for (int it = 1; it <= nsteps; ++it) {
    const int seg = (it - 1) / J->K;
    if ((it - 1) % J->K == 0) {
      rc = ckpt_io(J, seg, true);
      if (rc) return rc;
    }
    if (seg == S - 1) adj_record<T>(J, it - 1 - seg * J->K);
    one_step(F, it, nsteps + 1 - it, true);
  }
  dft_flush(F);
  CK(cudaEventRecord(J->ev[1], F->st));
  CK(cudaEventSynchronize(J->ev[1]));
  float x = 0.f;
  CK(cudaEventElapsedTime(&x, J->ev[0], J->ev[1]));
  J->ms[0] = x;
  J->rec_seg = S - 1;
  J->nsteps = nsteps;
  CK(cudaGetLastError());
  return IRIS_OK;
}

template <typename T> int adj_backward(iris_adjoint* J) {
  iris_engine* F = J->F;
  const iris_params& p = F->p;
  const int N = J->nsteps, S = (N + J->K - 1) / J->K;
  int rc = zero_state(J->A, J->fbytes, J->sbytes);
  if (rc) return rc;
  CK(cudaMemsetAsync(J->d_grad, 0, sizeof(double) * J->d.n, F->st));
  J->src_n = 0;
  J->src_scaled = false;
  double t_rec = 0, t_adj = 0;
  bool first = true;
  for (int seg = S - 1; seg >= 0; --seg) {
    const int s0 = seg * J->K + 1, s1 = std::min(N, (seg + 1) * J->K);
    float x = 0.f;
    if (J->rec_seg != seg) {
      CK(cudaEventRecord(J->ev[0], F->st));
      rc = ckpt_io(J, seg, false);
      if (rc) return rc;
      F->tf_end = 0;
      for (int it = s0; it <= s1; ++it) {
        adj_record<T>(J, it - s0);
        one_step(F, it, s1 + 1 - it, false);
      }
      CK(cudaEventRecord(J->ev[1], F->st));
      CK(cudaEventSynchronize(J->ev[1]));
      CK(cudaEventElapsedTime(&x, J->ev[0], J->ev[1]));
      t_rec += x;
      J->rec_seg = seg;
    }
    CK(cudaEventRecord(J->ev[0], F->st));
    for (int it = s1; it >= s0; --it) {
      if (it >= p.to_fourier && it % p.sample_fourier == 0) adj_source<T>(J, it);
      adj_step<T>(J, first, it - s0);
      first = false;
    }
    CK(cudaEventRecord(J->ev[1], F->st));
    CK(cudaEventSynchronize(J->ev[1]));
    CK(cudaEventElapsedTime(&x, J->ev[0], J->ev[1]));
    t_adj += x;
  }
  J->ms[1] = t_rec;
  J->ms[2] = t_adj;
  CK(cudaGetLastError());
  return IRIS_OK;
}

void adj_free(iris_adjoint* J) {
  if (J->F) iris_destroy(J->F);
  if (J->A) iris_destroy(J->A);
  void* ptrs[] = {J->acoef, J->d_w, J->d_grad, J->rec, J->d_design, J->d_src[0], J->d_src[1],
                  J->d_stw[0], J->d_stw[1], J->d_sgw[0], J->d_sgw[1], J->d_ssx[0], J->d_ssx[1]};
  for (void* q : ptrs)
    if (q) cudaFree(q);
  for (void* q : J->ckpt)
    if (q) cudaFree(q);
  for (cudaEvent_t e : {J->ev[0], J->ev[1], J->fork, J->join})
    if (e) cudaEventDestroy(e);
  if (J->st2) cudaStreamDestroy(J->st2);
}

}  // namespace

extern "C" {

int iris_adjoint_create(const iris_params* pin, const double* fw, const int design[6], int checkpoint_every,
                        const double* weights, iris_adjoint** out) {
  clear_error();
  if (!pin || !fw || !design || !out) return fail(IRIS_EINVAL, "null argument");
  *out = nullptr;
  const iris_params& p = *pin;
  if (checkpoint_every < 1) return fail(IRIS_EINVAL, "checkpoint_every must be >= 1");
  const int* D = design;
  if (D[0] < 1 || D[1] > p.nx || D[0] > D[1] || D[2] < 1 || D[3] > p.ny || D[2] > D[3] || D[4] < p.hi ||
      D[5] > p.hf || D[4] > D[5])
    return fail(IRIS_EINVAL, "design region must lie in [1,nx] x [1,ny] x [hi,hf]");
  if (p.hi <= p.pmlzi || p.hf >= p.pmlzf) return fail(IRIS_EINVAL, "the structure layer must lie outside the UPML slabs");
  if (p.box1[4] <= p.pmlzi || p.box1[5] >= p.pmlzf)
    return fail(IRIS_EINVAL, "the DFT z planes of box 1 must lie outside the UPML slabs");
  iris_adjoint* J = new iris_adjoint();
  auto bail = [&](int code) {
    adj_free(J);
    delete J;
    return code;
  };
  // the forward engine steps as the parameters ask (FP32: the fused pass by
  // default); the adjoint state is a member engine that only holds fields
  iris_params q = p;
  for (int i = 0; i < 6; ++i) q.box2[i] = q.box1[i];
  int rc = create_engine(&q, fw, false, true, &J->F);
  if (rc) return bail(rc);
  q.stencil = IRIS_STENCIL_SPLIT;
  rc = create_engine(&q, fw, true, true, &J->A);
  if (!rc) rc = tfsf_alloc(J->A, 16);  // callers may step it (iris_adjoint_engine)
  if (rc) return bail(rc);
  J->A->P = 0;  // it has no DFT buffers
  iris_engine* F = J->F;
  J->K = checkpoint_every;
  J->d = Design{D[0], D[2], D[4], D[1] - D[0] + 1, D[3] - D[2] + 1, D[5] - D[4] + 1, 0};
  J->d.n = (long)J->d.nx * J->d.ny * J->d.nz;
  J->fbytes = (size_t)3 * F->g.comp * F->esz;
  for (int s = 0; s < 2; ++s) J->sbytes[s] = (size_t)3 * F->pcomp[s] * F->esz;
  // objective weights, folded with the flux sign and scale and the DFT's dt
  const int nof = p.nof;
  J->w.assign(2 * (size_t)nof, 0.0);
  for (int k = 0; k < nof; ++k) J->w[nof + k] = 1.0;
  if (weights) J->w.assign(weights, weights + 2 * nof);
  std::vector<double> wd(2 * (size_t)nof);
  const double scale = p.eps0 * p.Q / (2.0 * p.dt);
  double wmax[2] = {0, 0};
  for (int side = 0; side < 2; ++side)
    for (int k = 0; k < nof; ++k) {
      const double v = J->w[side * nof + k];
      wd[side * nof + k] = (side == 0 ? -1.0 : 1.0) * scale * p.dt * v;
      if (v != 0.0) J->side_on[side] = true;
      if (v != 0.0 && std::isfinite(wd[side * nof + k])) wmax[side] = std::max(wmax[side], std::fabs(wd[side * nof + k]));
    }
  // adjoint UPML rows from the forward ones
  const std::vector<double>& c = F->coef_h;
  const size_t nrow = c.size() / NCOEF;
  std::vector<double> ac(c.size());
  const double e2 = p.eps0 * p.eps0;
  for (size_t r = 0; r < nrow; ++r) {
    const double* f = c.data() + NCOEF * r;
    double* a = ac.data() + NCOEF * r;
    for (int k = 0; k < 3; ++k) {
      a[AJ_A + k] = f[CD_A + k];
      a[AJ_AL + k] = f[CE_A + k];
      a[AJ_GE + k] = f[CE_B + k] * (f[C_FP + k] * f[CD_A + k] - f[C_FM + k]);
      a[AJ_BE + k] = f[CE_B + k] * f[C_FP + k] * f[CD_B + k] * e2;
      a[AJ_DE + k] = f[CD_B + k] * e2;
      a[AJ_GH + k] = f[CH_B + k] * (f[C_FP + k] * f[CD_A + k] - f[C_FM + k]);
      a[AJ_BH + k] = -f[CH_B + k] * f[C_FP + k] * f[CB_B + k];
      a[AJ_DH + k] = -f[CB_B + k];
    }
  }
  const size_t rsz = F->prec == IRIS_FP64 ? 8 : 4;
  const size_t csz = F->prec == IRIS_FP64 ? 16 : 8;
  auto dev_alloc = [&](void** q2, size_t b) { return cudaMalloc(q2, std::max<size_t>(b, 16)) == cudaSuccess; };
  if (!dev_alloc(&J->acoef, ac.size() * rsz) || !dev_alloc((void**)&J->d_w, sizeof(double) * 2 * nof) ||
      !dev_alloc((void**)&J->d_grad, sizeof(double) * J->d.n) ||
      !dev_alloc(&J->rec, (size_t)J->K * 3 * J->d.n * csz) || !dev_alloc(&J->d_design, J->d.n * rsz)) {
    cudaGetLastError();
    return bail(fail(IRIS_ENOMEM, "adjoint buffers: allocation failed"));
  }
  if (F->prec == IRIS_FP32) {
    for (int side = 0; side < 2; ++side) std::frexp(wmax[side], &J->kmax[side]);
    const size_t one = 4 * sizeof(double2) * F->fm[0][2].nloc;
    J->src_cap = (int)std::max<size_t>(1, std::min<size_t>(SRC_MAX, SRC_BYTES / std::max<size_t>(1, one)));
    for (int side = 0; side < 2; ++side)
      if (J->side_on[side] && (!dev_alloc((void**)&J->d_src[side], J->src_cap * one) ||
                               !dev_alloc((void**)&J->d_stw[side], J->src_cap * sizeof(int4) * nof) ||
                               !dev_alloc((void**)&J->d_sgw[side], sizeof(float) * nof) ||
                               !dev_alloc((void**)&J->d_ssx[side], 4 * sizeof(float) * F->fm[0][2].nloc))) {
        cudaGetLastError();
        return bail(fail(IRIS_ENOMEM, "adjoint buffers: allocation failed"));
      }
  }
  if (F->prec == IRIS_FP64) {
    if (cudaMemcpy(J->acoef, ac.data(), ac.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess)
      return bail(fail(IRIS_ECUDA, "adjoint rows upload failed"));
  } else {
    std::vector<float> af(ac.begin(), ac.end());
    if (cudaMemcpy(J->acoef, af.data(), af.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess)
      return bail(fail(IRIS_ECUDA, "adjoint rows upload failed"));
  }
  if (cudaMemcpy(J->d_w, wd.data(), sizeof(double) * 2 * nof, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaEventCreate(&J->ev[0]) != cudaSuccess || cudaEventCreate(&J->ev[1]) != cudaSuccess)
    return bail(fail(IRIS_ECUDA, "adjoint initialisation failed"));
  adj_setup_march(J);
  *out = J;
  return IRIS_OK;
}

void iris_adjoint_destroy(iris_adjoint* J) {
  if (!J) return;
  cudaSetDevice(J->F ? J->F->device : 0);
  if (J->F) cudaStreamSynchronize(J->F->st);
  adj_free(J);
  delete J;
}

int iris_adjoint_set_material(iris_adjoint* J, const double* re, const double* im) {
  clear_error();
  if (!J || !re) return fail(IRIS_EINVAL, "null argument");
  int rc = iris_set_material(J->F, re, im);
  if (rc) return rc;
  if (J->F->eps_complex) return fail(IRIS_EINVAL, "the adjoint form needs a real material");
  return IRIS_OK;
}

int iris_adjoint_set_design(iris_adjoint* J, const double* v) {
  clear_error();
  if (!J || !v) return fail(IRIS_EINVAL, "null argument");
  iris_engine* F = J->F;
  CK(cudaSetDevice(F->device));
  if (F->eps_complex) return fail(IRIS_EINVAL, "the adjoint form needs a real material");
  const unsigned nb = (unsigned)((J->d.n + 255) / 256);
  if (F->prec == IRIS_FP64) {
    CK(cudaMemcpyAsync(J->d_design, v, sizeof(double) * J->d.n, cudaMemcpyHostToDevice, F->st));
    k_adj_scatter<double><<<nb, 256, 0, F->st>>>((double*)F->eps, F->g, F->p.hi, J->d, (const double*)J->d_design);
  } else {
    std::vector<float> f(v, v + J->d.n);
    CK(cudaMemcpyAsync(J->d_design, f.data(), sizeof(float) * J->d.n, cudaMemcpyHostToDevice, F->st));
    k_adj_scatter<float><<<nb, 256, 0, F->st>>>((float*)F->eps, F->g, F->p.hi, J->d, (const float*)J->d_design);
  }
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(F->st));
  return IRIS_OK;
}

int iris_adjoint_forward(iris_adjoint* J, int nsteps, double* L, double* Jout) {
  iris::NvtxRange nvtx_("iris_adjoint_forward");
  clear_error();
  if (!J || nsteps < 1) return fail(IRIS_EINVAL, "bad argument");
  iris_engine* F = J->F;
  CK(cudaSetDevice(F->device));
  if (F->eps_complex) return fail(IRIS_EINVAL, "the adjoint form needs a real material");
  int rc = F->prec == IRIS_FP64 ? adj_forward<double>(J, nsteps) : adj_forward<float>(J, nsteps);
  if (rc) return rc;
  const int nof = F->p.nof;
  std::vector<double> flux(6 * (size_t)nof);
  rc = iris_flux(F, 0, flux.data());
  if (rc) return rc;
  double s = 0.0;
  for (int k = 0; k < nof; ++k) s += J->w[k] * flux[4 * nof + k] + J->w[nof + k] * flux[5 * nof + k];
  if (L) *L = s;
  if (Jout) std::copy(flux.begin(), flux.end(), Jout);
  return IRIS_OK;
}

int iris_adjoint_backward(iris_adjoint* J, double* grad) {
  iris::NvtxRange nvtx_("iris_adjoint_backward");
  clear_error();
  if (!J || !grad) return fail(IRIS_EINVAL, "null argument");
  if (J->nsteps < 1) return fail(IRIS_EINVAL, "no forward solve to differentiate");
  iris_engine* F = J->F;
  CK(cudaSetDevice(F->device));
  int rc = F->prec == IRIS_FP64 ? adj_backward<double>(J) : adj_backward<float>(J);
  if (rc) return rc;
  CK(cudaMemcpyAsync(grad, J->d_grad, sizeof(double) * J->d.n, cudaMemcpyDeviceToHost, F->st));
  CK(cudaStreamSynchronize(F->st));
  for (long q = 0; q < J->d.n; ++q)
    if (!std::isfinite(grad[q])) return fail(IRIS_ENAN, "non-finite gradient");
  return IRIS_OK;
}

int iris_adjoint_engine(iris_adjoint* J, int which, iris_engine** eng) {
  if (!J || !eng || (which != 0 && which != 1)) return fail(IRIS_EINVAL, "bad argument");
  *eng = which == 0 ? J->F : J->A;
  return IRIS_OK;
}

int iris_adjoint_apply(iris_adjoint* J, int nsteps) {
  clear_error();
  if (!J || nsteps < 0) return fail(IRIS_EINVAL, "bad argument");
  iris_engine* F = J->F;
  CK(cudaSetDevice(F->device));
  CK(cudaStreamSynchronize(J->A->st));
  const bool d = F->prec == IRIS_FP64;
  if (J->marched && nsteps > 0) {  // the caller's state may hold any images
    const AdjArgs<float> a = adj_args<float>(J, false, -1, false);
    k_adj_images<float><<<F->grd, F->blk, 0, F->st>>>(a);
  }
  for (int k = 0; k < nsteps; ++k) d ? adj_step<double>(J, k == 0, -1) : adj_step<float>(J, k == 0, -1);
  if (nsteps > 0) d ? adj_finalize<double>(J) : adj_finalize<float>(J);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(F->st));
  return IRIS_OK;
}

int iris_adjoint_timing(const iris_adjoint* J, double* ms) {
  if (!J || !ms) return fail(IRIS_EINVAL, "bad argument");
  for (int k = 0; k < 3; ++k) ms[k] = J->ms[k];
  return IRIS_OK;
}

}  // extern "C"
