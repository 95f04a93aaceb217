// The resident persistent kernel: small grids whose E and H fit in the SMs'
// shared memory step there for a whole span.  Not part of the public ABI.
#pragma once
#include <cuda_runtime.h>

#include "iris_device.cuh"

namespace iris {

// k_res: a span of steps in one cooperative launch, like k_tiny, with the
// state in shared memory instead of the L2.
//
// Ownership.  The grid is a list of rows (x runs) in (z, y) order; CTA c owns
// rows [r0, r1), E and H of its cells in shared memory: planes of
// [row][x = 0 .. nx+1], the x ghosts included (H at x = 0, E at x = nx+1), and
// D, B and the coefficients of its UPML rows (a UPML row takes about twice the
// memory and time of another, so CTAs in the slabs own about half the rows).
// When six components do not fit, E_x stays in its global array (NC = 5); when
// D and B do not, they do (db = 0).  y and z neighbours lie within ny rows: own rows are read from shared
// memory, the others from the global field arrays, where every CTA publishes
// the rows its neighbours read.  Bloch images in y and z are formed on the
// fly from the row they are images of; a phase of exactly 1 is a copy (on
// GB300 the FP64 products of the ghosts cost as much as the update).
//
// Order.  A phase first does the rows whose neighbours are all its own; a warp
// about to read other CTAs' rows waits for their flags of the phase before
// (one arrival word a CTA, release / acquire, bounded); the CTA ends the phase
// with one barrier and sets its flag: no grid-wide barrier, and the flags'
// latency (about a microsecond) hides behind the first part.  The neighbour relation is symmetric, so a CTA
// past its wait also knows that the rows it published for the phase before
// have been read.
//
// LL (FP64, every CTA's phase a single round of its threads: small grids,
// bound by the latency of this exchange): no flags and no rows in the global
// arrays; every number another CTA reads is published as a 16-byte packet with
// its step's tag, and the lane that needs it polls for it.  A phase then
// waits for one store to become visible instead of the CTA's last store, a
// barrier, a release and the load behind the acquire.  A packet needs one
// place only: the number it is a function of next is published back by the
// lanes that read it, and the lane that overwrites it has read all of those
// (curl E and curl H are transposes of one another).  A lane reads the packet
// of its own part p, or both parts where the row it reads is a Bloch image
// with a phase, and the two directions across a border agree on which
// (res_ll_ask); what a complex material needs of the other part comes from the
// neighbouring lane, so a number's publication follows from the reads of both
// lanes of its pair, not from their running in step.  The same order keeps a
// span's last H phase from overwriting ghosts that its first E phase still
// reads.  4x4x512: 5.9 us a step before, 4.4 so; 1x1x400 5.7 and 4.4.
//
// TF/SF.  The H correction is added as the H phase stores (nothing else reads
// that H in the phase); the E correction of step i is added when step i+1's E
// phase loads the cell, because the H phase reads E uncorrected, and to the
// samples and the final state.  Ghost cells that are corrected but never
// rewritten by a Bloch copy are accumulated at the end of the span, step by
// step.  All stored values equal the split passes' bit for bit.
//
// What bounds it: FP64, the FP64 pipes and the dependent chain of one number;
// FP32, instruction issue and shared-memory bandwidth (about 30 8-byte
// accesses a cell and step).

struct ResCta {
  int r0, r1;       // rows owned
  int nb0, nbn;     // neighbour CTAs: nbn of them from nb0 on, modulo the grid
  unsigned s0, sh, s1;  // sample points: E [s0, sh), H [sh, s1)
};

// TF/SF corrections as the phases apply them: component and plane of the E
// and the H correction, their sign, and whether the ghost column nx+1 and
// the ghost row ny+1 are in their range.
struct ResSrc {
  int on, cE, zE, cH, zH, sgn, gx, gy;
};

constexpr int RES_THREADS = 1024;    // threads a CTA at most
constexpr int RES_LL_THREADS = 512;  // LL (more registers a thread)
constexpr int RES_FLAG_STRIDE = 32;  // words between two CTAs' flags (128 bytes)
constexpr unsigned RES_GLOBAL = 1u << 30, RES_CORR = 1u << 31;

template <typename T> struct ResArgs {
  FieldArgs<T> a;
  ResSrc s;
  const TfsfVal<T>* tfv;  // TF/SF corrections per [step of the span][ix in 0..nx+1]
  const ResCta* cta;
  const uint2* samp;   // (element offset in shared memory | flags, ring position)
  typename V2<T>::t* S;
  long P;
  int* tk;
  int slot0, it0, n;
  int to_fourier, sample_fourier, dft;
  int db;              // D and B of the UPML rows in shared memory
  int rows, head;      // rows of the row tables, and their bytes
  int runs, nruns;     // FP32: warps take 32-cell runs of rows; entries of a run table
  int one[3];          // Bloch phase of x, y, z exactly 1
  unsigned* flag;
  int* err;
  ulonglong2* ll;          // LL: the packets, [E, H][component][storage index][part]
  unsigned long long ep;   // LL: tag of the step before the first
};

// The flag of a CTA and the wait for its neighbours' flags.
__device__ __forceinline__ unsigned res_ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void res_st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The calling warp waits until every neighbour has finished phase `want`;
// false (and the error word set) when it gave up.
__device__ __forceinline__ bool res_wait_warp(const unsigned* flag, int nb0, int nbn, unsigned want, int* err,
                                              long long limit) {
  bool ok = true;
  for (int l = (int)threadIdx.x & 31; l < nbn; l += 32) {
    int c = nb0 + l;
    if (c >= (int)gridDim.x) c -= (int)gridDim.x;
    const unsigned* f = flag + (long)c * RES_FLAG_STRIDE;
    if ((int)(res_ld_acquire(f) - want) >= 0) continue;
    const long long t0 = clock64();
    while ((int)(res_ld_acquire(f) - want) < 0)
      if (clock64() - t0 > limit) {
        ok = false;
        break;
      }
  }
  ok = __all_sync(0xffffffffu, ok);
  if (!ok && (threadIdx.x & 31) == 0) atomicExch(err, 6);
  __syncwarp();
  return ok;
}

// A field value written by another CTA: from L2 (own rows of E_x under NC = 5
// are read through L1, which this SM's own stores keep up to date).
__device__ __forceinline__ cx<float> ld_l2(const float2* p) {
  const float2 v = __ldcg(p);
  return {v.x, v.y};
}
__device__ __forceinline__ cx<double> ld_l2(const double2* p) {
  const double2 v = __ldcg(p);
  return {v.x, v.y};
}

// A Bloch image, rounded as cmul is where its result is stored: in FP32 the
// compiler would otherwise contract the product into the sum that uses it.
__device__ __forceinline__ cx<double> res_ph(bool one, cx<double> ph, cx<double> v) { return one ? v : cmul(ph, v); }
__device__ __forceinline__ cx<float> res_ph(bool one, cx<float> p, cx<float> v) {
  if (one) return v;
  return {__fmaf_rn(p.re, v.re, -__fmul_rn(p.im, v.im)), __fmaf_rn(p.im, v.re, __fmul_rn(p.re, v.im))};
}

// How a phase reads a row's neighbours and what it does with its results: in
// shared memory, filled once by the CTA (the E rows again after the first
// step, whose images come from the stored ghosts).
enum {
  RF_ZG = 1,      // the z neighbour row is read from the global arrays
  RF_YG = 2,      // the y neighbour row likewise
  RF_ZP = 4,      // ... and is a Bloch image with a phase other than 1
  RF_YP = 8,
  RF_PUB = 16,    // other CTAs read this row
  RF_UPML = 32,
  RF_MAT = 64,    // structure plane (E)
  RF_SUB = 128,   // above the structure: 1/eps3 (E)
  RF_CORR = 256,  // a TF/SF correction applies
  RF_PUB2 = 1024, // ... across y, which reads component 2 too
  RF_GHOST = 512  // the last step leaves y or z ghosts (H)
};
struct __align__(16) ResRow {
  int fl;      // RF_*
  int gb;      // storage index of x = 0
  int zo, yo;  // neighbour rows: offset from the cell in shared memory or in storage
};

// One CTA's view of the grid and of its shared memory.
template <typename T, int NC> struct ResView {
  using V = typename V2<T>::t;
  V* sm;
  ResRow* er;          // E phase rows
  ResRow* hr;          // H phase rows
  const uint2* zy;     // per own row: (z << 16) + y, and its index among the CTA's UPML rows
  V* d;                // D, then B: [component][UPML row][x - 1]
  const T* cf;         // coefficients [UPML row][NCOEF]
  int cs, W, nrows, nu;  // elements of a component; UPML rows
  __device__ __forceinline__ V* e(int k) const { return sm + (NC == 6 ? k : k - 1) * cs; }
  __device__ __forceinline__ V* h(int k) const { return sm + (NC == 6 ? 3 + k : 2 + k) * cs; }
};

// D (which = 0) or B (1) of a UPML row: f + k pc + x, x from 1, and its
// coefficients; in shared memory or in the global arrays.
template <typename T> struct ResUpml {
  typename V2<T>::t* f;
  long pc;
  const T* cf;
};
template <typename T, int NC>
__device__ __forceinline__ ResUpml<T> res_upml(const ResArgs<T>& A, const ResView<T, NC>& v, int lrow, int which) {
  const FieldArgs<T>& a = A.a;
  const uint2 zy = v.zy[lrow];
  const int nx = a.g.nx;
  if (A.db) {
    if (!bc_ok((int)zy.y < v.nu, which ? BC_H_SLAB : BC_E_SLAB, zy.y)) return {nullptr, 0, nullptr};
    return {v.d + (3 * which * v.nu + (int)zy.y) * nx - 1, (long)v.nu * nx, v.cf + NCOEF * (int)zy.y};
  }
  const int z = (int)(zy.x >> 16), y = (int)(zy.x & 0xffffu), slab = z <= a.pmlzi ? 0 : 1;
  const int zr = slab == 0 ? z - 1 : z - a.pmlzf, row = slab == 0 ? z - 1 : a.pmlzi + z - a.pmlzf;
  const long pi = ((long)zr * a.g.ny + (y - 1)) * (long)nx;
  if (!bc_ok(pi >= 0 && pi + nx <= a.pcomp[slab], which ? BC_H_SLAB : BC_E_SLAB, pi)) return {nullptr, 0, nullptr};
  return {(which ? a.pml_b[slab] : a.pml_d[slab]) + pi - 1, a.pcomp[slab], a.coef + NCOEF * row};
}

template <typename T>
__device__ __forceinline__ ResRow res_row_e(const ResArgs<T>& A, int W, int nrows, int lrow, int y, int z, bool first) {
  const FieldArgs<T>& a = A.a;
  const Geo& g = a.g;
  const int pl = (int)g.plane, pt = (int)g.pitch, ny = g.ny;
  ResRow r;
  r.fl = 0;
  r.gb = z * pl + y * pt + g.xo;
  if (lrow >= ny) {
    r.zo = -ny * W;
  } else {
    const bool img = z == 1 && !first;
    r.zo = img ? (g.nz - 1) * pl : -pl;
    r.fl |= RF_ZG | (img && !A.one[2] ? RF_ZP : 0);
  }
  const bool img = y == 1 && !first;
  const int dr = img ? ny - 1 : -1, lr = lrow + dr;
  const bool own = lr >= 0 && lr < nrows && (y > 1 || img);
  r.yo = own ? dr * W : dr * pt;
  r.fl |= (own ? 0 : RF_YG) | (img && !A.one[1] ? RF_YP : 0);
  const bool py = (lrow == 0 && y > 1) || (y == 1 && lrow + ny - 1 >= nrows);  // read across y by another CTA
  r.fl |= (lrow < ny || py ? RF_PUB : 0) | (py ? RF_PUB2 : 0);
  if (z <= a.pmlzi || z >= a.pmlzf) r.fl |= RF_UPML;
  else if (z >= a.hi && z <= a.hf) r.fl |= RF_MAT;
  else if (z > a.hf) r.fl |= RF_SUB;
  if (A.s.on && z == A.s.zE && !first) r.fl |= RF_CORR;
  return r;
}

template <typename T>
__device__ __forceinline__ ResRow res_row_h(const ResArgs<T>& A, int W, int nrows, int lrow, int y, int z) {
  const FieldArgs<T>& a = A.a;
  const Geo& g = a.g;
  const int pl = (int)g.plane, pt = (int)g.pitch, ny = g.ny;
  ResRow r;
  r.fl = 0;
  r.gb = z * pl + y * pt + g.xo;
  if (lrow + ny < nrows) {
    r.zo = ny * W;
  } else {
    const bool img = z == g.nz;
    r.zo = img ? -(g.nz - 1) * pl : pl;
    r.fl |= RF_ZG | (img && !A.one[2] ? RF_ZP : 0);
  }
  const bool img = y == ny;
  const int dr = img ? 1 - ny : 1, lr = lrow + dr;
  const bool own = lr >= 0 && lr < nrows;
  r.yo = own ? dr * W : dr * pt;
  r.fl |= (own ? 0 : RF_YG) | (img && !A.one[1] ? RF_YP : 0);
  const bool py = (lrow == nrows - 1 && y < ny) || (y == ny && lrow - ny + 1 < 0);  // read across y by another CTA
  r.fl |= (lrow + ny >= nrows || py ? RF_PUB : 0) | (py ? RF_PUB2 : 0);
  if (z <= a.pmlzi || z >= a.pmlzf) r.fl |= RF_UPML;
  if (A.s.on && z == A.s.zH) r.fl |= RF_CORR;
  if (y == ny || z == g.nz) r.fl |= RF_GHOST;
  return r;
}

// E phase of one cell in FP32: e_update with the neighbours from shared memory
// or the published rows, then the ghost at nx+1 and the rows other CTAs read.
// vE: the E correction pending from the step before.
template <bool CEPS, int NC>
__device__ __forceinline__ void res_e(const ResArgs<float>& A, const ResView<float, NC>& v, int x, int lrow,
                                      const TfsfVal<float>* vE) {
  using T = float;
  const FieldArgs<T>& a = A.a;
  const ResRow r = v.er[lrow];
  const int li = lrow * v.W + x, gi = r.gb + x, cp = (int)a.g.comp;
  if (!bc_ok(x >= 1 && x <= a.g.nx && lrow < v.nrows, BC_E_CELL, gi)) return;
  cx<T> h[3], hz0, hz1, hy0, hy2, e[3], c[3];
  if (NC == 5) e[0] = ld<float>(a.e + gi);
  if (r.fl & RF_ZG) {
    hz0 = ld_l2(a.h + (gi + r.zo));
    hz1 = ld_l2(a.h + (cp + gi + r.zo));
  } else {
    hz0 = ld<T>(v.h(0) + (li + r.zo));
    hz1 = ld<T>(v.h(1) + (li + r.zo));
  }
  if (r.fl & RF_YG) {
    hy0 = ld_l2(a.h + (gi + r.yo));
    hy2 = ld_l2(a.h + (2 * cp + gi + r.yo));
  } else {
    hy0 = ld<T>(v.h(0) + (li + r.yo));
    hy2 = ld<T>(v.h(2) + (li + r.yo));
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    h[k] = ld<T>(v.h(k) + li);
    if (NC == 6 || k > 0) e[k] = ld<T>(v.e(k) + li);
  }
  const cx<T> hx1 = ld<T>(v.h(1) + li - 1), hx2 = ld<T>(v.h(2) + li - 1);
  if (r.fl & (RF_ZP | RF_YP | RF_CORR)) {
    if (r.fl & RF_ZP) {
      hz0 = res_ph(false, a.pzm, hz0);
      hz1 = res_ph(false, a.pzm, hz1);
    }
    if (r.fl & RF_YP) {
      hy0 = res_ph(false, a.pym, hy0);
      hy2 = res_ph(false, a.pym, hy2);
    }
    if (r.fl & RF_CORR) {
      const auto t = vE[x];
      if (A.s.cE == 0) e[0] = tf_add(e[0], t.er, t.ei, A.s.sgn);
      else e[1] = tf_add(e[1], t.er, t.ei, A.s.sgn);
    }
  }
  c[0] = cadd(csub(csub(h[2], hy2), h[1]), hz1);
  c[1] = cadd(csub(csub(h[0], hz0), h[2]), hx2);
  c[2] = cadd(csub(csub(h[1], hx1), h[0]), hy0);
  if (r.fl & RF_UPML) {
    const ResUpml<T> u = res_upml(A, v, lrow, 0);
    if (!u.cf) return;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const cx<T> ck = rmul(a.eps0sq, c[k]);
      const cx<T> dold = ld<T>(u.f + k * u.pc + x);
      const cx<T> dn = cadd(rmul(u.cf[CD_A + k], dold), rmul(u.cf[CD_B + k], ck));
      st<T>(u.f + k * u.pc + x, dn);
      e[k] = cadd(rmul(u.cf[CE_A + k], e[k]),
                  rmul(u.cf[CE_B + k], csub(rmul(u.cf[C_FP + k], dn), rmul(u.cf[C_FM + k], dold))));
    }
  } else if (r.fl & RF_MAT) {
    e_apply<T, CEPS, 7, false, false>(a, a.pml_d, x, (int)(v.zy[lrow].x & 0xffffu), (int)(v.zy[lrow].x >> 16), c, e);
  } else {
    const T m = r.fl & RF_SUB ? a.m3 : a.m1;
#pragma unroll
    for (int k = 0; k < 3; ++k) e[k] = cadd(e[k], rmul(m, c[k]));
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (!(NC == 5 && k == 0)) st<T>(v.e(k) + li, e[k]);
    else st<T>(a.e + gi, e[k]);
  }
  if (r.fl & RF_PUB) {
#pragma unroll
    for (int k = NC == 5 ? 1 : 0; k < 3; ++k) st<T>(a.e + (k * cp + gi), e[k]);
  }
  if (x == 1) {
#pragma unroll
    for (int k = 1; k < 3; ++k) st<T>(v.e(k) + li + a.g.nx, res_ph(A.one[0], a.pxp, e[k]));
  }
}

// H phase of one cell in FP32: h_update likewise, the H correction of this
// step (vH), the ghost at x = 0 and the published rows.  last: the final step
// of the span also leaves the y and z ghosts of H (and their corrections) in
// the global arrays.
template <int NC>
__device__ __forceinline__ void res_h(const ResArgs<float>& A, const ResView<float, NC>& v, int x, int lrow,
                                      const TfsfVal<float>* vH, bool last) {
  using T = float;
  const FieldArgs<T>& a = A.a;
  const Geo& g = a.g;
  const ResRow r = v.hr[lrow];
  const int li = lrow * v.W + x, gi = r.gb + x, cp = (int)g.comp;
  if (!bc_ok(x >= 1 && x <= g.nx && lrow < v.nrows, BC_H_CELL, gi)) return;
  cx<T> ev[3], xp[3], yp[3], zp[3], h[3];
  if (NC == 5) ev[0] = ld<T>(a.e + gi);
  if (r.fl & RF_ZG) {
    zp[0] = ld_l2(a.e + (gi + r.zo));
    zp[1] = ld_l2(a.e + (cp + gi + r.zo));
  } else {
    zp[0] = NC == 5 ? ld<T>(a.e + (gi + (int)g.plane)) : ld<T>(v.e(0) + (li + r.zo));
    zp[1] = ld<T>(v.e(1) + (li + r.zo));
  }
  if (r.fl & RF_YG) {
    yp[0] = ld_l2(a.e + (gi + r.yo));
    yp[2] = ld_l2(a.e + (2 * cp + gi + r.yo));
  } else {
    // (NC = 5: an own y row is one row on, or ny - 1 rows back for an image)
    yp[0] = NC == 5 ? ld<T>(a.e + (gi + (r.yo > 0 ? 1 : 1 - g.ny) * (int)g.pitch)) : ld<T>(v.e(0) + (li + r.yo));
    yp[2] = ld<T>(v.e(2) + (li + r.yo));
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (NC == 6 || k > 0) ev[k] = ld<T>(v.e(k) + li);
    h[k] = ld<T>(v.h(k) + li);
  }
  xp[1] = ld<T>(v.e(1) + li + 1);
  xp[2] = ld<T>(v.e(2) + li + 1);
  if (r.fl & (RF_ZP | RF_YP)) {
    if (r.fl & RF_ZP) {
      zp[0] = res_ph(false, a.pzp, zp[0]);
      zp[1] = res_ph(false, a.pzp, zp[1]);
    }
    if (r.fl & RF_YP) {
      yp[0] = res_ph(false, a.pyp, yp[0]);
      yp[2] = res_ph(false, a.pyp, yp[2]);
    }
  }
  if (r.fl & RF_UPML) {
    const ResUpml<T> u = res_upml(A, v, lrow, 1);
    if (!u.cf) return;
    cx<T> c[3];
    c[0] = cadd(csub(csub(yp[2], ev[2]), zp[1]), ev[1]);
    c[1] = cadd(csub(csub(zp[0], ev[0]), xp[2]), ev[2]);
    c[2] = cadd(csub(csub(xp[1], ev[1]), yp[0]), ev[0]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const cx<T> bold = ld<T>(u.f + k * u.pc + x);
      const cx<T> bn = csub(rmul(u.cf[CD_A + k], bold), rmul(u.cf[CB_B + k], c[k]));
      st<T>(u.f + k * u.pc + x, bn);
      h[k] = cadd(rmul(u.cf[CE_A + k], h[k]),
                  rmul(u.cf[CH_B + k], csub(rmul(u.cf[C_FP + k], bn), rmul(u.cf[C_FM + k], bold))));
    }
  } else {
    h_update<T, false>(a, x, 1, 1, ev, xp, yp, zp, h);
  }
  auto fix = [&](cx<T>* q, int ix) {  // the correction of component cH
    const auto t = vH[ix];
    if (A.s.cH == 0) q[0] = tf_add(q[0], t.hr, t.hi, A.s.sgn);
    else q[1] = tf_add(q[1], t.hr, t.hi, A.s.sgn);
  };
  if (x == g.nx) {
    cx<T> q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) q[k] = res_ph(A.one[0], a.pxm, h[k]);
    if (r.fl & RF_CORR) fix(q, 0);
#pragma unroll
    for (int k = 0; k < 3; ++k) st<T>(v.h(k) + li - g.nx, q[k]);
  }
  if (last && (r.fl & RF_GHOST)) {
    const unsigned zy = v.zy[lrow].x;
    cx<T> q[3];
    if ((int)(zy & 0xffffu) == g.ny) {
#pragma unroll
      for (int k = 0; k < 3; ++k) q[k] = res_ph(false, a.pym, h[k]);
      if (r.fl & RF_CORR) fix(q, x);
#pragma unroll
      for (int k = 0; k < 3; ++k) st<T>(a.h + k * cp + gi - g.ny * (int)g.pitch, q[k]);
    }
    if ((int)(zy >> 16) == g.nz) {
#pragma unroll
      for (int k = 0; k < 3; ++k) st<T>(a.h + k * cp + gi - g.nz * (int)g.plane, res_ph(false, a.pzm, h[k]));
    }
  }
  if (r.fl & RF_CORR) fix(h, x);
#pragma unroll
  for (int k = 0; k < 3; ++k) st<T>(v.h(k) + li, h[k]);
  if (r.fl & RF_PUB) {
#pragma unroll
    for (int k = 0; k < 3; ++k) st<T>(a.h + (k * cp + gi), h[k]);
  }
}

// The same for 32 consecutive cells of a row that needs none of the special
// cases (the flags are the row's, so the warp's): lane l takes x, the lanes
// beyond nx idle.  What is left is 12 reads and 3 writes of shared memory and
// 24 FP32 operations a cell.
constexpr int RF_E_SLOW = RF_YG | RF_ZP | RF_YP | RF_UPML | RF_CORR;
constexpr int RF_H_SLOW = RF_YG | RF_ZP | RF_YP | RF_UPML | RF_CORR;

template <bool CEPS, int NC>
__device__ __forceinline__ void res_e_fast(const ResArgs<float>& A, const ResView<float, NC>& v, const ResRow& r, int x,
                                           int lrow) {
  const FieldArgs<float>& a = A.a;
  if (x > a.g.nx) return;
  const int li = lrow * v.W + x, gi = r.gb + x, cp = (int)a.g.comp;
  const float2 *H0 = v.h(0) + li, *H1 = v.h(1) + li, *H2 = v.h(2) + li;
  cx<float> e[3], hz0, hz1;
  if (NC == 5) e[0] = ld<float>(a.e + gi);
  if (r.fl & RF_ZG) {
    hz0 = ld_l2(a.h + (gi + r.zo));
    hz1 = ld_l2(a.h + (cp + gi + r.zo));
  } else {
    hz0 = ld<float>(H0 + r.zo);
    hz1 = ld<float>(H1 + r.zo);
  }
  float m = r.fl & RF_SUB ? a.m3 : a.m1;
  cx<float> mc;
  if (r.fl & RF_MAT) {
    if (CEPS) mc = ld<float>(a.eps_c + (gi - a.hi * (int)a.g.plane));
    else m = a.eps_r[gi - a.hi * (int)a.g.plane];
  }
  const cx<float> h0 = ld<float>(H0), h1 = ld<float>(H1), h2 = ld<float>(H2);
  const cx<float> hy0 = ld<float>(H0 + r.yo), hy2 = ld<float>(H2 + r.yo);
  const cx<float> hx1 = ld<float>(H1 - 1), hx2 = ld<float>(H2 - 1);
#pragma unroll
  for (int k = NC == 5 ? 1 : 0; k < 3; ++k) e[k] = ld<float>(v.e(k) + li);
  cx<float> c[3];
  c[0] = cadd(csub(csub(h2, hy2), h1), hz1);
  c[1] = cadd(csub(csub(h0, hz0), h2), hx2);
  c[2] = cadd(csub(csub(h1, hx1), h0), hy0);
  if (CEPS && (r.fl & RF_MAT)) {
#pragma unroll
    for (int k = 0; k < 3; ++k) e[k] = cadd(e[k], cmul(mc, c[k]));
  } else {
#pragma unroll
    for (int k = 0; k < 3; ++k) e[k] = cadd(e[k], rmul(m, c[k]));
  }
#pragma unroll
  for (int k = NC == 5 ? 1 : 0; k < 3; ++k) st<float>(v.e(k) + li, e[k]);
  if (NC == 5) st<float>(a.e + gi, e[0]);
  if (r.fl & RF_PUB) {  // component 2 is read across y only
    if (NC == 6) st<float>(a.e + gi, e[0]);
    st<float>(a.e + (cp + gi), e[1]);
    if (r.fl & RF_PUB2) st<float>(a.e + (2 * cp + gi), e[2]);
  }
  if (x == 1) {
#pragma unroll
    for (int k = 1; k < 3; ++k) st<float>(v.e(k) + li + a.g.nx, res_ph(A.one[0], a.pxp, e[k]));
  }
}

template <int NC>
__device__ __forceinline__ void res_h_fast(const ResArgs<float>& A, const ResView<float, NC>& v, const ResRow& r, int x,
                                           int lrow) {
  const FieldArgs<float>& a = A.a;
  const Geo& g = a.g;
  if (x > g.nx) return;
  const int li = lrow * v.W + x, gi = r.gb + x, cp = (int)g.comp;
  const float2 *E0 = NC == 5 ? nullptr : v.e(0) + li, *E1 = v.e(1) + li, *E2 = v.e(2) + li;
  cx<float> ev[3], xp[3], yp[3], zp[3], h[3];
  if (NC == 5) {
    ev[0] = ld<float>(a.e + gi);
    yp[0] = ld<float>(a.e + (gi + (r.yo > 0 ? 1 : 1 - g.ny) * (int)g.pitch));
    zp[0] = (r.fl & RF_ZG) ? ld_l2(a.e + (gi + r.zo)) : ld<float>(a.e + (gi + (int)g.plane));
  }
  if (r.fl & RF_ZG) {
    if (NC == 6) zp[0] = ld_l2(a.e + (gi + r.zo));
    zp[1] = ld_l2(a.e + (cp + gi + r.zo));
  } else {
    if (NC == 6) zp[0] = ld<float>(E0 + r.zo);
    zp[1] = ld<float>(E1 + r.zo);
  }
  if (NC == 6) {
    ev[0] = ld<float>(E0);
    yp[0] = ld<float>(E0 + r.yo);
  }
  ev[1] = ld<float>(E1);
  ev[2] = ld<float>(E2);
  yp[2] = ld<float>(E2 + r.yo);
  xp[1] = ld<float>(E1 + 1);
  xp[2] = ld<float>(E2 + 1);
#pragma unroll
  for (int k = 0; k < 3; ++k) h[k] = ld<float>(v.h(k) + li);
  h_update<float, false>(a, x, 1, 1, ev, xp, yp, zp, h);
#pragma unroll
  for (int k = 0; k < 3; ++k) st<float>(v.h(k) + li, h[k]);
  if (r.fl & RF_PUB) {
    st<float>(a.h + gi, h[0]);
    st<float>(a.h + (cp + gi), h[1]);
    if (r.fl & RF_PUB2) st<float>(a.h + (2 * cp + gi), h[2]);
  }
  if (x == g.nx) {
#pragma unroll
    for (int k = 0; k < 3; ++k) st<float>(v.h(k) + li - g.nx, res_ph(A.one[0], a.pxm, h[k]));
  }
}

// FP64: one work item is one real number, the real (p = 0) or imaginary part
// of component k of a cell.  GB300 issues an FP64 warp instruction on a
// sub-partition every 64 cycles whatever the lanes do, so what counts is the
// number of warp instructions and the length of a chain: every lane runs the
// same operations with its own component's operands (no path per component),
// and a cell's six numbers sit on six lanes.  With i, j the components after k
// in cyclic order the curls are
//   E_k: ((H_j - H_j(-1 on axis i)) - H_i) + H_i(-1 on axis j)
//   H_k: ((E_j(+1 on axis i) - E_j) - E_i(+1 on axis j)) + E_i,
// the association of e_update and h_update.
__device__ __forceinline__ double res_dl2(const double2* f, int i, int p) { return __ldcg((const double*)(f + i) + p); }
__device__ __forceinline__ double res_ds(const double2* f, int i, int p) { return ((const double*)(f + i))[p]; }
// LL: a number and its step's tag as one 16-byte packet, written and read whole.
__device__ __forceinline__ void res_ll_st(ulonglong2* q, double v, unsigned long long tag) {
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(q),
               "l"(__double_as_longlong(v)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ bool res_ll_ld(const ulonglong2* q, unsigned long long tag, double& v) {
  unsigned long long d, t;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
               : "=l"(d), "=l"(t)
               : "l"(q)
               : "memory");
  v = __longlong_as_double((long long)d);
  return t == tag;
}
// The packets q (null: none) with this tag, polled together for at most about
// limit clock cycles; false when it gave up.
__device__ __forceinline__ bool res_ll_get(const ulonglong2* const (&q)[4], unsigned long long tag, double (&v)[4],
                                           long long limit) {
  bool ok[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) ok[c] = !q[c] || res_ll_ld(q[c], tag, v[c]);
  if (ok[0] && ok[1] && ok[2] && ok[3]) return true;
  const long long t0 = clock64();
  while (!(ok[0] && ok[1] && ok[2] && ok[3])) {
    if (clock64() - t0 > limit) return false;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (!ok[c]) ok[c] = res_ll_ld(q[c], tag, v[c]);
  }
  return true;
}
// The packets of the number whose parts lie at b that a lane with part p reads
// (in q, q + 1): both where the row is an image with a phase, else its own.
__device__ __forceinline__ void res_ll_ask(const ulonglong2** q, const ulonglong2* b, bool image, int p) {
  q[0] = image ? b : b + p;
  if (image) q[1] = b + 1;
}
// What a phase of a step needs of LL: the tag of what it reads (0: nothing,
// the first step's E phase reads the state in memory) and of what it
// publishes, the wait's limit and where a wait that gave up is noted.
struct ResLl {
  unsigned long long want, pub;
  long long limit;
  int* stop;
};

// Part p of ph * w, as cmul rounds it.
__device__ __forceinline__ double res_dph(cx<double> ph, cx<double> w, int p) {
  return p == 0 ? axmby_(ph.re, w.re, ph.im, w.im) : axpby_(ph.re, w.im, ph.im, w.re);
}
// The other part of the same cell and component: on the neighbouring lane
// (items come in pairs and both lanes of a pair take the same branches).
__device__ __forceinline__ cx<double> res_pair(double own, int p) {
  const unsigned lane = threadIdx.x & 31u;
  const double oth = __shfl_xor_sync(3u << (lane & 30u), own, 1);
  return p == 0 ? cx<double>{own, oth} : cx<double>{oth, own};
}

template <bool CEPS, int NC, bool LL>
__device__ __forceinline__ void res_e64(const ResArgs<double>& A, const ResView<double, NC>& v, int k, int p, int x,
                                        int lrow, const TfsfVal<double>* vE, const ResLl& ll) {
  const FieldArgs<double>& a = A.a;
  const Geo& g = a.g;
  const ResRow r = v.er[lrow];
  const int li = lrow * v.W + x, gi = r.gb + x, cp = (int)g.comp;
  if (!bc_ok(x >= 1 && x <= g.nx && lrow < v.nrows, BC_E_CELL, gi)) return;
  const int i = k == 2 ? 0 : k + 1, j = k == 0 ? 2 : k - 1;
  const double2 *hi = v.h(i), *hj = v.h(j);
  // LL: the packets of component j down axis i and of component i down axis j
  // (read where they were asked for only; given initial values, the kernel came
  // out at 64 registers with spills instead of 118: 4x4x512 1438 us for 256 steps, 1419)
  double pk[4];
  if constexpr (LL) {
    if (ll.want) {
      const ulonglong2* q[4] = {};
      auto ask = [&](int ax, int c, int at) {
        if (ax != 0 && (r.fl & (ax == 1 ? RF_YG : RF_ZG)))
          res_ll_ask(q + at, A.ll + 2l * ((3 + c) * cp + gi + (ax == 1 ? r.yo : r.zo)),
                     (r.fl & (ax == 1 ? RF_YP : RF_ZP)) != 0, p);
      };
      ask(i, j, 0);
      ask(j, i, 2);
      if (!res_ll_get(q, ll.want, pk, ll.limit)) {
        atomicExch(A.err, 6);
        *(volatile int*)ll.stop = 1;
      }
    }
  }
  // part p of component c one cell down axis ax
  auto nb = [&](const double2* hc, int c, int ax) {
    if (ax == 0) return res_ds(hc, li - 1, p);
    const int off = ax == 1 ? r.yo : r.zo, gl = ax == 1 ? RF_YG : RF_ZG, im = ax == 1 ? RF_YP : RF_ZP;
    if (LL && (r.fl & gl) && ll.want) {
      const double u = c == j ? pk[0] : pk[2], w = c == j ? pk[1] : pk[3];
      return r.fl & im ? res_dph(ax == 1 ? a.pym : a.pzm, cx<double>{u, w}, p) : u;
    }
    if (r.fl & im) {
      const double2 w = (r.fl & gl) ? __ldcg(a.h + c * cp + gi + off) : hc[li + off];
      return res_dph(ax == 1 ? a.pym : a.pzm, cx<double>{w.x, w.y}, p);
    }
    return (r.fl & gl) ? res_dl2(a.h + c * cp, gi + off, p) : res_ds(hc, li + off, p);
  };
  double e = NC == 5 && k == 0 ? res_dl2(a.e, gi, p) : res_ds(v.e(k), li, p);
  const double c = da(ds(ds(res_ds(hj, li, p), nb(hj, j, i)), res_ds(hi, li, p)), nb(hi, i, j));
  if ((r.fl & RF_CORR) && k == A.s.cE) {
    const double t = p == 0 ? vE[x].er : vE[x].ei;
    e = A.s.sgn > 0 ? da(e, t) : ds(e, t);
  }
  if (r.fl & RF_UPML) {
    const ResUpml<double> u = res_upml(A, v, lrow, 0);
    if (!u.cf) return;
    const double* cf = u.cf + k;
    double* D = (double*)(u.f + k * u.pc + x) + p;
    const double dold = *D;
    const double dn = axpby_(cf[CD_A], dold, cf[CD_B], dm(a.eps0sq, c));
    *D = dn;
    e = axpby_(cf[CE_A], e, cf[CE_B], axmby_(cf[C_FP], dn, cf[C_FM], dold));
  } else if (r.fl & RF_MAT) {
    const int ie = gi - a.hi * (int)g.plane;
    if (CEPS) {
      const double2 w = a.eps_c[ie];
      const cx<double> cc = res_pair(c, p);
      const double o = p == 0 ? cc.im : cc.re;
      e = axpy_(w.x, c, axpy_(p == 0 ? -w.y : w.y, o, e));
    } else {
      e = axpy_(a.eps_r[ie], c, e);
    }
  } else {
    e = axpy_(r.fl & RF_SUB ? a.m3 : a.m1, c, e);
  }
  if (!(NC == 5 && k == 0)) ((double*)(v.e(k) + li))[p] = e;
  if (LL) {
    if (r.fl & RF_PUB) res_ll_st(A.ll + 2l * (k * cp + gi) + p, e, ll.pub);
  } else if ((r.fl & RF_PUB) || (NC == 5 && k == 0)) {
    ((double*)(a.e + k * cp + gi))[p] = e;
  }
  if (x == 1 && k > 0) {
    const double q = A.one[0] ? e : res_dph(a.pxp, res_pair(e, p), p);
    ((double*)(v.e(k) + li + g.nx))[p] = q;
  }
}

template <int NC, bool LL>
__device__ __forceinline__ void res_h64(const ResArgs<double>& A, const ResView<double, NC>& v, int k, int p, int x,
                                        int lrow, const TfsfVal<double>* vH, bool last, const ResLl& ll) {
  const FieldArgs<double>& a = A.a;
  const Geo& g = a.g;
  const ResRow r = v.hr[lrow];
  const int li = lrow * v.W + x, gi = r.gb + x, cp = (int)g.comp;
  if (!bc_ok(x >= 1 && x <= g.nx && lrow < v.nrows, BC_H_CELL, gi)) return;
  const int i = k == 2 ? 0 : k + 1, j = k == 0 ? 2 : k - 1;
  double pk[4];
  if constexpr (LL) {
    const ulonglong2* q[4] = {};
    auto ask = [&](int ax, int c, int at) {
      if (ax != 0 && (r.fl & (ax == 1 ? RF_YG : RF_ZG)))
        res_ll_ask(q + at, A.ll + 2l * (c * cp + gi + (ax == 1 ? r.yo : r.zo)),
                   (r.fl & (ax == 1 ? RF_YP : RF_ZP)) != 0, p);
    };
    ask(i, j, 0);
    ask(j, i, 2);
    if (!res_ll_get(q, ll.want, pk, ll.limit)) {
      atomicExch(A.err, 6);
      *(volatile int*)ll.stop = 1;
    }
  }
  // part p of component c of the cell, and of the cell one up axis ax
  auto own = [&](int c) { return NC == 5 && c == 0 ? res_dl2(a.e, gi, p) : res_ds(v.e(c), li, p); };
  auto nb = [&](int c, int ax) {
    if (ax == 0) return res_ds(v.e(c), li + 1, p);  // components 1 and 2 only
    const int off = ax == 1 ? r.yo : r.zo, gl = ax == 1 ? RF_YG : RF_ZG, im = ax == 1 ? RF_YP : RF_ZP;
    if (LL && (r.fl & gl)) {
      const double u = c == j ? pk[0] : pk[2], w = c == j ? pk[1] : pk[3];
      return r.fl & im ? res_dph(ax == 1 ? a.pyp : a.pzp, cx<double>{u, w}, p) : u;
    }
    // storage offset of the row (own rows' offsets are shared-memory ones)
    const int so = (r.fl & gl) ? off : ax == 1 ? (off > 0 ? 1 : 1 - g.ny) * (int)g.pitch : (int)g.plane;
    const bool far = (r.fl & gl) || (NC == 5 && c == 0);
    if (r.fl & im) {
      const double2 w = far ? __ldcg(a.e + c * cp + gi + so) : v.e(c)[li + off];
      return res_dph(ax == 1 ? a.pyp : a.pzp, cx<double>{w.x, w.y}, p);
    }
    return far ? res_dl2(a.e + c * cp, gi + so, p) : res_ds(v.e(c), li + off, p);
  };
  double h = res_ds(v.h(k), li, p);
  const double c = da(ds(ds(nb(j, i), own(j)), nb(i, j)), own(i));
  if (r.fl & RF_UPML) {
    const ResUpml<double> u = res_upml(A, v, lrow, 1);
    if (!u.cf) return;
    const double* cf = u.cf + k;
    double* B = (double*)(u.f + k * u.pc + x) + p;
    const double bold = *B;
    const double bn = axmby_(cf[CD_A], bold, cf[CB_B], c);
    *B = bn;
    h = axpby_(cf[CE_A], h, cf[CH_B], axmby_(cf[C_FP], bn, cf[C_FM], bold));
  } else {
    h = ymax_(h, a.dtcq2, c);
  }
  const bool ck = (r.fl & RF_CORR) && k == A.s.cH;
  auto fix = [&](double q, int ix) {
    if (!ck) return q;
    const double t = p == 0 ? vH[ix].hr : vH[ix].hi;
    return A.s.sgn > 0 ? da(q, t) : ds(q, t);
  };
  if (x == g.nx) {
    const double q = A.one[0] ? h : res_dph(a.pxm, res_pair(h, p), p);
    ((double*)(v.h(k) + li - g.nx))[p] = fix(q, 0);
  }
  if (last && (r.fl & RF_GHOST)) {
    const unsigned zy = v.zy[lrow].x;
    const cx<double> w = res_pair(h, p);
    if ((int)(zy & 0xffffu) == g.ny)
      ((double*)(a.h + k * cp + gi - g.ny * (int)g.pitch))[p] = fix(res_dph(a.pym, w, p), x);
    if ((int)(zy >> 16) == g.nz) ((double*)(a.h + k * cp + gi - g.nz * (int)g.plane))[p] = res_dph(a.pzm, w, p);
  }
  h = fix(h, x);
  ((double*)(v.h(k) + li))[p] = h;
  if (r.fl & RF_PUB) {
    if (LL) res_ll_st(A.ll + 2l * ((3 + k) * cp + gi) + p, h, ll.pub);
    else ((double*)(a.h + k * cp + gi))[p] = h;
  }
}

// Work items of a phase over a set of rows: cells (FP32), or the six numbers
// of every cell, component-major with the parts of a value on neighbouring
// lanes (FP64; SPLIT).  f(k, p, x, j): component, part (FP64), column and row
// j of the set.
template <bool SPLIT, typename F> __device__ __forceinline__ void res_items(int rows, int nx, F f) {
  const int cells = rows * nx;
  if (SPLIT) {
    for (int w = threadIdx.x; w < 6 * cells; w += blockDim.x) {
      const int q = w >> 1;
      const int k = q >= 2 * cells ? 2 : q >= cells ? 1 : 0, c = q - k * cells, j = c / nx;
      f(k, w & 1, c - j * nx + 1, j);
    }
  } else {
    int j = (int)threadIdx.x / nx, x = (int)threadIdx.x - j * nx;
    const int dj = (int)blockDim.x / nx, dx = (int)blockDim.x - dj * nx;
    while (j < rows) {
      f(0, 0, x + 1, j);
      j += dj;
      x += dx;
      if (x >= nx) {
        x -= nx;
        ++j;
      }
    }
  }
}

// FP32, rows whose last 32-cell run is not mostly empty: a warp takes one run
// of 32 cells of a row at a time, so the row's flags are the warp's.  The runs
// of a phase are walked in the order of a table: the rows that read own rows
// only, with the D runs of the others spread over its end, s positions apart
// (s odd or 1, so that different warps take them): by then the neighbours'
// flags have arrived, and the L2 latency of a run that reads another CTA's
// rows is covered by the warps that do not.  Position p of N: dependent run k
// (dep) or own run k.
struct ResOrder {
  int N, D, s;
  __device__ __forceinline__ bool at(int p, int& k) const {
    const int b = N - 1 - p, c = min(D, b / s + 1);  // dependent runs at positions >= p
    if (b % s == 0 && b / s < D) {
      k = D - c;
      return true;
    }
    k = p - (D - c);
    return false;
  }
};
__device__ __forceinline__ ResOrder res_order(int rows, int dep, int nr, int nw) {
  ResOrder o;
  o.N = rows * nr;
  o.D = dep * nr;
  o.s = 3 * o.D <= o.N - nw ? 3 : 1;
  return o;
}

template <typename T, bool CEPS, int NC, bool LL = false>
__global__ void __launch_bounds__(LL ? RES_LL_THREADS : RES_THREADS) k_res(ResArgs<T> A, long long limit) {
  using V = typename V2<T>::t;
  extern __shared__ __align__(16) unsigned char res_smem[];
  constexpr bool SPLIT = sizeof(T) == 8;
  __shared__ int stop_s;  // a wait gave up
  if (threadIdx.x == 0) stop_s = 0;
  const FieldArgs<T>& a = A.a;
  const Geo& g = a.g;
  const ResCta ct = A.cta[blockIdx.x];
  const int nx = g.nx, ny = g.ny, nrows = ct.r1 - ct.r0, W = nx + 2;
  const int cp = (int)g.comp, pl = (int)g.plane, pt = (int)g.pitch;
  ResView<T, NC> v;
  // row tables first (their size does not depend on the CTA), then the fields
  v.er = (ResRow*)res_smem;
  v.hr = v.er + A.rows;
  uint2* zy = (uint2*)(v.hr + A.rows);
  v.zy = zy;
  unsigned *oe = (unsigned*)(zy + A.rows), *oh = oe + A.nruns;  // run tables (row << 16) + first x (A.runs)
  v.sm = (V*)(res_smem + A.head);
  v.cs = nrows * W;
  v.W = W;
  v.nrows = nrows;
  // UPML rows: the first nlo and those from nhi on
  const int nlo = min(max(min(a.pmlzi, g.nz) * ny - ct.r0, 0), nrows);
  const int nhi = max(nlo, min(max((a.pmlzf - 1) * ny - ct.r0, 0), nrows));
  v.nu = nlo + nrows - nhi;
  v.d = v.sm + NC * v.cs;
  T* cf = (T*)(v.d + 6 * v.nu * nx);
  v.cf = cf;
  for (int j = threadIdx.x; j < nrows; j += blockDim.x) {
    const int r = ct.r0 + j, z = r / ny + 1, y = r - (z - 1) * ny + 1;
    zy[j] = make_uint2(((unsigned)z << 16) + (unsigned)y, (unsigned)(j < nlo ? j : j - nhi + nlo));
    v.er[j] = res_row_e(A, W, nrows, j, y, z, true);
    v.hr[j] = res_row_h(A, W, nrows, j, y, z);
  }
  // own state in, x ghosts included
  for (int w = threadIdx.x; w < nrows * W; w += blockDim.x) {
    const int j = w / W, x = w - j * W, r = ct.r0 + j, z = r / ny, y = r - z * ny;
    const int gi = (z + 1) * pl + (y + 1) * pt + x + g.xo;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (!(NC == 5 && k == 0)) v.e(k)[w] = a.e[k * cp + gi];
      v.h(k)[w] = a.h[k * cp + gi];
    }
  }
  __syncthreads();
  // D, B and the coefficients of UPML row u in or out
  auto upml_io = [&](bool in) {
    for (int w = threadIdx.x; w < v.nu * nx; w += blockDim.x) {
      const int u = w / nx, x = w - u * nx, j = u < nlo ? u : u - nlo + nhi;
      const int z = (int)(zy[j].x >> 16), y = (int)(zy[j].x & 0xffffu), slab = z <= a.pmlzi ? 0 : 1;
      const long pi = ((long)(slab == 0 ? z - 1 : z - a.pmlzf) * ny + (y - 1)) * nx + x;
      if (!bc_ok(pi >= 0 && pi < a.pcomp[slab], BC_E_SLAB, pi)) continue;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        V &d = a.pml_d[slab][k * a.pcomp[slab] + pi], &b = a.pml_b[slab][k * a.pcomp[slab] + pi];
        V &sd = v.d[k * v.nu * nx + w], &sb = v.d[(3 + k) * v.nu * nx + w];
        if (in) {
          sd = d;
          sb = b;
        } else {
          d = sd;
          b = sb;
        }
      }
    }
  };
  if (A.db) {
    upml_io(true);
    for (int w = threadIdx.x; w < v.nu * NCOEF; w += blockDim.x) {
      const int u = w / NCOEF, j = u < nlo ? u : u - nlo + nhi, z = (int)(zy[j].x >> 16);
      cf[w] = a.coef[NCOEF * (z <= a.pmlzi ? z - 1 : a.pmlzi + z - a.pmlzf) + w - u * NCOEF];
    }
    __syncthreads();
  }
  // Rows whose phase reads other CTAs' rows: E, the first ny and a y = 1 row
  // whose image row ny is not owned; H, the last ny and a y = ny row whose
  // image row 1 is not owned (at most one more row each).  A CTA whose phase
  // is a single round of its threads takes all rows after the wait: a second
  // round would cost another dependent chain.
  const bool whole = nrows * nx * (SPLIT ? 6 : 1) <= (int)blockDim.x;
  const int ne = whole ? nrows : min(ny, nrows), nh = whole ? 0 : max(0, nrows - ny);
  int badE = -1, badH = -1;
  if (!whole) {
    const int l1 = nrows - 1 - (ct.r1 - 1) % ny;  // the last row with y = 1
    if (l1 >= ny && l1 + ny - 1 >= nrows) badE = l1;
    const int ln = ny - 1 - ct.r0 % ny;           // the first row with y = ny
    if (ln < nh && ln - ny + 1 < 0) badH = ln;
  }
  ResLl ll{0, 0, limit, &stop_s};
  auto e_item = [&](int k, int p, int x, int lrow, const TfsfVal<T>* vE) {
    if constexpr (SPLIT) res_e64<CEPS, NC, LL>(A, v, k, p, x, lrow, vE, ll);
    else res_e<CEPS, NC>(A, v, x, lrow, vE);
  };
  auto h_item = [&](int k, int p, int x, int lrow, const TfsfVal<T>* vH, bool last) {
    if constexpr (SPLIT) res_h64<NC, LL>(A, v, k, p, x, lrow, vH, last, ll);
    else res_h<NC>(A, v, x, lrow, vH, last);
  };
  const bool runs = !SPLIT && A.runs;
  const int nr = (nx + 31) >> 5, nw = (int)blockDim.x >> 5, warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
  const int depE = ne + (badE >= 0 ? 1 : 0), depH = nrows - nh + (badH >= 0 ? 1 : 0);
  // row j of a phase's dependent rows and of its others
  auto e_dep = [&](int j) { return j < ne ? j : badE; };
  auto h_dep = [&](int j) { return nh + j < nrows ? nh + j : badH; };
  auto e_own = [&](int j) { return badE < 0 || j + ne < badE ? j + ne : j + ne + 1; };
  auto h_own = [&](int j) { return badH < 0 || j < badH ? j : j + 1; };
  if (runs) {
    const ResOrder qe = res_order(nrows, depE, nr, nw), qh = res_order(nrows, depH, nr, nw);
    for (int p = threadIdx.x; p < qe.N; p += blockDim.x) {
      int k;
      const bool de = qe.at(p, k);
      oe[p] = ((unsigned)(de ? e_dep(k / nr) : e_own(k / nr)) << 16) + (unsigned)(k % nr * 32 + 1);
      const bool dh = qh.at(p, k);
      oh[p] = ((unsigned)(dh ? h_dep(k / nr) : h_own(k / nr)) << 16) + (unsigned)(k % nr * 32 + 1);
    }
    __syncthreads();
  }
  // The neighbours' flags, waited for once a phase by each warp that reads
  // their rows.
  auto wait = [&](unsigned want) {
    if (!res_wait_warp(A.flag, ct.nb0, ct.nbn, want, A.err, limit)) *(volatile int*)&stop_s = 1;
  };
  // A phase's writes are done: publish them (by the last warp, which has the
  // least work); false when a wait gave up.
  auto done = [&](unsigned phase) {
    __syncthreads();
    if (LL && phase < 2u * A.n) return *(volatile int*)&stop_s == 0;
    if ((int)threadIdx.x == (int)blockDim.x - 32) res_st_release(A.flag + (long)blockIdx.x * RES_FLAG_STRIDE, phase);
    return *(volatile int*)&stop_s == 0;
  };
  auto e_phase = [&](int i, const TfsfVal<T>* vE) {
    const unsigned want = 2u * i;
    if constexpr (!SPLIT) {
      if (runs) {
        bool waited = i == 0;
        for (int p = warp; p < nrows * nr; p += nw) {
          const unsigned o = oe[p];
          const int l = (int)(o >> 16), x = (int)(o & 0xffffu) + lane;
          if (!waited && (l < ne || l == badE)) {
            wait(want);
            waited = true;
          }
          const ResRow r = v.er[l];
          if (!(r.fl & RF_E_SLOW)) res_e_fast<CEPS, NC>(A, v, r, x, l);
          else if (x <= nx) res_e<CEPS, NC>(A, v, x, l, vE);
        }
        return;
      }
    }
    res_items<SPLIT>(nrows - depE, nx, [&](int k, int p, int x, int j) { e_item(k, p, x, e_own(j), vE); });
    if (!LL && i > 0) wait(want);
    res_items<SPLIT>(depE, nx, [&](int k, int p, int x, int j) { e_item(k, p, x, e_dep(j), vE); });
  };
  auto h_phase = [&](int i, const TfsfVal<T>* vH, bool last) {
    const unsigned want = 2u * i + 1u;
    if constexpr (!SPLIT) {
      if (runs) {
        const int slow = last ? RF_H_SLOW | RF_GHOST : RF_H_SLOW;
        bool waited = false;
        for (int p = warp; p < nrows * nr; p += nw) {
          const unsigned o = oh[p];
          const int l = (int)(o >> 16), x = (int)(o & 0xffffu) + lane;
          if (!waited && (l >= nh || l == badH)) {
            wait(want);
            waited = true;
          }
          const ResRow r = v.hr[l];
          if (!(r.fl & slow)) res_h_fast<NC>(A, v, r, x, l);
          else if (x <= nx) res_h<NC>(A, v, x, l, vH, last);
        }
        return;
      }
    }
    res_items<SPLIT>(nrows - depH, nx, [&](int k, int p, int x, int j) { h_item(k, p, x, h_own(j), vH, last); });
    if (!LL) wait(want);
    res_items<SPLIT>(depH, nx, [&](int k, int p, int x, int j) { h_item(k, p, x, h_dep(j), vH, last); });
  };
  auto sampled = [&](int it) { return A.dft && it >= A.to_fourier && it % A.sample_fourier == 0; };
  // own sample points [q0, q1) into a ring slot (vE: the pending E correction);
  // four table entries at a time, so that their latencies overlap
  auto sample = [&](unsigned q0, unsigned q1, int slot, const TfsfVal<T>* vE) {
    V* out = A.S + (long)slot * A.P;
    for (unsigned q = q0 + threadIdx.x; q < q1; q += 4 * blockDim.x) {
      uint2 c[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) c[t] = q + t * blockDim.x < q1 ? A.samp[q + t * blockDim.x] : make_uint2(0u, 0u);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (q + t * blockDim.x >= q1) break;
        const unsigned off = c[t].x & ~(RES_GLOBAL | RES_CORR);
        const bool far = (c[t].x & RES_GLOBAL) != 0;
        if (!bc_ok(c[t].y < A.P && off < (far ? (unsigned)cp : (unsigned)(NC * v.cs)), BC_GATHER_DST, c[t].y)) continue;
        cx<T> s = far ? ld<T>(a.e + off) : ld<T>(v.sm + off);
        if ((c[t].x & RES_CORR) && vE) {
          const unsigned x = far ? off % (unsigned)pt - (unsigned)g.xo : off % (unsigned)v.cs % (unsigned)W;
          const auto u = vE[x];
          s = tf_add(s, u.er, u.ei, A.s.sgn);
        }
        st<T>(out + c[t].y, s);
      }
    }
  };
  int slot = A.slot0;
  bool h_due = false;  // the last step's H samples are still to be taken
  for (int i = 0; i < A.n; ++i) {
    const TfsfVal<T>* prev = A.s.on && i > 0 ? A.tfv + (long)(i - 1) * W : nullptr;
    const TfsfVal<T>* cur = A.s.on ? A.tfv + (long)i * W : nullptr;
    const int it = A.it0 + i;
    if (h_due) sample(ct.sh, ct.s1, slot - 1, nullptr);
    ll.want = i == 0 ? 0 : A.ep + i;
    ll.pub = A.ep + i + 1;
    e_phase(i, prev);
    ll.want = ll.pub;
    if (!done(2u * i + 1u)) return;
    h_due = sampled(it);
    if (h_due) {
      if (blockIdx.x == 0 && threadIdx.x == 0) A.tk[slot] = it + 1 - A.to_fourier;
      sample(ct.s0, ct.sh, slot, cur);
      ++slot;
    }
    if (i == 0)  // from the second step on, y and z images are formed from their rows
      for (int j = threadIdx.x; j < nrows; j += blockDim.x)
        v.er[j] = res_row_e(A, W, nrows, j, (int)(zy[j].x & 0xffffu), (int)(zy[j].x >> 16), false);
    h_phase(i, cur, i == A.n - 1);
    if (!done(2u * i + 2u)) return;
  }
  if (h_due) sample(ct.sh, ct.s1, slot - 1, nullptr);
  // the neighbours have read the last published rows: the final state with
  // its ghosts and the last step's E correction
  wait(2u * A.n);
  __syncthreads();
  if (*(volatile int*)&stop_s) return;
  if (A.db) upml_io(false);
  const TfsfVal<T>* lastv = A.s.on ? A.tfv + (long)(A.n - 1) * W : nullptr;
  res_items<false>(nrows, nx, [&](int, int, int x, int j) {
    const int z = (int)(v.zy[j].x >> 16), y = (int)(v.zy[j].x & 0xffffu), li = j * W + x;
    const int gi = z * pl + y * pt + x + g.xo;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const bool ck = lastv && z == A.s.zE && k == A.s.cE;
      auto fix = [&](cx<T> q, int ix, bool in) {
        if (!ck || !in) return q;
        const auto t = lastv[ix];
        return tf_add(q, t.er, t.ei, A.s.sgn);
      };
      const cx<T> e = NC == 5 && k == 0 ? ld_l2(a.e + gi) : ld<T>(v.e(k) + li);
      V* E = a.e + k * cp;
      st<T>(E + gi, fix(e, x, true));
      if (x == 1) st<T>(E + gi + nx, fix(res_ph(false, a.pxp, e), nx + 1, A.s.gx));
      if (y == 1) st<T>(E + gi + ny * pt, fix(res_ph(false, a.pyp, e), x, A.s.gy));
      if (z == 1) st<T>(E + gi + g.nz * pl, res_ph(false, a.pzp, e));
      if (x == nx) st<T>(E + gi - nx, fix(res_ph(false, a.pxm, e), 0, true));
      if (y == ny) st<T>(E + gi - ny * pt, fix(res_ph(false, a.pym, e), x, true));
      if (z == g.nz) st<T>(E + gi - g.nz * pl, res_ph(false, a.pzm, e));
      st<T>(a.h + k * cp + gi, ld<T>(v.h(k) + li));
      if (x == nx) st<T>(a.h + k * cp + gi - nx, ld<T>(v.h(k) + j * W));
    }
  });
  // ghost cells of the corrected planes that no Bloch copy writes: the
  // corrections of every step of the span, in order (E: the four corners of
  // the plane; H: also the column nx+1 and the row ny+1, within the ranges)
  if (A.s.on) {
    const int nb = 2 * (nx + 2) + 2 * ny;  // border cells of the plane
    for (int w = blockIdx.x + gridDim.x * threadIdx.x; w < nb; w += gridDim.x * blockDim.x) {
      int x, y;
      if (w < 2 * (nx + 2)) {
        y = w < nx + 2 ? 0 : ny + 1;
        x = w < nx + 2 ? w : w - (nx + 2);
      } else {
        const int q = w - 2 * (nx + 2);
        x = q < ny ? 0 : nx + 1;
        y = (q < ny ? q : q - ny) + 1;
      }
      if ((x == nx + 1 && !A.s.gx) || (y == ny + 1 && !A.s.gy)) continue;
      const bool corner = (x == 0 || x == nx + 1) && (y == 0 || y == ny + 1);
      if (corner) {
        V* p = a.e + A.s.cE * cp + A.s.zE * pl + y * pt + x + g.xo;
        cx<T> s = ld<T>(p);
        for (int i = 0; i < A.n; ++i) {
          const auto t = A.tfv[(long)i * W + x];
          s = tf_add(s, t.er, t.ei, A.s.sgn);
        }
        st<T>(p, s);
      }
      if (corner || x == nx + 1 || y == ny + 1) {
        V* p = a.h + A.s.cH * cp + A.s.zH * pl + y * pt + x + g.xo;
        cx<T> s = ld<T>(p);
        for (int i = 0; i < A.n; ++i) {
          const auto t = A.tfv[(long)i * W + x];
          s = tf_add(s, t.hr, t.hi, A.s.sgn);
        }
        st<T>(p, s);
      }
    }
  }
}

}  // namespace iris
