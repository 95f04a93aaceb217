// The fused E+H pass of the planes outside the UPML slabs (FP32), staged in
// shared memory: shared by the single-engine launch (iris_engine.cu) and the
// batched form (iris_batch.cu).  Not part of the public ABI.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "iris_device.cuh"

namespace iris {

// One tile column: W x R cells of the plane, marched in z over a chunk, from
// (E, H) into double buffers (E', H') as fused_column does, and with its
// arithmetic.  A CTA computes E' on the (W+1) x (R+1) cells that its own cells'
// H' needs (the last column and row write nothing) and H' one plane behind.
// What differs is how a plane gets to the threads: the boxes of H and E
// (three components each, the one-cell halo included) are copied two to three
// planes ahead into a ring of four planes in shared memory by 16-byte
// cp.async, and every operand is read from there; E' replaces E in its plane
// of the ring, where the next plane's H' reads its neighbours'.
// fused_column holds one plane ahead in registers: 49 KB a SM in flight, which
// at the 2.5 us a load takes under load is 82 % of the copy bandwidth.  Cells
// map to threads in flat order, MR_S a thread; W and R are compile-time (a few
// shapes, the one with the fewest tiles is taken), so that every offset in
// shared memory is an immediate, and the tiles that touch no border of the
// plane run code without its ghosts and images: with run-time shapes and
// border tests a cell cost 300 instructions and the pass was bound by them.
// (TMA boxes instead of cp.async, one or two planes ahead: 5.1 and 6.3 ms a
// 512x512x1024 pass against 4.8; rows of 36 elements of 8 bytes keep the TMA
// unit at 9 bytes a cycle.)
// Cells one past nx or ny are the Bloch images of x = 1, y = 1: their places in
// the boxes are filled from x = 1, y = 1, and only what they read across the
// border (H at x = 0, y = 0) has slots of its own.
// Measured on GB300 against fused_column, us a pass with the UPML slabs:
// 512x512x1024 4767 -> 4705, 256x256x512 794 -> 665, 160x160x512 316 -> 293,
// 256x256x128 347 -> 230; the march itself moves its 96 bytes a cell at 91 % of
// the measured copy bandwidth (222 planes of 512x512 in 0.98 ms).
// Boxes start at even elements (16 bytes): x = 1 is stored at an even index,
// W and the pitch are even.

constexpr int MR_T = 512, MR_S = 1;  // threads of a CTA (two an SM), cells a thread
// (256 threads of two cells, at 124 registers: 4.78 ms for a batch of 32 ragged
// cells against 4.52, large planes the same)
// Planes of a z chunk, at least: chunks this short cost 3 planes of loads each
// but end the launch evenly and keep the CTAs at different planes (marching
// 512x512x1024 in one chunk: 6.3 ms a pass, 31 planes a chunk 4.8, 21 4.7, 16
// 4.7; 256x256x512: 102 planes 0.79, 30 0.68, 10 0.66; 160x160x512: 102 0.35, 21 0.30, 10 0.29).
constexpr int MR_CHUNK = 14;

struct MarchArgs {
  FieldArgs<float> f;  // the old state
  float2* e_new;
  float2* h_new;
  int tx, ty;          // tiles of the plane
};
// The slabs' march: D is double buffered (image and overlap cells read the old
// D of cells another CTA owns), B is its owner's and stays in place.
struct MarchSlabArgs {
  MarchArgs m;
  float2* d_new[2];
};

// The adjoint's march (ADJ): the same column with the passes' roles exchanged,
// E' = E - dtcq2 curl_b H, then H' = H + curl_f W, W = m E' (m the structure's
// eps_inv, 1/eps1 or 1/eps3); W takes E's place in the ring.  E has no stored
// images.  The gradient term of the design cells, with the forward curl rec.
struct MarchGrad {
  int x0, y0, z0, nx, ny, nz;  // design cells
  long n;
  const float2* rec;  // [3][n]
  double* grad;       // [n], or null
};

__device__ __forceinline__ void march_cpa16(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void march_cpa8(unsigned dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

// T: threads of a CTA.  UPML: with the old D and B of its cells and the
// coefficient rows in the ring.
template <int W_, int R_, int T_ = MR_T, bool UPML_ = false> struct MarchTile {
  static constexpr int W = W_, R = R_, T = T_, WT = W + 1, NC = (W + 1) * (R + 1);
  static constexpr bool UPML = UPML_;
  static constexpr int BXH = (W + 4) / 2 * 2, BXE = (W + 2) / 2 * 2;  // columns of a box: x0-2 .., x0 ..
  static constexpr int HC = (R + 2) * BXH, EC = (R + 1) * BXE;        // elements of a component of a box
  static constexpr int HB = 3 * HC * 8, EB = 3 * EC * 8;              // bytes of a plane's box
  static constexpr int NI = W + R + 2;                                // image slots
  static constexpr int UB = UPML ? 6 * T * 8 + 2 * NCOEF * 4 : 0;     // bytes of a plane's D, B and coefficients
  static constexpr int SMEM = 4 * (HB + EB) + 4 * 2 * NI * 8 + 4 * UB;
  static constexpr int PH = 3 * HC / 2, PE = 3 * EC / 2;              // 16-byte pieces of a plane
  static_assert(W % 2 == 0 && NC <= T * MR_S && SMEM <= 112 * 1024 && (!UPML || MR_S == 1), "tile shape");
};

// Planes z0..z1 of tile (bx, by): every thread of the CTA.  EDGE: the tile
// touches a border of the plane.
template <typename TL, bool CEPS, bool EDGE, bool ADJ>
__device__ __forceinline__ void march_column(const MarchArgs& A, unsigned char* smem, int bx, int by, int z0, int z1,
                                             float2* const* d_new, const MarchGrad* J) {
  const FieldArgs<float>& a = A.f;
  const Geo& g = a.g;
  constexpr int HC = TL::HC, EC = TL::EC, BXH = TL::BXH, BXE = TL::BXE, NI = TL::NI;
  constexpr int JH = (TL::PH + TL::T - 1) / TL::T, JE = (TL::PE + TL::T - 1) / TL::T;
  constexpr bool UPML = TL::UPML;
  const int t = threadIdx.x;
  const int x0 = 1 + bx * TL::W, y0 = 1 + by * TL::R;
  unsigned char* const sh = smem;                              // 4 planes of H
  unsigned char* const se = smem + 4 * TL::HB;                 // 4 planes of E, then E'
  float2* const si = (float2*)(smem + 4 * (TL::HB + TL::EB));  // the images' H at x = 0 [row], y = 0 [R+1+col]: [4][2][NI]
  unsigned char* const su = smem + 4 * (TL::HB + TL::EB) + 4 * 2 * NI * 8;  // UPML: [4][D, B: [6][T]; E, H rows]
  if (!bc_ok(z0 >= (UPML ? 1 : 2) && z1 + (UPML ? 0 : 1) <= g.nz && z0 <= z1 + 1, BC_FUSED_CELL, ((long)z0 << 32) | (unsigned)z1)) return;
  const float2* E = a.e;
  const float2* H = a.h;
  const int pl = (int)g.plane, pt = (int)g.pitch, cp = (int)g.comp;
  // this thread's cells
  int ih[MR_S], ie[MR_S], ow[MR_S];  // offsets in the H and E boxes and in storage (plane 0)
  int oc[MR_S], ed[MR_S];  // EDGE: storage offset of the cell whose E' it is; 1 x = nx, 2 y = ny, 4 x = 1, 8 y = 1,
                           // 16 and 32 image in x and y
  bool act[MR_S], own[MR_S];
  float ep[MR_S];
  cx<float> epc[CEPS ? MR_S : 1];
  cx<float> ev[MR_S][3];  // E' of the plane below
#pragma unroll
  for (int s = 0; s < MR_S; ++s) {
    const int c = t + s * TL::T, row = c / TL::WT, col = c - row * TL::WT, x = x0 + col, y = y0 + row;
    act[s] = (s * TL::T + TL::T <= TL::NC || c < TL::NC) && (!EDGE || (x <= g.nx + 1 && y <= g.ny + 1));
    own[s] = act[s] && col < TL::W && row < TL::R && (!EDGE || (x <= g.nx && y <= g.ny));
    ih[s] = (row + 1) * BXH + col + 2;
    ie[s] = row * BXE + col;
    ow[s] = y * pt + x + g.xo;
    oc[s] = ow[s];
    ed[s] = 0;
    if (EDGE) {
      const bool ximg = x == g.nx + 1, yimg = y == g.ny + 1;
      oc[s] = (yimg ? 1 : y) * pt + (ximg ? 1 : x) + g.xo;
      ed[s] = (x == g.nx ? 1 : 0) + (y == g.ny ? 2 : 0) + (x == 1 ? 4 : 0) + (y == 1 ? 8 : 0) + (ximg ? 16 : 0) +
              (yimg ? 32 : 0);
    }
    ep[s] = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) ev[s][k] = {0.f, 0.f};
  }
  // this thread's 16-byte pieces of the boxes: storage offset on plane 0 (-1:
  // none, past the storage rows, which only cells that are not computed would
  // read); piece t + j TL::T lies (t + j TL::T) 16 bytes into a plane of the
  // ring.  EDGE: a piece at x = nx+1 comes from x = 1; where it begins at nx,
  // its second half does (bit j of a mask; the row starts at go - xi).
  int gh[JH], ge[JE];
  unsigned mh = 0u, me = 0u;
  auto piece = [&](int id, int total, int bc, int rows, int xs, int ys, bool& split) {
    const int per = bc / 2, k = id / (rows * per), q = id - k * rows * per, rr = q / per, cc = 2 * (q - rr * per);
    int x = xs + cc, y = ys + rr;
    split = false;
    if (EDGE) {
      if (id >= total || y > g.ny + 1 || x > g.nx + 1) return -1;
      if (y == g.ny + 1) y = 1;
      if (x == g.nx + 1) x = 1;
      else split = x == g.nx;
    } else if (id >= total) {
      return -1;
    }
    return k * cp + y * pt + x + g.xo;
  };
#pragma unroll
  for (int j = 0; j < JH; ++j) {
    bool sp;
    gh[j] = piece(t + j * TL::T, TL::PH, BXH, TL::R + 2, x0 - 2, y0 - 1, sp);
    if (sp) mh |= 1u << j;
  }
#pragma unroll
  for (int j = 0; j < JE; ++j) {
    bool sp;
    ge[j] = piece(t + j * TL::T, TL::PE, BXE, TL::R + 1, x0, y0, sp);
    if (sp) me |= 1u << j;
  }
  const unsigned uh = smem_u32(sh) + 16u * t, ue = smem_u32(se) + 16u * t;
  auto copy = [&](unsigned dst, const float2* src, bool split) {
    if (EDGE && split) {
      march_cpa8(dst, src);
      march_cpa8(dst + 8u, src + 1 - g.nx);
    } else {
      march_cpa16(dst, src);
    }
  };
  // UPML: this thread's cell within a plane of D and B
  const int px = EDGE && (ed[0] & 16) ? 1 : x0 + t % TL::WT, py = EDGE && (ed[0] & 32) ? 1 : y0 + t / TL::WT;
  auto in_slab = [&](int z) { return z <= a.pmlzi || z >= a.pmlzf; };
  // everything of plane p into its ring place p & 3: one commit group a plane
  auto ahead = [&](int p) {
    if (p <= z1 + 1) {
      const int zo = (UPML && p == g.nz + 1 ? 1 : p) * pl;
      if (UPML && p >= z0) {
        // the old D of this thread's E' cell on the plane, the B of its own
        // cell on the plane below, and both planes' coefficient rows
        unsigned char* const u = su + (p & 3) * TL::UB;
        const int ze = p == g.nz + 1 ? 1 : p, zb = p - 1;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int z = q == 0 ? ze : zb;
          if (!in_slab(z) || (q == 1 && zb < z0)) continue;
          const int slab = z <= a.pmlzi ? 0 : 1, zr = slab == 0 ? z - 1 : z - a.pmlzf;
          if (q == 0 ? act[0] : own[0]) {
            const long pi = ((long)zr * g.ny + (py - 1)) * (long)g.nx + (px - 1);
            const float2* src = (q == 0 ? a.pml_d[slab] : a.pml_b[slab]) + pi;
            if (bc_ok(pi >= 0 && pi < a.pcomp[slab], BC_FUSED_SLAB, pi))
#pragma unroll
              for (int k = 0; k < 3; ++k)
                march_cpa8(smem_u32(u) + 8u * ((3 * q + k) * TL::T + t), src + k * a.pcomp[slab]);
          }
          if ((t >> 5) == q && (t & 31) < NCOEF) {
            const float* src = a.coef + NCOEF * (slab == 0 ? z - 1 : a.pmlzi + z - a.pmlzf) + (t & 31);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(u) + 48u * TL::T +
                                                                          4u * (q * NCOEF + (t & 31))),
                         "l"(src)
                         : "memory");
          }
        }
      }
      const unsigned dh = uh + (unsigned)((p & 3) * TL::HB), de = ue + (unsigned)((p & 3) * TL::EB);
#pragma unroll
      for (int j = 0; j < JH; ++j)
        if ((!EDGE && (j + 1) * TL::T <= TL::PH) || gh[j] >= 0)
          copy(dh + 16u * TL::T * j, H + (gh[j] + zo), (mh >> j) & 1u);
      if (p >= z0) {
#pragma unroll
        for (int j = 0; j < JE; ++j)
          if ((!EDGE && (j + 1) * TL::T <= TL::PE) || ge[j] >= 0)
            copy(de + 16u * TL::T * j, E + (ge[j] + zo), (me >> j) & 1u);
        if (EDGE) {
#pragma unroll
          for (int s = 0; s < MR_S; ++s) {
            if (!act[s] || !(ed[s] & 48)) continue;
            const unsigned d = smem_u32(si + (p & 3) * 2 * NI);
            const int c = t + s * TL::T, row = c / TL::WT, col = c - row * TL::WT, q = zo + oc[s];
            if (ed[s] & 16) {
              march_cpa8(d + 8u * row, H + (cp + q - 1));
              march_cpa8(d + 8u * (NI + row), H + (2 * cp + q - 1));
            }
            if (ed[s] & 32) {
              march_cpa8(d + 8u * (TL::R + 1 + col), H + (q - pt));
              march_cpa8(d + 8u * (NI + TL::R + 1 + col), H + (2 * cp + q - pt));
            }
          }
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto eps_of = [&](int p) {  // the structure's eps_inv of plane p, loaded one plane ahead
    if (UPML && p == g.nz + 1) p = 1;
    if (p >= a.hi && p <= a.hf) {
#pragma unroll
      for (int s = 0; s < MR_S; ++s)
        if (act[s]) {
          if (CEPS) epc[s] = ld<float>(a.eps_c + ((p - a.hi) * pl + oc[s]));
          else ep[s] = a.eps_r[(p - a.hi) * pl + oc[s]];
        }
    }
  };
  auto get = [](const float2* p) {
    const float2 v = *p;
    return cx<float>{v.x, v.y};
  };
  ahead(z0 - 1);
  ahead(z0);
  ahead(z0 + 1);
  ahead(z0 + 2);
  eps_of(z0);
  asm volatile("cp.async.wait_group 2;" ::: "memory");
  __syncthreads();
  for (int z = z0; z <= z1 + 1; ++z) {
    const float2* hz = (const float2*)(sh + (z & 3) * TL::HB);
    const float2* hm = (const float2*)(sh + ((z + 3) & 3) * TL::HB);  // plane z-1
    float2* ez = (float2*)(se + (z & 3) * TL::EB);
    const float2* em = (const float2*)(se + ((z + 3) & 3) * TL::EB);  // E' of plane z-1
    const int zc = UPML && z == g.nz + 1 ? 1 : z;
    const bool mat = zc >= a.hi && zc <= a.hf;
    const float mz = zc < a.hi ? a.m1 : a.m3;
#pragma unroll
    for (int s = 0; s < MR_S; ++s) {
      if (!act[s]) continue;
      cx<float> h0, h1, h2, hx1, hx2, hy0, hy2, hz0, hz1, en[3], cu[3];
      {
        const float2* p = hz + ih[s];
        h0 = get(p);
        h1 = get(p + HC);
        h2 = get(p + 2 * HC);
        hx1 = get(p + HC - 1);
        hx2 = get(p + 2 * HC - 1);
        hy0 = get(p - BXH);
        hy2 = get(p + 2 * HC - BXH);
        hz0 = get(hm + ih[s]);
        hz1 = get(hm + ih[s] + HC);
#pragma unroll
        for (int k = 0; k < 3; ++k) en[k] = get(ez + ie[s] + k * EC);
      }
      if (EDGE && (ed[s] & 48)) {
        const int c = t + s * TL::T, row = c / TL::WT, col = c - row * TL::WT;
        const float2* p = si + (z & 3) * 2 * NI;
        if (ed[s] & 16) {
          hx1 = get(p + row);
          hx2 = get(p + NI + row);
        }
        if (ed[s] & 32) {
          hy0 = get(p + TL::R + 1 + col);
          hy2 = get(p + NI + TL::R + 1 + col);
        }
      }
      if (UPML && z == g.nz + 1) {  // the image of plane 1, above H's ghost plane
        hz0 = ld<float>(H + oc[s]);
        hz1 = ld<float>(H + (cp + oc[s]));
      }
      cu[0] = cadd(csub(csub(h2, hy2), h1), hz1);
      cu[1] = cadd(csub(csub(h0, hz0), h2), hx2);
      cu[2] = cadd(csub(csub(h1, hx1), h0), hy0);
      if (UPML && in_slab(zc)) {
        const float2* u = (const float2*)(su + (z & 3) * TL::UB);
        const cx<float> dv[3] = {get(u + t), get(u + TL::T + t), get(u + 2 * TL::T + t)};
        e_apply<float, CEPS, 7, !CEPS, true>(a, own[s] && z <= z1 ? d_new : nullptr, px, py, zc, cu, en, 0.f, dv,
                                             (const float*)(u + 6 * TL::T));
      } else if (ADJ) {
#pragma unroll
        for (int k = 0; k < 3; ++k) en[k] = cadd(en[k], rmul(-a.dtcq2, cu[k]));
      } else if (CEPS && mat) {
#pragma unroll
        for (int k = 0; k < 3; ++k) en[k] = cadd(en[k], cmul(epc[CEPS ? s : 0], cu[k]));
      } else {
        const float m = mat ? ep[s] : mz;
#pragma unroll
        for (int k = 0; k < 3; ++k) en[k] = cadd(en[k], rmul(m, cu[k]));
      }
      if (EDGE && (ed[s] & 48)) {
        cx<float> ph = {1.f, 0.f};
        if (ed[s] & 16) ph = cmul(ph, a.pxp);
        if (ed[s] & 32) ph = cmul(ph, a.pyp);
#pragma unroll
        for (int k = 0; k < 3; ++k) en[k] = cmul(ph, en[k]);
      }
      if (UPML && z == g.nz + 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) en[k] = cmul(a.pzp, en[k]);
      }
      if (ADJ) {
        if (own[s] && z <= z1) {
          const int i = z * pl + ow[s];
#pragma unroll
          for (int k = 0; k < 3; ++k) st<float>(A.e_new + (k * cp + i), en[k]);
          const int c = t + s * TL::T, dx = x0 + c % TL::WT - J->x0, dy = y0 + c / TL::WT - J->y0, dz = z - J->z0;
          if (J->grad && dz >= 0 && dz < J->nz && dx >= 0 && dx < J->nx && dy >= 0 && dy < J->ny) {
            const long q = ((long)dz * J->ny + dy) * J->nx + dx;
            float g1 = 0.f;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const cx<float> r = get(J->rec + k * J->n + q);
              g1 = add_(g1, add_(mul_(en[k].re, r.re), mul_(en[k].im, r.im)));
            }
            J->grad[q] += (double)g1;
          }
        }
        const float m = mat ? ep[s] : mz;
#pragma unroll
        for (int k = 0; k < 3; ++k) en[k] = rmul(m, en[k]);  // W from here on
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) ez[ie[s] + k * EC] = make_float2(en[k].re, en[k].im);
      if (own[s]) {
        const int i = z * pl + ow[s];
        if (z > z0) {
          // H'(z-1) of the cell: h_update from E'(z-1), its +x and +y neighbours and E'(z)
          cx<float> xp[3], yp[3], zp[3], hn[3];
          const float2* p = em + ie[s];
          xp[1] = get(p + EC + 1);
          xp[2] = get(p + 2 * EC + 1);
          yp[0] = get(p + BXE);
          yp[2] = get(p + 2 * EC + BXE);
          zp[0] = en[0];
          zp[1] = en[1];
          hn[0] = hz0;
          hn[1] = hz1;
          hn[2] = get(hm + ih[s] + 2 * HC);
          if (UPML) {
            hn[0] = get(hm + ih[s]);
            hn[1] = get(hm + ih[s] + HC);
            const float2* u = (const float2*)(su + (z & 3) * TL::UB);
            const cx<float> bv[3] = {get(u + 3 * TL::T + t), get(u + 4 * TL::T + t), get(u + 5 * TL::T + t)};
            h_update<float, true>(a, px, py, z - 1, ev[s], xp, yp, zp, hn, bv, (const float*)(u + 6 * TL::T) + NCOEF);
          } else if (ADJ) {
            hn[0] = cadd(hn[0], cadd(csub(csub(yp[2], ev[s][2]), zp[1]), ev[s][1]));
            hn[1] = cadd(hn[1], cadd(csub(csub(zp[0], ev[s][0]), xp[2]), ev[s][2]));
            hn[2] = cadd(hn[2], cadd(csub(csub(xp[1], ev[s][1]), yp[0]), ev[s][0]));
          } else {
            h_update<float, false>(a, 1, 1, 1, ev[s], xp, yp, zp, hn);
          }
          const int j = i - pl;
#pragma unroll
          for (int k = 0; k < 3; ++k) st<float>(A.h_new + (k * cp + j), hn[k]);
          if (UPML && z - 1 == g.nz) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              st<float>(A.e_new + (k * cp + j - g.nz * pl), cmul(a.pzm, ev[s][k]));
              st<float>(A.h_new + (k * cp + j - g.nz * pl), cmul(a.pzm, hn[k]));
            }
          }
          if (EDGE && (ed[s] & 1)) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              if (!ADJ) st<float>(A.e_new + (k * cp + j - g.nx), cmul(a.pxm, ev[s][k]));
              st<float>(A.h_new + (k * cp + j - g.nx), cmul(a.pxm, hn[k]));
            }
          }
          if (EDGE && (ed[s] & 2)) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              if (!ADJ) st<float>(A.e_new + (k * cp + j - g.ny * pt), cmul(a.pym, ev[s][k]));
              st<float>(A.h_new + (k * cp + j - g.ny * pt), cmul(a.pym, hn[k]));
            }
          }
        }
        if (!ADJ && z <= z1) {
#pragma unroll
          for (int k = 0; k < 3; ++k) st<float>(A.e_new + (k * cp + i), en[k]);
          if (UPML && z == 1) {
#pragma unroll
            for (int k = 0; k < 3; ++k) st<float>(A.e_new + (k * cp + i + g.nz * pl), cmul(a.pzp, en[k]));
          }
          if (EDGE && (ed[s] & 4)) {
#pragma unroll
            for (int k = 0; k < 3; ++k) st<float>(A.e_new + (k * cp + i + g.nx), cmul(a.pxp, en[k]));
          }
          if (EDGE && (ed[s] & 8)) {
#pragma unroll
            for (int k = 0; k < 3; ++k) st<float>(A.e_new + (k * cp + i + g.ny * pt), cmul(a.pyp, en[k]));
          }
        }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) ev[s][k] = en[k];
    }
    eps_of(z + 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // this thread's copies of plane z+1 have landed
    __syncthreads();  // everyone's have; E'(z) is complete; plane z-1 of the ring has been read
    ahead(z + 3);
  }
  // (a batch's next column refills the ring)
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
}

template <typename TL, bool CEPS, bool ADJ = false>
__device__ __forceinline__ void march_tile(const MarchArgs& A, unsigned char* smem, int bx, int by, int z0, int z1,
                                           float2* const* d_new = nullptr, const MarchGrad* J = nullptr) {
  if (bx == 0 || by == 0 || bx == A.tx - 1 || by == A.ty - 1)
    march_column<TL, CEPS, true, ADJ>(A, smem, bx, by, z0, z1, d_new, J);
  else
    march_column<TL, CEPS, false, ADJ>(A, smem, bx, by, z0, z1, d_new, J);
}

// The tile shapes, and the one taken for an nx x ny plane: the fewest bytes of
// boxes, a row counted as 24 elements longer than the tile (its halo, the
// sectors its ends share with other tiles, and the pieces of a warp's accesses
// a row's end splits).  512x512x256 and 256x256x512, us a pass: 54x8 1420 and
// 662, 44x10 1410 and 662, 32x14 1428 and 675, 24x19 1482 and 697, 16x29 1547
// and 725; wider ones (60x7, 72x6) lose on ragged planes.
#define IRIS_MARCH_SHAPES(F) F(0, 32, 14) F(1, 24, 19) F(2, 16, 29) F(3, 44, 10) F(4, 54, 8)
#define IRIS_MARCH_SMEM(ID, W, R) MarchTile<W, R>::SMEM,
constexpr int MARCH_MAX_SMEM = std::max({IRIS_MARCH_SHAPES(IRIS_MARCH_SMEM) 0});
#undef IRIS_MARCH_SMEM
// The slabs' march: the same column with the old D and B of its cells and the
// coefficients in the ring, tiles half the size (two CTAs of 256 threads an SM).
// Of a pass of 512x512x256 with slabs of 17 planes fused_column took 480 us at
// 38 % of the copy bandwidth, and the pass 1420 us; it takes 1321 so, 256x256x512
// 625 instead of 662, 256x256x96 159 instead of 167.
#define IRIS_SLAB_SHAPES(F) F(0, 32, 6) F(1, 24, 9) F(2, 16, 14) F(3, 40, 5)
constexpr int MS_T = 256;
template <int W, int R> using SlabTile = MarchTile<W, R, MS_T, true>;
#define IRIS_SLAB_SMEM(ID, W, R) SlabTile<W, R>::SMEM,
constexpr int SLAB_MAX_SMEM = std::max({IRIS_SLAB_SHAPES(IRIS_SLAB_SMEM) 0});
#undef IRIS_SLAB_SMEM
struct MarchShape {
  int id = -1, w = 0, r = 0, tx = 0, ty = 0;  // id < 0: none; cells of a tile, tiles of the plane
  size_t smem = 0;
};
inline MarchShape march_shape(int nx, int ny) {
  MarchShape best;
  double cost = 1e300;
#define IRIS_MARCH_TRY(ID, W, R)                                        \
  {                                                                     \
    const int tx = (nx + W - 1) / W, ty = (ny + R - 1) / R;             \
    const double c = (double)tx * ty * (W + 24) * (R + 1.5);            \
    if (c < cost) {                                                     \
      cost = c;                                                         \
      best.id = ID, best.w = W, best.r = R, best.tx = tx, best.ty = ty;                        \
      best.smem = MarchTile<W, R>::SMEM;                                \
    }                                                                   \
  }
  IRIS_MARCH_SHAPES(IRIS_MARCH_TRY)
#undef IRIS_MARCH_TRY
  return best;
}
inline MarchShape slab_shape(int nx, int ny) {
  MarchShape best;
  double cost = 1e300;
#define IRIS_SLAB_TRY(ID, W, R)                                         \
  {                                                                     \
    const int tx = (nx + W - 1) / W, ty = (ny + R - 1) / R;             \
    const double c = (double)tx * ty * (W + 24) * (R + 1.5);            \
    if (c < cost) {                                                     \
      cost = c;                                                         \
      best.id = ID, best.w = W, best.r = R, best.tx = tx, best.ty = ty;                        \
      best.smem = SlabTile<W, R>::SMEM;                                 \
    }                                                                   \
  }
  IRIS_SLAB_SHAPES(IRIS_SLAB_TRY)
#undef IRIS_SLAB_TRY
  return best;
}
// Tile rows and z chunks that a launch holds in grid.y and grid.z (of each of its
// two ranges).  Planes of more tile rows step with the column of iris_fused.cuh
// (both axes in one index, or a tile row to start from as an argument, cost the
// marches 0.3 to 3 %).
constexpr int MR_MAX_ROWS = 65535, MR_MAX_CHUNKS = 32767;
// Planes of a z chunk of len planes: MR_CHUNK to 2 MR_CHUNK - 1, or len; more
// where there would be too many chunks.
inline int march_chunk(int len) {
  const int n = std::min(MR_MAX_CHUNKS, std::max(1, len / MR_CHUNK));
  return (len + n - 1) / n;
}

// The same in the slabs: 12 to 23, or len (512x512x256, slabs of 17 planes, a
// pass: 1359 us in chunks of 5 planes, 1334 of 9, 1321 of 17; 256x256x96 163, 160, 159).
inline int slab_chunk(int len) {
  const int n = std::min(MR_MAX_CHUNKS, std::max(1, len / 12));
  return (len + n - 1) / n;
}

}  // namespace iris
