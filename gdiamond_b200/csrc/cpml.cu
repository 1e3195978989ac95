// cpml.cu -- convolutional PML (CPML) absorbing layers: per-step E and H kernels with the
// auxiliary psi fields of the layers.
//
// The reference absorbs with a graded pseudo-PML folded into Ca/Cb/Da/Db (a real-valued
// stretch, gDiamond/utils.h:585-660) in front of PEC faces that are never updated
// (gDiamond/gdiamond.hpp:1193-1221); outgoing waves are partly reflected.  A CPML layer instead
// replaces each spatial difference d in the curl by d / kappa + psi, with the recursive
// convolution psi <- b psi + a d (complex-frequency-shifted stretch s = kappa + sigma /
// (alpha + i w), in the normalised units of the reference: eps0 = mu0 = c = 1):
//
//   Ex <- Ca Ex + Cb [ (dyHz/ky + psi_exy) - (dzHy/kz + psi_exz) - Jx dx ],   dyHz = Hz(j) - Hz(j-1)
//
// and likewise for the other five components.  Profiles along each axis are tabulated at the E
// positions (integer n) and the H positions (n + 1/2).  Outside every layer a component's update
// is the reference's formula, operation for operation, so the interior stays bit-identical to
// the non-PML solver; psi is stored only in the slabs of its axis (2L + 1 positions).
//
// Whole grids step with cpml_half<H>: one E and one H launch per step, for one grid or for a
// group of grids of a batch (blockIdx.z = grid).  Monitor values are staged for the deferred DFT.
// cpml_region recomputes listed cells for the shell companion of the tiled kernel.
#include <algorithm>
#include <cstring>

#include "fdtd_kernels.cuh"

namespace fdtd {

namespace {

__device__ __forceinline__ void e_coefs(const uint16_t* mat, const Material* tab, long long idx,
                                        float* ca, float* cb) {
  const Material m = tab[mat[idx]];
  ca[0] = m.a.x; cb[0] = m.a.y; ca[1] = m.a.z; cb[1] = m.a.w; ca[2] = m.b.x; cb[2] = m.b.y;
}

__device__ __forceinline__ void h_coefs(const uint16_t* mat, const Material* tab, long long idx,
                                        float* da, float* db) {
  const Material m = tab[mat[idx]];
  da[0] = m.b.z; db[0] = m.b.w; da[1] = m.c.x; db[1] = m.c.y; da[2] = m.c.z; db[2] = m.c.w;
}

// psi slab element of axis a at slot s for cell (i, j, k)
__device__ __forceinline__ long long psi_at(const Grid& g, int a, int S, int s, int i, int j, int k) {
  if (a == 0) return s + (long long)S * (j + (long long)g.ny * k);
  if (a == 1) return i + (long long)g.nx * (s + (long long)S * k);
  return i + (long long)g.nx * (j + (long long)g.ny * s);
}

// The CPML form of one difference d along axis a at table position n: updates psi in place and
// returns d / kappa + psi; outside the layer (slot < 0) returns d itself.
__device__ __forceinline__ float stretched(float d, const CpmlAxis& ax, bool h, int n,
                                           float* psi, long long pidx) {
  const int s = h ? ax.slot_h[n] : ax.slot_e[n];
  if (s < 0) return d;
  const float b = h ? ax.bh[n] : ax.be[n], a = h ? ax.ah[n] : ax.ae[n];
  const float ik = h ? ax.ikh[n] : ax.ike[n];
  const float p = add(mul(b, psi[pidx]), mul(a, d));
  psi[pidx] = p;
  return add(mul(d, ik), p);
}

__device__ __forceinline__ bool src_sum(const Sources& S, int comp, int i, int j, int k,
                                        long long t, float* v) {
  return source_value(S, comp, i, j, k, t, v);
}

__device__ __forceinline__ bool interior(const Grid& g, int i, int j, int k) {
  return i >= 1 && i <= g.nx - 2 && j >= 1 && j <= g.ny - 2 && k >= 1 && k <= g.nz - 2;
}

// E update of interior cell (i, j, k) at step t: E and H of step t from Fi, the new E into Fo
// (Fi == Fo: in place).
__device__ __forceinline__ void e_cell(const Grid& g, const FieldPtrs& Fi, const FieldPtrs& Fo,
                                       const uint16_t* mat, const Material* tab,
                                       const Sources& S, long long t,
                                       float dx, const CpmlDev& P, int i, int j, int k) {
  const long long sy = g.pitch, sz = g.plane, idx = i + j * sy + k * sz;
  float* const* f = Fi.f;
  const float hx = f[3][idx], hy = f[4][idx], hz = f[5][idx];
  const float dyHz = sub(hz, f[5][idx - sy]), dzHy = sub(hy, f[4][idx - sz]);
  const float dzHx = sub(hx, f[3][idx - sz]), dxHz = sub(hz, f[5][idx - 1]);
  const float dxHy = sub(hy, f[4][idx - 1]), dyHx = sub(hx, f[3][idx - sy]);
  const CpmlAxis& X = P.ax[0];
  const CpmlAxis& Y = P.ax[1];
  const CpmlAxis& Z = P.ax[2];
  float cx, cy, cz;
  if (X.slot_e[i] < 0 && Y.slot_e[j] < 0 && Z.slot_e[k] < 0) {  // the reference's update
    cx = sub(dyHz, dzHy);
    cy = sub(dzHx, dxHz);
    cz = sub(dxHy, dyHx);
  } else {
    const int sxs = X.slot_e[i] < 0 ? 0 : X.slot_e[i], sys = Y.slot_e[j] < 0 ? 0 : Y.slot_e[j];
    const int szs = Z.slot_e[k] < 0 ? 0 : Z.slot_e[k];
    cx = sub(stretched(dyHz, Y, false, j, P.psi_e[0], psi_at(g, 1, Y.S, sys, i, j, k)),
             stretched(dzHy, Z, false, k, P.psi_e[1], psi_at(g, 2, Z.S, szs, i, j, k)));
    cy = sub(stretched(dzHx, Z, false, k, P.psi_e[2], psi_at(g, 2, Z.S, szs, i, j, k)),
             stretched(dxHz, X, false, i, P.psi_e[3], psi_at(g, 0, X.S, sxs, i, j, k)));
    cz = sub(stretched(dxHy, X, false, i, P.psi_e[4], psi_at(g, 0, X.S, sxs, i, j, k)),
             stretched(dyHx, Y, false, j, P.psi_e[5], psi_at(g, 1, Y.S, sys, i, j, k)));
  }
  if (S.n) {
    float v;
    if (src_sum(S, 0, i, j, k, t, &v)) cx = sub(cx, mul(v, dx));
    if (src_sum(S, 1, i, j, k, t, &v)) cy = sub(cy, mul(v, dx));
    if (src_sum(S, 2, i, j, k, t, &v)) cz = sub(cz, mul(v, dx));
  }
  float ca[3], cb[3];
  e_coefs(mat, tab, idx, ca, cb);
  const float ex = f[0][idx], ey = f[1][idx], ez = f[2][idx];
  Fo.f[0][idx] = yee(ca[0], ex, cb[0], cx);
  Fo.f[1][idx] = yee(ca[1], ey, cb[1], cy);
  Fo.f[2][idx] = yee(ca[2], ez, cb[2], cz);
}

// H update of interior cell (i, j, k) at step t, after every E update of the step: H of step t
// from Fi, the new E from Fo, the new H into Fo (Fi == Fo: in place).
__device__ __forceinline__ void h_cell(const Grid& g, const FieldPtrs& Fi, const FieldPtrs& Fo,
                                       const uint16_t* mat, const Material* tab,
                                       const Sources& S, long long t,
                                       float dx, const CpmlDev& P, int i, int j, int k) {
  const long long sy = g.pitch, sz = g.plane, idx = i + j * sy + k * sz;
  float* const* f = Fo.f;
  const float ex = f[0][idx], ey = f[1][idx], ez = f[2][idx];
  const float dzEy = sub(f[1][idx + sz], ey), dyEz = sub(f[2][idx + sy], ez);
  const float dxEz = sub(f[2][idx + 1], ez), dzEx = sub(f[0][idx + sz], ex);
  const float dyEx = sub(f[0][idx + sy], ex), dxEy = sub(f[1][idx + 1], ey);
  const CpmlAxis& X = P.ax[0];
  const CpmlAxis& Y = P.ax[1];
  const CpmlAxis& Z = P.ax[2];
  float cx, cy, cz;
  if (X.slot_h[i] < 0 && Y.slot_h[j] < 0 && Z.slot_h[k] < 0) {  // the reference's update
    cx = sub(dzEy, dyEz);
    cy = sub(dxEz, dzEx);
    cz = sub(dyEx, dxEy);
  } else {
    const int sxs = X.slot_h[i] < 0 ? 0 : X.slot_h[i], sys = Y.slot_h[j] < 0 ? 0 : Y.slot_h[j];
    const int szs = Z.slot_h[k] < 0 ? 0 : Z.slot_h[k];
    cx = sub(stretched(dzEy, Z, true, k, P.psi_h[0], psi_at(g, 2, Z.S, szs, i, j, k)),
             stretched(dyEz, Y, true, j, P.psi_h[1], psi_at(g, 1, Y.S, sys, i, j, k)));
    cy = sub(stretched(dxEz, X, true, i, P.psi_h[2], psi_at(g, 0, X.S, sxs, i, j, k)),
             stretched(dzEx, Z, true, k, P.psi_h[3], psi_at(g, 2, Z.S, szs, i, j, k)));
    cz = sub(stretched(dyEx, Y, true, j, P.psi_h[4], psi_at(g, 1, Y.S, sys, i, j, k)),
             stretched(dxEy, X, true, i, P.psi_h[5], psi_at(g, 0, X.S, sxs, i, j, k)));
  }
  if (S.n) {
    float v;
    if (src_sum(S, 3, i, j, k, t, &v)) cx = sub(cx, mul(v, dx));
    if (src_sum(S, 4, i, j, k, t, &v)) cy = sub(cy, mul(v, dx));
    if (src_sum(S, 5, i, j, k, t, &v)) cz = sub(cz, mul(v, dx));
  }
  float da[3], db[3];
  h_coefs(mat, tab, idx, da, db);
  const float hx = Fi.f[3][idx], hy = Fi.f[4][idx], hz = Fi.f[5][idx];
  Fo.f[3][idx] = yee(da[0], hx, db[0], cx);
  Fo.f[4][idx] = yee(da[1], hy, db[1], cy);
  Fo.f[5][idx] = yee(da[2], hz, db[2], cz);
}

// ------------------------------------------------------------------ whole-grid half steps
// A thread owns kCpmlV = 2 consecutive x cells (a cell pair, one 8-byte access per field) of one
// row and marches along z, so the z-neighbours of the curls are its own registers of the plane
// before and everything that depends on x and y alone (addresses, layer slots and profiles of x
// and y, face tests) is computed once per march instead of once per cell.  The pairs of a row
// that touch an x layer (XL) are marched by blocks of their own: no warp runs the x-layer code
// for a few of its lanes.  The y layers are uniform along a row, the z layers along a plane.
//
// Bound: memory (38 bytes per cell and half step plus the layers' psi) off the layers, latency in
// them.  The pointers stay in the constant bank (kernel parameters) instead of registers; psi is
// loaded where it is used, one axis after the other: that makes a chain of the layers' loads but
// leaves 64 registers and 32 warps per SM, where loading everything first needs 80.  B200, both half
// steps: 32 grids of 96^3 with 8 layer cells 0.55 ms a step (51 Gcell-updates/s; one thread per
// cell without a march 1.57 ms; all loads first 0.58), 256^3 with 10 layer cells 0.28 ms (59; 0.52;
// 0.30).  Four cells per thread (128 registers, 12 warps) took 0.74 and 0.33 ms; loading a plane
// ahead, prefetching into L2, and stepping a batch in groups that fit the L2 cache gained nothing.
constexpr int V = kCpmlV;
constexpr int kHalfThreads = 128;

struct Cells {
  float v[V];
};
__device__ __forceinline__ Cells ldv(const float* p) {
  const float2 f = *reinterpret_cast<const float2*>(p);
  return {{f.x, f.y}};
}
__device__ __forceinline__ void stv(float* p, const Cells& q) {
  *reinterpret_cast<float2*>(p) = make_float2(q.v[0], q.v[1]);
}
__device__ __forceinline__ Cells subv(const Cells& a, const Cells& b) {
  Cells r;
#pragma unroll
  for (int e = 0; e < V; ++e) r.v[e] = sub(a.v[e], b.v[e]);
  return r;
}

// psi of V cells of one row along y or z; vec: whole-pair accesses are aligned.  Cells outside
// `upd` (faces, padding) have no psi.
__device__ __forceinline__ Cells ld_psi(const float* psi, bool vec, const bool* upd) {
  if (vec) return ldv(psi);
  Cells p;
#pragma unroll
  for (int e = 0; e < V; ++e) p.v[e] = upd[e] ? psi[e] : 0.0f;
  return p;
}
__device__ __forceinline__ void st_psi(float* psi, const Cells& p, bool vec, const bool* upd) {
  if (vec) {
    stv(psi, p);
    return;
  }
#pragma unroll
  for (int e = 0; e < V; ++e)
    if (upd[e]) psi[e] = p.v[e];
}
// d <- d / kappa + psi for one profile entry; p becomes the new psi in the cells of `upd`.
__device__ __forceinline__ void stretch(Cells& d, float b, float a, float ik, Cells& p,
                                        const bool* upd) {
#pragma unroll
  for (int e = 0; e < V; ++e) {
    const float n = add(mul(b, p.v[e]), mul(a, d.v[e]));
    p.v[e] = upd[e] ? n : p.v[e];
    d.v[e] = add(mul(d.v[e], ik), n);
  }
}

// E (H = false) or H half step of step t over planes [k0, k1) of cells i0 .. i0+V-1 of row j, in
// place.  P: layers; s: sources, monitors, material and per-cell coefficients.
template <bool H, bool XL>
__device__ __forceinline__ void march_row(const CpmlHot& h, const CpmlSim& s, long long t, int i0,
                                          int j, int k0, int k1) {
  const Grid& g = h.g;
  const bool jrow = j >= 1 && j <= g.ny - 2;
  bool upd[V];
#pragma unroll
  for (int e = 0; e < V; ++e) upd[e] = jrow && i0 + e >= 1 && i0 + e <= g.nx - 2;
  const bool vec = (g.nx & (V - 1)) == 0;
  const CpmlAxis &X = h.P.ax[0], &Y = h.P.ax[1], &Z = h.P.ax[2];
  // x layers: a layer's slots are consecutive, xs + e for the cells with xin[e]
  int xs = 0;
  bool xin[V] = {};
  float xb[V], xa[V], xi[V];
  if (XL) {
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const int i = min(i0 + e, g.nx - 1), sl = H ? X.slot_h[i] : X.slot_e[i];
      xin[e] = upd[e] && sl >= 0;
      if (xin[e]) xs = sl - e;
      xb[e] = H ? X.bh[i] : X.be[i];
      xa[e] = H ? X.ah[i] : X.ae[i];
      xi[e] = H ? X.ikh[i] : X.ike[i];
    }
  }
  const int ys = H ? Y.slot_h[j] : Y.slot_e[j];
  const float yb = H ? Y.bh[j] : Y.be[j], ya = H ? Y.ah[j] : Y.ae[j], yi = H ? Y.ikh[j] : Y.ike[j];
  const int lean_id = s.lean ? s.lean_id : -1;
  const float lean_c = H ? s.lean_db : s.lean_cb;
  // planes that some source or monitor of this half step touches
  int slo = 1 << 30, shi = -1, mlo = 1 << 30, mhi = -1;
  for (int n = 0; n < s.S.n; ++n)
    if ((s.S.s[n].comp >= 3) == H) slo = min(slo, s.S.s[n].k), shi = max(shi, s.S.s[n].k);
  for (int n = 0; n < s.M.n; ++n)
    if ((s.M.m[n].comp >= 3) == H) mlo = min(mlo, s.M.m[n].k), mhi = max(mhi, s.M.m[n].k);

  // offset of the row's cells in a plane; the planes' bases are uniform
  const uint32_t o = (uint32_t)(i0 + j * g.pitch);
  const uint32_t oy = H ? o + (uint32_t)g.pitch : o - (uint32_t)g.pitch;
  // E: components 0, 1 of H at plane k-1; H: components 0, 1 of E at plane k
  Cells c0 = {}, c1 = {};
  if (jrow && k0 + (H ? 0 : -1) >= 0) {
    const long long b = (long long)(k0 + (H ? 0 : -1)) * g.plane;
    c0 = ldv(h.F.f[H ? 0 : 3] + b + o);
    c1 = ldv(h.F.f[H ? 1 : 4] + b + o);
  }
  for (int k = k0; k < k1; ++k) {
    const long long base = (long long)k * g.plane;
    const long long bnew = base + (H ? g.plane : 0);
    // fields differenced (s0, s1, s2) and advanced (d0, d1, d2)
    const float* const s0 = h.F.f[H ? 0 : 3] + base;
    const float* const s1 = h.F.f[H ? 1 : 4] + base;
    const float* const s2 = h.F.f[H ? 2 : 5] + base;
    const float* const n0p = h.F.f[H ? 0 : 3] + bnew;
    const float* const n1p = h.F.f[H ? 1 : 4] + bnew;
    float* const d0 = h.F.f[H ? 3 : 0] + base;
    float* const d1 = h.F.f[H ? 4 : 1] + base;
    float* const d2 = h.F.f[H ? 5 : 2] + base;
    if (jrow) {
      if (k >= 1 && k <= g.nz - 2) {
        Cells f0 = ldv(d0 + o), f1 = ldv(d1 + o), f2 = ldv(d2 + o);
        const Cells v2 = ldv(s2 + o);
        const Cells n0 = ldv(n0p + o), n1 = ldv(n1p + o);
        const Cells y0 = ldv(s0 + oy), y2 = ldv(s2 + oy);
        float x1 = 0.0f, x2 = 0.0f;
        if (H ? i0 + V < g.nx : i0 > 0) {
          x1 = s1[o + (H ? V : -1)];
          x2 = s2[o + (H ? V : -1)];
        }
        ushort2 id = {};
        if (h.mat) id = *reinterpret_cast<const ushort2*>(h.mat + base + o);
        const int zs = H ? Z.slot_h[k] : Z.slot_e[k];
        float* const* psi = H ? h.P.psi_h : h.P.psi_e;
        // curl = (dy2 - dz1, dz0 - dx2, dx1 - dy0) for E, the negative for H
        Cells dy2 = H ? subv(y2, v2) : subv(v2, y2), dy0 = H ? subv(y0, c0) : subv(n0, y0);
        Cells dz1 = subv(n1, c1), dz0 = subv(n0, c0), dx2, dx1;
#pragma unroll
        for (int e = 0; e < V; ++e) {
          if (!H) {
            dx2.v[e] = sub(v2.v[e], e ? v2.v[e - 1] : x2);
            dx1.v[e] = sub(n1.v[e], e ? n1.v[e - 1] : x1);
          } else {
            dx2.v[e] = sub(e < V - 1 ? v2.v[e + 1] : x2, v2.v[e]);
            dx1.v[e] = sub(e < V - 1 ? c1.v[e + 1] : x1, c1.v[e]);
          }
        }
        if (ys >= 0) {
          float* const a2 = psi[H ? 1 : 0] + (long long)g.nx * Y.S * k + (uint32_t)(i0 + g.nx * ys);
          float* const a0 = psi[H ? 4 : 5] + (long long)g.nx * Y.S * k + (uint32_t)(i0 + g.nx * ys);
          Cells p2 = ld_psi(a2, vec, upd), p0 = ld_psi(a0, vec, upd);
          stretch(dy2, yb, ya, yi, p2, upd);
          stretch(dy0, yb, ya, yi, p0, upd);
          st_psi(a2, p2, vec, upd);
          st_psi(a0, p0, vec, upd);
        }
        if (zs >= 0) {
          const float b = H ? Z.bh[k] : Z.be[k], a = H ? Z.ah[k] : Z.ae[k];
          const float ik = H ? Z.ikh[k] : Z.ike[k];
          float* const a1 = psi[H ? 0 : 1] + (long long)g.nx * g.ny * zs + (uint32_t)(i0 + g.nx * j);
          float* const a0 = psi[H ? 3 : 2] + (long long)g.nx * g.ny * zs + (uint32_t)(i0 + g.nx * j);
          Cells p1 = ld_psi(a1, vec, upd), p0 = ld_psi(a0, vec, upd);
          stretch(dz1, b, a, ik, p1, upd);
          stretch(dz0, b, a, ik, p0, upd);
          st_psi(a1, p1, vec, upd);
          st_psi(a0, p0, vec, upd);
        }
        if (XL) {
          float* const a2 = psi[H ? 2 : 3] + (long long)X.S * g.ny * k + (xs + X.S * j);
          float* const a1 = psi[H ? 5 : 4] + (long long)X.S * g.ny * k + (xs + X.S * j);
          Cells p2, p1;
#pragma unroll
          for (int e = 0; e < V; ++e) {
            p2.v[e] = xin[e] ? a2[e] : 0.0f;
            p1.v[e] = xin[e] ? a1[e] : 0.0f;
          }
#pragma unroll
          for (int e = 0; e < V; ++e)
            if (xin[e]) {
              a2[e] = p2.v[e] = add(mul(xb[e], p2.v[e]), mul(xa[e], dx2.v[e]));
              a1[e] = p1.v[e] = add(mul(xb[e], p1.v[e]), mul(xa[e], dx1.v[e]));
              dx2.v[e] = add(mul(dx2.v[e], xi[e]), p2.v[e]);
              dx1.v[e] = add(mul(dx1.v[e], xi[e]), p1.v[e]);
            }
        }
        // E: (dyHz - dzHy, dzHx - dxHz, dxHy - dyHx); H: (dzEy - dyEz, dxEz - dzEx, dyEx - dxEy)
        Cells u0 = H ? subv(dz1, dy2) : subv(dy2, dz1);
        Cells u1 = H ? subv(dx2, dz0) : subv(dz0, dx2);
        Cells u2 = H ? subv(dy0, dx1) : subv(dx1, dy0);
        if (k >= slo && k <= shi) {
          const float dx = s.dx;
#pragma unroll
          for (int e = 0; e < V; ++e) {
            float v;
            if (source_value(s.S, H ? 3 : 0, i0 + e, j, k, t, &v)) u0.v[e] = sub(u0.v[e], mul(v, dx));
            if (source_value(s.S, H ? 4 : 1, i0 + e, j, k, t, &v)) u1.v[e] = sub(u1.v[e], mul(v, dx));
            if (source_value(s.S, H ? 5 : 2, i0 + e, j, k, t, &v)) u2.v[e] = sub(u2.v[e], mul(v, dx));
          }
        }
        if (h.mat) {
          const int ids[V] = {id.x, id.y};
          if (id.x == lean_id && id.y == lean_id) {
#pragma unroll
            for (int e = 0; e < V; ++e) {  // the a coefficients are 1 and 1 * f == f
              f0.v[e] = upd[e] ? add(f0.v[e], mul(lean_c, u0.v[e])) : f0.v[e];
              f1.v[e] = upd[e] ? add(f1.v[e], mul(lean_c, u1.v[e])) : f1.v[e];
              f2.v[e] = upd[e] ? add(f2.v[e], mul(lean_c, u2.v[e])) : f2.v[e];
            }
          } else {
#pragma unroll
            for (int e = 0; e < V; ++e) {
              const Material* m = h.tab + ids[e];
              const float2 q = __ldg(reinterpret_cast<const float2*>(&m->b) + (H ? 1 : 0));
              const float4 w = __ldg(H ? &m->c : &m->a);
              // E: {Cax, Cbx, Cay, Cby} = w, {Caz, Cbz} = q; H: {Dax, Dbx} = q, {Day .. Dbz} = w
              const float m0 = H ? yee(q.x, f0.v[e], q.y, u0.v[e]) : yee(w.x, f0.v[e], w.y, u0.v[e]);
              const float m1 = H ? yee(w.x, f1.v[e], w.y, u1.v[e]) : yee(w.z, f1.v[e], w.w, u1.v[e]);
              const float m2 = H ? yee(w.z, f2.v[e], w.w, u2.v[e]) : yee(q.x, f2.v[e], q.y, u2.v[e]);
              f0.v[e] = upd[e] ? m0 : f0.v[e];
              f1.v[e] = upd[e] ? m1 : f1.v[e];
              f2.v[e] = upd[e] ? m2 : f2.v[e];
            }
          }
        } else {
          const int c = H ? 6 : 0;
          const Cells a0 = ldv(s.coef[c] + base + o), b0 = ldv(s.coef[c + 3] + base + o);
          const Cells a1 = ldv(s.coef[c + 1] + base + o), b1 = ldv(s.coef[c + 4] + base + o);
          const Cells a2 = ldv(s.coef[c + 2] + base + o), b2 = ldv(s.coef[c + 5] + base + o);
#pragma unroll
          for (int e = 0; e < V; ++e) {
            f0.v[e] = upd[e] ? yee(a0.v[e], f0.v[e], b0.v[e], u0.v[e]) : f0.v[e];
            f1.v[e] = upd[e] ? yee(a1.v[e], f1.v[e], b1.v[e], u1.v[e]) : f1.v[e];
            f2.v[e] = upd[e] ? yee(a2.v[e], f2.v[e], b2.v[e], u2.v[e]) : f2.v[e];
          }
        }
        stv(d0 + o, f0);
        stv(d1 + o, f1);
        stv(d2 + o, f2);
        c0 = n0;
        c1 = n1;
      } else if (k + (H ? 1 : 0) < g.nz) {  // a z face: nothing changes, carry the neighbours on
        c0 = ldv(n0p + o);
        c1 = ldv(n1p + o);
      }
    }
    if (k >= mlo && k <= mhi) {  // face cells too: the fold reads every cell of the plane
      for (int n = 0; n < s.M.n; ++n) {
        const MonitorDev& m = s.M.m[n];
        if ((m.comp >= 3) != H || m.k != k) continue;
        const float* f = h.F.f[m.comp] + base + o;
#pragma unroll
        for (int e = 0; e < V; ++e)
          if (i0 + e < g.nx) dft_record(m, t, i0 + e, j, g, f[e]);
      }
    }
  }
}

// Work of CTA b of the blocks of one z-chunk: first the quads off the x layers, then those that
// touch one.
template <bool H>
__device__ __forceinline__ void half_block(const CpmlHot& h, const CpmlSim& s, long long t, int b,
                                           int k0, int k1) {
  const Grid& g = h.g;
  const int nq = (g.nx + V - 1) / V, nl = h.ql[H], nlay = nl + h.qr[H], nint = nq - nlay;
  const int bint = (nint * g.ny + kHalfThreads - 1) / kHalfThreads;
  if (b < bint) {
    const int q = b * kHalfThreads + (int)threadIdx.x;
    const int j = q / nint;
    if (j < g.ny) march_row<H, false>(h, s, t, V * (nl + q - j * nint), j, k0, k1);
  } else if (nlay > 0) {
    const int q = (b - bint) * kHalfThreads + (int)threadIdx.x;
    const int j = q / nlay, l = q - j * nlay;
    if (j < g.ny) march_row<H, true>(h, s, t, V * (l < nl ? l : l + nint), j, k0, k1);
  }
}

// One grid (arguments in the parameters): blockIdx.x = cells, blockIdx.y = z-chunk of zc planes.
template <bool H>
__global__ void __launch_bounds__(kHalfThreads, 8) cpml_half(const __grid_constant__ CpmlHot h,
                                                          const __grid_constant__ CpmlSim s,
                                                          long long t, int zc) {
  const int k0 = (int)blockIdx.y * zc;
  half_block<H>(h, s, t, (int)blockIdx.x, k0, min(h.g.nz, k0 + zc));
}

// The grids of one launch of a batch.  Every launch, and every node of a captured graph, carries the
// parameters it is declared with, so there are a few sizes.  Above 4 KB (9 grids) they are dear: a
// first call of 900 steps captures and starts its graph in 4 to 6 ms for 2 or 8 grids, in 11 ms with
// the 13 KB of 32 grids (and 14 with the 6.6 KB of 16).
template <int G>
struct CpmlGroup {
  CpmlHot h[G];
};

// A group of grids of a batch: blockIdx.z = grid of the group.
template <bool H, int G>
__global__ void __launch_bounds__(kHalfThreads, 8)
    cpml_half_batch(const __grid_constant__ CpmlGroup<G> grp, const CpmlSim* __restrict__ sims,
                    long long t_offset, int zc) {
  const CpmlHot& h = grp.h[blockIdx.z];
  const CpmlSim& s = sims[blockIdx.z];
  const int k0 = (int)blockIdx.y * zc;
  if (k0 >= h.g.nz) return;
  half_block<H>(h, s, s.t0 + t_offset, (int)blockIdx.x, k0, min(h.g.nz, k0 + zc));
}

// The shell companion: blockIdx.x indexes the block list; cells inside `inner` return.
template <bool H>
__global__ void __launch_bounds__(128) cpml_region(Grid g, FieldPtrs Fi, FieldPtrs Fo,
                                                   const uint16_t* mat, const Material* tab,
                                                   Sources S, Monitors M, CpmlDev P, long long t,
                                                   float dx, const int4* blocks, CpmlBox inner) {
  const int4 b = blocks[blockIdx.x];
  const int i = b.x * 32 + threadIdx.x, j = b.y * 4 + threadIdx.y, k = b.z;
  if (i >= g.nx || j >= g.ny || k >= g.nz) return;
  if (i >= inner.lo[0] && i < inner.hi[0] && j >= inner.lo[1] && j < inner.hi[1] &&
      k >= inner.lo[2] && k < inner.hi[2])
    return;
  const long long idx = i + (long long)j * g.pitch + (long long)k * g.plane;
  const int c0 = H ? 3 : 0;
  if (interior(g, i, j, k)) {
    if (H)
      h_cell(g, Fi, Fo, mat, tab, S, t, dx, P, i, j, k);
    else
      e_cell(g, Fi, Fo, mat, tab, S, t, dx, P, i, j, k);
  } else if (Fi.f[c0] != Fo.f[c0]) {  // faces never change: carry them into the output set
    for (int c = c0; c < c0 + 3; ++c) Fo.f[c][idx] = Fi.f[c][idx];
  }
  for (int n = 0; n < M.n; ++n) {
    const MonitorDev& m = M.m[n];
    if ((m.comp >= 3) == H && m.k == k) dft_record(m, t, i, j, g, Fo.f[m.comp][idx]);
  }
}

}  // namespace

cudaError_t launch_cpml_region(bool h_half, const Grid& g, const FieldPtrs& Fi,
                               const FieldPtrs& Fo, const uint16_t* mat, const Material* tab,
                               const Sources& S, const Monitors& M, const CpmlDev& P,
                               long long t, float dx, const int4* blocks, int nblocks,
                               const CpmlBox& inner, cudaStream_t st) {
  if (nblocks <= 0) return cudaSuccess;
  if (!mat) return cudaErrorInvalidValue;
  if (h_half)
    cpml_region<true><<<nblocks, dim3(32, 4), 0, st>>>(g, Fi, Fo, mat, tab, S, M, P, t, dx,
                                                        blocks, inner);
  else
    cpml_region<false><<<nblocks, dim3(32, 4), 0, st>>>(g, Fi, Fo, mat, tab, S, M, P, t, dx,
                                                         blocks, inner);
  return cudaGetLastError();
}

namespace {

// Blocks that cover one z-chunk of grid h (the more of the E and the H half step).
int cpml_blocks(const CpmlHot& h) {
  int most = 0;
  for (int k = 0; k < 2; ++k) {
    const int nlay = h.ql[k] + h.qr[k], nint = (h.g.nx + V - 1) / V - nlay;
    most = std::max(most, (nint * h.g.ny + kHalfThreads - 1) / kHalfThreads +
                              (nlay * h.g.ny + kHalfThreads - 1) / kHalfThreads);
  }
  return most;
}

// Planes per z-chunk: a longer march amortises its set-up and the extra plane it loads, but every SM
// should have several blocks.  Where even single planes do not give them, a march only makes a chain
// of its planes' loads: 32^3 cells with 6 layer cells take 12.7 us a step with single planes, 24.4
// with four (the floor of the loop before), 96^3 with 8 layer cells 25.1 with two and 27.3 with four.
int cpml_planes(long long blocks, int nz) {
  int zc = 16;
  while (zc > 1 && blocks * ((nz + zc - 1) / zc) < 148 * 8) zc /= 2;
  return zc;
}

template <int G>
cudaError_t launch_group(const CpmlHot* hot, int n, const CpmlSim* sims, long long t_offset,
                         int zc, dim3 grd, cudaStream_t st) {
  CpmlGroup<G> grp;
  memset(&grp, 0, sizeof(grp));
  std::copy(hot, hot + n, grp.h);
  cpml_half_batch<false, G><<<grd, kHalfThreads, 0, st>>>(grp, sims, t_offset, zc);
  cpml_half_batch<true, G><<<grd, kHalfThreads, 0, st>>>(grp, sims, t_offset, zc);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_cpml_batch_step(const CpmlHot* hot, int n, const CpmlSim* sims,
                                   long long t_offset, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (n > kCpmlGroup) return cudaErrorInvalidValue;
  long long blocks = 0;
  int most = 0, max_nz = 0;
  for (int q = 0; q < n; ++q) {
    const int b = cpml_blocks(hot[q]);
    blocks += b;
    most = std::max(most, b);
    max_nz = std::max(max_nz, hot[q].g.nz);
  }
  const int zc = std::max(cpml_planes(blocks, max_nz), (max_nz + 65534) / 65535);
  const dim3 grd((unsigned)most, (unsigned)((max_nz + zc - 1) / zc), (unsigned)n);
  if (n <= 2) return launch_group<2>(hot, n, sims, t_offset, zc, grd, st);
  if (n <= 8) return launch_group<8>(hot, n, sims, t_offset, zc, grd, st);
  return launch_group<kCpmlGroup>(hot, n, sims, t_offset, zc, grd, st);
}

cudaError_t launch_cpml_step(const CpmlHot& h, const CpmlSim& s, long long t, cudaStream_t st,
                             int* launches) {
  const int nb = cpml_blocks(h);
  const int zc = std::max(cpml_planes(nb, h.g.nz), (h.g.nz + 65534) / 65535);
  const dim3 grd((unsigned)nb, (unsigned)((h.g.nz + zc - 1) / zc));
  cpml_half<false><<<grd, kHalfThreads, 0, st>>>(h, s, t, zc);
  cpml_half<true><<<grd, kHalfThreads, 0, st>>>(h, s, t, zc);
  *launches += 2;
  return cudaGetLastError();
}

}  // namespace fdtd
