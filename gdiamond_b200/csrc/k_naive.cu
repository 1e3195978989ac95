// k_naive.cu -- separate E and H launches per step, in place, over the whole grid.
//
// The B200 counterpart of the reference's naive GPU kernels updateE_3Dmap_fix /
// updateH_3Dmap_fix (gDiamond/kernels.cuh:337-394) and of the per-step DFT kernel
// update_field_FFT_xy (gDiamond/kernels.cuh:87-113).  Differences by design: the pitched
// layout, per-step source values read from a device waveform table (no per-step memcpy), FP64
// monitor sums, and the coefficients read either from 12 per-cell arrays or from a material
// map + table.  Every multiply/add is separately rounded, so results are bit-identical to the
// reference's CPU update.
#include <algorithm>

#include "fdtd_kernels.cuh"

namespace fdtd {

struct CoefArrays {
  const float* c[12];  // pitched per-cell arrays, Cax Cay Caz Cbx Cby Cbz Dax Day Daz Dbx Dby Dbz
};

// Arithmetic of one field type, every operation separately rounded.
template <typename T>
struct Arith;
template <>
struct Arith<float> {
  __device__ static float sub(float a, float b) { return __fsub_rn(a, b); }
  __device__ static float mul(float a, float b) { return __fmul_rn(a, b); }
  __device__ static float add(float a, float b) { return __fadd_rn(a, b); }
};
template <>
struct Arith<double> {
  __device__ static double sub(double a, double b) { return __dsub_rn(a, b); }
  __device__ static double mul(double a, double b) { return __dmul_rn(a, b); }
  __device__ static double add(double a, double b) { return __dadd_rn(a, b); }
};

// Source term in type T: the FP32 waveform samples of all covering sources summed in T.
template <typename T>
__device__ __forceinline__ bool source_value_t(const Sources& S, int comp, int i, int j, int k,
                                               long long t, T* v) {
  T acc = 0;
  bool any = false;
  for (int n = 0; n < S.n; ++n) {
    const SourceDev& s = S.s[n];
    if (s.comp != comp) continue;
    const bool hit = (s.kind == 0) ? (s.i == i && s.j == j && s.k == k) : (s.k == k);
    if (hit) {
      acc = Arith<T>::add(acc, (T)(t < S.tw ? S.wave[n * S.tw + t] : 0.0f));
      any = true;
    }
  }
  *v = acc;
  return any;
}

// A pair of x-neighbours: one 8- or 16-byte access.
template <typename T>
struct Pair {
  T x, y;
};
template <typename T>
__device__ __forceinline__ Pair<T> ld(const T* p) {
  if constexpr (sizeof(T) == 4) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    return {v.x, v.y};
  } else {
    const double2 v = *reinterpret_cast<const double2*>(p);
    return {v.x, v.y};
  }
}
template <typename T>
__device__ __forceinline__ void st(T* p, const Pair<T>& v) {
  if constexpr (sizeof(T) == 4)
    *reinterpret_cast<float2*>(p) = make_float2(v.x, v.y);
  else
    *reinterpret_cast<double2*>(p) = make_double2(v.x, v.y);
}
template <typename T>
__device__ __forceinline__ Pair<T> sub(const Pair<T>& a, const Pair<T>& b) {
  return {Arith<T>::sub(a.x, b.x), Arith<T>::sub(a.y, b.y)};
}

constexpr int kNaiveThreads = 128;

// E (H = false) or H half step, in place.  T = float or double (FP64 storage: the error reference
// of reduced-precision runs; coefficients and waveforms are widened).  A thread owns an x-pair of
// one row and marches up through zc planes: the z-neighbours of the curls are its registers of
// the plane before, and addresses, face tests and source tests are paid once per march.  The E half
// step goes up through the grid and the H half step down, so that each starts on what the other
// touched last (in L2).  Bound: memory (9 field values per cell and half step).  160^3 FP64, 40
// steps and a 16-frequency monitor: 4.0 ms, 5.3 with one cell per thread (5.0 of them with the
// reversed H half step alone).
// blockIdx.x = pairs of a plane, blockIdx.y = z-chunk.
template <typename T, bool H, bool kMat>
__global__ void __launch_bounds__(kNaiveThreads)
    naive_half(const Grid g, const FieldPtrs Fp, const CoefArrays A, const uint16_t* mat,
               const Material* tab, const __grid_constant__ Sources S, long long t, float dx_f,
               int zc) {
  using R = Arith<T>;
  T* const* F = reinterpret_cast<T* const*>(Fp.f);
  const int npx = (g.nx + 1) / 2;
  const int q = (int)(blockIdx.x * kNaiveThreads + threadIdx.x);
  const int j = q / npx, i0 = 2 * (q - j * npx);
  if (j < 1 || j > g.ny - 2) return;  // (rows past the last one too)
  const bool u0 = i0 >= 1 && i0 <= g.nx - 2, u1 = i0 + 1 <= g.nx - 2;
  const int chunk = H ? (int)(gridDim.y - 1 - blockIdx.y) : (int)blockIdx.y;
  const int k0 = max(1, chunk * zc), k1 = min(g.nz - 1, chunk * zc + zc);
  if (k0 >= k1) return;
  const T dx = (T)dx_f;
  int slo = 1 << 30, shi = -1;
  for (int n = 0; n < S.n; ++n)
    if ((S.s[n].comp >= 3) == H) slo = min(slo, S.s[n].k), shi = max(shi, S.s[n].k);
  // fields differenced (s) and advanced (d)
  const T* const s0 = F[H ? 0 : 3];
  const T* const s1 = F[H ? 1 : 4];
  const T* const s2 = F[H ? 2 : 5];
  T* const d0 = F[H ? 3 : 0];
  T* const d1 = F[H ? 4 : 1];
  T* const d2 = F[H ? 5 : 2];
  const long long sy = H ? (long long)g.pitch : -(long long)g.pitch;
  long long idx = i0 + (long long)j * g.pitch + (long long)k0 * g.plane;
  // E: components 0, 1 of H at plane k-1; H: components 0, 1 of E at plane k
  Pair<T> c0 = ld(s0 + idx - (H ? 0 : g.plane)), c1 = ld(s1 + idx - (H ? 0 : g.plane));
  for (int k = k0; k < k1; ++k, idx += g.plane) {
    const Pair<T> v2 = ld(s2 + idx);
    const Pair<T> n0 = ld(s0 + idx + (H ? g.plane : 0)), n1 = ld(s1 + idx + (H ? g.plane : 0));
    const Pair<T> y0 = ld(s0 + idx + sy), y2 = ld(s2 + idx + sy);
    T x1 = 0, x2 = 0;  // the neighbour across the pair's edge
    if (H ? i0 + 2 < g.nx : i0 > 0) {
      x1 = s1[idx + (H ? 2 : -1)];
      x2 = s2[idx + (H ? 2 : -1)];
    }
    Pair<T> f0 = ld(d0 + idx), f1 = ld(d1 + idx), f2 = ld(d2 + idx);
    // E: (dyHz - dzHy, dzHx - dxHz, dxHy - dyHx); H: (dzEy - dyEz, dxEz - dzEx, dyEx - dxEy)
    Pair<T> cx, cy, cz;
    if (!H) {
      const Pair<T> dx2 = sub(v2, Pair<T>{x2, v2.x}), dx1 = sub(n1, Pair<T>{x1, n1.x});
      cx = sub(sub(v2, y2), sub(n1, c1));
      cy = sub(sub(n0, c0), dx2);
      cz = sub(dx1, sub(n0, y0));
    } else {
      const Pair<T> dx2 = sub(Pair<T>{v2.y, x2}, v2), dx1 = sub(Pair<T>{c1.y, x1}, c1);
      cx = sub(sub(n1, c1), sub(y2, v2));
      cy = sub(dx2, sub(n0, c0));
      cz = sub(sub(y0, c0), dx1);
    }
    if (k >= slo && k <= shi) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        T v;
        T& ax = e ? cx.y : cx.x;
        T& ay = e ? cy.y : cy.x;
        T& az = e ? cz.y : cz.x;
        if (source_value_t<T>(S, H ? 3 : 0, i0 + e, j, k, t, &v)) ax = R::sub(ax, R::mul(v, dx));
        if (source_value_t<T>(S, H ? 4 : 1, i0 + e, j, k, t, &v)) ay = R::sub(ay, R::mul(v, dx));
        if (source_value_t<T>(S, H ? 5 : 2, i0 + e, j, k, t, &v)) az = R::sub(az, R::mul(v, dx));
      }
    }
    float2 ca[3], cb[3];  // Ca, Cb (Da, Db) of the pair per component
    if (kMat) {
      const ushort2 id = *reinterpret_cast<const ushort2*>(mat + idx);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const Material* m = tab + (e ? id.y : id.x);
        const float2 h = __ldg(reinterpret_cast<const float2*>(&m->b) + (H ? 1 : 0));
        const float4 w = __ldg(H ? &m->c : &m->a);
        // E: {Cax, Cbx, Cay, Cby} = w, {Caz, Cbz} = h; H: {Dax, Dbx} = h, {Day .. Dbz} = w
        const float a0 = H ? h.x : w.x, b0 = H ? h.y : w.y, a1 = H ? w.x : w.z;
        const float b1 = H ? w.y : w.w, a2 = H ? w.z : h.x, b2 = H ? w.w : h.y;
        (e ? ca[0].y : ca[0].x) = a0;
        (e ? cb[0].y : cb[0].x) = b0;
        (e ? ca[1].y : ca[1].x) = a1;
        (e ? cb[1].y : cb[1].x) = b1;
        (e ? ca[2].y : ca[2].x) = a2;
        (e ? cb[2].y : cb[2].x) = b2;
      }
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        ca[c] = *reinterpret_cast<const float2*>(A.c[(H ? 6 : 0) + c] + idx);
        cb[c] = *reinterpret_cast<const float2*>(A.c[(H ? 9 : 3) + c] + idx);
      }
    }
    auto advance = [&](Pair<T>& f, const Pair<T>& c, const float2& a, const float2& b) {
      const T vx = R::add(R::mul((T)a.x, f.x), R::mul((T)b.x, c.x));
      const T vy = R::add(R::mul((T)a.y, f.y), R::mul((T)b.y, c.y));
      f.x = u0 ? vx : f.x;  // faces and the pad column keep their value
      f.y = u1 ? vy : f.y;
    };
    advance(f0, cx, ca[0], cb[0]);
    advance(f1, cy, ca[1], cb[1]);
    advance(f2, cz, ca[2], cb[2]);
    st(d0 + idx, f0);
    st(d1 + idx, f1);
    st(d2 + idx, f2);
    c0 = n0;
    c1 = n1;
  }
}

// One thread per plane cell of every monitor: grid (ceil(nx/32), ceil(ny/8), nmon), block (32, 8)
template <typename T>
__global__ void __launch_bounds__(256) naive_dft(Grid g, FieldPtrs Fp, Monitors M, long long t) {
  T* const* F = reinterpret_cast<T* const*>(Fp.f);
  const int i = blockIdx.x * 32 + threadIdx.x;
  const int j = blockIdx.y * 8 + threadIdx.y;
  if (i >= g.nx || j >= g.ny || (int)blockIdx.z >= M.n) return;
  const MonitorDev& m = M.m[blockIdx.z];
  const double v = (double)F[m.comp][i + (long long)j * g.pitch + (long long)m.k * g.plane];
  const double2* tab = m.tab + t * m.nf;
  const long long np = (long long)g.nx * g.ny;
  const long long p = i + (long long)j * g.nx;
  for (int f = 0; f < m.nf; ++f) {
    const double2 cs = tab[f];
    double* re = m.re + f * np + p;
    double* im = m.im + f * np + p;
    *re = dadd(*re, dmul(dmul(v, cs.x), m.scale));
    *im = dsub(*im, dmul(dmul(v, cs.y), m.scale));
  }
}

template <typename T>
void naive_step_t(const Grid& g, const FieldPtrs& F, const CoefArrays& A, const uint16_t* mat,
                  const Material* tab, const Sources& S, const Monitors& M, long long t, float dx,
                  cudaStream_t st, int* launches) {
  const long long pairs = (long long)((g.nx + 1) / 2) * g.ny;
  const long long nb = (pairs + kNaiveThreads - 1) / kNaiveThreads;
  // planes per march: at least 8 blocks per SM before it gets longer, and single planes where pairs of
  // them leave fewer than 4 (a march is then only a chain of loads: FP64 48^3 8.1 us a step with one
  // plane, 11.3 with two; 80^3 14.3 and 12.3)
  const auto blocks = [&](int planes) { return nb * ((g.nz + planes - 1) / planes); };
  int zc = 16;
  while (zc > 2 && blocks(zc) < 148 * 8) zc /= 2;
  if (blocks(zc) < 148 * 4) zc = 1;
  zc = std::max(zc, (g.nz + 65534) / 65535);
  const dim3 grd((unsigned)nb, (unsigned)((g.nz + zc - 1) / zc));
  if (mat) {
    naive_half<T, false, true><<<grd, kNaiveThreads, 0, st>>>(g, F, A, mat, tab, S, t, dx, zc);
    naive_half<T, true, true><<<grd, kNaiveThreads, 0, st>>>(g, F, A, mat, tab, S, t, dx, zc);
  } else {
    naive_half<T, false, false><<<grd, kNaiveThreads, 0, st>>>(g, F, A, mat, tab, S, t, dx, zc);
    naive_half<T, true, false><<<grd, kNaiveThreads, 0, st>>>(g, F, A, mat, tab, S, t, dx, zc);
  }
  *launches += 2;
  if (M.n) {
    const dim3 b2(32, 8), g2((g.nx + 31) / 32, (g.ny + 7) / 8, M.n);
    naive_dft<T><<<g2, b2, 0, st>>>(g, F, M, t);
    *launches += 1;
  }
}

cudaError_t launch_naive_step(const Grid& g, const FieldPtrs& F, const float* const* coef,
                              const uint16_t* mat, const Material* tab, const Sources& S,
                              const Monitors& M, long long t, float dx, cudaStream_t st,
                              int* launches, bool fp64) {
  CoefArrays A;
  for (int c = 0; c < 12; ++c) A.c[c] = coef ? coef[c] : nullptr;
  if (fp64)
    naive_step_t<double>(g, F, A, mat, tab, S, M, t, dx, st, launches);
  else
    naive_step_t<float>(g, F, A, mat, tab, S, M, t, dx, st, launches);
  return cudaGetLastError();
}

}  // namespace fdtd
