// dft_fold.cu -- the deferred half of the running DFT monitors.
//
// The tiled kernels do not touch a monitor's FP64 sums: every step they write the monitor
// plane's FP32 values into slot t % kDftSlots of the monitor's staging ring (dft_record).  A fold
// adds a window of n <= kDftSlots consecutive steps to the sums:
//   re[f][p] += (v_t[p] * cos_t[f]) * scale,  im[f][p] -= (v_t[p] * sin_t[f]) * scale
// for t ascending, with separately rounded FP64 operations -- the same operations in the same
// order per (f, p) as accumulating once per step (the FP64 form of the reference's
// update_field_FFT_xy, kernels.cuh:87-113), so the sums are bit-identical to it.  What changes
// is the memory traffic: a step costs 4 bytes per monitor cell written and read back instead of
// a read-modify-write of 2 * nf doubles (1 KB at 32 frequencies), and the sums are read and
// written once per window.
//
// A thread owns two plane cells and kFoldF frequencies: their sums stay in registers for the whole
// window, the staged values of consecutive cells are coalesced, and each (cos, sin) pair of a
// step, a broadcast load, serves both cells.  Bound: FP64 issue with many monitors or frequencies,
// the latency of a step's loads with few (256 x 256 cells, 8 frequencies: 256 blocks, 7 warps per SM).
#include "fdtd_kernels.cuh"

namespace fdtd {

namespace {

constexpr int kFoldThreads = 128;
constexpr int kFoldF = 8;  // frequencies per thread

constexpr int kFoldP = 2;  // plane cells per thread, kFoldThreads apart

// Adds n staged steps from t0 on to the sums of NF frequencies from f0 on, for the plane cells p[].
// NF is a constant: a run-time count splits the step into a branch per frequency, with no independent
// work between them (5 frequencies of 6 monitors of 400 x 400 cells: 1.46 ms a window of 128 steps with
// a run-time count, 0.87 with constants).
template <int NF, bool SCALED>
__device__ __forceinline__ void fold_cells(const MonitorDev& m, long long np,
                                           const long long (&p)[kFoldP], bool two, int f0,
                                           long long t0, int n) {
  // (always NF; as a run-time guard of the first loads it makes the compiler keep the loop's registers
  // apart from theirs: without it 8 frequencies take 1.3 times as long)
  const int nfc = min(kFoldF, m.nf - f0);
  double re[kFoldP][NF], im[kFoldP][NF];
#pragma unroll
  for (int c = 0; c < kFoldP; ++c)
#pragma unroll
    for (int q = 0; q < NF; ++q) {
      re[c][q] = q < nfc ? m.re[(long long)(f0 + q) * np + p[c]] : 0.0;
      im[c][q] = q < nfc ? m.im[(long long)(f0 + q) * np + p[c]] : 0.0;
    }
  const float* const st0 = m.stage + p[0];
  const float* const st1 = m.stage + p[1];
  const double scale = m.scale;
  const int nf = m.nf;
  const double2* tab0 = m.tab + t0 * nf + f0;
  const int slot0 = (int)(t0 & (kDftSlots - 1));
#pragma unroll 2
  for (int s = 0; s < n; ++s) {
    const long long o = (long long)((slot0 + s) & (kDftSlots - 1)) * np;
    const double v[kFoldP] = {(double)st0[o], (double)st1[o]};
    const double2* tab = tab0 + (long long)s * nf;
#pragma unroll
    for (int q = 0; q < NF; ++q) {
      const double2 cs = __ldg(&tab[q]);
#pragma unroll
      for (int k = 0; k < kFoldP; ++k) {
        double c = dmul(v[k], cs.x), d = dmul(v[k], cs.y);
        if (SCALED) {
          c = dmul(c, scale);
          d = dmul(d, scale);
        }
        re[k][q] = dadd(re[k][q], c);
        im[k][q] = dsub(im[k][q], d);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < kFoldP; ++c)
#pragma unroll
    for (int q = 0; q < NF; ++q)
      if (c == 0 || two) {
        m.re[(long long)(f0 + q) * np + p[c]] = re[c][q];
        m.im[(long long)(f0 + q) * np + p[c]] = im[c][q];
      }
}

template <int NF>
__device__ __forceinline__ void fold_group(const MonitorDev& m, long long np,
                                           const long long (&p)[kFoldP], bool two, int f0,
                                           long long t0, int n) {
  // x * 1.0 == x: without a scale two of the six operations per step and frequency fall away
  if (m.scale == 1.0)
    fold_cells<NF, false>(m, np, p, two, f0, t0, n);
  else
    fold_cells<NF, true>(m, np, p, two, f0, t0, n);
}

__device__ __forceinline__ void fold_monitor(const MonitorDev& m, const Grid& g, long long t0,
                                             int n) {
  const long long np = (long long)g.nx * g.ny;
  const long long p0 = (long long)blockIdx.x * (kFoldThreads * kFoldP) + threadIdx.x;
  const int f0 = (int)blockIdx.y * kFoldF;
  if (m.stage == nullptr || p0 >= np || f0 >= m.nf) return;
  // a thread without a second cell folds its first one twice and stores it once
  const bool two = p0 + kFoldThreads < np;
  const long long p[kFoldP] = {p0, two ? p0 + kFoldThreads : p0};
  static_assert(kFoldF == 8, "the cases below");
  switch (min(kFoldF, m.nf - f0)) {
    case 1: fold_group<1>(m, np, p, two, f0, t0, n); break;
    case 2: fold_group<2>(m, np, p, two, f0, t0, n); break;
    case 3: fold_group<3>(m, np, p, two, f0, t0, n); break;
    case 4: fold_group<4>(m, np, p, two, f0, t0, n); break;
    case 5: fold_group<5>(m, np, p, two, f0, t0, n); break;
    case 6: fold_group<6>(m, np, p, two, f0, t0, n); break;
    case 7: fold_group<7>(m, np, p, two, f0, t0, n); break;
    default: fold_group<8>(m, np, p, two, f0, t0, n); break;
  }
}

// One grid: blockIdx.z is the monitor.
__global__ void __launch_bounds__(kFoldThreads) dft_fold(const __grid_constant__ Monitors M,
                                                         const Grid g, long long t0, int n) {
  if ((int)blockIdx.z < M.n) fold_monitor(M.m[blockIdx.z], g, t0, n);
}

// A batch: blockIdx.z is grid * kMaxMonitors + monitor; the grid's arguments (monitors, step counter
// t0 at the start of the batch step) are the ones the batched kernel reads (TiledArgs, or CpmlSim for
// CPML batches).
// The window starts t_offset steps later.
template <class Args>
__global__ void __launch_bounds__(kFoldThreads) dft_fold_batch(const Args* grids,
                                                               long long t_offset, int n) {
  const Args& a = grids[blockIdx.z / kMaxMonitors];
  const int k = (int)blockIdx.z % kMaxMonitors;
  if (k < a.M.n) fold_monitor(a.M.m[k], a.g, a.t0 + t_offset, n);
}

dim3 fold_grid(long long max_np, int max_nf, int nz) {
  constexpr int per = kFoldThreads * kFoldP;
  return dim3((unsigned)((max_np + per - 1) / per),
              (unsigned)((max_nf + kFoldF - 1) / kFoldF), (unsigned)nz);
}

// Launches of as many grids as blockIdx.z can number.
template <class Args>
cudaError_t fold_batch(const Args* grids, int ngrids, long long max_np, int max_nf,
                       long long t_offset, int n, cudaStream_t st) {
  constexpr int per = 65535 / kMaxMonitors;
  for (int g0 = 0; g0 < ngrids; g0 += per) {
    const int ng = ngrids - g0 < per ? ngrids - g0 : per;
    dft_fold_batch<Args><<<fold_grid(max_np, max_nf, ng * kMaxMonitors), kFoldThreads, 0, st>>>(
        grids + g0, t_offset, n);
  }
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_dft_fold(const Monitors& M, const Grid& g, long long t0, int n,
                            cudaStream_t st) {
  if (M.n <= 0 || n <= 0) return cudaSuccess;
  if (n > kDftSlots || t0 < 0) return cudaErrorInvalidValue;
  int max_nf = 0;
  for (int k = 0; k < M.n; ++k) max_nf = max_nf > M.m[k].nf ? max_nf : M.m[k].nf;
  dft_fold<<<fold_grid((long long)g.nx * g.ny, max_nf, M.n), kFoldThreads, 0, st>>>(M, g, t0, n);
  return cudaGetLastError();
}

cudaError_t launch_dft_fold_batch(const TiledArgs* grids, int ngrids, long long max_np,
                                  int max_nf, long long t_offset, int n, cudaStream_t st) {
  if (ngrids <= 0 || max_nf <= 0 || n <= 0) return cudaSuccess;
  if (n > kDftSlots || t_offset < 0) return cudaErrorInvalidValue;
  return fold_batch(grids, ngrids, max_np, max_nf, t_offset, n, st);
}

cudaError_t launch_dft_fold_cpml_batch(const CpmlSim* sims, int nsims, long long max_np,
                                       int max_nf, long long t_offset, int n, cudaStream_t st) {
  if (nsims <= 0 || max_nf <= 0 || n <= 0) return cudaSuccess;
  if (n > kDftSlots || t_offset < 0) return cudaErrorInvalidValue;
  return fold_batch(sims, nsims, max_np, max_nf, t_offset, n, st);
}

}  // namespace fdtd
