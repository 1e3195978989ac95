// mlp_train.cu -- one training epoch of the surrogate MLP ensemble in one launch.
//
// A minibatch step of the ensemble is a chain of small dependent products (64 rows, widths up to
// 256): as separate launches (gather, 4 forward products, loss, 4 x {weight gradient, column sum,
// input gradient}, Adam: 20 of them) each one costs a launch, a cold start and a tail for about a
// microsecond of work.  Here a cluster of 16 CTAs (8 for more than 4 members) takes one member
// through every minibatch of the epoch.  The members are independent, so nothing waits outside
// its cluster.  4 members of 6-256-256-256-64, 4096 rows in batches of 64: 37 us a step instead of
// 154 (8 CTAs 58, 16 CTAs of 256 threads 45); bound by the latency of the chain (issue slots 38 %
// busy, fixed-latency and barrier stalls).
//
// Split: CTA c owns a slice of 16-column groups of every layer's outputs.  It computes those
// columns forward (its rows of W_l) and backward (its columns of G_{l-1}), keeps the matching rows
// of dW_l in registers and applies Adam to exactly the rows of W_l that only it reads forward.
// Activations and gradients cross CTAs through global memory (L2) as BF16, ordered by the
// cluster barrier: one per layer forward, one per hidden layer backward.  Between the arrival
// and the wait of a backward barrier a CTA computes dW_l and the bias gradients, so only the
// input-gradient products are on the critical path.  A barrier also separates the last read of
// W_l in a step (dX_l, by all CTAs) from its update.
//
// Arithmetic is that of the separate kernels in mlp.cu, operation for operation: mma.sync with
// FP32 accumulators over k in steps of 16, the same epilogues, column sums in row order, the same
// Adam update.  A tcgen05 tile has 128 rows; a minibatch of 64 would leave half of it empty and
// the products are bound by latency, not by tensor throughput.
#include "fdtd_common.cuh"
#include "mlp.cuh"

namespace fdtd {
namespace mlp {
namespace {

constexpr int kThreads = 512;  // 16 warps
constexpr int kWarps = kThreads / 32;
constexpr int kUnits = kTrainMaxWidth / 8 / kWarps;  // 8-column units of dW per warp, at most
constexpr int kRows = kTrainMaxRows, kWidth = kTrainMaxWidth;
constexpr int LD = kWidth + 8;   // row stride of the row-operand tiles (BF16), conflict-free
constexpr int LDW = 32 + 8;      // row stride of a column slice of W
constexpr uint32_t OFF_B = kRows * LD * 2;
constexpr uint32_t OFF_W = OFF_B + kRows * LD * 2;
constexpr uint32_t OFF_G = OFF_W + kWidth * LDW * 2;
constexpr uint32_t OFF_R = OFF_G + kRows * 33 * 4;
constexpr uint32_t kSmem = OFF_R + kRows * 4;
static_assert(32 * LD <= kWidth * LDW, "the forward slice of W fits the backward one's space");
static_assert(kSmem <= 227 * 1024, "shared memory per CTA");

__device__ __forceinline__ void cp16(void* s, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <bool T>
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const __nv_bfloat16* p) {
  if (T)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}
template <bool T>
__device__ __forceinline__ void ldsm2(uint32_t (&r)[2], const __nv_bfloat16* p) {
  if (T)
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                 : "=r"(r[0]), "=r"(r[1]) : "r"(smem_u32(p)));
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
                 : "=r"(r[0]), "=r"(r[1]) : "r"(smem_u32(p)));
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Rows [0, rows) x columns [0, cols) of src (row stride ld elements, cols % 8 == 0, 16-byte
// aligned rows) into s (row stride lds); rows up to rows_pad become zero.  Asynchronous.
__device__ __forceinline__ void copy_rows(__nv_bfloat16* s, int lds, const __nv_bfloat16* src,
                                          int ld, int rows, int rows_pad, int cols) {
  const int cpr = cols / 8;
  if (cpr == 0) return;
  const int dr = kThreads / cpr, dc = kThreads - dr * cpr;  // row and chunk steps of a thread
  int r = (int)threadIdx.x / cpr, c = (int)threadIdx.x - r * cpr;
  while (r < rows_pad) {
    if (r < rows)
      cp16(s + r * lds + 8 * c, src + (long long)r * ld + 8 * c);
    else
      *reinterpret_cast<uint4*>(s + r * lds + 8 * c) = make_uint4(0, 0, 0, 0);
    r += dr;
    c += dc;
    if (c >= cpr) {
      c -= cpr;
      ++r;
    }
  }
}

// The minibatch's inputs as BF16: rows of X by index, columns padded with zeros to 16.
__device__ __forceinline__ void gather_rows(__nv_bfloat16* s, const float* X, const int* row, int in,
                                            int rows, int rows_pad, int cols_pad) {
  for (int q = threadIdx.x; q < rows_pad * cols_pad; q += kThreads) {
    const int r = q / cols_pad, c = q - r * cols_pad;
    const float v = r < rows && c < in ? X[(long long)row[r] * in + c] : 0.0f;
    s[r * LD + c] = __float2bfloat16_rn(v);
  }
}

// acc[j] += A (16 rows from row m0 of sA, k contiguous) x the 8 columns from n0 + 8 j of B, over K
// (multiple of 16); BT: B is stored [k][n] (row stride LDW), else [n][k] (row stride LD).
template <bool BT, int NJ>
__device__ __forceinline__ void product(float (&acc)[NJ][4], const __nv_bfloat16* sA, int m0,
                                        const __nv_bfloat16* sB, int n0, int K) {
  const int lane = threadIdx.x & 31;
  const __nv_bfloat16* pa = sA + (m0 + (lane & 15)) * LD + (lane >> 4) * 8;
  const __nv_bfloat16* pb[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j)
    pb[j] = BT ? sB + (lane & 15) * LDW + n0 + 8 * j
               : sB + (n0 + 8 * j + (lane & 7)) * LD + ((lane >> 3) & 1) * 8;
#pragma unroll 4
  for (int k = 0; k < K; k += 16) {
    uint32_t a[4], b[2];
    ldsm4<false>(a, pa + k);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      ldsm2<BT>(b, BT ? pb[j] + k * LDW : pb[j] + k);
      mma(acc[j], a, b);
    }
  }
}

// Column slice of CTA c in a layer of n outputs (n % 16 == 0): [first, first + count).
template <int CTAS>
__device__ __forceinline__ void slice(int n, int c, int* first, int* count) {
  const int groups = n / 16, per = (groups + CTAS - 1) / CTAS;
  const int g0 = min(c * per, groups), g1 = min(g0 + per, groups);
  *first = 16 * g0;
  *count = 16 * (g1 - g0);
}

// Bias gradient of the CTA's columns (summed in row order from sG, row stride 33) and its update.
__device__ __forceinline__ void bias_step(const TrainArgs& a, long long po, int l, int first,
                                          int count, int M, const float* sG, const AdamStep& ad) {
  const int c = (int)threadIdx.x - (kThreads - 32);  // the last warp
  if (c < 0 || c >= count) return;
  float s = 0.0f;
#pragma unroll 8
  for (int r = 0; r < M; ++r) s += sG[r * 33 + c];
  const long long i = po + a.b_off[l] + first + c;
  float w = a.params[i], m = a.adam_m[i], v = a.adam_v[i];
  adam_update(w, m, v, s, ad);
  a.params[i] = w;
  a.adam_m[i] = m;
  a.adam_v[i] = v;
  a.wbf[i] = __float2bfloat16_rn(w);
}

template <int CTAS>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(kThreads, 1)
    train_epoch(const __grid_constant__ TrainArgs a) {
  constexpr int NJ = 16 / CTAS;  // 8-column tiles a warp computes at a time; 16-row tiles of dW
  constexpr int RT = 16 / CTAS;
  extern __shared__ __align__(16) unsigned char smem[];
  __nv_bfloat16* sA = reinterpret_cast<__nv_bfloat16*>(smem);
  __nv_bfloat16* sB = reinterpret_cast<__nv_bfloat16*>(smem + OFF_B);
  __nv_bfloat16* sW = reinterpret_cast<__nv_bfloat16*>(smem + OFF_W);
  float* sG = reinterpret_cast<float*>(smem + OFF_G);
  int* sRow = reinterpret_cast<int*>(smem + OFF_R);
  const int c = (int)blockIdx.x % CTAS, e = (int)blockIdx.x / CTAS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
  const long long po = e * a.P;
  const int L = a.L, in0 = a.dims[0], in_pad = (in0 + 15) / 16 * 16, out = a.dims[L];

  double loss_sum = 0.0;  // lane 0: the warp's squared errors of the whole epoch
  for (int step = 0; step < a.steps; ++step) {
    const long long r0 = (long long)step * a.batch;
    const int M = (int)min((long long)a.batch, a.n - r0), M16 = (M + 15) / 16 * 16, mt = M16 / 16;
    const AdamStep ad{a.lr, a.b1, a.b2, a.eps, a.corr[step].x, a.corr[step].y};
    __syncthreads();  // the previous step's readers of the shared tiles are done
    for (int r = tid; r < M; r += kThreads) sRow[r] = a.perm[e * a.n + r0 + r];
    __syncthreads();
    // ------------------------------------------------------------------ forward
    for (int l = 0; l < L; ++l) {
      const int K = a.dims[l], K16 = l == 0 ? in_pad : K, N = a.dims[l + 1];
      int first, count;
      slice<CTAS>(N, c, &first, &count);
      // W rows of the slice do not wait for the other CTAs: only this one updates them
      if (l == 0) {
        for (int q = tid; q < count * in_pad; q += kThreads) {
          const int r = q / in_pad, k = q - r * in_pad;
          sW[r * LD + k] = k < in0 ? a.wbf[po + a.w_off[0] + (long long)(first + r) * in0 + k]
                                   : __float2bfloat16(0.0f);
        }
        gather_rows(sA, a.X, sRow, in0, M, M16, in_pad);
      } else {
        copy_rows(sW, LD, a.wbf + po + a.w_off[l] + (long long)first * K, K, count, count, K);
        cluster_wait();
        copy_rows(sA, LD, a.act[l] + (long long)e * a.cap * K, K, M, M16, K);
      }
      cp_wait();
      __syncthreads();
      float loss = 0.0f;
      const int tiles = mt * (count / (8 * NJ));  // 16 rows x 8 NJ columns each
      for (int t = warp; t < tiles; t += kWarps) {
        const int m0 = (t % mt) * 16, n0 = (t / mt) * 8 * NJ;
        float2 bv[NJ], yv[NJ][2];  // loaded ahead of the product that hides their latency
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const int col = first + n0 + 8 * j + 2 * tig;
          bv[j] = *reinterpret_cast<const float2*>(a.params + po + a.b_off[l] + col);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = m0 + gid + 8 * h;
            if (l + 1 == L && r < M)
              yv[j][h] = *reinterpret_cast<const float2*>(a.Y + (long long)sRow[r] * out + col);
          }
        }
        float acc[NJ][4] = {};
        product<false, NJ>(acc, sA, m0, sW, n0, K16);
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = m0 + gid + 8 * h, lc = n0 + 8 * j + 2 * tig, col = first + lc;
            if (r >= M) continue;
            const float v0 = acc[j][2 * h] + bv[j].x, v1 = acc[j][2 * h + 1] + bv[j].y;
            const long long o = ((long long)e * a.cap + r) * N + col;
            if (l + 1 < L) {
              *reinterpret_cast<float2*>(a.z[l] + o) = make_float2(v0, v1);
              *reinterpret_cast<__nv_bfloat162*>(a.act[l + 1] + o) =
                  __halves2bfloat162(__float2bfloat16_rn(gelu(v0)), __float2bfloat16_rn(gelu(v1)));
            } else {  // the loss's gradient
              const float scale = 2.0f / ((float)M * (float)N);
              const float d0 = v0 - yv[j][h].x, d1 = v1 - yv[j][h].y;
              loss += d0 * d0 + d1 * d1;
              const float g0 = scale * d0, g1 = scale * d1;
              *reinterpret_cast<__nv_bfloat162*>(a.gbf[l] + ((long long)e * kRows + r) * N + col) =
                  __halves2bfloat162(__float2bfloat16_rn(g0), __float2bfloat16_rn(g1));
              sG[r * 33 + lc] = g0;
              sG[r * 33 + lc + 1] = g1;
            }
          }
      }
      if (l + 1 == L && tiles > 0) {
        for (int q = 16; q > 0; q >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, q);
        loss_sum += (double)loss;
      }
      __syncthreads();  // sA and sW are read; sG is complete
      cluster_arrive();
    }
    {
      int first, count;
      slice<CTAS>(out, c, &first, &count);
      bias_step(a, po, L - 1, first, count, M, sG, ad);
    }
    // ------------------------------------------------------------------ backward
    for (int l = L - 1; l >= 0; --l) {
      const int in = a.dims[l], o = a.dims[l + 1], in16 = l == 0 ? in_pad : in;
      int rfirst, rcount;  // rows of W_l (columns of G_l) this CTA owns
      slice<CTAS>(o, c, &rfirst, &rcount);
      int cfirst = 0, ccount = 0;  // columns of G_{l-1} it owns
      if (l > 0) {
        slice<CTAS>(in, c, &cfirst, &ccount);
        copy_rows(sB, LD, a.act[l] + (long long)e * a.cap * in, in, M, M16, in);
        copy_rows(sW, LDW, a.wbf + po + a.w_off[l] + cfirst, in, o, o, ccount);
      } else {
        gather_rows(sB, a.X, sRow, in0, M, M16, in_pad);
      }
      if (l == L - 1) cluster_wait();  // below, the wait for dX_l is also the next layer's
      copy_rows(sA, LD, a.gbf[l] + (long long)e * kRows * o, o, M, M16, o);
      cp_wait();
      __syncthreads();
      if (l > 0) {  // G_{l-1} = (G_l W_l) * GELU'(z_{l-1})
        const int tiles = mt * (ccount / (8 * NJ));
        for (int t = warp; t < tiles; t += kWarps) {
          const int m0 = (t % mt) * 16, n0 = (t / mt) * 8 * NJ;
          float2 zv[NJ][2];  // loaded ahead of the product that hides their latency
#pragma unroll
          for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int r = m0 + gid + 8 * h;
              if (r < M)
                zv[j][h] = *reinterpret_cast<const float2*>(
                    a.z[l - 1] + ((long long)e * a.cap + r) * in + cfirst + n0 + 8 * j + 2 * tig);
            }
          float acc[NJ][4] = {};
          product<true, NJ>(acc, sA, m0, sW, n0, o);
#pragma unroll
          for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int r = m0 + gid + 8 * h, lc = n0 + 8 * j + 2 * tig;
              if (r >= M) continue;
              const long long q = ((long long)e * kRows + r) * in + cfirst + lc;
              const float g0 = acc[j][2 * h] * gelu_grad(zv[j][h].x);
              const float g1 = acc[j][2 * h + 1] * gelu_grad(zv[j][h].y);
              *reinterpret_cast<__nv_bfloat162*>(a.gbf[l - 1] + q) =
                  __halves2bfloat162(__float2bfloat16_rn(g0), __float2bfloat16_rn(g1));
              sG[r * 33 + lc] = g0;
              sG[r * 33 + lc + 1] = g1;
            }
        }
        __syncthreads();
        cluster_arrive();
      }
      // dW_l, rows rfirst.. (at most RT 16-row tiles), this warp's 8-column units
      const int units = (in16 + 7) / 8, per = (units + kWarps - 1) / kWarps;
      // The parameters and moments that this thread updates are its own: all of them are loaded
      // now, behind the products and the barrier (one load after another's store would wait for
      // it, for every element).
      const bool even = (in & 1) == 0;
      float2 pw[RT][kUnits][2], pm[RT][kUnits][2], pv[RT][kUnits][2];
      auto mine = [&](int i, int u, int h, long long* q) {
        const int col = (warp * per + u) * 8 + 2 * tig;
        *q = po + a.w_off[l] + (long long)(rfirst + 16 * i + gid + 8 * h) * in + col;
        return 16 * i < rcount && u < per && col < in;
      };
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int u = 0; u < kUnits; ++u)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            long long q;
            if (even && mine(i, u, h, &q)) {
              pw[i][u][h] = *reinterpret_cast<const float2*>(a.params + q);
              pm[i][u][h] = *reinterpret_cast<const float2*>(a.adam_m + q);
              pv[i][u][h] = *reinterpret_cast<const float2*>(a.adam_v + q);
            }
          }
      float w[RT][kUnits][4] = {};
      for (int k = 0; k < M16; k += 16) {
        uint32_t fb[kUnits][2];
#pragma unroll
        for (int u = 0; u < kUnits; ++u)
          if (u < per && warp * per + u < units)
            ldsm2<true>(fb[u], sB + (k + (lane & 15)) * LD + (warp * per + u) * 8);
#pragma unroll
        for (int i = 0; i < RT; ++i)
          if (16 * i < rcount) {
            uint32_t fa[4];
            // matrices (k 0-7, m 0-7), (k 0-7, m 8-15), (k 8-15, m 0-7), (k 8-15, m 8-15)
            ldsm4<true>(fa, sA + (k + (lane & 7) + ((lane >> 4) & 1) * 8) * LD + rfirst + 16 * i +
                                ((lane >> 3) & 1) * 8);
#pragma unroll
            for (int u = 0; u < kUnits; ++u)
              if (u < per && warp * per + u < units) mma(w[i][u], fa, fb[u]);
          }
      }
      if (l > 0) {
        bias_step(a, po, l - 1, cfirst, ccount, M, sG, ad);
        cluster_wait();  // every CTA has read W_l: it may change; G_{l-1} is complete
      }
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int u = 0; u < kUnits; ++u)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            long long q;
            if (!mine(i, u, h, &q)) continue;
            if (even) {
              float2 nw = pw[i][u][h], nm = pm[i][u][h], nv = pv[i][u][h];
              adam_update(nw.x, nm.x, nv.x, w[i][u][2 * h], ad);
              adam_update(nw.y, nm.y, nv.y, w[i][u][2 * h + 1], ad);
              *reinterpret_cast<float2*>(a.params + q) = nw;
              *reinterpret_cast<float2*>(a.adam_m + q) = nm;
              *reinterpret_cast<float2*>(a.adam_v + q) = nv;
              *reinterpret_cast<__nv_bfloat162*>(a.wbf + q) =
                  __halves2bfloat162(__float2bfloat16_rn(nw.x), __float2bfloat16_rn(nw.y));
            } else {
#pragma unroll
              for (int b = 0; b < 2; ++b)
                if ((warp * per + u) * 8 + 2 * tig + b < in) {
                  float nw = a.params[q + b], nm = a.adam_m[q + b], nv = a.adam_v[q + b];
                  adam_update(nw, nm, nv, w[i][u][2 * h + b], ad);
                  a.params[q + b] = nw;
                  a.adam_m[q + b] = nm;
                  a.adam_v[q + b] = nv;
                  a.wbf[q + b] = __float2bfloat16_rn(nw);
                }
            }
          }
      __syncthreads();  // sA, sB, sW and sG are free; the updated rows are visible to this CTA
    }
  }
  if (lane == 0 && loss_sum != 0.0) atomicAdd(&a.loss[e], (float)loss_sum);
}

template <int CTAS>
cudaError_t set_attributes() {
  cudaError_t e = cudaFuncSetAttribute(
      train_epoch<CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
  if (e == cudaSuccess && CTAS > 8)
    e = cudaFuncSetAttribute(train_epoch<CTAS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

// Clusters of CTAS that the current device holds at a time (0: none, or unknown); asked once a
// device.
template <int CTAS>
int clusters() {
  static std::atomic<int> known[kAttrDevices] = {};  // count + 1
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (dev < kAttrDevices && known[dev].load() > 0) return known[dev].load() - 1;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = CTAS;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CTAS);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (set_attributes<CTAS>() != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, train_epoch<CTAS>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  if (dev < kAttrDevices) known[dev].store(n + 1);
  return n;
}

template <int CTAS>
cudaError_t launch(const TrainArgs& a, int members, cudaStream_t st) {
  static AttributesSet done;
  return launch_with(done, set_attributes<CTAS>, train_epoch<CTAS>, dim3(CTAS * members),
                     dim3(kThreads), kSmem, st, a);
}

}  // namespace

// Large ensembles take turns: a B200 holds 15 clusters of 8, and every turn is the chain of a whole
// epoch, while the launch-per-product path runs all members at once.  Of that path's time a
// minibatch step takes 0.64 to 0.93 in three turns (31 to 45 members), 0.80 to 1.02 in four with two
// or more hidden layers and 0.77 to 1.08 with one (6-256-16), 0.91 to 1.26 in five (61 to 64).
bool train_epoch_supported(const int* dims, int L, int batch, int members) {
  if (L < 2 || L > kFusedMaxLayers || batch > kTrainMaxRows || dims[0] > 64) return false;
  for (int l = 1; l <= L; ++l)
    if (dims[l] % 16 != 0 || dims[l] > kTrainMaxWidth) return false;
  return members <= 4 || members <= (L > 2 ? 4 : 3) * clusters<8>();
}

// A member's cluster: 16 CTAs (more than the portable 8) for small ensembles, whose members then
// all run at once, where the device has a GPC with 16 free SMs; 8 otherwise.
cudaError_t launch_train_epoch(const TrainArgs& a, int members, cudaStream_t st) {
  return members <= 4 && clusters<16>() > 0 ? launch<16>(a, members, st)
                                            : launch<8>(a, members, st);
}

}  // namespace mlp
}  // namespace fdtd
