// materials.cu -- compress 12 per-cell coefficient arrays into a material map on the GPU.
//
// The reference keeps Ca/Cb/Da/Db as 12 per-cell FP32 arrays (gDiamond/gdiamond.hpp:891-904,
// filled by set_FDTD_matrices_3D_structure, gDiamond/utils.h:542-690) and re-reads all 48
// bytes per cell in every step.  Real grids hold few distinct 12-tuples (vacuum, a handful of
// dielectrics, the graded PML shell), so the solver stores a uint16 id per cell plus a table
// of distinct tuples.  This file builds that map on the device:
//   1. insert: hash each cell's 12 words (bitwise) into an open-addressing table of 2^20
//      64-bit keys; a key's representative is its first cell (lowest index);
//   2. assign: number the keys in the order of their representatives (bucketed by ranges of cells,
//      then counted within the bucket) and copy each one's tuple into the table.  Neighbouring
//      cells of a graded layer then have neighbouring table entries, and a warp's coefficient
//      loads touch a few cache lines instead of one per cell;
//   3. map: write each cell's id and compare its 12 words with the table entry, so a 64-bit
//      hash collision is detected (the map is then rejected) instead of silently merged; count
//      the cells of each id and report the id held by the most cells (the kernels' fast path
//      keeps that material's coefficients in registers).
// Probing is bounded; overflow or more than 65536 tuples reject the map (the per-cell arrays
// and the naive kernel are used instead).
#include "fdtd_kernels.cuh"

namespace fdtd {

namespace {

constexpr int kSlotBits = 20;
constexpr uint32_t kSlots = 1u << kSlotBits;
constexpr unsigned long long kEmpty = ~0ull;
constexpr int kMaxProbe = 4096;
constexpr int kMaxMaterials = 65536;
constexpr int kBuckets = 4096;  // of representatives, by ranges of cells

struct Scratch {
  unsigned long long keys[kSlots];
  unsigned long long rep[kSlots];
  uint32_t ids[kSlots];
  unsigned int nuniq;  // keys inserted
  unsigned int nid;    // ids handed out
  unsigned int flags;  // 1 = probe overflow, 2 = hash collision
  unsigned int mode;   // id held by the most cells (the lowest such id on a tie)
  unsigned int count[kMaxMaterials];  // cells per id
  uint32_t slot[kMaxMaterials];            // occupied slots, in no order
  unsigned long long first[kMaxMaterials]; // their representatives
  unsigned long long sorted[kMaxMaterials];  // the representatives by bucket
  uint32_t start[kBuckets + 1];              // first entry of a bucket (before: their counts)
  uint32_t cursor[kBuckets];
};

struct Coef12 {
  const float* c[12];  // pitched
};

__device__ __forceinline__ unsigned long long hash12(const uint32_t* w) {
  unsigned long long h = 0x9E3779B97F4A7C15ull;
#pragma unroll
  for (int a = 0; a < 12; ++a) {
    h ^= (unsigned long long)w[a] + 0x632BE59BD9B4E019ull + (h << 6) + (h >> 2);
    h *= 0xFF51AFD7ED558CCDull;
    h ^= h >> 33;
  }
  return h == kEmpty ? 0ull : h;
}

__device__ __forceinline__ void load12(const Coef12& C, long long idx, uint32_t* w) {
#pragma unroll
  for (int a = 0; a < 12; ++a) w[a] = __float_as_uint(C.c[a][idx]);
}

__device__ __forceinline__ long long cell_index(const Grid& g, long long lin) {
  const long long i = lin % g.nx, r = lin / g.nx;
  const long long j = r % g.ny, k = r / g.ny;
  return i + j * g.pitch + k * g.plane;
}

__global__ void k_reset(Scratch* s) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < kSlots) {
    s->keys[q] = kEmpty;
    s->rep[q] = kEmpty;
    s->ids[q] = 0xFFFFFFFFu;
  }
  if (q < (uint32_t)kMaxMaterials) s->count[q] = 0;
  if (q <= (uint32_t)kBuckets) s->start[q] = 0;
  if (q == 0) s->nuniq = s->nid = s->flags = s->mode = 0;
}

__global__ void k_insert(Grid g, Coef12 C, Scratch* s, long long n) {
  for (long long lin = blockIdx.x * (long long)blockDim.x + threadIdx.x; lin < n;
       lin += (long long)gridDim.x * blockDim.x) {
    const long long idx = cell_index(g, lin);
    uint32_t w[12];
    load12(C, idx, w);
    const unsigned long long h = hash12(w);
    uint32_t slot = (uint32_t)h & (kSlots - 1);
    bool done = false;
    for (int probe = 0; probe < kMaxProbe && !done; ++probe) {
      const unsigned long long cur = *((volatile unsigned long long*)&s->keys[slot]);
      if (cur == h) { done = true; break; }
      if (cur == kEmpty) {
        const unsigned long long old = atomicCAS(&s->keys[slot], kEmpty, h);
        if (old == kEmpty) atomicAdd(&s->nuniq, 1u);
        if (old == kEmpty || old == h) { done = true; break; }
      }
      slot = (slot + 1) & (kSlots - 1);
    }
    if (!done) {
      atomicOr(&s->flags, 1u);
      continue;
    }
    if ((unsigned long long)idx < *((volatile unsigned long long*)&s->rep[slot]))
      atomicMin(&s->rep[slot], (unsigned long long)idx);
  }
}

// Lists the occupied slots and their representatives and counts these in buckets of 2^shift cells.
__global__ void k_list(Scratch* s, int shift) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= kSlots || s->keys[q] == kEmpty) return;
  const unsigned int n = atomicAdd(&s->nid, 1u);
  if (n >= (unsigned)kMaxMaterials) return;  // rejected on the host
  s->slot[n] = q;
  s->first[n] = s->rep[q];
  atomicAdd(&s->start[s->rep[q] >> shift], 1u);
}

// Counts to first entries; one block of 1024 threads.
__global__ void __launch_bounds__(1024) k_scan(Scratch* s) {
  constexpr int P = kBuckets / 1024;
  __shared__ uint32_t sum[1024];
  const int t = threadIdx.x;
  uint32_t c[P], mine = 0;
#pragma unroll
  for (int q = 0; q < P; ++q) mine += c[q] = s->start[t * P + q];
  sum[t] = mine;
  for (int d = 1; d < 1024; d *= 2) {
    __syncthreads();
    const uint32_t add = t >= d ? sum[t - d] : 0;
    __syncthreads();
    sum[t] += add;
  }
  uint32_t at = sum[t] - mine;
#pragma unroll
  for (int q = 0; q < P; ++q) {
    s->start[t * P + q] = s->cursor[t * P + q] = at;
    at += c[q];
  }
  if (t == 1023) s->start[kBuckets] = at;
}

__global__ void __launch_bounds__(256) k_scatter(Scratch* s, int nuniq, int shift) {
  const int n = blockIdx.x * 256 + threadIdx.x;
  if (n >= nuniq) return;
  const unsigned long long r = s->first[n];
  s->sorted[atomicAdd(&s->cursor[r >> shift], 1u)] = r;
}

// Entry n of the list gets the id that counts the representatives before its own: those of the
// buckets before its bucket and the smaller ones in it (counting all of them by comparison took
// 0.17 ms for 32768 materials, as long as the rest of a 32^3 map).
__global__ void __launch_bounds__(256) k_assign(Coef12 C, Scratch* s, Material* table, int nuniq,
                                                int shift) {
  const int n = blockIdx.x * 256 + threadIdx.x;
  if (n >= nuniq) return;
  const unsigned long long r = s->first[n];
  const uint32_t q0 = s->start[r >> shift], q1 = s->start[(r >> shift) + 1];
  uint32_t id = q0;
  for (uint32_t q = q0; q < q1; ++q) id += s->sorted[q] < r ? 1u : 0u;
  s->ids[s->slot[n]] = id;
  float v[12];
#pragma unroll
  for (int a = 0; a < 12; ++a) v[a] = C.c[a][r];
  // {Cax, Cbx, Cay, Cby}, {Caz, Cbz, Dax, Dbx}, {Day, Dby, Daz, Dbz}
  Material m;
  m.a = make_float4(v[0], v[3], v[1], v[4]);
  m.b = make_float4(v[2], v[5], v[6], v[9]);
  m.c = make_float4(v[7], v[10], v[8], v[11]);
  table[id] = m;
}

__global__ void k_map(Grid g, Coef12 C, Scratch* s, const Material* table, uint16_t* mat,
                      long long n) {
  for (long long lin = blockIdx.x * (long long)blockDim.x + threadIdx.x; lin < n;
       lin += (long long)gridDim.x * blockDim.x) {
    const long long idx = cell_index(g, lin);
    uint32_t w[12];
    load12(C, idx, w);
    const unsigned long long h = hash12(w);
    uint32_t slot = (uint32_t)h & (kSlots - 1);
    int probe = 0;
    while (probe < kMaxProbe && s->keys[slot] != h) {
      slot = (slot + 1) & (kSlots - 1);
      ++probe;
    }
    if (probe == kMaxProbe) { atomicOr(&s->flags, 1u); continue; }
    const uint32_t id = s->ids[slot];
    if (id >= (uint32_t)kMaxMaterials) continue;  // rejected on the host
    const Material m = table[id];
    const uint32_t t[12] = {__float_as_uint(m.a.x), __float_as_uint(m.a.z),
                            __float_as_uint(m.b.x), __float_as_uint(m.a.y),
                            __float_as_uint(m.a.w), __float_as_uint(m.b.y),
                            __float_as_uint(m.b.z), __float_as_uint(m.c.x),
                            __float_as_uint(m.c.z), __float_as_uint(m.b.w),
                            __float_as_uint(m.c.y), __float_as_uint(m.c.w)};
    bool same = true;
#pragma unroll
    for (int a = 0; a < 12; ++a) same = same && (t[a] == w[a]);
    if (!same) atomicOr(&s->flags, 2u);
    mat[idx] = (uint16_t)id;
    // cells per id: one atomic per group of lanes holding the same id
    const unsigned peers = __match_any_sync(__activemask(), id);
    if ((threadIdx.x & 31) == (unsigned)(__ffs(peers) - 1)) atomicAdd(&s->count[id], __popc(peers));
  }
}

// The id with the most cells (lowest id on a tie): one CTA of 1024 threads.
__global__ void k_mode(Scratch* s, int nmat) {
  __shared__ unsigned long long best[32];
  unsigned long long b = 0;  // (count << 32) | (0xFFFFFFFF - id): max picks most cells, lowest id
  for (int q = threadIdx.x; q < nmat; q += blockDim.x)
    b = max(b, ((unsigned long long)s->count[q] << 32) | (0xFFFFFFFFu - (unsigned)q));
  for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
  if ((threadIdx.x & 31) == 0) best[threadIdx.x >> 5] = b;
  __syncthreads();
  if (threadIdx.x < 32) {
    b = best[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    if (threadIdx.x == 0) s->mode = 0xFFFFFFFFu - (unsigned)(b & 0xFFFFFFFFu);
  }
}

}  // namespace

namespace {

// One warp per block of kUniX x kUniY x kUniZ cells: each lane tests 32 of its 1024 cells.
__global__ void k_uniform_blocks(Grid g, const uint16_t* mat, int id, uint8_t* out, int nbx,
                                 int nby, long long nblk) {
  const long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x & 31;
  if (w >= nblk) return;  // warp-uniform
  const int bx = (int)(w % nbx), by = (int)((w / nbx) % nby), bz = (int)(w / ((long long)nbx * nby));
  bool ok = true;
  for (int q = lane; q < kUniX * kUniY * kUniZ; q += 32) {
    const int i = bx * kUniX + q % kUniX, j = by * kUniY + (q / kUniX) % kUniY;
    const int k = bz * kUniZ + q / (kUniX * kUniY);
    if (i < g.nx && j < g.ny && k < g.nz)
      ok = ok && mat[i + (long long)j * g.pitch + (long long)k * g.plane] == (uint16_t)id;
  }
  ok = __all_sync(0xffffffffu, ok);
  if (lane == 0) out[w] = ok ? 1 : 0;
}

}  // namespace

cudaError_t build_uniform_blocks(const Grid& g, const uint16_t* mat, int id, uint8_t* out,
                                 cudaStream_t st) {
  const int nbx = (g.nx + kUniX - 1) / kUniX, nby = (g.ny + kUniY - 1) / kUniY;
  const int nbz = (g.nz + kUniZ - 1) / kUniZ;
  const long long nblk = (long long)nbx * nby * nbz;
  const int threads = 256;
  const long long blocks = (nblk * 32 + threads - 1) / threads;
  k_uniform_blocks<<<(unsigned)blocks, threads, 0, st>>>(g, mat, id, out, nbx, nby, nblk);
  return cudaGetLastError();
}

size_t material_scratch_bytes() { return sizeof(Scratch); }

cudaError_t build_material_map(const Grid& g, const float* const* coef12, uint16_t* mat,
                               Material* table, void* scratch, size_t scratch_bytes,
                               cudaStream_t st, DedupResult* out) {
  out->ok = false;
  out->nmat = 0;
  if (scratch_bytes < sizeof(Scratch)) return cudaErrorInvalidValue;
  Scratch* s = static_cast<Scratch*>(scratch);
  Coef12 C;
  for (int a = 0; a < 12; ++a) C.c[a] = coef12[a];
  const long long n = (long long)g.nx * g.ny * g.nz;
  const int threads = 256;
  const int blocks = 148 * 16;
  k_reset<<<(kSlots + threads - 1) / threads, threads, 0, st>>>(s);
  k_insert<<<blocks, threads, 0, st>>>(g, C, s, n);
  unsigned int hdr[3];
  cudaError_t e = cudaMemcpyAsync(hdr, &s->nuniq, sizeof(hdr), cudaMemcpyDeviceToHost, st);
  if (e != cudaSuccess) return e;
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
  if (hdr[2] != 0 || hdr[0] > (unsigned)kMaxMaterials) return cudaGetLastError();
  const int nuniq = (int)hdr[0];
  int shift = 0;
  while ((g.plane * g.nz - 1) >> shift >= kBuckets) ++shift;
  k_list<<<(kSlots + threads - 1) / threads, threads, 0, st>>>(s, shift);
  k_scan<<<1, 1024, 0, st>>>(s);
  k_scatter<<<(nuniq + 255) / 256, 256, 0, st>>>(s, nuniq, shift);
  k_assign<<<(nuniq + 255) / 256, 256, 0, st>>>(C, s, table, nuniq, shift);
  k_map<<<blocks, threads, 0, st>>>(g, C, s, table, mat, n);
  k_mode<<<1, 1024, 0, st>>>(s, (int)hdr[0]);
  unsigned int hdr4[4];
  if ((e = cudaMemcpyAsync(hdr4, &s->nuniq, sizeof(hdr4), cudaMemcpyDeviceToHost, st)) !=
      cudaSuccess)
    return e;
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
  out->nmat = (int)hdr4[0];
  out->ok = hdr4[2] == 0 && hdr4[0] <= (unsigned)kMaxMaterials;
  out->dominant = (int)hdr4[3];
  return cudaGetLastError();
}

}  // namespace fdtd
