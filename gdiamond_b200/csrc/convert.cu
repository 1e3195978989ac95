// convert.cu -- field transfers of the C-ABI on the device: conversion of stored field arrays
// (FP16 / BF16 with a per-component scale, FP64) to and from FP32 / FP64 (pitched layout on both
// sides; one thread per element of a row, grid (ceil(nx/128), ny, nz)), copies of rows between
// pitched and packed arrays, and clearing of several arrays in one launch.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "fdtd_kernels.cuh"

namespace fdtd {
namespace {

template <typename S>
__device__ __forceinline__ double load_as(const void* p, long long i);
template <>
__device__ __forceinline__ double load_as<float>(const void* p, long long i) {
  return (double)static_cast<const float*>(p)[i];
}
template <>
__device__ __forceinline__ double load_as<__half>(const void* p, long long i) {
  return (double)__half2float(static_cast<const __half*>(p)[i]);
}
template <>
__device__ __forceinline__ double load_as<__nv_bfloat16>(const void* p, long long i) {
  return (double)__bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
}
template <>
__device__ __forceinline__ double load_as<double>(const void* p, long long i) {
  return static_cast<const double*>(p)[i];
}

template <typename S, typename D>
__global__ void to_wide(Grid g, const void* src, float scale, D* dst) {
  const int i = blockIdx.x * 128 + threadIdx.x;
  if (i >= g.nx) return;
  const long long idx = i + (long long)blockIdx.y * g.pitch + (long long)blockIdx.z * g.plane;
  // FP32 and FP64 are stored unscaled; scaling by a power of two is exact in FP32.
  const double v = load_as<S>(src, idx);
  dst[idx] = (sizeof(S) == 2) ? (D)((float)v * scale) : (D)v;
}

template <typename S>
__global__ void from_f32(Grid g, const float* src, float inv_scale, S* dst) {
  const int i = blockIdx.x * 128 + threadIdx.x;
  if (i >= g.nx) return;
  const long long idx = i + (long long)blockIdx.y * g.pitch + (long long)blockIdx.z * g.plane;
  const float v = src[idx];
  if constexpr (sizeof(S) == 2) {
    if constexpr (std::is_same<S, __half>::value)
      dst[idx] = __float2half_rn(v * inv_scale);
    else
      *reinterpret_cast<uint16_t*>(dst + idx) = bf16_rne_bits(v * inv_scale);
  } else {
    dst[idx] = (S)v;
  }
}

// Rows of cpr chunks of type V between arrays of row strides ss and ds bytes.  A thread moves U
// chunks, all loads before the stores: bound by memory.  The 2-D copies of the runtime, which
// this replaces, move 3.5 TB/s (read and written) with aligned rows and 1.7 with odd ones; this
// kernel 6.2 and 4.4 (512x512x384 and 251x243x190 cells, 4 bytes).
template <typename V, int U>
__global__ void __launch_bounds__(256) copy_rows_kernel(const char* src, long long ss, char* dst,
                                                        long long ds, uint32_t cpr,
                                                        uint32_t total) {
  const uint32_t i0 = blockIdx.x * (256u * U) + threadIdx.x;
  V v[U];
  long long d[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t i = i0 + u * 256u;
    const uint32_t r = i / cpr, c = i - r * cpr;
    d[u] = (long long)r * ds + (long long)c * (int)sizeof(V);
    if (i < total)
      v[u] = *reinterpret_cast<const V*>(src + (long long)r * ss + (long long)c * (int)sizeof(V));
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (i0 + u * 256u < total) *reinterpret_cast<V*>(dst + d[u]) = v[u];
}

template <typename V>
cudaError_t copy_rows_as(const char* src, long long ss, char* dst, long long ds, long long row,
                         long long rows, cudaStream_t st) {
  constexpr int U = sizeof(V) == 16 ? 4 : 8;
  const long long cpr = row / (long long)sizeof(V);
  const long long per = std::max<long long>(1, (1LL << 30) / cpr);  // rows of one launch
  for (long long r0 = 0; r0 < rows; r0 += per) {
    const uint32_t total = (uint32_t)(std::min(per, rows - r0) * cpr);
    copy_rows_kernel<V, U><<<(total + 256 * U - 1) / (256 * U), 256, 0, st>>>(
        src + r0 * ss, ss, dst + r0 * ds, ds, (uint32_t)cpr, total);
  }
  return cudaGetLastError();
}

// Stored values of rows of nx elements (row stride `pitch` elements) widened to FP32 in a packed
// array, as to_wide does; eight elements per thread.
template <typename S>
__global__ void __launch_bounds__(256) widen_rows(const S* src, int pitch, uint32_t nx,
                                                  uint32_t total, float scale, float* dst) {
  constexpr int U = 8;
  const uint32_t i0 = blockIdx.x * (256u * U) + threadIdx.x;
  double v[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t i = i0 + u * 256u;
    const uint32_t r = i / nx, c = i - r * nx;
    if (i < total) v[u] = load_as<S>(src, (long long)r * pitch + c);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t i = i0 + u * 256u;
    if (i < total) dst[i] = sizeof(S) == 2 ? (float)v[u] * scale : (float)v[u];
  }
}

template <typename S>
cudaError_t widen_as(const S* src, int pitch, int nx, long long rows, float scale, float* dst,
                     cudaStream_t st) {
  const long long per = std::max<long long>(1, (1LL << 30) / nx);  // rows of one launch
  for (long long r0 = 0; r0 < rows; r0 += per) {
    const uint32_t total = (uint32_t)(std::min(per, rows - r0) * nx);
    widen_rows<S><<<(total + 2047) / 2048, 256, 0, st>>>(src + r0 * pitch, pitch, (uint32_t)nx,
                                                         total, scale, dst + r0 * nx);
  }
  return cudaGetLastError();
}

// 16-byte stores of zero over every range (all are whole device allocations: 256-byte aligned),
// blockIdx.y = range; the last bytes singly.
__global__ void __launch_bounds__(256) clear_kernel(const __grid_constant__ ClearList L) {
  char* p = static_cast<char*>(L.p[blockIdx.y]);
  const unsigned long long n = L.bytes[blockIdx.y], n16 = n / 16;
  const unsigned long long step = (unsigned long long)gridDim.x * 256;
  unsigned long long i = blockIdx.x * 256ull + threadIdx.x;
  if (i < n - 16 * n16) p[16 * n16 + i] = 0;
  for (; i < n16; i += step) reinterpret_cast<uint4*>(p)[i] = make_uint4(0, 0, 0, 0);
}

dim3 conv_grid(const Grid& g) { return dim3((g.nx + 127) / 128, g.ny, g.nz); }

}  // namespace

cudaError_t copy_rows(const void* src, long long src_stride, void* dst, long long dst_stride,
                      long long row, long long rows, cudaStream_t st) {
  if (row <= 0 || rows <= 0) return cudaSuccess;
  const char* s = static_cast<const char*>(src);
  char* d = static_cast<char*>(dst);
  if (src_stride == row && dst_stride == row) {  // contiguous: rows of any length will do
    const long long bytes = row * rows;
    long long r = 1LL << 26;
    while (r > 1 && bytes % r) r >>= 1;
    if (r >= 16) {
      row = src_stride = dst_stride = r;
      rows = bytes / r;
    }
  }
  // the widest chunk that both sides' rows start and end on
  const unsigned long long a = (unsigned long long)(uintptr_t)s | (uintptr_t)d | row |
                               (rows > 1 ? src_stride | dst_stride : 0);
  if (a % 16 == 0) return copy_rows_as<uint4>(s, src_stride, d, dst_stride, row, rows, st);
  if (a % 8 == 0) return copy_rows_as<uint2>(s, src_stride, d, dst_stride, row, rows, st);
  if (a % 4 == 0) return copy_rows_as<uint32_t>(s, src_stride, d, dst_stride, row, rows, st);
  if (a % 2 == 0) return copy_rows_as<uint16_t>(s, src_stride, d, dst_stride, row, rows, st);
  return copy_rows_as<uint8_t>(s, src_stride, d, dst_stride, row, rows, st);
}

cudaError_t widen_field_packed(const Grid& g, const void* src, int storage, float scale,
                               float* dst, cudaStream_t st) {
  const long long rows = (long long)g.ny * g.nz;
  switch (storage) {
    case 1: return widen_as((const __half*)src, g.pitch, g.nx, rows, scale, dst, st);
    case 2: return widen_as((const __nv_bfloat16*)src, g.pitch, g.nx, rows, scale, dst, st);
    case 3: return widen_as((const double*)src, g.pitch, g.nx, rows, scale, dst, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t clear_ranges(const ClearList& L, cudaStream_t st) {
  if (L.n <= 0) return cudaSuccess;
  unsigned long long most = 0;
  for (int q = 0; q < L.n; ++q) most = std::max(most, L.bytes[q]);
  const unsigned long long blocks = (most / 16 + 256 * 8 - 1) / (256 * 8);
  const dim3 grid((unsigned)std::min<unsigned long long>(std::max(blocks, 1ull), 148 * 8),
                  (unsigned)L.n);
  clear_kernel<<<grid, 256, 0, st>>>(L);
  return cudaGetLastError();
}

cudaError_t convert_field_to_f32(const Grid& g, const void* src, int storage, float scale,
                                 float* dst, cudaStream_t st) {
  switch (storage) {
    case 0: to_wide<float, float><<<conv_grid(g), 128, 0, st>>>(g, src, scale, dst); break;
    case 1: to_wide<__half, float><<<conv_grid(g), 128, 0, st>>>(g, src, scale, dst); break;
    case 2: to_wide<__nv_bfloat16, float><<<conv_grid(g), 128, 0, st>>>(g, src, scale, dst); break;
    case 3: to_wide<double, float><<<conv_grid(g), 128, 0, st>>>(g, src, scale, dst); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t convert_field_to_f64(const Grid& g, const void* src, int storage, float scale,
                                 double* dst, cudaStream_t st) {
  switch (storage) {
    case 0: to_wide<float, double><<<conv_grid(g), 128, 0, st>>>(g, src, scale, dst); break;
    case 1: to_wide<__half, double><<<conv_grid(g), 128, 0, st>>>(g, src, scale, dst); break;
    case 2: to_wide<__nv_bfloat16, double><<<conv_grid(g), 128, 0, st>>>(g, src, scale, dst); break;
    case 3: to_wide<double, double><<<conv_grid(g), 128, 0, st>>>(g, src, scale, dst); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t convert_field_from_f32(const Grid& g, const float* src, int storage, float inv_scale,
                                   void* dst, cudaStream_t st) {
  switch (storage) {
    case 0: from_f32<float><<<conv_grid(g), 128, 0, st>>>(g, src, inv_scale, (float*)dst); break;
    case 1: from_f32<__half><<<conv_grid(g), 128, 0, st>>>(g, src, inv_scale, (__half*)dst); break;
    case 2:
      from_f32<__nv_bfloat16><<<conv_grid(g), 128, 0, st>>>(g, src, inv_scale,
                                                             (__nv_bfloat16*)dst);
      break;
    case 3: from_f32<double><<<conv_grid(g), 128, 0, st>>>(g, src, inv_scale, (double*)dst); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace fdtd
