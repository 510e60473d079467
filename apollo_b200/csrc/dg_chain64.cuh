// Copies shared by the float64 kernels whose warps work on tiles of eight
// elements (dg_stage64.cu, dg_deriv64.cu): asynchronous copies to shared
// memory and vector accesses of a lane's run of node values.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "dg_device.cuh"

namespace apollo {

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
// n doubles (one node's fields) by 16-byte copies where n is even (both sides
// then start on a 16-byte boundary), 8-byte ones otherwise
template <int n> __device__ __forceinline__ void cp_async_node(double* dst, const double* src) {
  if constexpr (n % 2 == 0) {
#pragma unroll
    for (int c = 0; c < n; c += 2) cp_async16(dst + c, src + c);
  } else {
#pragma unroll
    for (int c = 0; c < n; ++c) cp_async8(dst + c, src + c);
  }
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
// all but the n newest groups have arrived
template <int n> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(n) : "memory");
}

// The eight elements 8 tile .. 8 tile + 7 of an array [n][per] into dst
// [8][per], rows past the end repeating the last element; src starts on a
// 16-byte boundary (eight elements of doubles then always do).
template <int per>
__device__ __forceinline__ void copy_tile(double* dst, const double* __restrict__ src, int tile, int n, int lane) {
  if (tile * 8 + 8 <= n) {
    const double* s = src + (size_t)tile * 8 * per;
#pragma unroll 4
    for (int i = lane; i < 4 * per; i += 32) cp_async16(dst + 2 * i, s + 2 * i);
  } else {
    for (int i = lane; i < 8 * per; i += 32) {
      const int e = i / per;
      cp_async8(dst + i, src + (size_t)min(tile * 8 + e, n - 1) * per + (i - e * per));
    }
  }
}

// n consecutive doubles, 16-byte accesses when ALIGNED (both counts even)
template <int n, bool ALIGNED>
__device__ __forceinline__ void load_run(const double* __restrict__ p, double* v) {
  if constexpr (ALIGNED && n % 2 == 0) {
#pragma unroll
    for (int i = 0; i < n; i += 2) {
      const double2 t = *reinterpret_cast<const double2*>(p + i);
      v[i] = t.x;
      v[i + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < n; ++i) v[i] = p[i];
  }
}
template <int n, bool ALIGNED>
__device__ __forceinline__ void store_run(double* __restrict__ p, const double* v) {
  if constexpr (ALIGNED && n % 2 == 0) {
#pragma unroll
    for (int i = 0; i < n; i += 2) *reinterpret_cast<double2*>(p + i) = make_double2(v[i], v[i + 1]);
  } else {
#pragma unroll
    for (int i = 0; i < n; ++i) p[i] = v[i];
  }
}

// A lane's node values of accumulator block b of one element, v[field][0, 1]
// (PK: the order's Pack64, which says how the block holds its nodes).
template <int M, class PK>
__device__ __forceinline__ void load_block(const double* __restrict__ e, int b, int lc, double (*v)[2]) {
  constexpr bool EVEN = (PK::NP * M) % 2 == 0;
  double t[2 * M];
#pragma unroll
  for (int f = 0; f < 2 * M; ++f) t[f] = 0.0;
  if (PK::paired(b)) {
    const int n0 = 8 * b + 2 * lc;
    if (n0 + 1 < PK::NP) load_run<2 * M, EVEN>(e + n0 * M, t);
    else if (n0 < PK::NP) load_run<M, EVEN>(e + n0 * M, t);
  } else {
    const int n0 = 8 * b + lc;
    if (n0 < PK::NP) load_run<M, false>(e + n0 * M, t);
  }
#pragma unroll
  for (int f = 0; f < M; ++f) {
    v[f][0] = t[f];
    v[f][1] = t[M + f];
  }
}
template <int M, class PK>
__device__ __forceinline__ void store_block(double* __restrict__ e, int b, int lc, const double (*v)[2]) {
  constexpr bool EVEN = (PK::NP * M) % 2 == 0;
  double t[2 * M];
#pragma unroll
  for (int f = 0; f < M; ++f) {
    t[f] = v[f][0];
    t[M + f] = v[f][1];
  }
  if (PK::paired(b)) {
    const int n0 = 8 * b + 2 * lc;
    if (n0 + 1 < PK::NP) store_run<2 * M, EVEN>(e + n0 * M, t);
    else if (n0 < PK::NP) store_run<M, EVEN>(e + n0 * M, t);
  } else {
    const int n0 = 8 * b + lc;
    if (n0 < PK::NP) store_run<M, false>(e + n0 * M, t);
  }
}

}  // namespace apollo
