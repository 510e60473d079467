// Copies shared by the float64 kernels whose warps work on tiles of eight
// elements (dg_stage64.cu, dg_deriv64.cu): asynchronous copies to shared
// memory and vector accesses of a lane's run of node values.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "dg_device.cuh"
#include "dg_dmma.cuh"

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

// Overlap with the kernel before in the stream (programmatic dependent launch):
// a kernel launched with `overlap` may start while that one still runs, does
// what depends on none of its results (operators, connectivity), and waits for
// its completion here; allow_next lets the kernel after start in the same way.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
template <class... P, class... A>
cudaError_t launch_kernel(void (*k)(P...), int grid, int threads, size_t smem, cudaStream_t s, bool overlap, A... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&c, k, args...);
}

// Row strides (doubles) of a tile in shared memory, padded so that the lanes of
// one access phase (two rows of four lanes for 16 bytes, four rows for 8) fall
// on different banks: a whole element's nodes (per = NP M; an odd count is
// copied without padding, 16 bytes at a time), a row's face nodes (3 (N+1) M),
// and its geometry.
constexpr int elem_stride(int per, int m) {
  if (per % 2) return per;
  if (m % 2 == 0) return per % 4 == 2 ? per : per + 2;
  return per + (12 - per % 8) % 8;
}
constexpr int face_stride(int per, int m) { return m % 2 == 0 ? (per % 4 == 2 ? per : per + 2) : per | 1; }
constexpr int kGeoStride = 18;

// The eight elements 8 tile .. 8 tile + 7 of an array [n][per] into dst, one
// every `stride` doubles, rows past the end repeating the last element; src
// starts on a 16-byte boundary (eight elements of doubles then always do).
template <int per, int stride>
__device__ __forceinline__ void copy_tile(double* dst, const double* __restrict__ src, int tile, int n, int lane) {
  if (tile * 8 + 8 <= n) {
    const double* s = src + (size_t)tile * 8 * per + 2 * lane;
    double* t = dst + 2 * lane;
    if constexpr (per % 2) {  // not padded: 4 per pieces of 16 bytes in a row
#pragma unroll
      for (int u = 0; u < (4 * per + 31) / 32; ++u)
        if (u < 4 * per / 32 || 32 * u + lane < 4 * per) cp_async16(t + 64 * u, s + 64 * u);
    } else {  // row by row, so that every address is the lane's plus a constant
#pragma unroll
      for (int u = 0; u < (per / 2 + 31) / 32; ++u)
        if (u < per / 64 || 32 * u + lane < per / 2) {
#pragma unroll
          for (int r = 0; r < 8; ++r) cp_async16(t + r * stride + 64 * u, s + r * per + 64 * u);
        }
    }
  } else {
    for (int i = lane; i < 8 * per; i += 32) {
      const int e = i / per;
      cp_async8(dst + e * stride + (i - e * per), src + (size_t)min(tile * 8 + e, n - 1) * per + (i - e * per));
    }
  }
}

// Where a (row, face) pair's nodes come from: element (or ghost slot) x, y =
// its face | 4: in reverse order | 8: a ghost slot of face-node blocks.
__device__ __forceinline__ int2 face_source(int2 conn, int own, int face, int K) {
  if (conn.y < 0) return make_int2(own, face);  // boundary: its own nodes stand in
  return make_int2(conn.x, conn.y | 4 | (conn.x >= K ? 8 : 0));
}
// Bulk copies from shared to global memory (16-byte boundaries and sizes): the
// writes of a tile's rows as the lanes that issue them see fit; read_done
// before the shared memory is reused, all_done before the block ends.
__device__ __forceinline__ void bulk_store(double* dst, const double* src, int bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(dst),
               "r"((unsigned)__cvta_generic_to_shared(src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_read_done() { asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_all_done() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
// a full tile [8][stride] of elements of `per` doubles to global memory
template <int per, int stride>
__device__ __forceinline__ void bulk_store_tile(double* dst, const double* src, int lane) {
  fence_async_proxy();
  __syncwarp();
  if constexpr (per % 2 == 0) {
    if (lane < 8) bulk_store(dst + lane * per, src + lane * stride, per * 8);
  } else {
    static_assert(per == stride, "rows of an odd count are not padded");
    if (lane == 0) bulk_store(dst, src, 8 * per * 8);
  }
  bulk_commit();
}

// n consecutive doubles, 16-byte accesses when n is even (a node of an even
// number of fields starts on such a boundary)
template <int n>
__device__ __forceinline__ void load_run(const double* __restrict__ p, double* v) {
  if constexpr (n % 2 == 0) {
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
template <int n>
__device__ __forceinline__ void store_run(double* __restrict__ p, const double* v) {
  if constexpr (n % 2 == 0) {
#pragma unroll
    for (int i = 0; i < n; i += 2) *reinterpret_cast<double2*>(p + i) = make_double2(v[i], v[i + 1]);
  } else {
#pragma unroll
    for (int i = 0; i < n; ++i) p[i] = v[i];
  }
}

// n consecutive doubles of shared memory, read here and not kept in registers
// from an earlier read
template <int n> __device__ __forceinline__ void shared_run(const double* p, double* v) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  if constexpr (n % 2 == 0) {
#pragma unroll
    for (int i = 0; i < n; i += 2)
      asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];\n" : "=d"(v[i]), "=d"(v[i + 1]) : "r"(a + 8 * i));
  } else {
#pragma unroll
    for (int i = 0; i < n; ++i) asm volatile("ld.shared.f64 %0, [%1];\n" : "=d"(v[i]) : "r"(a + 8 * i));
  }
}

// A lane's node values of accumulator block b of one element, v[field][j] at
// node 8 b + 4 j + lc (PK: the order's Pack64).
template <int M, class PK>
__device__ __forceinline__ void load_block(const double* __restrict__ e, int b, int lc, double (*v)[2]) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int n = 8 * b + 4 * j + lc;
    double t[M];
#pragma unroll
    for (int f = 0; f < M; ++f) t[f] = 0.0;
    if (n < PK::NP) load_run<M>(e + n * M, t);
#pragma unroll
    for (int f = 0; f < M; ++f) v[f][j] = t[f];
  }
}
template <int M, class PK>
__device__ __forceinline__ void store_block(double* __restrict__ e, int b, int lc, const double (*v)[2]) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int n = 8 * b + 4 * j + lc;
    double t[M];
#pragma unroll
    for (int f = 0; f < M; ++f) t[f] = v[f][j];
    if (n < PK::NP) store_run<M>(e + n * M, t);
  }
}

// A lane's node accumulators of one element: a[b][f][j] at node 8 b + 4 j + lc,
// and this lane's share of the TL nodes past the last block.
template <int M, class PK> struct Nodes {
  double a[PK::NB][M][2];
  double t[PK::TL > 0 ? PK::TL : 1][M];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int b = 0; b < PK::NB; ++b)
#pragma unroll
      for (int f = 0; f < M; ++f) a[b][f][0] = a[b][f][1] = 0.0;
#pragma unroll
    for (int n = 0; n < PK::TL; ++n)
#pragma unroll
      for (int f = 0; f < M; ++f) t[n][f] = 0.0;
  }
  // += the contraction of two A operands with a "nodes" entry in memory (the
  // fields of a mask, the same in the whole warp; the others' operands are zero)
  __device__ __forceinline__ void add(const double* entry, int lane, const double* A0, const double* A1,
                                      unsigned fields = ~0u) {
#pragma unroll
    for (int b = 0; b < PK::NB; ++b) {
      const double2 w = reinterpret_cast<const double2*>(entry)[b * 32 + lane];
#pragma unroll
      for (int f = 0; f < M; ++f)
        if (fields >> f & 1) dmma_8x8x4(a[b][f], A0[f], w.x);
#pragma unroll
      for (int f = 0; f < M; ++f)
        if (fields >> f & 1) dmma_8x8x4(a[b][f], A1[f], w.y);
    }
#pragma unroll
    for (int n = 0; n < PK::TL; ++n) {
      const double2 w = reinterpret_cast<const double2*>(entry + PK::NB * 64)[n * 4 + (lane & 3)];
#pragma unroll
      for (int f = 0; f < M; ++f) t[n][f] = fma(A1[f], w.y, fma(A0[f], w.x, t[n][f]));
    }
  }
  // += with the first of the pair only
  __device__ __forceinline__ void add1(const double* entry, int lane, const double* A0) {
#pragma unroll
    for (int b = 0; b < PK::NB; ++b) {
      const double w = entry[(b * 32 + lane) * 2];
#pragma unroll
      for (int f = 0; f < M; ++f) dmma_8x8x4(a[b][f], A0[f], w);
    }
#pragma unroll
    for (int n = 0; n < PK::TL; ++n) {
      const double w = entry[PK::NB * 64 + (n * 4 + (lane & 3)) * 2];
#pragma unroll
      for (int f = 0; f < M; ++f) t[n][f] = fma(A0[f], w, t[n][f]);
    }
  }
  // the four lanes' shares together (all lanes of the warp)
  __device__ __forceinline__ void finish() {
#pragma unroll
    for (int n = 0; n < PK::TL; ++n)
#pragma unroll
      for (int f = 0; f < M; ++f) {
        t[n][f] += __shfl_xor_sync(0xffffffffu, t[n][f], 1);
        t[n][f] += __shfl_xor_sync(0xffffffffu, t[n][f], 2);
      }
  }
  // block b of NBT as load_block has it
  __device__ __forceinline__ void get(int b, int lc, double (*v)[2]) const {
#pragma unroll
    for (int f = 0; f < M; ++f) {
      if (b < PK::NB) {
        v[f][0] = a[b < PK::NB ? b : 0][f][0];
        v[f][1] = a[b < PK::NB ? b : 0][f][1];
      } else {
        v[f][0] = PK::TL == 2 && lc == 1 ? t[PK::TL == 2 ? 1 : 0][f] : t[0][f];
        v[f][1] = 0.0;
      }
    }
  }
};

}  // namespace apollo
