// CSR x dense row slices (fp16 A and B, fp32 accumulation), shared by the CSR
// product kernel and the CSR pass of the hybrid product.
//
// A warp computes one row of A times a 256-column slice of B: every lane owns 8
// consecutive columns. For each entry the warp reads that B row's slice as one
// 512-byte load (16 bytes per lane), with several entries' loads in flight
// before their FMAs.
#pragma once
#include <cuda_fp16.h>
#include <cstdint>
#include <type_traits>

namespace spmm {

__device__ __forceinline__ void fma8(float (&acc)[8], float a, uint4 b) {
  const __half2* h = reinterpret_cast<const __half2*>(&b);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 f = __half22float2(h[k]);
    acc[2 * k] = fmaf(a, f.x, acc[2 * k]);
    acc[2 * k + 1] = fmaf(a, f.y, acc[2 * k + 1]);
  }
}

// acc[0..7] += sum over entries e in [e0, e1) of vals[e] * B[col_idx[e]][n..n+7],
// in order, U entries' B loads in flight. Warp-uniform e0 / e1; `valid` (this
// lane's columns lie inside B) may differ per lane. Lanes read 32 entries'
// indices and values together, 32 entries ahead of their use, so that a B load
// waits for no index, and the last entries of a row load together like any
// others (one by one, with their indices read first, a row's last U - 1 entries
// took as long as 2 U (U - 1) others).
template <int U>   // 4 or 8
__device__ __forceinline__ void csr_row_slice(const int* __restrict__ col_idx, const __half* __restrict__ vals,
                                              const __half* __restrict__ B, long long ldb, int e0, int e1, int n,
                                              bool valid, float (&acc)[8]) {
  const int lane = threadIdx.x & 31;
  const __half* src = B + (valid ? n : n - 8 * lane);   // past N: the slice's first column
  int next_k = 0;
  __half next_a = __float2half(0.f);
  if (e0 + lane < e1) {
    next_k = __ldg(col_idx + e0 + lane);
    next_a = __ldg(vals + e0 + lane);
  }
  for (int base = e0; base < e1; base += 32) {
    const int cnt = min(32, e1 - base), ks = next_k;
    const float as = __half2float(next_a);
    if (base + 32 + lane < e1) {
      next_k = __ldg(col_idx + base + 32 + lane);
      next_a = __ldg(vals + base + 32 + lane);
    }
    // V entries from i on, of which the first n are there (no condition on a load:
    // past the last entry its row again)
    auto entries = [&](auto count, int i, int n) {
      constexpr int V = decltype(count)::value;
      uint4 b[V];
#pragma unroll
      for (int t = 0; t < V; ++t) {
        const unsigned k = (unsigned)__shfl_sync(0xffffffffu, ks, i + min(t, n - 1));
        b[t] = __ldg(reinterpret_cast<const uint4*>(src + (unsigned long long)k * (unsigned)ldb));
      }
#pragma unroll
      for (int t = 0; t < V; ++t) {
        const float a = __shfl_sync(0xffffffffu, as, (i + t) & 31);
        if (t < n) fma8(acc, a, b[t]);
      }
    };
    int i = 0;
    for (; cnt - i >= U; i += U) entries(std::integral_constant<int, U>{}, i, U);
    // the rest in the smallest step that holds it: a row of one entry in eight loads
    // took 4.3 us where one takes 3.2 (5056 x 832, 0.1 %, N 64)
    const int rest = cnt - i;
    if (rest > U / 2)
      entries(std::integral_constant<int, U>{}, i, rest);
    else if (U > 4 && rest > 2)
      entries(std::integral_constant<int, U / 2>{}, i, rest);
    else if (rest == 2)
      entries(std::integral_constant<int, 2>{}, i, 2);
    else if (rest == 1)
      entries(std::integral_constant<int, 1>{}, i, 1);
  }
}

// The CSR part of one output tile of the hybrid product: rows [row0, row0 + rows)
// and columns [n0, n1) of C (n1 - n0 a multiple of 8) gain A_csr x B in place.
// Called by the four epilogue warps of a CTA (`wq` = 0..3) after their stores of
// the tile are ordered by a barrier; each warp takes every fourth row.
__device__ __forceinline__ void csr_tile_pass(const int* __restrict__ row_ptr, const int* __restrict__ col_idx,
                                              const __half* __restrict__ vals, const __half* __restrict__ B,
                                              long long ldb, float* C, long long ldc, long long row0, int rows,
                                              int n0, int n1, int wq, int lane) {
  for (int r = wq; r < rows; r += 4) {
    const long long row = row0 + r;
    const int e0 = __ldg(row_ptr + row), e1 = __ldg(row_ptr + row + 1);
    if (e0 >= e1) continue;
    for (int nb = n0; nb < n1; nb += 256) {
      const int n = nb + lane * 8;
      const bool valid = n < n1;
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      csr_row_slice<8>(col_idx, vals, B, ldb, e0, e1, n, valid, acc);
      if (valid) {
        float4* c = reinterpret_cast<float4*>(C + row * ldc + n);
        float4 x = __ldcg(c), y = __ldcg(c + 1);
        x.x += acc[0];
        x.y += acc[1];
        x.z += acc[2];
        x.w += acc[3];
        y.x += acc[4];
        y.y += acc[5];
        y.z += acc[6];
        y.w += acc[7];
        c[0] = x;
        c[1] = y;
      }
    }
  }
}

}  // namespace spmm
