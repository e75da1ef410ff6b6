// Epilogue pieces shared by the tensor-core screens (bf16_search.cu,
// exact_screen.cu): an epilogue thread owns one query (one TMEM lane) and
// turns 32 accumulator columns at a time into candidate-list pushes; a warp
// trims a list by a radix select over registers.
#pragma once

#include "tc_util.cuh"

namespace fknn {

constexpr int STAGE_ROW = 36;  // floats per lane row of the push staging area

// max of 32 values as a tree of three-input maxima (16 instructions)
__device__ __forceinline__ float max32(const float *v) {
  float a[10];
#pragma unroll
  for (int k = 0; k < 10; ++k) a[k] = fmax3(v[3 * k], v[3 * k + 1], v[3 * k + 2]);
  const float b0 = fmax3(a[0], a[1], a[2]), b1 = fmax3(a[3], a[4], a[5]), b2 = fmax3(a[6], a[7], a[8]);
  const float b3 = fmax3(a[9], v[30], v[31]);
  return fmax3(b0, b1, fmaxf(b2, b3));
}

__device__ __forceinline__ float max32(const uint32_t (&r)[32]) {
  float v[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
  return max32(v);
}

// bit j set iff v[j] >= t, built as four independent chains
__device__ __forceinline__ uint32_t ge_mask32(const float *v, float t) {
  uint32_t p[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int g = 0; g < 4; ++g) p[g] |= (v[g * 8 + j] >= t ? 1u : 0u) << (g * 8 + j);
  return (p[0] | p[1]) | (p[2] | p[3]);
}

// Screens 32 accumulator columns c .. c+31 of one query (this lane): every
// column j inside the slab [r0, r1) with acc >= cq is appended to the
// query's list with its screening distance qn - 2 sc acc.  The lane's
// candidates form a bit mask; their values are read back from the lane's
// shared-memory staging row, so the push loop runs once per candidate.
__device__ __forceinline__ int screen_chunk(const uint32_t (&r)[32], int c, int r0, int r1, float cq, float qn,
                                            float sc, uint32_t p0, float *row, Candidate *list, int cnt) {
  if (r0 >= c + 32 || r1 <= c) return cnt;
  float v[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
  if (!(r0 <= c && r1 >= c + 32)) {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (c + j < r0 || c + j >= r1) v[j] = -INFINITY;
  }
  if (max32(v) >= cq) {
    uint32_t mask = ge_mask32(v, cq);
#pragma unroll
    for (int j = 0; j < 32; j += 4)
      *reinterpret_cast<float4 *>(row + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    while (mask) {
      const int j = __ffs(mask) - 1;
      mask &= mask - 1;
      Candidate cd;
      cd.ds = fmaf(-2.f * sc, row[j], qn);
      cd.pos = p0 + c + j;
      list[cnt++] = cd;
    }
  }
  return cnt;
}

// kth smallest (1-based) of the n keys held NPL per lane (element
// j*32 + lane in key[j]; keys past n ignored): a warp radix select that
// starts below the bits all keys share and takes up to 8 bits per pass from
// a shared-memory histogram.  Keys are order-preserving images of floats.
template <int NPL>
__device__ __forceinline__ uint32_t warp_kth_regs(const uint32_t (&key)[NPL], int n, int kth, uint32_t *hist) {
  const int lane = threadIdx.x & 31;
  uint32_t mn = 0xffffffffu, mx = 0u;
#pragma unroll
  for (int j = 0; j < NPL; ++j)
    if (j * 32 + lane < n) {
      mn = min(mn, key[j]);
      mx = max(mx, key[j]);
    }
  mn = __reduce_min_sync(0xffffffffu, mn);
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (mn == mx) return mn;
  int hi = 32 - __clz(mn ^ mx);  // bits [hi-1, 0] still differ
  uint32_t mask = hi == 32 ? 0u : ~((1u << hi) - 1u);
  uint32_t prefix = mn & mask;
  int remaining = kth;
  while (hi > 0) {
    const int w = min(8, hi), shift = hi - w;
    const uint32_t nb = 1u << w;
    for (uint32_t i = lane; i < 256; i += 32) hist[i] = 0;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < NPL; ++j)
      if (j * 32 + lane < n && (key[j] & mask) == prefix) atomicAdd(&hist[(key[j] >> shift) & (nb - 1)], 1u);
    __syncwarp();
    uint32_t local[8], sum = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      local[j] = hist[lane * 8 + j];
      sum += local[j];
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    const uint32_t excl = inc - sum;
    const uint32_t hit = __ballot_sync(0xffffffffu, excl < (uint32_t)remaining && inc >= (uint32_t)remaining);
    const int owner = __ffs(hit) - 1;
    uint32_t bin = 0, before = 0;
    if (lane == owner) {
      uint32_t c = excl;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (c + local[j] >= (uint32_t)remaining) {
          bin = lane * 8 + j;
          before = c;
          break;
        } else {
          c += local[j];
        }
    }
    bin = __shfl_sync(0xffffffffu, bin, owner);
    before = __shfl_sync(0xffffffffu, before, owner);
    remaining -= (int)before;
    prefix |= bin << shift;
    mask |= (nb - 1) << shift;
    hi = shift;
    __syncwarp();
  }
  return prefix;
}

}  // namespace fknn
