// Small device helpers: mbarrier + bulk-copy PTX, bounded waits, sorts,
// the reference's sequential L2.
#pragma once

#include "fknn_internal.cuh"

namespace fknn {

// Every spin-wait gives up after WAIT_NS nanoseconds of the global timer
// (checked every 64 polls), with an iteration cap behind it in case the
// timer does not advance.
constexpr uint64_t WAIT_NS = 1000000000ull;
constexpr uint32_t WAIT_LIMIT = 1u << 28;

// Error bits written to the per-call device flag.
constexpr int ERR_WAIT_TIMEOUT = 1 << 8;
constexpr int ERR_BAD_QUERY_TYPE = 1 << 0;
constexpr int ERR_BAD_QUERY_VALUE = 1 << 1;
constexpr int ERR_BAD_QUERY_VEC = 1 << 2;
constexpr int ERR_PLAN_BOUND = 1 << 3;  // a device-built plan met a buffer bound (reported, never written past)

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// 1-D bulk copy global -> shared (the TMA bulk engine), completion counted
// on an mbarrier.  dst, src 16-byte aligned; bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait: returns false (and raises ERR_WAIT_TIMEOUT) if the phase
// has not completed within WAIT_NS.  The timer is first read after 64 polls:
// reading it costs more than most waits last.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, int *err) {
  if (mbar_try_wait(bar, parity)) return true;
  uint64_t t0 = 0;
#pragma unroll 1
  for (uint32_t it = 1; it < WAIT_LIMIT; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 63u) == 0u) {
      const uint64_t t = global_ns();
      if (t0 == 0) t0 = t;
      else if (t - t0 > WAIT_NS) break;
    }
  }
  atomicOr(err, ERR_WAIT_TIMEOUT);
  return false;
}

__device__ __forceinline__ uint32_t ld_volatile_u32(const uint32_t *p) { return *(const volatile uint32_t *)p; }

__device__ __forceinline__ uint64_t exact_key(float d, uint32_t id) {
  return ((uint64_t)f32_sortable(d) << 32) | id;
}

// In-shared-memory bitonic sort of n (power of two) elements, ascending,
// all threads of the block participate.
template <typename K>
__device__ void block_bitonic_sort(K *key, int n) {
  for (int size = 2; size <= n; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < (n >> 1); i += blockDim.x) {
        int lo = 2 * stride * (i / stride) + (i % stride);
        int hi = lo + stride;
        bool asc = (lo & size) == 0;
        K a = key[lo], b = key[hi];
        if ((a > b) == asc) {
          key[lo] = b;
          key[hi] = a;
        }
      }
      __syncthreads();
    }
  }
}

// L2SqrSQ8_sym (pyglass/glass/simd/distance.hpp:329-366) as an exact int32
// over 112-byte codes: |q - c|^2 = |q|^2 + |c|^2 - 2 q.c with dp4a; qw is the
// query code as words, qq its squared norm.  Bytes 100..111 are padding and
// not looked at (a graph's codes carry their squared norm there).
__device__ __forceinline__ int sq8_dist(const int *__restrict__ qw, int qq, const int8_t *__restrict__ code) {
  const int4 *c4 = reinterpret_cast<const int4 *>(code);
  int cc = 0, qc = 0;
#pragma unroll
  for (int w = 0; w < 28 / 4; ++w) {
    const int4 v = c4[w];
    cc = __dp4a(v.x, v.x, cc);
    qc = __dp4a(qw[4 * w + 0], v.x, qc);
    if (w == DIM / 16) break;
    cc = __dp4a(v.y, v.y, cc);
    cc = __dp4a(v.z, v.z, cc);
    cc = __dp4a(v.w, v.w, cc);
    qc = __dp4a(qw[4 * w + 1], v.y, qc);
    qc = __dp4a(qw[4 * w + 2], v.z, qc);
    qc = __dp4a(qw[4 * w + 3], v.w, qc);
  }
  return qq + cc - 2 * qc;
}


// Offsets of one query's candidate lists in the merge: warp 0 reads the
// item counts (item_slot[item0 + i] selects the item, lane L of tq the
// list) 32 at a time and scans them with shuffles.  prefix[i] = first
// position of item i, *total = their sum, or over_value when there are more
// than max_items items (item_slot NULL: the items are item0 .. item0 +
// nitems - 1).  Caller: the whole block, then __syncthreads().
__device__ __forceinline__ void list_offsets(const uint32_t *__restrict__ item_slot, uint32_t item0, uint32_t nitems,
                                             const uint32_t *__restrict__ out_cnt, uint32_t L, uint32_t tq,
                                             uint32_t *prefix, int *total, uint32_t max_items, int over_value) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  if (nitems > max_items) {
    if (lane == 0) *total = over_value;
    return;
  }
  uint32_t carry = 0;
  for (uint32_t base = 0; base < nitems; base += 32) {
    const uint32_t i = base + lane;
    const uint32_t c = i < nitems ? out_cnt[(uint64_t)(item_slot ? item_slot[item0 + i] : item0 + i) * tq + L] : 0u;
    uint32_t inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    if (i < nitems) prefix[i] = carry + inc - c;
    carry += __shfl_sync(0xffffffffu, inc, 31);
  }
  if (lane == 0) *total = (int)carry;
}

// kth smallest (1-based, kth <= n) of key[0 .. n) in shared memory, as its
// f32_sortable image: a radix select of the whole block that starts below
// the bits all keys share.  red: 4 words of shared memory.
template <int THREADS>
__device__ uint32_t block_kth(const float *key, int n, uint32_t kth, uint32_t *hist, uint32_t *red) {
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) {
    red[0] = 0xffffffffu;
    red[1] = 0;
  }
  __syncthreads();
  uint32_t mn = 0xffffffffu, mx = 0;
  for (int i = tid; i < n; i += THREADS) {
    const uint32_t u = f32_sortable(key[i]);
    mn = min(mn, u);
    mx = max(mx, u);
  }
  mn = __reduce_min_sync(0xffffffffu, mn);
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) {
    atomicMin(&red[0], mn);
    atomicMax(&red[1], mx);
  }
  __syncthreads();
  mn = red[0];
  mx = red[1];
  int hi = mn == mx ? 0 : 32 - __clz(mn ^ mx);
  uint32_t mask = hi == 32 ? 0u : ~((1u << hi) - 1u);
  uint32_t prefix = mn & mask, remaining = kth;
  while (hi > 0) {
    const int w = min(8, hi), shift = hi - w;
    for (int i = tid; i < 256; i += THREADS) hist[i] = 0;
    __syncthreads();
    for (int i = tid; i < n; i += THREADS) {
      const uint32_t u = f32_sortable(key[i]);
      if ((u & mask) == prefix) atomicAdd(&hist[(u >> shift) & ((1u << w) - 1)], 1u);
    }
    __syncthreads();
    if (tid < 32) {
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
      uint32_t c = inc - sum;
      if (c < remaining && inc >= remaining) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (c < remaining && c + local[j] >= remaining) {
            red[2] = lane * 8 + j;
            red[3] = c;
          }
          c += local[j];
        }
      }
    }
    __syncthreads();
    prefix |= red[2] << shift;
    remaining -= red[3];
    mask |= ((1u << w) - 1) << shift;
    hi = shift;
  }
  __syncthreads();
  return prefix;
}

// distance.h:62-72 normal_l2(base, query): v = x - q; v *= v; r += v, every
// operation rounded to float, in dimension order, never fused.  The row is
// 16-byte aligned: four dimensions per load.
__device__ __forceinline__ float seq_l2_row(const float *__restrict__ x, const float *q) {
  const float4 *x4 = reinterpret_cast<const float4 *>(x);
  float r = 0.f;
#pragma unroll 5
  for (int d = 0; d < DIM / 4; ++d) {
    const float4 v = __ldg(x4 + d);
    const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float t = __fsub_rn(e[j], q[4 * d + j]);
      t = __fmul_rn(t, t);
      r = __fadd_rn(r, t);
    }
  }
  return r;
}

}  // namespace fknn
