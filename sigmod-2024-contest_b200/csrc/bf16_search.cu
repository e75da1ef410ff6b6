// Reduced-precision form: BF16 tensor-core screen (tcgen05, FP32 accumulate
// in TMEM) into a widened candidate list of k' per query, FP32 re-rank from
// the original vectors with the reference's arithmetic (distance.h:62-72),
// FP64 recompute of the candidates within 1e-6 relative of the k-th FP32
// distance so the boundary order follows exact arithmetic.
//
// Layouts (both operands K-major, no swizzle, core matrices of 8 rows x 16 B):
//   query half A: 128 queries x 112 bf16, element (q, k) at
//                 ((k/8)*16 + q/8)*64 + (q%8)*8 + k%8
//   row block  B: 256 rows x 112 bf16, element (r, k) at
//                 ((k/8)*32 + r/8)*64 + (r%8)*8 + k%8
// Dims 0..99 carry the vector; on the row side dims 100/101 carry
// -|x|^2/2 split into a bf16 high part and a bf16 remainder, on the query
// side dims 100/101 are 1.0.  The MMA therefore produces
// acc = q.x - |x|^2/2, and ds = |q|^2 - 2*acc approximates |q - x|^2 with no
// per-row term left for the epilogue: a row is a candidate for query q iff
// acc >= (|q|^2 - T_q)/2, one compare per TMEM value.
#include <algorithm>
#include <cfloat>
#include <chrono>
#include <cstring>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "screen_util.cuh"

namespace fknn {

namespace {

constexpr int BQ = 256;                       // queries per tile: two halves of 128 = MMA M = TMEM lanes
constexpr int BM = BQ / 2;
constexpr int BR = 256;                       // rows per block = MMA N
constexpr int BP = 128;                       // columns an epilogue warp screens
constexpr int BS = 2;                         // shared-memory stages for row blocks
constexpr int B_ACCS = 2;                     // accumulators
constexpr int B_EPI = 4 * (BR / BP);          // epilogue warps 0 .. 7: TMEM lanes 32 (w % 4) .., columns BP (w / 4) ..
constexpr int B_LISTS = B_EPI * 32;           // working lists of a half: one per epilogue thread
constexpr int B_LOAD_WARP = B_EPI;
constexpr int B_MMA_WARP = B_EPI + 1;
constexpr int B_THREADS = (B_EPI + 2) * 32;
constexpr uint32_t TMEM_COLS = B_ACCS * BR;
constexpr int B_SLOTS = 8;                    // 32-column chunks an epilogue warp stages at a time
constexpr int B_ROW = 36;                     // words of a staged chunk: 32 columns, 4 of its query
constexpr int B_SLACK = 24;                   // entries past the k'-th that a trim may keep

// Operand formats of the tensor-core screen.  Both operands are K-major,
// no swizzle, in core matrices of 8 rows x 16 bytes; every MMA consumes 32
// bytes of K per row (two core-matrix columns), so the descriptors of both
// formats are alike and only the MMA kind, its K and the bytes per row differ.
struct FmtBF16 {
  static constexpr bool kFP8 = false;
  static constexpr int K = 112;                 // 100 dims, 2 norm terms, zero padding
  static constexpr int ROW_BYTES = K * 2;
  static constexpr int MMAS = K / 16;           // kind::f16: K = 16 per MMA
  // F32 accumulate, BF16 A and B, K-major, N = BR, M = BM
  static constexpr uint32_t IDESC =
      (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BR >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
};
struct FmtFP8 {
  static constexpr bool kFP8 = true;
  static constexpr int K = 128;                 // 100 dims, 3 norm terms, zero padding
  static constexpr int ROW_BYTES = K;
  static constexpr int MMAS = K / 32;           // kind::f8f6f4: K = 32 per MMA
  // F32 accumulate, E4M3 A and B, K-major, N = BR, M = BM
  static constexpr uint32_t IDESC =
      (1u << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(BR >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
};
template <class F>
struct Tiles {
  static constexpr uint32_t A = (uint32_t)BM * F::ROW_BYTES;  // half a tile's queries
  static constexpr uint32_t B = (uint32_t)BR * F::ROW_BYTES;  // a row block
};

// byte offset of (row r, byte b of the row) in a row block
__device__ __forceinline__ uint32_t rb_byte(uint32_t r, uint32_t b) {
  return ((b >> 4) * (BR / 8) + (r >> 3)) * 128 + (r & 7) * 16 + (b & 15);
}

template <class F>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
  if constexpr (F::kFP8) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(F::IDESC), "r"(accumulate));
  } else {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(F::IDESC), "r"(accumulate));
  }
}

// ------------------------------------------------------------- build ---

__global__ void k_build_bf16_blocks(const float *__restrict__ vecs, const float *__restrict__ norms,
                                    const uint32_t *__restrict__ perm, uint64_t n, __nv_bfloat16 *__restrict__ out) {
  const uint64_t b = blockIdx.x;
  constexpr int BK = FmtBF16::K;
  __nv_bfloat16 *o = out + b * (Tiles<FmtBF16>::B / 2);
  for (uint32_t i = threadIdx.x; i < (uint32_t)BR * BK; i += blockDim.x) {
    const uint32_t r = i / BK, k = i % BK;
    const uint64_t p = b * BR + r;
    float v = 0.f;
    if (p < n) {
      const uint32_t id = perm[p];
      if (k < (uint32_t)DIM) {
        v = vecs[(uint64_t)id * DIM + k];
      } else if (k == DIM || k == DIM + 1) {
        const float h = -0.5f * norms[id];
        const float hi = __bfloat162float(__float2bfloat16_rn(h));
        v = (k == DIM) ? hi : h - hi;
      }
    }
    o[rb_byte(r, 2 * k) / 2] = __float2bfloat16_rn(v);
  }
}

// Where a tile's lanes come from: the host plan's per-tile arrays, or a
// device plan's sorted queries (tile t = positions tile_first[t] ..
// + tiles[t].nq of order_q, slabs from the query descriptors).
struct LaneSrc {
  const int32_t *lane_q = nullptr;
  const uint32_t *lane_s = nullptr, *lane_e = nullptr;
  const uint32_t *tile_first = nullptr, *order_q = nullptr;
  const QueryDesc *desc = nullptr;
  const uint32_t *ntile = nullptr;  // device plan: the tile count
};

__device__ __forceinline__ int32_t lane_query(const LaneSrc &ls, const Tile &tl, uint32_t t, int L, uint32_t &s,
                                              uint32_t &e) {
  if (ls.lane_q) {
    const int32_t qi = ls.lane_q[t * BQ + L];
    if (qi >= 0) {
      s = ls.lane_s[t * BQ + L];
      e = ls.lane_e[t * BQ + L];
    }
    return qi;
  }
  if ((uint32_t)L >= tl.nq) return -1;
  const int32_t qi = (int32_t)ls.order_q[ls.tile_first[t] + L];
  s = ls.desc[qi].s;
  e = ls.desc[qi].e;
  return qi;
}

// One block per tile (grid-strided over a device plan's tile count).
__global__ void k_tile_stage_bf16(const float *__restrict__ q, LaneSrc ls, const Tile *__restrict__ tiles,
                                  uint32_t ntile_h, const QueryDesc *__restrict__ desc,
                                  __nv_bfloat16 *__restrict__ out, float2 *__restrict__ lane_qs) {
  constexpr int BK = FmtBF16::K;
  const uint32_t ntile = ls.ntile ? *ls.ntile : ntile_h;
  __shared__ int32_t lq[BQ];
  for (uint32_t t = blockIdx.x; t < ntile; t += gridDim.x) {
    const Tile tl = tiles[t];
    __nv_bfloat16 *o = out + (uint64_t)t * 2 * (Tiles<FmtBF16>::A / 2);
    for (uint32_t l = threadIdx.x; l < (uint32_t)BQ; l += blockDim.x) {
      uint32_t s_, e_;
      const int32_t qi = lane_query(ls, tl, t, (int)l, s_, e_);
      lq[l] = qi;
      lane_qs[t * BQ + l] = make_float2(qi >= 0 ? desc[qi].qn : 0.f, 1.f);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < (uint32_t)BQ * BK; i += blockDim.x) {
      const uint32_t l = i / BK, k = i % BK;
      const int32_t qi = lq[l];
      float v = 0.f;
      if (qi >= 0) {
        if (k < (uint32_t)DIM) v = q[(uint64_t)qi * DIM + k];
        else if (k == DIM || k == DIM + 1) v = 1.f;
      }
      o[(l / BM) * (Tiles<FmtBF16>::A / 2) + cm_index(l % BM, k)] = __float2bfloat16_rn(v);
    }
    __syncthreads();
  }
}

// FP8-e4m3 per-dimension-scaled codes, the tensor-core analogue of the
// per-dimension SQ8 codes of sq8_quant.hpp:30-63 (mi/dif per dimension).
// Each dimension is centred at c = (max + min)/2 and scaled by
// s = (max - min)/2 / 448 so its range fills e4m3 (|x'| <= 448):
//   row side : x'_k = e4m3((x_k - c_k) / s_k), k < 100; dims 100..102 hold
//              -|x - c|^2/2 as e4m3 high, middle and low parts
//   query    : A_k = e4m3(lambda * (q_k - c_k) * s_k); dims 100..102 = lambda,
//              lambda a power of two in [2^-9, 2^8] with max|A_k| <= 448
// so acc = lambda * ((q - c).(x - c) - |x - c|^2/2) and
// ds = |q - c|^2 - 2 acc / lambda approximates |q - x|^2.
__global__ void k_dim_minmax(const float *__restrict__ vecs, uint64_t n, uint32_t *__restrict__ mn,
                             uint32_t *__restrict__ mx) {
  __shared__ uint32_t smn[DIM], smx[DIM];
  for (int d = threadIdx.x; d < DIM; d += blockDim.x) {
    smn[d] = 0xffffffffu;
    smx[d] = 0u;
  }
  __syncthreads();
  const uint64_t total = n * DIM;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t u = f32_sortable(vecs[i]);
    const int d = (int)(i % DIM);
    atomicMin(&smn[d], u);
    atomicMax(&smx[d], u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < DIM; d += blockDim.x) {
    atomicMin(&mn[d], smn[d]);
    atomicMax(&mx[d], smx[d]);
  }
}

__global__ void k_fp8_params(const uint32_t *__restrict__ mn, const uint32_t *__restrict__ mx,
                             float *__restrict__ center, float *__restrict__ scale) {
  const int d = threadIdx.x;
  if (d >= DIM) return;
  const float a = sortable_f32(mn[d]), b = sortable_f32(mx[d]);
  center[d] = 0.5f * (a + b);
  scale[d] = fmaxf(0.5f * (b - a), 1e-30f) / 448.f;
}

__global__ void k_build_fp8_blocks(const float *__restrict__ vecs, const uint32_t *__restrict__ perm, uint64_t n,
                                   const float *__restrict__ center, const float *__restrict__ scale,
                                   unsigned char *__restrict__ out) {
  const uint64_t b = blockIdx.x;
  unsigned char *o = out + b * Tiles<FmtFP8>::B;
  __shared__ float cn[BR];
  // centred norms of the block's rows (float FMA chain)
  for (uint32_t r = threadIdx.x; r < (uint32_t)BR; r += blockDim.x) {
    const uint64_t p = b * BR + r;
    float s = 0.f;
    if (p < n) {
      const float *x = vecs + (uint64_t)perm[p] * DIM;
      for (int k = 0; k < DIM; ++k) {
        const float t = x[k] - center[k];
        s = fmaf(t, t, s);
      }
    }
    cn[r] = s;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < (uint32_t)BR * FmtFP8::K; i += blockDim.x) {
    const uint32_t r = i / FmtFP8::K, k = i % FmtFP8::K;
    const uint64_t p = b * BR + r;
    float v = 0.f;
    if (p < n) {
      if (k < (uint32_t)DIM) {
        v = (vecs[(uint64_t)perm[p] * DIM + k] - center[k]) / scale[k];
      } else if (k <= DIM + 2) {
        const float h = -0.5f * cn[r];
        const float hi = float(__nv_fp8_e4m3(h));
        const float mid = float(__nv_fp8_e4m3(h - hi));
        v = (k == DIM) ? hi : (k == DIM + 1) ? mid : h - hi - mid;
      }
    }
    o[rb_byte(r, k)] = __nv_fp8_e4m3(v).__x;
  }
}

__global__ void k_tile_stage_fp8(const float *__restrict__ q, LaneSrc ls, const Tile *__restrict__ tiles,
                                 uint32_t ntile_h, const float *__restrict__ center, const float *__restrict__ scale,
                                 unsigned char *__restrict__ out, float2 *__restrict__ lane_qs) {
  const uint32_t ntile = ls.ntile ? *ls.ntile : ntile_h;
  __shared__ float lam[BQ];
  __shared__ int32_t lq[BQ];
  for (uint32_t t = blockIdx.x; t < ntile; t += gridDim.x) {
    const Tile tl = tiles[t];
    unsigned char *o = out + (uint64_t)t * 2 * Tiles<FmtFP8>::A;
    for (uint32_t l = threadIdx.x; l < (uint32_t)BQ; l += blockDim.x) {
      uint32_t s_, e_;
      const int32_t qi = lane_query(ls, tl, t, (int)l, s_, e_);
      lq[l] = qi;
      float qn = 0.f, mw = 0.f;
      if (qi >= 0) {
        const float *x = q + (uint64_t)qi * DIM;
        for (int k = 0; k < DIM; ++k) {
          const float u = x[k] - center[k];
          qn = fmaf(u, u, qn);
          mw = fmaxf(mw, fabsf(u * scale[k]));
        }
      }
      // largest power of two with lambda * max|w| <= 448, within e4m3's exact powers
      int e = 8;
      if (mw > 0.f) e = min(8, max(-9, (int)floorf(log2f(448.f / mw))));
      const float lambda = ldexpf(1.f, e);
      lam[l] = lambda;
      lane_qs[t * BQ + l] = make_float2(qn, 1.f / lambda);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < (uint32_t)BQ * FmtFP8::K; i += blockDim.x) {
      const uint32_t l = i / FmtFP8::K, k = i % FmtFP8::K;
      const int32_t qi = lq[l];
      float v = 0.f;
      if (qi >= 0) {
        if (k < (uint32_t)DIM) v = lam[l] * (q[(uint64_t)qi * DIM + k] - center[k]) * scale[k];
        else if (k <= DIM + 2) v = lam[l];
      }
      o[(l / BM) * Tiles<FmtFP8>::A + cm_byte(l % BM, k)] = __nv_fp8_e4m3(v).__x;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------ screen ---

template <class F>
struct BScreenSmem {
  unsigned char a[2][Tiles<F>::A];
  unsigned char b[BS][Tiles<F>::B];
  struct {
    float row[B_SLOTS][B_ROW];  // staged chunks
    uint32_t hist[256];         // the histogram of a trim
  } w[B_EPI];
  float4 q[BQ];      // per query: lowest accumulator value of a candidate, slab (bits), what a pilot keeps: the best of
                     // every so many rows (BP, 32, 8 or 1)
  float2 qs[BQ];     // |q|^2 (centred for FP8), -2 / lambda
  float thr[BQ];     // current bound T on the k'-th screening distance
  int32_t lq[BQ];
  int cnt[2][B_LISTS];
  uint64_t full[BS], empty[BS], accfull[B_ACCS], accempty[B_ACCS], afull;
  uint32_t tmem_base;
  uint32_t next[2];  // the next processing slot, by item parity (work queue)
};
static_assert(sizeof(BScreenSmem<FmtBF16>) <= 227 * 1024, "one screen CTA per SM");

struct ScreenArgs {
  const WorkItem *items;
  const Tile *tiles;
  const unsigned char *atiles;  // [tile][half], operand tiles of 128 queries
  LaneSrc ls;
  const float2 *lane_qs;        // per tile lane: |q|^2 (centred for FP8), 1 / lambda
  const unsigned char *blocks_t, *blocks_c;
  uint32_t *T_global;           // per query: upper bound on its k'-th screening distance (f32_sortable)
  uint32_t *ovf;                // per query: non-zero = left to the exact scan
  Candidate *work;              // [CTA][half][B_LISTS][capb]
  Candidate *out;               // [item][BQ][ocap]
  uint32_t *out_cnt;            // [item][BQ]
  uint32_t kprime, capb, ocap, refresh;
  uint32_t halves;              // working lists per CTA: 1 where no tile has more than BM queries
  uint32_t kseed;               // pilot: k' of the search
  uint32_t stride;              // > 1: a pilot pass over every stride-th row block
  uint32_t withhold;
  uint32_t nitems;
  const uint32_t *nitems_d;     // device plan: the item count (NULL: nitems)
  const uint32_t *order;        // processing slot -> item (NULL: the same)
  uint32_t *queue;              // zero at the launch: next slot past the grid's first ones
  int *err;
};

// candidate iff qn - 2*sc*acc <= T  <=>  acc >= (qn - T) / (2 sc); with no
// bound yet every column of the slab is one.  f2 = -2 sc, a power of two.
__device__ __forceinline__ float acc_bound(float T, float2 qs) {
  return T == INFINITY ? -FLT_MAX : (T - qs.x) / qs.y;
}

// Trim of one list (n entries) of query L: the k'-th screening distance, or
// one a little above it, bounds what is kept; the bound is shared through
// T_global and with the CTA's other lists of the query.  Whole warp; returns
// the number kept (0 where ties do not fit: the exact scan answers the query).
template <class F, int NPL>
__device__ __noinline__ int b_trim(Candidate *list, int n, BScreenSmem<F> &sm, int L, uint32_t kprime,
                                      uint32_t capb, uint32_t *T_global, uint32_t *ovf) {
  const int lane = threadIdx.x & 31;
  const int32_t qi = sm.lq[L];
  float T = sm.thr[L];
  const float Tg = sortable_f32(ld_volatile_u32(T_global + qi));
  uint32_t key[NPL], pos[NPL];
#pragma unroll
  for (int j = 0; j < NPL; ++j) {
    const int i = j * 32 + lane;
    uint2 c = make_uint2(0xffffffffu, 0u);
    if (i < n) c = *reinterpret_cast<const uint2 *>(list + i);
    key[j] = i < n ? f32_sortable(__uint_as_float(c.x)) : 0xffffffffu;
    pos[j] = c.y;
  }
  if (n >= (int)kprime)
    T = fminf(T, sortable_f32(warp_kth_upper<NPL>(key, n, (int)kprime, B_SLACK, sm.w[threadIdx.x >> 5].hist)));
  if (Tg < T) T = Tg;
  if (lane == 0 && T < Tg) atomicMin(T_global + qi, f32_sortable(T));
  const uint32_t tk = f32_sortable(T);
  int kept = 0;
  const uint32_t lt = (1u << lane) - 1u;
  uint2 *dst = reinterpret_cast<uint2 *>(list);
  __syncwarp();
#pragma unroll
  for (int j = 0; j < NPL; ++j) {
    if (j * 32 >= n) break;
    const bool keep = j * 32 + lane < n && key[j] <= tk;
    const uint32_t b = __ballot_sync(0xffffffffu, keep);
    if (keep) dst[kept + __popc(b & lt)] = make_uint2(__float_as_uint(sortable_f32(key[j])), pos[j]);
    kept += __popc(b);
  }
  __syncwarp();
  if (kept > (int)capb - BP) {  // a tie flood
    if (lane == 0) ovf[qi] = 1u;
    T = -INFINITY;
    kept = 0;
  }
  if (lane == 0) {
    sm.thr[L] = T;
    sm.q[L].x = acc_bound(T, sm.qs[L]);
  }
  __syncwarp();
  return kept;
}

// The item's result for a query whose lists (one in every BM from work and cnt
// on, more than ocap entries in all) have to be bounded: their k'-th screening
// distance by a radix select that reads them again for every digit (rare: a
// seeded query has far fewer).  Whole warp; returns the entries written, more
// than ocap only where ties do not fit.
template <class F>
__device__ __noinline__ int b_select(const Candidate *work, const int *cnt, BScreenSmem<F> &sm, int L, uint32_t kprime,
                                     uint32_t capb, uint32_t ocap, uint32_t *T_global, Candidate *out) {
  const int lane = threadIdx.x & 31;
  uint32_t *hist = sm.w[threadIdx.x >> 5].hist;
  auto each = [&](auto &&f) {  // every entry, the warp together
#pragma unroll 1
    for (int l = 0; l < B_LISTS; l += BM) {
      const uint2 *list = reinterpret_cast<const uint2 *>(work + (uint64_t)l * capb);
      const int n = cnt[l];
#pragma unroll 1
      for (int i = 0; i < n; i += 32) f(i + lane < n, i + lane < n ? list[i + lane] : make_uint2(0u, 0u));
    }
  };
  uint32_t mask = 0, prefix = 0, want = kprime;
#pragma unroll 1
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (int i = lane; i < 256; i += 32) hist[i] = 0;
    __syncwarp();
    each([&](bool on, uint2 c) {
      const uint32_t u = f32_sortable(__uint_as_float(c.x));
      if (on && (u & mask) == prefix) atomicAdd(&hist[u >> shift & 255], 1u);
    });
    __syncwarp();
    uint32_t before = 0, bin = 0;
#pragma unroll 1
    for (uint32_t b = 0; b < 256; b += 32) {  // the bin of the want-th key of the prefix
      const uint32_t c = hist[b + lane];
      uint32_t inc = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      const uint32_t hit = __ballot_sync(0xffffffffu, before + inc >= want);
      if (hit) {
        const int w = __ffs(hit) - 1;
        bin = b + w;
        before += __shfl_sync(0xffffffffu, inc - c, w);
        break;
      }
      before += __shfl_sync(0xffffffffu, inc, 31);
    }
    want -= before;
    prefix |= bin << shift;
    mask |= 255u << shift;
    __syncwarp();
  }
  if (lane == 0) atomicMin(T_global + sm.lq[L], prefix);
  int kept = 0;
  each([&](bool on, uint2 c) {
    const bool keep = on && f32_sortable(__uint_as_float(c.x)) <= prefix;
    const uint32_t b = __ballot_sync(0xffffffffu, keep);
    const uint32_t o = kept + __popc(b & ((1u << lane) - 1u));
    if (keep && o < ocap) *reinterpret_cast<uint2 *>(out + o) = c;
    kept += __popc(b);
  });
  return kept;
}

// Stages one chunk of a lane's columns, and what an append needs of its
// query: the bound, ds = qn + f2 v, and the slab's columns and lane packed.
__device__ __forceinline__ void stage32(float *row, const uint32_t (&r)[32], float bound, float f2, float qn,
                                        uint32_t pack) {
#pragma unroll
  for (int j = 0; j < 32; j += 4)
    *reinterpret_cast<uint4 *>(row + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
  *reinterpret_cast<uint4 *>(row + 32) = make_uint4(__float_as_uint(bound), __float_as_uint(f2), __float_as_uint(qn), pack);
}
// r0, r1 in [0, 256], lane
__device__ __forceinline__ uint32_t pack_query(int r0, int r1, int lane, int col) {
  return (uint32_t)r0 | (uint32_t)r1 << 9 | (uint32_t)lane << 18 | (uint32_t)col / 32 << 23;
}

// Persistent, one CTA per SM, pulling work items (longest first) from a
// queue: warps 0-7 are the epilogue, warp 8 copies row blocks in, warp 9 issues
// MMAs.  A tile of more than 128 queries multiplies every row block with
// both halves of its queries, so a block crosses from L2 once for 256 queries.
// The products go to the two accumulators in turn, and every epilogue warp
// takes its columns of each into registers and releases it at once: what a
// warp does about candidates, which few blocks hold and then for a while, runs
// while the next product is made (with an accumulator and half the warps for
// each query half, every one of them waited for the slowest).
// N = 256: an MMA of 128 columns takes 91 cycles here, one of 256 takes 128.
// Bound by the epilogue's latency: a warp needs about 1,200 cycles a product
// (the MMAs 896) and 640 more when one of its queries has a candidate; sixteen
// epilogue warps of 64 columns each (96 registers a thread) measured the same.  Screens of a call, pilot
// included, before (tiles of 128 x 128, two CTAs per SM) and now: 50 queries
// over 1e6 rows 0.92 and 0.17 ms, 4,096 over 2e6 4.35 and 2.04 ms, 100,000 over
// 4e6 41.1 and 36 to 38 ms.
// Barrier phases run on across items: g counts the row blocks of this CTA's
// earlier items, u the products.
template <class F, int NPL>
__global__ void __launch_bounds__(B_THREADS, 1) k_screen_tc(ScreenArgs A) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  BScreenSmem<F> &sm = *reinterpret_cast<BScreenSmem<F> *>(smem_raw);
  constexpr uint32_t TA = Tiles<F>::A, TB = Tiles<F>::B;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t nitems = A.nitems_d ? *A.nitems_d : A.nitems;
  if (blockIdx.x >= nitems) return;  // (uniform: before any barrier or TMEM use)

  if (tid == 0) {
    for (int s = 0; s < BS; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    for (int a = 0; a < B_ACCS; ++a) {
      mbar_init(&sm.accfull[a], 1);
      mbar_init(&sm.accempty[a], B_EPI);
    }
    mbar_init(&sm.afull, 1);
    fence_mbar_init();
  }
  if (warp == B_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  uint32_t g = 0, iter = 0, u = 0;
  // a bounded wait gave up: the CTA's later items only mark their queries
  // (combined over the block at each item's closing barrier, so uniform)
  bool aborted = false;
  for (uint32_t slot = blockIdx.x; slot < nitems; ++iter) {
    const uint32_t item_id = A.order ? A.order[slot] : slot;
    const WorkItem it = A.items[item_id];
    const Tile tl = A.tiles[it.tile];
    const bool both = tl.nq > (uint32_t)BM;
    // every stride-th row block of the item (stride 1: all of them)
    const uint32_t nsub = (it.blk1 - it.blk0 + A.stride - 1) / A.stride;
    const uint32_t nprod = both ? 2 * nsub : nsub;
    bool gave_up = false;  // this thread saw a wait give up in this item

    if (warp == B_LOAD_WARP) {
      // ------------------------------------------------ producer
      if (lane == 0 && !aborted) {
        const unsigned char *blocks = tl.order == ORDER_TIME ? A.blocks_t : A.blocks_c;
        bool ok = true;
        const uint32_t na = both ? 2 * TA : TA;
        mbar_arrive_expect_tx(&sm.afull, na);
        bulk_g2s(sm.a[0], A.atiles + (uint64_t)it.tile * 2 * TA, na, &sm.afull);
        uint32_t issued = 0;
        // test hook (fknn_index_test_withhold_copy): the first work item issues
        // no row-block copy, so its MMA issuer's and epilogue's waits run out
        const uint32_t nsub_issue = (A.withhold && item_id == 0) ? 0u : nsub;
#pragma unroll 1
        for (uint32_t sub = 0; sub < nsub_issue; ++sub) {
          const uint32_t gs = g + sub;
          const int st = gs % BS;
          if (gs >= BS && !mbar_wait_bounded(&sm.empty[st], ((gs / BS) - 1) & 1, A.err)) {
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(&sm.full[st], TB);
          bulk_g2s(sm.b[st], blocks + (uint64_t)(it.blk0 + sub * A.stride) * TB, TB, &sm.full[st]);
          ++issued;
        }
        // every issued copy has landed before the item ends
        ok = mbar_wait_bounded(&sm.afull, iter & 1, A.err) && ok;
#pragma unroll 1
        for (uint32_t i = issued > BS ? issued - BS : 0; i < issued; ++i)
          ok = mbar_wait_bounded(&sm.full[(g + i) % BS], ((g + i) / BS) & 1, A.err) && ok;
        if (!ok || issued != nsub) gave_up = true;
      }
      __syncwarp();
    } else if (warp == B_MMA_WARP) {
      // ------------------------------------------------ MMA issuer
      if (lane == 0 && !aborted) {
        uint32_t done = 0, v = u;
        bool ok = mbar_wait_bounded(&sm.afull, iter & 1, A.err);
        const uint32_t a0 = smem_u32(sm.a[0]);
#pragma unroll 1
        for (uint32_t sub = 0; sub < nsub && ok; ++sub) {
          const uint32_t gs = g + sub;
          const int st = gs % BS;
          if (!mbar_wait_bounded(&sm.full[st], (gs / BS) & 1, A.err)) break;
          const uint32_t b0 = smem_u32(sm.b[st]);
#pragma unroll 1
          for (int half = 0; half < (both ? 2 : 1); ++half, ++v) {
            const uint32_t ab = v % B_ACCS;
            if (v >= B_ACCS && !mbar_wait_bounded(&sm.accempty[ab], (v / B_ACCS - 1) & 1, A.err)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t d = tmem + ab * BR, ah = a0 + half * TA;
#pragma unroll
            for (int kk = 0; kk < F::MMAS; ++kk) {
              const uint64_t da = umma_desc(ah + kk * 2 * (BM / 8) * 128, (BM / 8) * 128, 128);
              const uint64_t db = umma_desc(b0 + kk * 2 * (BR / 8) * 128, (BR / 8) * 128, 128);
              umma<F>(d, da, db, kk > 0);
            }
            umma_commit(&sm.accfull[ab]);  // the accumulator is ready for the epilogue
          }
          if (!ok) break;
          umma_commit(&sm.empty[st]);  // the row block may be overwritten once these MMAs finish
          ++done;
        }
        // no MMA of this item is in flight when the next item (or the dealloc) comes
        if (v > u) mbar_wait_bounded(&sm.accfull[(v - 1) % B_ACCS], ((v - 1) / B_ACCS) & 1, A.err);
        if (done != nsub) gave_up = true;
      }
      __syncwarp();
    } else {
      // ------------------------------------------------ epilogue: lane = query = TMEM lane
      const int c0 = warp / 4 * BP;  // its columns
      const int row = tid & (BM - 1);
      const bool pilot = A.stride > 1;
      if (tid < (both ? BQ : BM)) {
        uint32_t s = 0, e = 0;
        const int32_t qi = lane_query(A.ls, tl, it.tile, tid, s, e);
        float T = -INFINITY;
        if (qi >= 0) {
          T = sortable_f32(ld_volatile_u32(A.T_global + qi));
          if (ld_volatile_u32(A.ovf + qi)) T = -INFINITY;
        }
        float2 qs = A.lane_qs[it.tile * BQ + tid];
        qs.y *= -2.f;
        sm.lq[tid] = qi;
        sm.thr[tid] = T;
        sm.qs[tid] = qs;
        // In the pilot a slab keeps the best of every BP, 32 or 8 of its sampled
        // rows, or every row, as its length leaves enough of them for the rank:
        // what has no seed pushes rows by the hundred in the main pass.  (2,000
        // queries over slabs of 20,000 rows, k' = 400: 3.88 ms with maxima of 32
        // at least, 0.68 so; 8,000 rows, k' = 200: 1.59 and 0.61.  10,000 queries
        // over a skewed base of 3e5 rows: screens 2.17 and 1.69 ms, 5.46 and 2.98
        // at k' = 400.  4,096 over 2e6, few such slabs: 2.11 and 2.15.  Maxima of
        // 32 from 1.0 or 2.5 to a rank on: 20.1 to 21.3 and 19.8 ms of screens
        // over 1e6 rows at k' = 400, but 2.24 for the 4,096.)
        const uint32_t sampled = (e - s) / A.stride, rank = exact_seed_rank(A.kseed, 1, A.stride);
        sm.q[tid] = make_float4(acc_bound(T, qs), __uint_as_float(s), __uint_as_float(e),
                                (float)(sampled / BP >= 4 * rank         ? BP
                                        : sampled / 32 >= rank * 8 / 5   ? 32
                                        : sampled / 8 >= rank + rank / 5 ? 8
                                                                         : 1));
      }
      asm volatile("bar.sync 1, %0;" ::"n"(B_EPI * 32) : "memory");
      Candidate *const work = A.work + (uint64_t)blockIdx.x * A.halves * B_LISTS * A.capb;
      auto &wsm = sm.w[warp];
      const uint32_t lt = (1u << lane) - 1u;
      int cnt0 = 0, cnt1 = 0;  // entries of this thread's lists
      bool ok = !aborted;
      uint32_t until_refresh = A.refresh;  // row blocks between reads of the shared bound
      for (uint32_t v = 0; v < nprod && ok; ++v) {
        const uint32_t ab = (u + v) % B_ACCS, sub = both ? v / 2 : v;
        const int half = both ? (int)(v & 1) : 0, L = half * BM + row;
        const float4 q = sm.q[L];
        const uint32_t s = __float_as_uint(q.y), e = __float_as_uint(q.z);
        const uint32_t p0 = (it.blk0 + sub * A.stride) * BR;
        const int r0 = (int)min(max(s, p0), p0 + BR) - (int)p0;
        const int r1 = (int)min(max(e, p0), p0 + BR) - (int)p0;
        const float bound = r0 < r1 ? q.x : INFINITY;
        // warp-uniform: the lanes' timers may disagree at the deadline
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(&sm.accfull[ab], ((u + v) / B_ACCS) & 1, A.err))) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t tb = tmem + ((uint32_t)((warp & 3) * 32) << 16) + ab * BR + c0;
        // A chunk of 32 columns whose maximum reaches the bound holds a
        // candidate, or a row outside the slab that raises it (the appends look
        // closer).  Two chunks are in registers at a time; all four at once
        // measured the same.
        int cnt = half ? cnt1 : cnt0;
        const float2 qs = sm.qs[L];
        bool any = pilot;
        const bool fine = pilot && __any_sync(0xffffffffu, q.w <= 32.f);
        float best = -INFINITY;
#pragma unroll 1
        for (int c = 0; c < BP; c += 64) {
          uint32_t ra[32], rb[32];
          tmem_ld32_issue(tb + c, ra);
          tmem_ld32_issue(tb + c + 32, rb);
          tmem_wait_ld(ra);
          tmem_wait_ld(rb);
          if (c == BP - 64) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive1(&sm.accempty[ab]);
          }
          float ga[4], gb[4];
          const float ma = max32(ra, ga), mb = max32(rb, gb);
          best = fmax3(best, ma, mb);
          if (pilot && !fine) continue;
          uint32_t todo = (ma >= bound ? 1u : 0u) | (mb >= bound ? 2u : 0u);
          if (!__any_sync(0xffffffffu, todo != 0)) continue;
          any = true;
          Candidate *const lists = work + (half * B_LISTS + warp * 32) * A.capb;
          const int col0 = c0 + c;
          if (pilot && q.w > 1.f) {
            Candidate *const mine = lists + lane * A.capb;
            if (q.w == 32.f) {
              if ((todo & 1u) && col0 >= r0 && col0 + 32 <= r1) mine[cnt++] = {fmaf(qs.y, ma, qs.x), p0 + col0};
              if ((todo & 2u) && col0 + 32 >= r0 && col0 + 64 <= r1) mine[cnt++] = {fmaf(qs.y, mb, qs.x), p0 + col0 + 32};
            } else if (q.w == 8.f) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const float m = j < 4 ? ga[j] : gb[j - 4];
                const int c8 = col0 + 8 * j;
                if (m >= bound && c8 >= r0 && c8 + 8 <= r1) mine[cnt++] = {fmaf(qs.y, m, qs.x), p0 + c8};
              }
            }
            todo = 0;
          }
          // One that passes on its own, as in most chunks: it is the maximum,
          // and its lane appends it by itself if it is inside the slab.  The
          // rest are staged in shared memory and appended by the warp.
          if (todo & 1u) {
            const uint32_t all = ge_mask32(ra, ga, bound), in = all & range_mask(r0 - col0, r1 - col0);
            if (in == 0 || (all & (all - 1)) == 0) todo ^= 1u;
            if (in && !(todo & 1u)) lists[lane * A.capb + cnt++] = {fmaf(qs.y, ma, qs.x), p0 + col0 + __ffs(in) - 1};
          }
          if (todo & 2u) {
            const uint32_t all = ge_mask32(rb, gb, bound), in = all & range_mask(r0 - col0 - 32, r1 - col0 - 32);
            if (in == 0 || (all & (all - 1)) == 0) todo ^= 2u;
            if (in && !(todo & 2u)) lists[lane * A.capb + cnt++] = {fmaf(qs.y, mb, qs.x), p0 + col0 + 31 + __ffs(in)};
          }
          while (__any_sync(0xffffffffu, todo != 0)) {
            // staged in shared memory, in order of chunk, then lane
            const uint32_t ba = __ballot_sync(0xffffffffu, todo & 1u), bb = __ballot_sync(0xffffffffu, todo & 2u);
            const int ia = __popc(ba & lt), ib = __popc(ba) + __popc(bb & lt);
            const uint32_t pack = pack_query(r0, r1, lane, col0);
            if ((todo & 1u) && ia < B_SLOTS) stage32(wsm.row[ia], ra, bound, qs.y, qs.x, pack), todo ^= 1u;
            if ((todo & 2u) && ib < B_SLOTS) stage32(wsm.row[ib], rb, bound, qs.y, qs.x, pack + (1u << 23)), todo ^= 2u;
            const int ns = min(__popc(ba) + __popc(bb), B_SLOTS);
            __syncwarp();
            // and appended: a column per lane, two lanes' chunks at a time
            constexpr int W = 2;
#pragma unroll 1
            for (int i = 0; i < ns; i += W) {
              float ds[W];
              uint32_t m[W], col[W];
              int src[W];
              bool pass[W];
#pragma unroll
              for (int j = 0; j < W; ++j) {
                const float *x = wsm.row[min(i + j, ns - 1)];
                const float val = x[lane];
                const float4 t = *reinterpret_cast<const float4 *>(x + 32);
                const uint32_t pk = __float_as_uint(t.w);
                col[j] = (pk >> 23) * 32 + lane;
                src[j] = (pk >> 18) & 31;
                pass[j] = i + j < ns && val >= t.x && col[j] >= (pk & 511) && col[j] < (pk >> 9 & 511);
                ds[j] = fmaf(t.y, val, t.z);
              }
#pragma unroll
              for (int j = 0; j < W; ++j) m[j] = __ballot_sync(0xffffffffu, pass[j]);
#pragma unroll
              for (int j = 0; j < W; ++j) {
                const int n = __shfl_sync(0xffffffffu, cnt, src[j]);
                if (pass[j]) lists[src[j] * A.capb + n + __popc(m[j] & lt)] = {ds[j], p0 + col[j]};
                if (lane == src[j]) cnt += __popc(m[j]);
              }
            }
            __syncwarp();  // the rows are free again
          }
        }
        if (any) {
          if (pilot && q.w == (float)BP && best >= bound && c0 >= r0 && c0 + BP <= r1)
            work[(half * B_LISTS + tid) * A.capb + cnt++] = {fmaf(qs.y, best, qs.x), p0 + c0};
          Candidate *const lists = work + (half * B_LISTS + warp * 32) * A.capb;
          // lists that could overflow next are trimmed (a product adds at most BP)
          uint32_t msk = __ballot_sync(0xffffffffu, cnt > (int)A.capb - BP);
#pragma unroll 1
          for (; msk; msk &= msk - 1) {
            const int b = __ffs(msk) - 1;
            const int n = b_trim<F, NPL>(lists + (uint64_t)b * A.capb, __shfl_sync(0xffffffffu, cnt, b), sm,
                                         half * BM + (warp & 3) * 32 + b, A.kprime, A.capb, A.T_global, A.ovf);
            if (lane == b) cnt = n;
          }
          if (half) cnt1 = cnt;
          else cnt0 = cnt;
        }
        // other items of the same query tighten the shared bound meanwhile
        // (every refresh-th row block of the item)
        if (A.refresh && half == (both ? 1 : 0) && --until_refresh == 0) {
          until_refresh = A.refresh;
#pragma unroll 1
          for (int i = tid; i < (both ? BQ : BM); i += B_EPI * 32) {
            const int32_t qi = sm.lq[i];
            if (qi < 0) continue;
            const float Tg = sortable_f32(ld_volatile_u32(A.T_global + qi));
            if (Tg < sm.thr[i]) {
              sm.thr[i] = Tg;
              sm.q[i].x = acc_bound(Tg, sm.qs[i]);
            }
          }
        }
      }
      if (!ok) {
        // this item's queries are answered by the exact scan
#pragma unroll 1
        for (int i = row; i < (both ? BQ : BM); i += BM)
          if (sm.lq[i] >= 0) A.ovf[sm.lq[i]] = 1u;
        cnt0 = cnt1 = 0;
        gave_up = true;
      }
      sm.cnt[0][tid] = cnt0;
      sm.cnt[1][tid] = cnt1;
      // every list of the item is complete (and visible)
      asm volatile("bar.sync 1, %0;" ::"n"(B_EPI * 32) : "memory");
      // a query's lists become the item's result
      const int per = (both ? BQ : BM) / B_EPI;
      const int q0 = warp * per, l0 = q0 % BM, hf = q0 / BM;  // its first query
      int n = 0;
      if (lane < per && sm.thr[q0 + lane] != -INFINITY)  // (marked: the exact scan answers it)
#pragma unroll 1
        for (int l = 0; l < B_LISTS; l += BM) n += sm.cnt[hf][l0 + lane + l];
      const uint64_t o0 = (uint64_t)item_id * BQ + q0;
#pragma unroll 1
      for (int b = 0; b < per; ++b) {
        const int nb = __shfl_sync(0xffffffffu, n, b);
        if (nb == 0) continue;
        Candidate *src = work + (uint64_t)(hf * B_LISTS + l0 + b) * A.capb, *dst = A.out + (o0 + b) * A.ocap;
        int *c = &sm.cnt[hf][l0 + b];
        if (nb > (int)A.ocap) {
          const int kept = b_select<F>(src, c, sm, q0 + b, A.kprime, A.capb, A.ocap, A.T_global, dst);
          if (lane == b) n = kept;
          continue;
        }
        int at = 0;
#pragma unroll 1
        for (int l = 0; l < B_LISTS; l += BM) {
          const uint2 *x = reinterpret_cast<const uint2 *>(src + (uint64_t)l * A.capb);
#pragma unroll 1
          for (int i = lane; i < c[l]; i += 32) reinterpret_cast<uint2 *>(dst)[at + i] = x[i];
          at += c[l];
        }
      }
      if (n > (int)A.ocap) {  // more ties than fit
        A.ovf[sm.lq[q0 + lane]] = 1u;
        n = 0;
      }
      if (lane < per) A.out_cnt[o0 + lane] = (uint32_t)n;
    }
    g += nsub;
    u += nprod;
    // double-buffered by item parity: a slow thread may still read the slot
    // of this barrier while thread 0 writes the one after
    if (tid == 0) sm.next[iter & 1] = atomicAdd(A.queue, 1u) + gridDim.x;
    tc_fence_before();
    // the item's shared state (queries, counts, bounds) is reused by the next
    aborted = __syncthreads_or(aborted || gave_up) != 0;
    tc_fence_after();
    slot = sm.next[iter & 1];
  }
  if (warp == B_MMA_WARP)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
}

// ------------------------------------------------------------ re-rank --

constexpr int RR_THREADS = 256;
constexpr int RR_CAP = 8192;        // screening candidates the large merge holds
constexpr int RR_CAP_SMALL = 1024;  // ... and the common one (8 blocks per SM)
constexpr int RR_LARGE_BLOCKS = 3;  // ... of the large one
constexpr int RR_KMAX = 1024;       // largest k'
constexpr int RR_ITEMS = 256;       // work items of a tile (the lists' offsets)

template <int CAP>
struct RerankSmem {
  float key[CAP];
  uint32_t val[CAP];
  uint64_t ekey[RR_KMAX];
  float qv[DIM];
  uint32_t cnt_prefix[RR_ITEMS + 1];
  uint32_t hist[256], red[4];
  int total, kept, ties;
};

struct MergeArgs {
  const uint32_t *big_q, *big_tile, *big_lane;
  const Tile *tiles;
  const uint32_t *item_slot;
  const Candidate *out;
  const uint32_t *out_cnt;
  const QueryDesc *desc;
  const float *q, *vecs;
  const uint32_t *perm_t, *perm_c, *ovf;
  uint32_t *ovf_list, *ovf_count;
  uint32_t k, kprime, capb;
  const uint32_t *seeded;
  uint32_t *ids;
  float *dists;
  uint32_t *n_f64;
  const uint32_t *nbig_d;  // device plan: the big-query count (NULL: the launch's nbig)
};

// One big query b (index into the plan's big-query arrays): gather its
// lists, keep the k' best screening distances, re-rank them in FP32.  Bound by
// latency: barriers and the gather of k' rows of 400 B (4,096 queries over 2e6
// rows, k' = 200: 0.70 ms with sorts of up to 8,192 candidates, 0.31 ms now).  A
// query with more than CAP candidates goes to `spill` (the large merge) or,
// from the large merge, to the exact scan.  Returns are block-uniform.
template <int CAP>
__device__ void merge_one(const MergeArgs &A, uint32_t b, RerankSmem<CAP> &sm, uint32_t *spill,
                          uint32_t *spill_count) {
  const uint32_t *big_tile = A.big_tile, *big_lane = A.big_lane, *item_slot = A.item_slot, *out_cnt = A.out_cnt;
  const Tile *tiles = A.tiles;
  const Candidate *out = A.out;
  const QueryDesc *desc = A.desc;
  const float *q = A.q, *vecs = A.vecs;
  const uint32_t *perm_t = A.perm_t, *perm_c = A.perm_c, *seeded = A.seeded;
  uint32_t *ovf_list = A.ovf_list, *ovf_count = A.ovf_count, *ids = A.ids, *n_f64 = A.n_f64;
  float *dists = A.dists;
  const uint32_t k = A.k, kprime = A.kprime, capb = A.capb;
  const int tid = threadIdx.x;
  const uint32_t qi = A.big_q[b];
  if (A.ovf[qi]) {
    if (tid == 0) ovf_list[atomicAdd(ovf_count, 1u)] = qi;
    return;
  }
  const Tile tl = tiles[big_tile[b]];
  const uint32_t L = big_lane[b];
  const uint32_t nitems = tl.item1 - tl.item0;
  const QueryDesc dsc = desc[qi];
  for (int d = tid; d < DIM; d += RR_THREADS) sm.qv[d] = q[(uint64_t)qi * DIM + d];
  // candidate counts of the query's items (a tile has at most a few dozen)
  // more items than prefix slots: the exact scan answers the query
  list_offsets(item_slot, tl.item0, nitems, out_cnt, L, BQ, sm.cnt_prefix, &sm.total, RR_ITEMS, RR_CAP + 1);
  if (tid == 0) sm.kept = sm.ties = 0;
  __syncthreads();
  const int M = sm.total;
  if (M > CAP && spill && M <= RR_CAP) {  // the large merge takes it
    if (tid == 0) spill[atomicAdd(spill_count, 1u)] = b;
    return;
  }
  // a pilot bound that kept fewer than k' rows was set too low: the exact
  // scan answers the query
  if (M > CAP || (seeded[qi] && M < (int)kprime)) {
    if (tid == 0) ovf_list[atomicAdd(ovf_count, 1u)] = qi;
    return;
  }
  // a warp copies a list at a time
  for (uint32_t i = tid / 32; i < nitems; i += RR_THREADS / 32) {
    const uint64_t item = item_slot ? item_slot[tl.item0 + i] : tl.item0 + i;
    const uint32_t base = sm.cnt_prefix[i];
    const uint32_t c = (i + 1 < nitems ? sm.cnt_prefix[i + 1] : (uint32_t)M) - base;
    const Candidate *src = out + (item * BQ + L) * capb;
    for (uint32_t j = tid & 31; j < c; j += 32) {
      const Candidate cd = src[j];
      sm.key[base + j] = cd.ds;
      sm.val[base + j] = cd.pos;
    }
  }
  __syncthreads();
  // FP32 re-rank of the k' best screened rows with the reference's arithmetic
  // (of those at the k'-th screening distance itself, the first ones of the order)
  const int C = min(M, (int)kprime);
  const uint32_t *perm = dsc.order == ORDER_TIME ? perm_t : perm_c;
  uint32_t kth = 0xffffffffu;
  if (M > C) kth = block_kth<RR_THREADS>(sm.key, M, (uint32_t)C, sm.hist, sm.red);
  for (int i = tid; i < M; i += RR_THREADS) {
    const uint32_t u = f32_sortable(sm.key[i]);
    if (u < kth || M == C) sm.ekey[atomicAdd(&sm.kept, 1)] = sm.val[i];
    else if (u == kth) atomicAdd(&sm.ties, 1);
  }
  __syncthreads();
  if (M > C) {
    const int below = sm.kept;
    const bool fit = below + sm.ties == C;  // as a rule the k'-th alone: no walk over all M by its one thread
    const float tie = sortable_f32(kth);
    __syncthreads();
    for (int i = tid; i < M; i += RR_THREADS)
      if (f32_sortable(sm.key[i]) == kth) {
        if (fit) {
          sm.ekey[atomicAdd(&sm.kept, 1)] = sm.val[i];
          continue;
        }
        int at = below;
        for (int j = 0; j < M; ++j) at += sm.key[j] == tie && sm.val[j] < sm.val[i] ? 1 : 0;
        if (at < C) sm.ekey[at] = sm.val[i];
      }
    __syncthreads();
  }
  for (int i = tid; i < C; i += RR_THREADS) {
    const uint32_t id = perm[(uint32_t)sm.ekey[i]];
    sm.ekey[i] = exact_key(seq_l2_row(vecs + (uint64_t)id * DIM, sm.qv), id);
  }
  // order: a key's place is the number of smaller ones (they are distinct),
  // counted by its thread; above 2 keys a thread the sort is faster
  if (C <= 2 * RR_THREADS) {
    uint64_t e[2];
    int rank[2] = {0, 0};
    __syncthreads();
    e[0] = tid < C ? sm.ekey[tid] : ~0ull;
    e[1] = tid + RR_THREADS < C ? sm.ekey[tid + RR_THREADS] : ~0ull;
    for (int j = 0; j < C; ++j) {
      const uint64_t x = sm.ekey[j];
      rank[0] += x < e[0] ? 1 : 0;
      rank[1] += x < e[1] ? 1 : 0;
    }
    __syncthreads();
    if (tid < C) sm.ekey[rank[0]] = e[0];
    if (tid + RR_THREADS < C) sm.ekey[rank[1]] = e[1];
    __syncthreads();
  } else {
    int cp2 = 32;
    while (cp2 < C) cp2 <<= 1;
    for (int i = C + tid; i < cp2; i += RR_THREADS) sm.ekey[i] = ~0ull;
    __syncthreads();
    block_bitonic_sort(sm.ekey, cp2);
  }
  // FP64 at the k-th boundary: candidates within 1e-6 relative of the k-th
  // FP32 distance are ordered by their exact double distance
  if (tid == 0 && C > 0) {
    const int kk = min((int)k, C);
    const float D = sortable_f32((uint32_t)(sm.ekey[kk - 1] >> 32));
    const float lo = D - 1e-6f * D, hi = D + 1e-6f * D;
    int i0 = kk - 1, i1 = kk;
    while (i0 > 0 && sortable_f32((uint32_t)(sm.ekey[i0 - 1] >> 32)) >= lo) --i0;
    while (i1 < C && sortable_f32((uint32_t)(sm.ekey[i1] >> 32)) <= hi) ++i1;
    if (i1 - i0 > 1) {
      double d64[64];
      const int nb = min(i1 - i0, 64);
      for (int j = 0; j < nb; ++j) {
        const uint32_t id = (uint32_t)sm.ekey[i0 + j];
        const float *x = vecs + (uint64_t)id * DIM;
        double s = 0.0;
        for (int d = 0; d < DIM; ++d) {
          const double t = (double)x[d] - (double)sm.qv[d];
          s += t * t;
        }
        d64[j] = s;
      }
      for (int a = 1; a < nb; ++a) {  // insertion sort by (d64, id)
        const double dv = d64[a];
        const uint64_t kv = sm.ekey[i0 + a];
        int b = a - 1;
        while (b >= 0 && (d64[b] > dv || (d64[b] == dv && (uint32_t)sm.ekey[i0 + b] > (uint32_t)kv))) {
          d64[b + 1] = d64[b];
          sm.ekey[i0 + b + 1] = sm.ekey[i0 + b];
          --b;
        }
        d64[b + 1] = dv;
        sm.ekey[i0 + b + 1] = kv;
      }
      atomicAdd(n_f64, (uint32_t)nb);
    }
  }
  __syncthreads();
  for (uint32_t j = tid; j < k; j += RR_THREADS) {
    uint32_t id = 0xffffffffu;
    float d = INFINITY;
    if ((int)j < C) {
      id = (uint32_t)sm.ekey[j];
      d = sortable_f32((uint32_t)(sm.ekey[j] >> 32));
    }
    ids[(uint64_t)qi * k + j] = id;
    if (dists) dists[(uint64_t)qi * k + j] = d;
  }
}

// work == nullptr: block b merges big query b (grid = number of big
// queries); else the blocks stride over the *work_count entries of work.
template <int CAP>
__global__ void __launch_bounds__(RR_THREADS)
    k_merge_rerank(MergeArgs A, uint32_t nbig, const uint32_t *__restrict__ work,
                   const uint32_t *__restrict__ work_count, uint32_t *__restrict__ spill,
                   uint32_t *__restrict__ spill_count) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  RerankSmem<CAP> &sm = *reinterpret_cast<RerankSmem<CAP> *>(smem_raw);
  const uint32_t nwork = work ? *work_count : (A.nbig_d ? *A.nbig_d : nbig);
  for (uint32_t w = blockIdx.x; w < nwork; w += gridDim.x) {
    merge_one<CAP>(A, work ? work[w] : w, sm, spill, spill_count);
    __syncthreads();  // shared memory is reused by the next query
  }
}

struct SeedBound {
  __device__ float operator()(float ds, const QueryDesc &) const { return ds; }
};

// A search's per-query state and counters, in one buffer of words: the bounds
// (filled with +inf), what starts at zero, and the lists.
struct TcState {
  uint32_t *T_global, *T_pilot;                    // nq each, adjacent
  uint32_t *ovf, *ovf_pilot, *seeded;              // nq each, adjacent, before the counters
  uint32_t *ovf_count, *n_f64, *spill_count, *queue;  // queue: pilot, main
  uint32_t *ovf_list, *spill;                      // nq each
  static size_t bytes(uint32_t nq) { return ((size_t)nq * 7 + 16) * 4; }
  TcState(uint32_t *d, uint32_t nq) {
    T_global = d;
    T_pilot = T_global + nq;
    ovf = T_pilot + nq;
    ovf_pilot = ovf + nq;
    seeded = ovf_pilot + nq;
    ovf_count = seeded + nq;
    n_f64 = ovf_count + 1;
    spill_count = ovf_count + 2;
    queue = ovf_count + 4;
    ovf_list = ovf_count + 16;
    spill = ovf_list + nq;
  }
  int reset(uint32_t nq, cudaStream_t st) const {
    int rc;
    if ((rc = launch_fill_u32(T_global, nq * 2, f32_sortable(INFINITY), st))) return rc;
    FKNN_CUDA(cudaMemsetAsync(ovf, 0, ((size_t)nq * 3 + 16) * 4, st));
    return FKNN_OK;
  }
};

// Work items of a plan.  Several per SM even out tiles of unequal length; with
// few queries there are few tiles, cut alike, and every further item only adds
// its own start, end and lists (100 queries over 1e6 rows: 0.46 ms at one item
// per SM, 0.54 at four; 5,000 over 1e5 rows 1.50 and 1.06).
inline uint32_t target_items(const fknn_index *idx, const fknn_tuning &tune, int mode, uint32_t nq) {
  return (uint32_t)idx->num_sms * items_per_sm(tune, mode, nq);
}

// Work items a tile may have: what the merge holds of their lists, and the
// scratch (8 GB).  Behind a seeded bound all of a query's lists together hold
// 3 k' entries or so, and a query too short to be seeded meets few items.
inline uint32_t max_items(uint64_t per_item, uint64_t tiles) {
  return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(RR_ITEMS, (8ull << 30) / (per_item * tiles)));
}

// The pilot's stride.  There is always a pilot: a screen without one pushes
// rows by the hundred before it has a bound, which costs this epilogue more
// than the pilot does (1,000 queries over 1e6 rows, k' = 200: screens of 5.7 ms
// without, 0.7 with it; 20,000 queries 13.9 and 6.0).
inline uint32_t pilot_stride(const fknn_tuning &tune, const fknn_tuning &dflt) {
  return tune.pilot_stride > 1 ? tune.pilot_stride : dflt.pilot_stride;
}

// Entries of a query in an item's result when memory is short: k' and a few
// ties, which a select makes of the working lists.
inline uint32_t tight_cap(uint32_t kprime, uint32_t capb) { return std::min(capb, (kprime + 64 + 31) / 32 * 32); }

// Scratch of the lists: nitems results of BQ queries, and working lists for
// every CTA.  Where the index's HBM budget or the memory left does not hold
// that, the caller plans again with one item per tile, and here as many CTAs
// as fit (tight).
inline int list_scratch(fknn_index *idx, uint32_t nitems, uint32_t halves, uint32_t capb, uint32_t ocap, bool tight,
                        Candidate **out, uint32_t **cnt, Candidate **work, uint32_t *grid) {
  int rc = ws_get(idx, 6, (size_t)nitems * BQ * ocap * sizeof(Candidate), (void **)out);
  if (!rc) rc = ws_get(idx, 7, (size_t)nitems * BQ * 4, (void **)cnt);
  if (!rc)
    for (*grid = std::min<uint32_t>(nitems, (uint32_t)idx->num_sms);; *grid = (*grid + 1) / 2) {
      rc = ws_get(idx, 11, (size_t)*grid * halves * B_LISTS * capb * sizeof(Candidate), (void **)work);
      if (rc != FKNN_ENOMEM || !tight || *grid == 1) break;
      cudaGetLastError();
    }
  return rc;
}

// What a tight plan does without is given back (slot 4: the exact path's lists).
inline void drop_lists(fknn_index *idx) {
  cudaGetLastError();  // (a refused allocation is not this call's error)
  for (int slot : {4, 6, 7, 11}) ws_drop(idx, slot);
}

// the trim holds a whole list in registers: 32 x NPL >= capb
template <class F>
static void (*screen_kernel(uint32_t capb))(ScreenArgs) {
  return capb <= 384 ? k_screen_tc<F, 12> : capb <= 512 ? k_screen_tc<F, 16> : capb <= 768 ? k_screen_tc<F, 24>
       : capb <= 1024 ? k_screen_tc<F, 32> : k_screen_tc<F, 40>;
}

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace

int build_bf16(fknn_index *idx, cudaStream_t st) {
  const uint64_t nblk = (idx->n + BR - 1) / BR;
  for (int o = 0; o < 2; ++o) {
    int rc = dev_alloc(idx, &idx->bf16_blocks[o], nblk * Tiles<FmtBF16>::B);
    if (rc) return rc;
    k_build_bf16_blocks<<<(unsigned)nblk, 256, 0, st>>>(idx->vecs, idx->norms, idx->ord[o].perm, idx->n,
                                                        (__nv_bfloat16 *)idx->bf16_blocks[o]);
    g_launches += 1;
  }
  FKNN_CUDA(cudaGetLastError());
  return FKNN_OK;
}

int build_fp8(fknn_index *idx, cudaStream_t st) {
  const uint64_t nblk = (idx->n + BR - 1) / BR;
  int rc = dev_alloc(idx, (void **)&idx->fp8_scale, 2 * DIM * sizeof(float));  // centre[100], scale[100]
  if (rc) return rc;
  uint32_t *mm;
  if ((rc = ws_get(idx, 15, 2 * DIM * sizeof(uint32_t), (void **)&mm))) return rc;
  FKNN_CUDA(cudaMemsetAsync(mm, 0xff, DIM * sizeof(uint32_t), st));
  FKNN_CUDA(cudaMemsetAsync(mm + DIM, 0, DIM * sizeof(uint32_t), st));
  k_dim_minmax<<<148 * 4, 256, 0, st>>>(idx->vecs, idx->n, mm, mm + DIM);
  k_fp8_params<<<1, 128, 0, st>>>(mm, mm + DIM, idx->fp8_scale, idx->fp8_scale + DIM);
  g_launches += 2;
  for (int o = 0; o < 2; ++o) {
    if ((rc = dev_alloc(idx, &idx->fp8_blocks[o], nblk * Tiles<FmtFP8>::B))) return rc;
    k_build_fp8_blocks<<<(unsigned)nblk, 256, 0, st>>>(idx->vecs, idx->ord[o].perm, idx->n, idx->fp8_scale,
                                                       idx->fp8_scale + DIM, (unsigned char *)idx->fp8_blocks[o]);
    g_launches += 1;
  }
  FKNN_CUDA(cudaGetLastError());
  return FKNN_OK;
}

// The pilot, its seeds and the screen proper.  The pilot keeps the best of
// every 128, 32 or 8 rows of every stride-th row block: as the few rows that
// matter lie in different groups as a rule, the r-th best of these is little
// above the r-th of the sample's rows (and never below it), at a fraction of the
// entries.  Where even that leaves too few for the rank it keeps every row.
template <class K>
static void launch_screens(K screen, ScreenArgs X, SeedArgs Z, const TcState &S, uint32_t kprime, uint32_t stride,
                           uint32_t refresh, bool withhold, uint32_t grid, uint32_t nbig_max, size_t smem,
                           cudaStream_t st) {
  X.T_global = S.T_pilot;
  X.ovf = S.ovf_pilot;
  // (the sample of a short slab is up to twice its nominal share)
  X.kprime = exact_seed_rank(kprime, 2, stride);
  X.kseed = kprime;
  X.refresh = 0;
  X.stride = stride;
  X.withhold = 0;
  X.queue = S.queue;
  screen<<<grid, B_THREADS, smem, st>>>(X);
  Z.tiles = X.tiles;
  Z.items = X.items;
  Z.out = X.out;
  Z.out_cnt = X.out_cnt;
  Z.tq = BQ;
  Z.list_cap = X.ocap;
  Z.blk_rows = BR;
  Z.stride = stride;
  Z.k = kprime;
  Z.T_global = S.T_global;
  Z.seeded = S.seeded;
  launch_screen_seed(Z, nbig_max, SeedBound(), st);
  g_launches += 1;
  X.T_global = S.T_global;
  X.ovf = S.ovf;
  X.kprime = kprime;
  X.refresh = (refresh + 1) / 2;  // (given in sub-tiles of 128 rows)
  X.stride = 1;
  X.withhold = withhold ? 1u : 0u;
  X.queue = S.queue + 1;
  screen<<<grid, B_THREADS, smem, st>>>(X);
  g_launches += 1;
}

template <class F>
static int search_tc(fknn_index *idx, const float *d_q, const float *d_meta, uint32_t nq, uint32_t k, uint32_t kprime,
                     uint32_t *d_ids, float *d_dists, cudaStream_t st, fknn_search_stats *stats) {
  const uint64_t n = idx->n;
  constexpr uint32_t TA = Tiles<F>::A;
  int rc;
  QueryDesc *d_desc, *h_desc;
  float *h_meta;
  if ((rc = prepare_queries(idx, d_q, d_meta, nq, st, &d_desc, &h_desc, &h_meta))) return rc;
  uint32_t nsmall_early = 0;
  if ((rc = launch_small_scans(idx, h_desc, d_desc, nq, d_q, k, d_ids, d_dists, st, &nsmall_early))) return rc;
  constexpr int mode = F::kFP8 ? FKNN_MODE_FP8_RERANK : FKNN_MODE_BF16_RERANK;
  const fknn_tuning tune = idx->tuning[mode];
  // candidate slots per (item, query): k' plus the pushes between trims; a
  // list holds at most 1280 (32 lanes x 40 registers in the trim)
  const uint32_t capb =
      (uint32_t)std::min<size_t>(1280, align_up(kprime + std::max<uint32_t>(tune.list_slack, 2 * BP), 128));
  auto t0 = std::chrono::steady_clock::now();
  Plan &P = idx->plan;
  PlanShape shape;
  shape.tq = BQ;
  shape.blk_rows = BR;
  shape.small_slab = SMALL_SLAB;
  shape.min_chunk_blocks = (tune.min_chunk_blocks + 1) / 2;  // (given in 128-row blocks)
  const uint64_t tiles_est = std::max<uint64_t>(1, (nq + BQ - 1) / BQ);
  Candidate *d_out = nullptr, *d_work = nullptr;
  uint32_t *d_ocnt = nullptr, *d_state, nitems = 0, sgrid = 0, ocap = capb, halves = 1;
  unsigned char *d_at = nullptr, *d_blob;
  float2 *d_lqs = nullptr;
  if ((rc = ws_get(idx, 5, TcState::bytes(nq), (void **)&d_state))) return rc;
  for (int tight = 0;; ++tight) {
    // results (items x 256 x ocap x 8 B) stay within ~8 GB
    ocap = tight ? tight_cap(kprime, capb) : capb;
    const uint64_t per_item = (uint64_t)BQ * ocap * sizeof(Candidate);
    shape.max_items_per_tile = tight ? 1u : max_items(per_item, tiles_est);
    shape.target_items = tight ? 1u : target_items(idx, tune, mode, nq);
    make_plan(h_desc, h_meta, nq, n, shape, P);
    nitems = (uint32_t)P.items.size();
    for (const Tile &t : P.tiles)
      if (t.nq > (uint32_t)BM) halves = 2;
    if (!nitems) break;
    // (the lists last: when tight, they take what is left)
    rc = ws_get(idx, 3, plan_blob_bytes(P), (void **)&d_blob);
    if (!rc) rc = ws_get(idx, 4, P.tiles.size() * 2 * TA, (void **)&d_at);
    if (!rc) rc = ws_get(idx, 10, P.tiles.size() * BQ * sizeof(float2), (void **)&d_lqs);
    if (!rc) rc = list_scratch(idx, nitems, halves, capb, ocap, tight, &d_out, &d_ocnt, &d_work, &sgrid);
    if (!rc) break;
    if (rc != FKNN_ENOMEM || tight) return rc;
    drop_lists(idx);
  }
  auto t1 = std::chrono::steady_clock::now();
  const uint32_t ntile = (uint32_t)P.tiles.size();
  const uint32_t nbig = (uint32_t)P.big.size(), nsmall = (uint32_t)P.small.size();
  std::vector<uint32_t> &slot = P.w_slot;
  slot.resize(nitems);
  {
    std::vector<uint32_t> &fill = P.w_fill;
    fill.resize(ntile);
    for (uint32_t t = 0; t < ntile; ++t) fill[t] = P.tiles[t].item0;
    for (uint32_t s = 0; s < nitems; ++s) slot[fill[P.items[s].tile]++] = s;
  }
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t o = off;
    off = align_up(off + bytes, 256);
    return o;
  };
  const size_t o_small = take(nsmall * 4), o_big = take(nbig * 4), o_btile = take(nbig * 4),
               o_blane = take(nbig * 4), o_tiles = take(ntile * sizeof(Tile)),
               o_items = take(nitems * sizeof(WorkItem)), o_lq = take((size_t)ntile * BQ * 4),
               o_ls = take((size_t)ntile * BQ * 4), o_le = take((size_t)ntile * BQ * 4), o_slot = take(nitems * 4);
  const size_t blob = off;
  unsigned char *h_blob;
  if ((rc = hs_get(idx, 3, blob + 256, (void **)&h_blob))) return rc;
  if ((rc = ws_get(idx, 3, blob + 256, (void **)&d_blob))) return rc;
  auto put = [&](size_t o, const void *src, size_t bytes) {
    if (bytes) std::memcpy(h_blob + o, src, bytes);
  };
  put(o_small, P.small.data(), nsmall * 4);
  put(o_big, P.big.data(), nbig * 4);
  put(o_btile, P.big_tile.data(), nbig * 4);
  put(o_blane, P.big_lane.data(), nbig * 4);
  put(o_tiles, P.tiles.data(), ntile * sizeof(Tile));
  put(o_items, P.items.data(), nitems * sizeof(WorkItem));
  put(o_lq, P.lane_q.data(), (size_t)ntile * BQ * 4);
  put(o_ls, P.lane_s.data(), (size_t)ntile * BQ * 4);
  put(o_le, P.lane_e.data(), (size_t)ntile * BQ * 4);
  put(o_slot, slot.data(), nitems * 4);
  if (blob) FKNN_CUDA(cudaMemcpyAsync(d_blob, h_blob, blob, cudaMemcpyHostToDevice, st));
  const TcState S(d_state, nq);
  if ((rc = S.reset(nq, st))) return rc;
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
  if (stats)
    for (auto &e : ev) FKNN_CUDA(cudaEventCreate(&e));
  const OrderData &OT = idx->ord[ORDER_TIME], &OC = idx->ord[ORDER_CAT];
  if (nitems) {
    LaneSrc ls;
    ls.lane_q = (const int32_t *)(d_blob + o_lq);
    ls.lane_s = (const uint32_t *)(d_blob + o_ls);
    ls.lane_e = (const uint32_t *)(d_blob + o_le);
    if constexpr (F::kFP8)
      k_tile_stage_fp8<<<ntile, 256, 0, st>>>(d_q, ls, (const Tile *)(d_blob + o_tiles), ntile, idx->fp8_scale,
                                              idx->fp8_scale + DIM, d_at, d_lqs);
    else
      k_tile_stage_bf16<<<ntile, 256, 0, st>>>(d_q, ls, (const Tile *)(d_blob + o_tiles), ntile, d_desc,
                                               (__nv_bfloat16 *)d_at, d_lqs);
    // per device context, so set on every call (cheap)
    auto screen = screen_kernel<F>(capb);
    FKNN_CUDA(cudaFuncSetAttribute(screen, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(BScreenSmem<F>)));
    FKNN_CUDA(cudaFuncSetAttribute(k_merge_rerank<RR_CAP_SMALL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(RerankSmem<RR_CAP_SMALL>)));
    FKNN_CUDA(cudaFuncSetAttribute(k_merge_rerank<RR_CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(RerankSmem<RR_CAP>)));
    if (stats) FKNN_CUDA(cudaEventRecord(ev[0], st));
    void *const *blocks = F::kFP8 ? idx->fp8_blocks : idx->bf16_blocks;
    const uint32_t stride = pilot_stride(tune, DEFAULT_TUNING[mode]);
    ScreenArgs X;
    X.items = (const WorkItem *)(d_blob + o_items);
    X.tiles = (const Tile *)(d_blob + o_tiles);
    X.atiles = d_at;
    X.ls = ls;
    X.lane_qs = d_lqs;
    X.blocks_t = (const unsigned char *)blocks[ORDER_TIME];
    X.blocks_c = (const unsigned char *)blocks[ORDER_CAT];
    X.out = d_out;
    X.out_cnt = d_ocnt;
    X.work = d_work;
    X.capb = capb;
    X.ocap = ocap;
    X.halves = halves;
    X.nitems = nitems;
    X.nitems_d = nullptr;
    X.order = nullptr;
    X.err = idx->d_flag;
    SeedArgs Z;
    Z.big_q = (const uint32_t *)(d_blob + o_big);
    Z.big_tile = (const uint32_t *)(d_blob + o_btile);
    Z.big_lane = (const uint32_t *)(d_blob + o_blane);
    Z.nbig = nbig;
    Z.nbig_d = nullptr;
    Z.item_slot = (const uint32_t *)(d_blob + o_slot);
    Z.desc = d_desc;
    launch_screens(screen, X, Z, S, kprime, stride, tune.bound_refresh, idx->test_withhold, sgrid, nbig,
                   sizeof(BScreenSmem<F>), st);
    idx->test_withhold = false;
    if (stats) FKNN_CUDA(cudaEventRecord(ev[1], st));
    MergeArgs A;
    A.big_q = (const uint32_t *)(d_blob + o_big);
    A.big_tile = (const uint32_t *)(d_blob + o_btile);
    A.big_lane = (const uint32_t *)(d_blob + o_blane);
    A.tiles = (const Tile *)(d_blob + o_tiles);
    A.item_slot = (const uint32_t *)(d_blob + o_slot);
    A.out = d_out;
    A.out_cnt = d_ocnt;
    A.desc = d_desc;
    A.q = d_q;
    A.vecs = idx->vecs;
    A.perm_t = OT.perm;
    A.perm_c = OC.perm;
    A.ovf = S.ovf;
    A.ovf_list = S.ovf_list;
    A.ovf_count = S.ovf_count;
    A.k = k;
    A.kprime = kprime;
    A.capb = ocap;
    A.seeded = S.seeded;
    A.ids = d_ids;
    A.dists = d_dists;
    A.n_f64 = S.n_f64;
    A.nbig_d = nullptr;
    // queries with more candidates than the common merge holds go to the large one
    k_merge_rerank<RR_CAP_SMALL><<<nbig, RR_THREADS, sizeof(RerankSmem<RR_CAP_SMALL>), st>>>(
        A, nbig, nullptr, nullptr, S.spill, S.spill_count);
    k_merge_rerank<RR_CAP><<<idx->num_sms * RR_LARGE_BLOCKS, RR_THREADS, sizeof(RerankSmem<RR_CAP>), st>>>(
        A, 0, S.spill, S.spill_count, nullptr, nullptr);
    g_launches += 3;
  }
  if (stats) FKNN_CUDA(cudaEventRecord(ev[2], st));
  if (nbig)
    if ((rc = launch_exact_scan(idx, S.ovf_list, S.ovf_count, 0, 0, d_desc, d_q, k, d_ids, d_dists, st))) return rc;
  if (nsmall_early && (rc = join_small_scans(idx, st))) return rc;
  FKNN_CUDA(cudaGetLastError());
  if (stats) {
    FKNN_CUDA(cudaEventRecord(ev[3], st));
    FKNN_CUDA(cudaEventSynchronize(ev[3]));
    float ms = 0.f;
    if (nitems) {
      FKNN_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[1]));
      stats->ms_screen = ms;
      FKNN_CUDA(cudaEventElapsedTime(&ms, ev[1], ev[2]));
      stats->ms_merge = ms;
    }
    FKNN_CUDA(cudaEventElapsedTime(&ms, ev[2], ev[3]));
    stats->ms_scan = ms;
    for (auto &e : ev) cudaEventDestroy(e);
    stats->pairs_screened = P.pairs_screened;
    stats->pairs_passing = P.pairs_passing;
    stats->pairs_contraction = P.pairs_contraction;
    stats->n_tiles = ntile;
    stats->n_work_items = nitems;
    stats->n_small = nsmall;
    stats->ms_plan = std::chrono::duration<float, std::milli>(t1 - t0).count();
    uint32_t h2[2] = {0, 0};
    FKNN_CUDA(cudaMemcpyAsync(h2, S.ovf_count, 8, cudaMemcpyDeviceToHost, st));
    FKNN_CUDA(cudaStreamSynchronize(st));
    stats->n_overflow = h2[0];
    stats->n_boundary_f64 = h2[1];
  }
  return FKNN_OK;
}

// The same search with the plan built on the device (device_plan.cu) and
// every launch of fixed size, captured once into a CUDA graph and replayed
// while nq, k, k', the tuning, the pointers and the scratch buffers stay
// the same.  Screens run persistent over the device item count; merges and
// scans read their counts from device memory.
template <class F>
static int search_tc_graph(fknn_index *idx, const float *d_q, const float *d_meta, uint32_t nq, uint32_t k,
                           uint32_t kprime, uint32_t *d_ids, float *d_dists, cudaStream_t st,
                           fknn_search_stats *stats) {
  constexpr uint32_t TA = Tiles<F>::A;
  int rc;
  constexpr int mode = F::kFP8 ? FKNN_MODE_FP8_RERANK : FKNN_MODE_BF16_RERANK;
  const fknn_tuning tune = idx->tuning[mode];
  const uint32_t capb =
      (uint32_t)std::min<size_t>(1280, align_up(kprime + std::max<uint32_t>(tune.list_slack, 2 * BP), 128));
  PlanShape shape;
  shape.tq = BQ;
  shape.blk_rows = BR;
  shape.small_slab = SMALL_SLAB;
  shape.min_chunk_blocks = (tune.min_chunk_blocks + 1) / 2;  // (given in 128-row blocks)
  // all buffers exist before the capture (a capture may not allocate)
  QueryDesc *d_desc;
  void *d_plan;
  unsigned char *d_at;
  float2 *d_lqs;
  Candidate *d_out, *d_work;
  uint32_t *d_ocnt, *d_state, sgrid, ocap;
  DevPlanSizes z;
  if ((rc = ws_get(idx, 2, (size_t)nq * sizeof(QueryDesc), (void **)&d_desc))) return rc;
  if ((rc = ws_get(idx, 5, TcState::bytes(nq), (void **)&d_state))) return rc;
  for (int tight = 0;; ++tight) {
    ocap = tight ? tight_cap(kprime, capb) : capb;
    shape.target_items = tight ? 1u : target_items(idx, tune, mode, nq);
    z = device_plan_sizes(idx, nq, shape);
    shape.max_items_per_tile =
        tight ? 1u : max_items((uint64_t)BQ * ocap * sizeof(Candidate), z.ntile_max);
    void *h;  // the radix sort's histogram slot at its largest: the plan sorts the queries and the work items
    const size_t keys = std::max<size_t>(nq, z.nitems_max);
    rc = ws_get(idx, 15, ((keys + 4095) / 4096) * 256 * sizeof(uint32_t) + 256, &h);
    if (!rc) rc = ws_get(idx, 19, device_plan_bytes(nq, z), &d_plan);
    if (!rc) rc = ws_get(idx, 4, (size_t)z.ntile_max * 2 * TA, (void **)&d_at);
    if (!rc) rc = ws_get(idx, 10, (size_t)z.ntile_max * BQ * sizeof(float2), (void **)&d_lqs);
    // (the lists last: when tight, they take what is left)
    if (!rc) rc = list_scratch(idx, z.nitems_max, 2, capb, ocap, tight, &d_out, &d_ocnt, &d_work, &sgrid);
    if (!rc) break;
    if (rc != FKNN_ENOMEM || tight) return rc;
    drop_lists(idx);
  }
  const TcState S(d_state, nq);
  const uint32_t stride = pilot_stride(tune, DEFAULT_TUNING[mode]);
  DevPlan P;
  device_plan_layout(P, d_plan, nq, z);
  auto screen = screen_kernel<F>(capb);
  FKNN_CUDA(cudaFuncSetAttribute(screen, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BScreenSmem<F>)));
  FKNN_CUDA(cudaFuncSetAttribute(k_merge_rerank<RR_CAP_SMALL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(RerankSmem<RR_CAP_SMALL>)));
  FKNN_CUDA(cudaFuncSetAttribute(k_merge_rerank<RR_CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(RerankSmem<RR_CAP>)));
  GraphCache &G = idx->graph;
  const bool withhold = idx->test_withhold;
  idx->test_withhold = false;
  const std::vector<uint64_t> key = {
      (uint64_t)F::kFP8, nq, k, kprime, capb, ocap, sgrid, shape.target_items, tune.list_slack,
      tune.items_per_sm, tune.min_chunk_blocks, tune.bound_refresh, stride, (uint64_t)withhold, (uint64_t)(uintptr_t)d_q, (uint64_t)(uintptr_t)d_meta,
      (uint64_t)(uintptr_t)d_ids, (uint64_t)(uintptr_t)d_dists, (uint64_t)(uintptr_t)d_desc,
      (uint64_t)(uintptr_t)d_plan, (uint64_t)(uintptr_t)d_at, (uint64_t)(uintptr_t)d_lqs, (uint64_t)(uintptr_t)d_out,
      (uint64_t)(uintptr_t)d_work,
      (uint64_t)(uintptr_t)d_ocnt, (uint64_t)(uintptr_t)d_state,
      (uint64_t)(uintptr_t)idx->ws[15].p};
  if (!G.exec || G.key != key) {
    G.release();
    for (auto &e : G.ev) FKNN_CUDA(cudaEventCreate(&e));
    if (!G.cap) FKNN_CUDA(cudaStreamCreateWithFlags(&G.cap, cudaStreamNonBlocking));
    if (!G.side) FKNN_CUDA(cudaStreamCreateWithFlags(&G.side, cudaStreamNonBlocking));
    if (!G.fork) FKNN_CUDA(cudaEventCreateWithFlags(&G.fork, cudaEventDisableTiming));
    if (!G.join) FKNN_CUDA(cudaEventCreateWithFlags(&G.join, cudaEventDisableTiming));
    const uint32_t l0 = g_launches;
    const cudaStream_t user_st = st;
    st = G.cap;  // captured nodes carry no stream: the replay goes to the caller's
    FKNN_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    // everything below is enqueued only; a failure ends the capture first
    auto body = [&]() -> int {
      int r;
      if ((r = enqueue_query_prep(idx, d_q, d_meta, nq, d_desc, st))) return r;
      if ((r = device_plan_build(idx, d_desc, d_meta, P, shape, st))) return r;
      // the short-slab exact scans need only the plan's list: a branch of
      // the graph beside the contraction (their rows of ids / dists are
      // disjoint from the merge's)
      FKNN_CUDA(cudaEventRecord(G.fork, st));
      FKNN_CUDA(cudaStreamWaitEvent(G.side, G.fork, 0));
      if ((r = launch_exact_scan(idx, P.small, P.cnt + DP_NSMALL, 0, nq / 4, d_desc, d_q, k, d_ids, d_dists,
                                 G.side)))
        return r;
      FKNN_CUDA(cudaEventRecord(G.join, G.side));
      if ((r = S.reset(nq, st))) return r;
      const OrderData &OT = idx->ord[ORDER_TIME], &OC = idx->ord[ORDER_CAT];
      LaneSrc ls;
      ls.tile_first = P.tile_first;
      ls.order_q = P.vals;
      ls.desc = d_desc;
      ls.ntile = P.cnt + DP_NTILE;
      const unsigned tgrid = std::min<uint32_t>(z.ntile_max, (uint32_t)idx->num_sms * 4);
      if constexpr (F::kFP8)
        k_tile_stage_fp8<<<tgrid, 256, 0, st>>>(d_q, ls, P.tiles, 0, idx->fp8_scale, idx->fp8_scale + DIM, d_at,
                                                d_lqs);
      else
        k_tile_stage_bf16<<<tgrid, 256, 0, st>>>(d_q, ls, P.tiles, 0, d_desc, (__nv_bfloat16 *)d_at, d_lqs);
      g_launches += 1;
      FKNN_CUDA(cudaEventRecordWithFlags(G.ev[0], st, cudaEventRecordExternal));  // an event node of the graph
      void *const *blocks = F::kFP8 ? idx->fp8_blocks : idx->bf16_blocks;
      ScreenArgs X;
      X.items = P.items;
      X.tiles = P.tiles;
      X.atiles = d_at;
      X.ls = ls;
      X.lane_qs = d_lqs;
      X.blocks_t = (const unsigned char *)blocks[ORDER_TIME];
      X.blocks_c = (const unsigned char *)blocks[ORDER_CAT];
      X.out = d_out;
      X.out_cnt = d_ocnt;
      X.work = d_work;
      X.capb = capb;
      X.ocap = ocap;
      X.halves = 2;
      X.nitems = 0;
      X.nitems_d = P.cnt + DP_NITEMS;
      X.order = P.ord_val;
      X.err = idx->d_flag;
      SeedArgs Z;
      Z.big_q = P.big_q;
      Z.big_tile = P.big_tile;
      Z.big_lane = P.big_lane;
      Z.nbig = 0;
      Z.nbig_d = P.cnt + DP_NBIG;
      Z.item_slot = nullptr;  // a tile's items are consecutive
      Z.desc = d_desc;
      launch_screens(screen, X, Z, S, kprime, stride, tune.bound_refresh, withhold, sgrid, nq, sizeof(BScreenSmem<F>),
                     st);
      FKNN_CUDA(cudaEventRecordWithFlags(G.ev[1], st, cudaEventRecordExternal));  // an event node of the graph
      MergeArgs A;
      A.big_q = P.big_q;
      A.big_tile = P.big_tile;
      A.big_lane = P.big_lane;
      A.tiles = P.tiles;
      A.item_slot = nullptr;  // a tile's items are consecutive
      A.out = d_out;
      A.out_cnt = d_ocnt;
      A.desc = d_desc;
      A.q = d_q;
      A.vecs = idx->vecs;
      A.perm_t = OT.perm;
      A.perm_c = OC.perm;
      A.ovf = S.ovf;
      A.ovf_list = S.ovf_list;
      A.ovf_count = S.ovf_count;
      A.k = k;
      A.kprime = kprime;
      A.capb = ocap;
      A.seeded = S.seeded;
      A.ids = d_ids;
      A.dists = d_dists;
      A.n_f64 = S.n_f64;
      A.nbig_d = P.cnt + DP_NBIG;
      k_merge_rerank<RR_CAP_SMALL><<<std::min<uint32_t>(nq, (uint32_t)idx->num_sms * 32), RR_THREADS,
                                     sizeof(RerankSmem<RR_CAP_SMALL>), st>>>(A, 0, nullptr, nullptr, S.spill,
                                                                             S.spill_count);
      k_merge_rerank<RR_CAP><<<idx->num_sms * RR_LARGE_BLOCKS, RR_THREADS, sizeof(RerankSmem<RR_CAP>), st>>>(
          A, 0, S.spill, S.spill_count, nullptr, nullptr);
      g_launches += 2;
      FKNN_CUDA(cudaEventRecordWithFlags(G.ev[2], st, cudaEventRecordExternal));  // an event node of the graph
      if ((r = launch_exact_scan(idx, S.ovf_list, S.ovf_count, 0, 0, d_desc, d_q, k, d_ids, d_dists, st))) return r;
      FKNN_CUDA(cudaStreamWaitEvent(st, G.join, 0));
      FKNN_CUDA(cudaEventRecordWithFlags(G.ev[3], st, cudaEventRecordExternal));  // an event node of the graph
      FKNN_CUDA(cudaGetLastError());
      return FKNN_OK;
    };
    const int brc = body();
    cudaGraph_t graph = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(st, &graph);
    st = user_st;
    if (brc || ce != cudaSuccess) {
      if (graph) cudaGraphDestroy(graph);
      G.release();
      cudaGetLastError();
      return brc ? brc : cuda_fail(ce, "cudaStreamEndCapture");
    }
    const cudaError_t ie = cudaGraphInstantiate(&G.exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) {
      G.exec = nullptr;
      G.release();
      return cuda_fail(ie, "cudaGraphInstantiate");
    }
    G.key = key;
    G.launches = g_launches - l0;
    st = user_st;
  }
  g_launches = G.launches;
  FKNN_CUDA(cudaGraphLaunch(G.exec, st));
  int flag = 0;
  FKNN_CUDA(cudaMemcpyAsync(&flag, idx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, st));
  FKNN_CUDA(cudaStreamSynchronize(st));
  if ((rc = check_query_flag_value(flag & ~ERR_WAIT_TIMEOUT))) return rc;
  if (stats) {
    float ms = 0.f;
    FKNN_CUDA(cudaEventElapsedTime(&ms, G.ev[0], G.ev[1]));
    stats->ms_screen = ms;
    FKNN_CUDA(cudaEventElapsedTime(&ms, G.ev[1], G.ev[2]));
    stats->ms_merge = ms;
    FKNN_CUDA(cudaEventElapsedTime(&ms, G.ev[2], G.ev[3]));
    stats->ms_scan = ms;
    uint32_t c[16];
    FKNN_CUDA(cudaMemcpy(c, P.cnt, sizeof(c), cudaMemcpyDeviceToHost));
    uint32_t h2[2] = {0, 0};
    FKNN_CUDA(cudaMemcpy(h2, S.ovf_count, 8, cudaMemcpyDeviceToHost));
    auto u64 = [&](int i) { return (uint64_t)c[i] | ((uint64_t)c[i + 1] << 32); };
    stats->pairs_screened = u64(10);
    stats->pairs_passing = u64(12);
    stats->pairs_contraction = u64(14);
    stats->n_tiles = c[DP_NTILE];
    stats->n_work_items = c[DP_NITEMS];
    stats->n_small = c[DP_NSMALL];
    stats->ms_plan = 0.f;
    stats->n_overflow = h2[0];
    stats->n_boundary_f64 = h2[1];
  }
  return FKNN_OK;
}

int search_bf16(fknn_index *idx, const float *d_q, const float *d_meta, uint32_t nq, uint32_t k, uint32_t kprime,
                uint32_t *d_ids, float *d_dists, cudaStream_t st, fknn_search_stats *stats) {
  return search_tc<FmtBF16>(idx, d_q, d_meta, nq, k, kprime, d_ids, d_dists, st, stats);
}

int search_bf16_graph(fknn_index *idx, const float *d_q, const float *d_meta, uint32_t nq, uint32_t k,
                      uint32_t kprime, uint32_t *d_ids, float *d_dists, cudaStream_t st, fknn_search_stats *stats) {
  return search_tc_graph<FmtBF16>(idx, d_q, d_meta, nq, k, kprime, d_ids, d_dists, st, stats);
}

int search_fp8_graph(fknn_index *idx, const float *d_q, const float *d_meta, uint32_t nq, uint32_t k,
                     uint32_t kprime, uint32_t *d_ids, float *d_dists, cudaStream_t st, fknn_search_stats *stats) {
  return search_tc_graph<FmtFP8>(idx, d_q, d_meta, nq, k, kprime, d_ids, d_dists, st, stats);
}

int search_fp8(fknn_index *idx, const float *d_q, const float *d_meta, uint32_t nq, uint32_t k, uint32_t kprime,
               uint32_t *d_ids, float *d_dists, cudaStream_t st, fknn_search_stats *stats) {
  return search_tc<FmtFP8>(idx, d_q, d_meta, nq, k, kprime, d_ids, d_dists, st, stats);
}

}  // namespace fknn
