// Epilogue pieces shared by the tensor-core screens (bf16_search.cu,
// exact_screen.cu): an epilogue thread owns one query (one TMEM lane) and
// turns 32 accumulator columns at a time into candidate-list pushes; a warp
// trims a list by a radix select over registers.
#pragma once

#include <algorithm>

#include "tc_util.cuh"

namespace fknn {

constexpr int STAGE_ROW = 36;  // floats per lane row of the push staging area

// max of 32 values as a tree of three-input maxima, and those of the four groups of 8
__device__ __forceinline__ float max32(const uint32_t (&r)[32], float (&g)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t *x = r + 8 * k;
    g[k] = fmax3(fmax3(__uint_as_float(x[0]), __uint_as_float(x[1]), __uint_as_float(x[2])),
                 fmax3(__uint_as_float(x[3]), __uint_as_float(x[4]), __uint_as_float(x[5])),
                 fmaxf(__uint_as_float(x[6]), __uint_as_float(x[7])));
  }
  return fmaxf(fmax3(g[0], g[1], g[2]), g[3]);
}

// bit j set iff r[j] >= t, given the groups' maxima: one group as a rule
__device__ __forceinline__ uint32_t ge_mask32(const uint32_t (&r)[32], const float (&g)[4], float t) {
  uint32_t in = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (g[k] >= t)
#pragma unroll
      for (int j = 8 * k; j < 8 * k + 8; ++j) in |= (__uint_as_float(r[j]) >= t ? 1u : 0u) << j;
  return in;
}

// bit j set iff r0 <= j < r1
__device__ __forceinline__ uint32_t range_mask(int r0, int r1) {
  const int a = max(r0, 0), b = min(r1, 32);
  return a >= b ? 0u : (0xffffffffu >> (32 - b)) & (0xffffffffu << a);
}

// one epilogue warp's scratch: staged candidate chunks, or the histogram of a trim
template <int SLOTS>
struct ScreenWarp {
  union {
    float row[SLOTS][STAGE_ROW];
    uint32_t hist[256];
  };
  float4 q[32];
  int info[SLOTS];  // first column | lane
};


// Candidates: the lanes (queries) whose 32-column chunk holds some stage its
// values in slots of their warp (x_stage); once the accumulator is released
// the warp takes a slot at a time, a column per lane, and appends the passing
// ones with one ballot (x_flush).  Each lane walking its own registers instead
// diverges, and measured slower.  Both are out of line and reload the chunk:
// they run for a few chunks of a sub-tile at most, and a copy per chunk pushes
// the other roles' code out of the instruction caches.
//   pass: column in [r0, r1) and v >= bound;  ds = qn + f2 v
struct ScreenQuery {
  float bound, f2, qn;
  int range;  // r0 << 16 | r1
};
template <int SLOTS>
__device__ __noinline__ int x_flush(ScreenWarp<SLOTS> &w, int ns, uint32_t p0, Candidate *lists, uint32_t list_cap,
                                    int cnt) {
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  __syncwarp();
#pragma unroll 1
  for (int i = 0; i < ns; ++i) {
    const int inf = w.info[i], src = inf & 31, c = (inf & ~31) + lane;
    const float v = w.row[i][lane];
    const float4 t = w.q[src];
    const int n = __shfl_sync(0xffffffffu, cnt, src), rg = __float_as_int(t.w);
    const bool pass = v >= t.x && c >= (rg >> 16) && c < (rg & 0xffff);
    const uint32_t m = __ballot_sync(0xffffffffu, pass);
    if (pass) {
      Candidate cd;
      cd.ds = fmaf(t.y, v, t.z);
      cd.pos = p0 + c;
      lists[src * list_cap + n + __popc(m & lt)] = cd;
    }
    if (lane == src) cnt += __popc(m);
  }
  __syncwarp();  // the slots are free again, the list entries visible to the warp
  return cnt;
}
// chunk of columns c .. c + 31, lanes fm; returns cnt << 8 | the slots in use
// (cnt changes when the slots run out)
template <int SLOTS>
__device__ __noinline__ int x_stage(uint32_t taddr, int c, uint32_t fm, ScreenQuery q, uint32_t p0,
                                    ScreenWarp<SLOTS> &w, int ns, Candidate *lists, uint32_t list_cap, int cnt) {
  const int lane = threadIdx.x & 31;
  uint32_t r[32];
  tmem_ld32_issue(taddr + c, r);
  w.q[lane] = make_float4(q.bound, q.f2, q.qn, __int_as_float(q.range));
  tmem_wait_ld(r);
  while (fm) {  // warp-uniform
    if (ns == SLOTS) {
      cnt = x_flush(w, ns, p0, lists, list_cap, cnt);
      ns = 0;
    }
    const int at = ns + __popc(fm & ((1u << lane) - 1u));
    const bool mine = ((fm >> lane) & 1u) && at < SLOTS;
    if (mine) {
#pragma unroll
      for (int j = 0; j < 32; j += 4)
        *reinterpret_cast<uint4 *>(&w.row[at][j]) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
      w.info[at] = c | lane;
    }
    const uint32_t took = __ballot_sync(0xffffffffu, mine);
    ns += __popc(took);
    fm &= ~took;
  }
  return cnt << 8 | ns;
}


// An upper bound on the kth smallest (1-based, kth <= n) of the n keys held
// NPL per lane (element j * 32 + lane in key[j]), at most `slack` keys above
// it: a warp radix select from the highest differing bit that stops as soon
// as the digit it is in ends near enough (one pass of three, as a rule).
template <int NPL>
__device__ __forceinline__ uint32_t warp_kth_upper(const uint32_t (&key)[NPL], int n, int kth, int slack,
                                                   uint32_t *hist) {
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
  int hi = mn == mx ? 0 : 32 - __clz(mn ^ mx);  // bits [hi-1, 0] still differ
  uint32_t mask = hi == 32 ? 0u : ~((1u << hi) - 1u);
  uint32_t prefix = mn & mask;
  int below = 0;  // keys smaller than the prefix's range
  while (hi > 0) {
    const int w = min(8, hi), shift = hi - w;
    for (int i = lane; i < 256; i += 32) hist[i] = 0;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < NPL; ++j)
      if (j * 32 + lane < n && (key[j] & mask) == prefix) atomicAdd(&hist[(key[j] >> shift) & ((1u << w) - 1)], 1u);
    __syncwarp();
    const uint4 a = reinterpret_cast<const uint4 *>(hist)[lane * 2], b = reinterpret_cast<const uint4 *>(hist)[lane * 2 + 1];
    const uint32_t local[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    int sum = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) sum += (int)local[j];
    int inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    const int want = kth - below;
    int c = inc - sum, bin = -1, upto = 0;
    if (c < want && inc >= want) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (bin < 0 && c + (int)local[j] >= want) {
          bin = lane * 8 + j;
          upto = c;  // keys before the bin
        }
        if (bin < 0) c += (int)local[j];
      }
      upto = upto << 16 | (int)local[bin & 7];
    }
    const int owner = __ffs(__ballot_sync(0xffffffffu, bin >= 0)) - 1;
    bin = __shfl_sync(0xffffffffu, bin, owner);
    upto = __shfl_sync(0xffffffffu, upto, owner);
    __syncwarp();
    prefix |= (uint32_t)bin << shift;
    mask |= ((1u << w) - 1) << shift;
    hi = shift;
    if (below + (upto >> 16) + (upto & 0xffff) <= kth + slack) break;
    below += upto >> 16;
  }
  return prefix | ~mask;
}

// Bounds from a pilot pass (every stride-th row block of each item): the r-th
// smallest screening distance over the union of a query's pilot lists is an
// estimate from above of the k-th of all its rows, which the merge checks.  r
// follows from the share of the query's own slab that was sampled.  NT threads
// per query, a list to each of their warps at a time (a thousand items have as
// many lists: one list at a time for all threads took 211 us of a 50-query
// call over 464 items); bound() turns the r-th distance into the value stored.
struct SeedArgs {
  const uint32_t *big_q, *big_tile, *big_lane;
  uint32_t nbig;
  const uint32_t *nbig_d;       // device plan: the big-query count (NULL: nbig)
  const Tile *tiles;
  const WorkItem *items;
  const uint32_t *item_slot;    // NULL: a tile's items are consecutive
  const Candidate *out;         // [item][tq][list_cap]
  const uint32_t *out_cnt;      // [item][tq]
  uint32_t tq, list_cap, blk_rows;
  const QueryDesc *desc;
  uint32_t stride, k;
  uint32_t *T_global;           // f32_sortable; untouched where the lists hold less than r entries
  uint32_t *seeded;             // NULL, or set to 1 where a bound was stored
};

template <int NT, class Bound>
__global__ void __launch_bounds__(256) k_screen_seed(SeedArgs A, Bound bound) {
  __shared__ uint32_t hist[256 / NT][256];
  __shared__ uint32_t red[256 / NT][4];  // total, min, max of the keys; digit found
  const int grp = threadIdx.x / NT, t = threadIdx.x % NT, lane = threadIdx.x & 31;
  const uint32_t nbig = A.nbig_d ? *A.nbig_d : A.nbig;
  auto sync = [&]() {
    if (NT == 32) __syncwarp();
    else __syncthreads();
  };
  uint32_t *h = hist[grp], *rd = red[grp];
  for (uint32_t b = blockIdx.x * (256 / NT) + grp; b < nbig; b += gridDim.x * (256 / NT)) {  // (group-uniform)
    const uint32_t qi = A.big_q[b], L = A.big_lane[b];
    const Tile tl = A.tiles[A.big_tile[b]];
    // the sampled rows of the query's slab, and the rank of the seed among them
    const QueryDesc dq = A.desc[qi];
    uint32_t rows = 0;
    for (uint32_t i = tl.item0 + t; i < tl.item1 && dq.e > dq.s; i += NT) {
      const WorkItem it = A.items[A.item_slot ? A.item_slot[i] : i];
      const uint32_t b0 = dq.s / A.blk_rows, b1 = (dq.e - 1) / A.blk_rows;  // the slab's first and last block
      const uint32_t p0 = it.blk0 + (b0 > it.blk0 ? (b0 - it.blk0 + A.stride - 1) / A.stride * A.stride : 0u);
      const uint32_t p1 = min(it.blk1, b1 + 1);
      if (p0 >= p1) continue;
      const uint32_t n = (p1 - 1 - p0) / A.stride + 1;  // sampled blocks that meet the slab
      rows += n * A.blk_rows;
      if (p0 == b0) rows -= dq.s - b0 * A.blk_rows;
      if (p0 + (n - 1) * A.stride == b1) rows -= (uint32_t)((uint64_t)(b1 + 1) * A.blk_rows - dq.e);
    }
    // every list of the query, a warp to a list
    auto each = [&](auto &&f) {
      for (uint32_t i = tl.item0 + t / 32; i < tl.item1; i += NT / 32) {
        const uint64_t item = A.item_slot ? A.item_slot[i] : i;
        const uint32_t c = A.out_cnt[item * A.tq + L];
        const Candidate *src = A.out + (item * A.tq + L) * A.list_cap;
        for (uint32_t j = lane; j < c; j += 32) f(f32_sortable(src[j].ds));
      }
    };
    sync();  // (red is reused)
    if (t == 0) {
      rd[0] = 0;
      rd[1] = 0xffffffffu;
      rd[2] = 0;
      rd[3] = 0;
    }
    sync();
    uint32_t n = 0, mn = 0xffffffffu, mx = 0;
    each([&](uint32_t u) {
      ++n;
      mn = min(mn, u);
      mx = max(mx, u);
    });
    n = __reduce_add_sync(0xffffffffu, n);
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    rows = __reduce_add_sync(0xffffffffu, rows);
    if (lane == 0) {
      atomicAdd(&rd[3], rows);
      atomicAdd(&rd[0], n);
      atomicMin(&rd[1], mn);
      atomicMax(&rd[2], mx);
    }
    sync();
    n = rd[0];
    mn = rd[1];
    mx = rd[2];
    const uint32_t r = exact_seed_rank(A.k, rd[3], dq.e - dq.s);
    if (n < r) continue;  // group-uniform
    // radix select from the highest bit in which the keys differ
    int hi = mn == mx ? 0 : 32 - __clz(mn ^ mx);
    uint32_t mask = hi == 32 ? 0u : ~((1u << hi) - 1u);
    uint32_t prefix = mn & mask, remaining = r;
    while (hi > 0) {
      const int w = min(8, hi), shift = hi - w;
      for (int i = t; i < 256; i += NT) h[i] = 0;
      sync();
      each([&](uint32_t u) {
        if ((u & mask) == prefix) atomicAdd(&h[(u >> shift) & ((1u << w) - 1)], 1u);
      });
      sync();
      if (t < 32) {
        uint32_t local[8], sum = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          local[j] = h[lane * 8 + j];
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
              rd[2] = lane * 8 + j;
              rd[3] = c;
            }
            c += local[j];
          }
        }
      }
      sync();
      prefix |= rd[2] << shift;
      remaining -= rd[3];
      mask |= ((1u << w) - 1) << shift;
      hi = shift;
      sync();
    }
    if (t == 0) {
      A.T_global[qi] = f32_sortable(bound(sortable_f32(prefix), dq));
      if (A.seeded) A.seeded[qi] = 1u;
    }
  }
}

// A warp per query where there are enough queries to fill the GPU that way
// (their lists are then few), else a block per query.  nmax: at least the
// number of queries.
template <class Bound>
inline void launch_screen_seed(const SeedArgs &A, uint32_t nmax, Bound bound, cudaStream_t st) {
  const uint32_t gmax = 148 * 16;
  if (nmax >= 4096) k_screen_seed<32><<<std::min((nmax + 7) / 8, gmax), 256, 0, st>>>(A, bound);
  else k_screen_seed<256><<<std::min(nmax, gmax), 256, 0, st>>>(A, bound);
  g_launches += 1;
}

}  // namespace fknn
