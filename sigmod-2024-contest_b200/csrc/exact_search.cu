// Exact FP32 filtered top-k (the B200 form of utils.h:80-158 Bruteforce).
//
// Pipeline for one batch of queries:
//   1. k_query_prep   predicate -> contiguous slab [s, e) of one row order
//                     (binary search on the sorted attribute columns), ||q||^2
//   2. host planner   slabs <= SMALL_SLAB -> row-by-row exact scan; others
//                     sorted and grouped into 256-query tiles, split into
//                     (tile, row chunk) work items
//   3. k_exact_screen tensor-core contraction q.x of float accuracy (two
//                     fp16 pieces a side) over the 64-row blocks
//                     (exact_screen.cu); ds = |x|^2+|q|^2-2q.x; rows whose ds
//                     can still reach the running k-th bound are kept in a
//                     per-(item, query) candidate list; the bound is shared
//                     across CTAs.  A pilot pass over every pilot_stride-th
//                     row block seeds the bounds (k_screen_seed).
//   4. k_merge        per query: union of its items' lists, k-th bound, then
//                     exact re-score of the survivors with the reference's
//                     sequential arithmetic, (dist, id) order, top-k out.  A
//                     query whose seed lay below its k-th is found here and
//                     screened and merged once more without one.
//   5. k_exact_scan   small slabs and any query whose candidates overflowed:
//                     exact distances row by row, block select on (dist, id).
// Ids and distances equal the reference's bit for bit: every row that can
// be in the top k (screening error bound in screen_eps) is re-scored with
// normal_l2's exact operation sequence and ordered by (dist, id) like the
// ResultMaxHeap of utils.h:35-78.
#include <algorithm>
#include <functional>
#include <thread>
#include <chrono>
#include <cmath>
#include <cstring>
#include <numeric>

#include "device_util.cuh"

namespace fknn {

namespace {

// ---------------------------------------------------------------- prep --

// Query checks: type in {0,1,2,3} (searcher.hpp:39-42 rejects the rest),
// v inside int32 for types 1/3 (read as int32, utils.h:99), window bounds
// not NaN for types 2/3, vector values finite and <= 1e15.
__global__ void k_validate_queries(const float *__restrict__ q, const float *__restrict__ meta, uint32_t nq,
                                   int *flag) {
  const uint64_t total = (uint64_t)nq * DIM;
  int bad = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total;
       i += (uint64_t)gridDim.x * blockDim.x) {
    if (!(fabsf(q[i]) <= 1e15f)) bad |= ERR_BAD_QUERY_VEC;
    if (i < nq) {
      const float *m = meta + i * 4;
      float t = m[0];
      if (!(t == 0.f || t == 1.f || t == 2.f || t == 3.f)) bad |= ERR_BAD_QUERY_TYPE;
      if ((t == 1.f || t == 3.f) && !(fabsf(m[1]) < 2147483648.f)) bad |= ERR_BAD_QUERY_VALUE;
      if ((t == 2.f || t == 3.f) && (m[2] != m[2] || m[3] != m[3])) bad |= ERR_BAD_QUERY_VALUE;
    }
  }
  if (bad) atomicOr(flag, bad);
}

// The first position in [lo, hi) that is not below (pred: monotone, true
// first), by the whole warp: 32 probes a step, so a million positions take
// four memory latencies where halving takes twenty.
template <class Pred>
__device__ __forceinline__ uint32_t warp_partition(uint32_t lo, uint32_t hi, Pred pred) {
  const uint32_t lane = threadIdx.x & 31;
  while (hi > lo) {
    const uint32_t chunk = (hi - lo + 31) / 32;
    const uint64_t p = (uint64_t)lo + (lane + 1ull) * chunk - 1;
    const uint32_t c = __popc(__ballot_sync(0xffffffffu, p < hi && pred((uint32_t)p)));
    const uint64_t end = (uint64_t)lo + (c + 1ull) * chunk - 1;
    lo += c * chunk;  // the probe after is not below, or past the end
    if (lo > hi) lo = hi;
    hi = (uint32_t)min((uint64_t)hi, end);
  }
  return lo;
}

// The same by one thread, halving.
template <class Pred>
__device__ __forceinline__ uint32_t thread_partition(uint32_t lo, uint32_t hi, Pred pred) {
  while (lo < hi) {
    const uint32_t m = lo + ((hi - lo) >> 1);
    if (pred(m)) lo = m + 1;
    else hi = m;
  }
  return lo;
}

// Predicate -> slab.  type 0: all rows (time order); 1: label == v (category
// order); 2: l <= ts <= r (time order); 3: both (category order, the window
// inside the label's slab).  The semantics are utils.h:110-137's.  WARP: by the
// whole warp, else by each thread.
template <bool WARP>
__device__ __forceinline__ void resolve_slab(const float *m, uint32_t n, const float *ts_t, const int32_t *lab_c,
                                             const float *ts_c, int32_t &order, uint32_t &s, uint32_t &e) {
  const uint32_t type = (uint32_t)m[0];
  auto partition = [](uint32_t lo, uint32_t hi, auto pred) {
    return WARP ? warp_partition(lo, hi, pred) : thread_partition(lo, hi, pred);
  };
  auto window = [&](const float *ts, uint32_t lo, uint32_t hi) {
    const float l = m[2], r = m[3];
    s = partition(lo, hi, [&](uint32_t p) { return ts[p] < l; });
    e = partition(lo, hi, [&](uint32_t p) { return ts[p] <= r; });
  };
  order = type == 0 || type == 2 ? ORDER_TIME : ORDER_CAT;
  if (type == 0) {
    s = 0;
    e = n;
  } else if (type == 2) {
    window(ts_t, 0, n);
  } else {
    const int32_t v = (int32_t)m[1];
    s = partition(0, n, [&](uint32_t p) { return lab_c[p] < v; });
    e = partition(s, n, [&](uint32_t p) { return lab_c[p] <= v; });
    if (type == 3) window(ts_c, s, e);
  }
  if (e < s) e = s;
}

// A warp per query (WARP) below QP_MANY queries, else a thread: the one has the
// shorter chain of memory latencies, the other a fifth of the loads.  Counts
// over 1e6 rows, whole calls, by warps and by threads: 25 and 40 us (4,000
// queries), 32 and 41 (16,000), 37 and 42 (32,000), 67 and 40 (100,000), 1,253
// and 240 (3e6).  64 bits: nq warps have up to 2^37 threads.
constexpr int QP_THREADS = 256;
constexpr uint32_t QP_MANY = 32768;
template <bool WARP>
__device__ __forceinline__ uint64_t query_of() {
  const uint64_t t = (uint64_t)blockIdx.x * QP_THREADS + threadIdx.x;
  return WARP ? t / 32 : t;
}
inline unsigned query_blocks(uint32_t nq) {
  const uint64_t threads = nq < QP_MANY ? (uint64_t)nq * 32 : nq;
  return (unsigned)((threads + QP_THREADS - 1) / QP_THREADS);
}

template <bool WARP>
__global__ void __launch_bounds__(QP_THREADS)
    k_query_prep(const float *__restrict__ q, const float *__restrict__ meta, uint32_t nq, uint32_t n,
                 const float *__restrict__ ts_t, const int32_t *__restrict__ lab_c, const float *__restrict__ ts_c,
                 QueryDesc *__restrict__ desc) {
  const uint64_t i = query_of<WARP>();
  if (i >= nq) return;
  const float *x = q + i * DIM;
  const uint32_t lane = threadIdx.x & 31;
  float v[4];
  if (WARP)
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = 32 * j + lane < DIM ? x[32 * j + lane] : 0.f;
  QueryDesc dsc;
  resolve_slab<WARP>(meta + i * 4, n, ts_t, lab_c, ts_c, dsc.order, dsc.s, dsc.e);
  // |q|^2 in dimension order (every lane the same chain)
  float s = 0.f;
  if (WARP) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const float t = __shfl_sync(0xffffffffu, v[d / 32], d % 32);
      s = fmaf(t, t, s);
    }
  } else {
#pragma unroll 10
    for (int d = 0; d < DIM; ++d) s = fmaf(x[d], x[d], s);
  }
  dsc.qn = s;
  if (!WARP || lane == 0) desc[i] = dsc;
}

template <bool WARP>
__global__ void __launch_bounds__(QP_THREADS)
    k_count(const float *__restrict__ meta, uint32_t nq, uint32_t n, const float *__restrict__ ts_t,
            const int32_t *__restrict__ lab_c, const float *__restrict__ ts_c, uint32_t *__restrict__ counts) {
  const uint64_t i = query_of<WARP>();
  if (i >= nq) return;
  int32_t o;
  uint32_t s, e;
  resolve_slab<WARP>(meta + i * 4, n, ts_t, lab_c, ts_c, o, s, e);
  if (!WARP || (threadIdx.x & 31) == 0) counts[i] = e - s;
}

// --------------------------------------------------------------- merge --

constexpr int MG_THREADS = 128;

template <int MCAP>
struct MergeSmem {
  float key[MCAP];
  uint32_t val[MCAP];
  uint64_t ekey[RESCORE_CAP];
  float qv[DIM];
  uint32_t cnt_prefix[MAX_ITEMS_PER_TILE + 1];
  uint32_t hist[256];
  uint32_t red[4];
  int total, surv;
};

struct ExactMergeArgs {
  const uint32_t *big_q, *big_tile, *big_lane;
  const Tile *tiles;
  const uint32_t *item_slot;
  const Candidate *out;
  const uint32_t *out_cnt;
  const QueryDesc *desc;
  const float *q, *vecs;
  const uint32_t *perm_t, *perm_c;
  uint32_t *T_global;
  const uint32_t *ovf;
  uint32_t *ovf_list, *ovf_count;  // queries for the exact scan
  // queries whose seeded bound may lie below their k-th (NULL: bounds are not seeded)
  uint32_t *redo_list, *redo_count, *redo_skip;
  uint32_t k;
  uint32_t *ids;
  float *dists;
};

// One big query b (index into the plan's big-query arrays): gather its
// lists, bound the k-th distance over their union, re-score the survivors
// with the reference's arithmetic, order them by (dist, id).  A query with
// more than MCAP candidates goes to `spill` (the large merge) or, from the
// large merge, to the exact scan.  Returns are block-uniform.
template <int MCAP>
__device__ void exact_merge_one(const ExactMergeArgs &A, uint32_t b, MergeSmem<MCAP> &sm, uint32_t *spill,
                                uint32_t *spill_count) {
  const int tid = threadIdx.x;
  const uint32_t k = A.k;
  const uint32_t qi = A.big_q[b];
  if (A.ovf[qi]) {
    if (tid == 0) A.ovf_list[atomicAdd(A.ovf_count, 1u)] = qi;
    return;
  }
  const Tile tl = A.tiles[A.big_tile[b]];
  const uint32_t L = A.big_lane[b];
  const uint32_t nitems = tl.item1 - tl.item0;
  const QueryDesc dsc = A.desc[qi];
  const float qn = dsc.qn;
  for (int d = tid; d < DIM; d += MG_THREADS) sm.qv[d] = A.q[(uint64_t)qi * DIM + d];
  // 1. gather the lists: item offsets, then a warp copies a list at a time
  list_offsets(A.item_slot, tl.item0, nitems, A.out_cnt, L, EXACT_TQ, sm.cnt_prefix, &sm.total, MAX_ITEMS_PER_TILE,
               MERGE_CAP + 1);
  if (tid == 0) sm.surv = 0;
  __syncthreads();
  const int M = sm.total;
  if (M > MCAP) {
    if (tid == 0) {
      if (spill && M <= MERGE_CAP) spill[atomicAdd(spill_count, 1u)] = b;
      else A.ovf_list[atomicAdd(A.ovf_count, 1u)] = qi;
    }
    return;
  }
  for (uint32_t i = tid / 32; i < nitems; i += MG_THREADS / 32) {
    const uint64_t item = A.item_slot[tl.item0 + i];
    const uint32_t base = sm.cnt_prefix[i];
    const uint32_t c = (i + 1 < nitems ? sm.cnt_prefix[i + 1] : (uint32_t)M) - base;
    const Candidate *src = A.out + (item * EXACT_TQ + L) * EXACT_CAP;
    for (uint32_t j = tid & 31; j < c; j += 32) {
      const Candidate cd = src[j];
      sm.key[base + j] = cd.ds;
      sm.val[base + j] = cd.pos;
    }
  }
  __syncthreads();
  // 2. k-th bound over the union.  A seeded bound admitted every row that
  //    can be in the top k iff the union's k-th is proven to lie below it
  const float Tg = sortable_f32(A.T_global[qi]);
  float T = Tg;
  bool proven = false;
  if (M >= (int)k) {
    const float h = screen_hi(sortable_f32(block_kth<MG_THREADS>(sm.key, M, k, sm.hist, sm.red)), qn);
    proven = h <= Tg + 5e-7f * fabsf(Tg);  // (screen_hi's own slack of 1e-6 covers the tolerance)
    T = fminf(T, h);
  }
  if (A.redo_list && !proven) {
    if (tid == 0) {
      A.redo_list[atomicAdd(A.redo_count, 1u)] = b;
      A.redo_skip[qi] = 0u;
      A.T_global[qi] = f32_sortable(INFINITY);
    }
    return;
  }
  // 3. survivors
  for (int i = tid; i < M; i += MG_THREADS) {
    if (screen_lo(sm.key[i], qn) <= T) {
      const int slot = atomicAdd(&sm.surv, 1);
      if (slot < RESCORE_CAP) sm.ekey[slot] = (dsc.order == ORDER_TIME ? A.perm_t : A.perm_c)[sm.val[i]];
    }
  }
  __syncthreads();
  const int S = sm.surv;
  if (S > RESCORE_CAP) {
    if (tid == 0) A.ovf_list[atomicAdd(A.ovf_count, 1u)] = qi;
    return;
  }
  // 4. exact re-score (distance.h:62-72 order of operations)
  for (int i = tid; i < S; i += MG_THREADS) {
    const uint32_t id = (uint32_t)sm.ekey[i];
    sm.ekey[i] = exact_key(seq_l2_row(A.vecs + (uint64_t)id * DIM, sm.qv), id);
  }
  __syncthreads();
  // 5. each survivor's rank is the number of smaller keys (keys are distinct:
  //    a row appears once), counted by its thread
  for (int i = tid; i < S; i += MG_THREADS) {
    const uint64_t e = sm.ekey[i];
    uint32_t rank = 0;
    for (int j = 0; j < S; ++j) rank += sm.ekey[j] < e ? 1u : 0u;
    if (rank < k) {
      A.ids[(uint64_t)qi * k + rank] = (uint32_t)e;
      if (A.dists) A.dists[(uint64_t)qi * k + rank] = sortable_f32((uint32_t)(e >> 32));
    }
  }
  for (uint32_t j = (uint32_t)S + tid; j < k; j += MG_THREADS) {
    A.ids[(uint64_t)qi * k + j] = 0xffffffffu;
    if (A.dists) A.dists[(uint64_t)qi * k + j] = INFINITY;
  }
}

// work == nullptr: block b merges big query b (grid = number of big
// queries); else the blocks stride over the *work_count entries of work.
template <int MCAP>
__global__ void __launch_bounds__(MG_THREADS)
    k_merge(ExactMergeArgs A, uint32_t nbig, const uint32_t *__restrict__ work, const uint32_t *__restrict__ work_count,
            uint32_t *__restrict__ spill, uint32_t *__restrict__ spill_count) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  MergeSmem<MCAP> &sm = *reinterpret_cast<MergeSmem<MCAP> *>(smem_raw);
  const uint32_t nwork = work ? *work_count : nbig;
  for (uint32_t w = blockIdx.x; w < nwork; w += gridDim.x) {
    exact_merge_one<MCAP>(A, work ? work[w] : w, sm, spill, spill_count);
    __syncthreads();  // shared memory is reused by the next query
  }
}

// ----------------------------------------------------------- exact scan --

// Bound by latency: a slab of 4,096 rows is 1.6 MB, and one block reads it.  So
// a thread has 25 loads of a row in flight, and the keys stay in shared memory
// until the k smallest are selected (a radix select, then every survivor counts
// its place).  A few queries have blocks of 512 threads, whose eight rows cover
// the longest slab that is planned for here (longer ones, of queries whose
// candidates overflowed, select whenever the buffer fills); from SCAN_MANY
// queries on blocks of 256, of which an SM holds five in place of three.  Calls of slabs
// of 2,000 to 4,096 rows, by 512 and by 256 threads: 179 and 208 us (100
// queries), 199 and 222 (300), 257 and 246 (600), 944 and 767 (4,000); of up to
// 64 rows 748 and 453 (30,000), where 649 was the time with sorts of 1,024 keys.
constexpr uint32_t SCAN_MANY = 512;
template <int NT, int CAP>
struct ScanSmem {
  uint64_t buf[CAP];  // keys
  uint64_t sel[KMAX_TILE];
  float qv[DIM];
  uint32_t hist[256];
  unsigned long long mn, mx;
  uint32_t bin, before, count;
  int cnt, kept;
  uint64_t thr;
};

// The k smallest of the cnt > k distinct keys in buf to sel, in no order.
template <int NT, int CAP>
__device__ void scan_select(ScanSmem<NT, CAP> &sm, int cnt, uint32_t k) {
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) {
    sm.mn = ~0ull;
    sm.mx = 0;
    sm.kept = 0;
  }
  __syncthreads();
  uint64_t mn = ~0ull, mx = 0;
  for (int i = tid; i < cnt; i += NT) {
    mn = min(mn, sm.buf[i]);
    mx = max(mx, sm.buf[i]);
  }
  atomicMin(&sm.mn, (unsigned long long)mn);
  atomicMax(&sm.mx, (unsigned long long)mx);
  __syncthreads();
  // radix select from the highest bit in which the keys differ, until the
  // digit it is in holds one key
  int hi = 64 - __clzll((long long)(sm.mn ^ sm.mx));
  uint64_t mask = hi == 64 ? 0ull : ~((1ull << hi) - 1ull), prefix = sm.mn & mask;
  uint32_t want = k;
  while (hi > 0) {
    const int w = min(8, hi), shift = hi - w;
    for (int i = tid; i < 256; i += NT) sm.hist[i] = 0;
    __syncthreads();
    for (int i = tid; i < cnt; i += NT) {
      const uint64_t u = sm.buf[i];
      if ((u & mask) == prefix) atomicAdd(&sm.hist[(u >> shift) & ((1u << w) - 1)], 1u);
    }
    __syncthreads();
    if (tid < 32) {
      uint32_t local[8], sum = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        local[j] = sm.hist[lane * 8 + j];
        sum += local[j];
      }
      uint32_t inc = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      uint32_t c = inc - sum;
      if (c < want && inc >= want) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (c < want && c + local[j] >= want) {
            sm.bin = lane * 8 + j;
            sm.before = c;
            sm.count = local[j];
          }
          c += local[j];
        }
      }
    }
    __syncthreads();
    prefix |= (uint64_t)sm.bin << shift;
    mask |= ((1ull << w) - 1ull) << shift;
    want -= sm.before;
    hi = shift;
    if (sm.count == 1) break;
  }
  for (int i = tid; i < cnt; i += NT) {
    const uint64_t u = sm.buf[i];
    if ((u & mask) <= prefix) sm.sel[atomicAdd(&sm.kept, 1)] = u;
  }
  __syncthreads();
}

template <int NT, int CAP>
__global__ void __launch_bounds__(NT)
    k_exact_scan(const uint32_t *__restrict__ list, const uint32_t *__restrict__ d_count, uint32_t h_count,
                 const QueryDesc *__restrict__ desc, const float *__restrict__ q, const float *__restrict__ blocks_t,
                 const float *__restrict__ blocks_c, const uint32_t *__restrict__ perm_t,
                 const uint32_t *__restrict__ perm_c, uint32_t k, uint32_t *__restrict__ ids,
                 float *__restrict__ dists) {
  __shared__ ScanSmem<NT, CAP> sm;
  const uint32_t count = d_count ? *d_count : h_count;
  const int tid = threadIdx.x;
  for (uint32_t li = blockIdx.x; li < count; li += gridDim.x) {
    const uint32_t qi = list[li];
    const QueryDesc dsc = desc[qi];
    const float *blocks = dsc.order == ORDER_TIME ? blocks_t : blocks_c;
    const uint32_t *perm = dsc.order == ORDER_TIME ? perm_t : perm_c;
    for (int d = tid; d < DIM; d += NT) sm.qv[d] = q[(uint64_t)qi * DIM + d];
    if (tid == 0) {
      sm.cnt = 0;
      sm.thr = ~0ull;
    }
    __syncthreads();
    int held = 0;  // keys in buf: counted at the step's barrier, for sm.cnt grows again as soon as a warp has passed it
    for (uint64_t base = dsc.s; base < dsc.e; base += NT) {
      const uint64_t p = base + tid;
      bool push = false;
      if (p < dsc.e) {
        const float *x = blocks + (p / BLK) * BLK_FLOATS + (p % BLK);
        const uint32_t id = perm[p];
        float r = 0.f;
#pragma unroll 1
        for (int d0 = 0; d0 < DIM; d0 += 25) {
          float v[25];
#pragma unroll
          for (int d = 0; d < 25; ++d) v[d] = __ldg(x + (d0 + d) * BLK);
#pragma unroll
          for (int d = 0; d < 25; ++d) {  // seq_l2_row's operations
            float t = __fsub_rn(v[d], sm.qv[d0 + d]);
            t = __fmul_rn(t, t);
            r = __fadd_rn(r, t);
          }
        }
        const uint64_t key = exact_key(r, id);
        push = key < sm.thr;
        if (push) sm.buf[atomicAdd(&sm.cnt, 1)] = key;
      }
      held += __syncthreads_count(push);
      if (held > CAP - NT && base + NT < dsc.e) {  // (block-uniform)
        scan_select(sm, held, k);
        uint64_t mx = 0;
        for (uint32_t i = tid; i < k; i += NT) {
          sm.buf[i] = sm.sel[i];
          mx = max(mx, sm.sel[i]);
        }
        if (tid == 0) {
          sm.cnt = (int)k;
          sm.mx = 0;
        }
        __syncthreads();
        atomicMax(&sm.mx, (unsigned long long)mx);
        __syncthreads();
        if (tid == 0) sm.thr = sm.mx;
        held = (int)k;
        __syncthreads();
      }
    }
    int c = held;
    const uint64_t *keys = sm.buf;
    if (c > (int)k) {
      scan_select(sm, c, k);
      keys = sm.sel;
      c = (int)k;
    }
    // a key's place is the number of smaller ones (they are distinct)
    for (int i = tid; i < c; i += NT) {
      const uint64_t e = keys[i];
      uint32_t rank = 0;
      for (int j = 0; j < c; ++j) rank += keys[j] < e ? 1u : 0u;
      ids[(uint64_t)qi * k + rank] = (uint32_t)e;
      if (dists) dists[(uint64_t)qi * k + rank] = sortable_f32((uint32_t)(e >> 32));
    }
    for (uint32_t j = (uint32_t)c + tid; j < k; j += NT) {
      ids[(uint64_t)qi * k + j] = 0xffffffffu;
      if (dists) dists[(uint64_t)qi * k + j] = INFINITY;
    }
    __syncthreads();
  }
}

// ------------------------------------ predicate compaction (no-alloc form) --
//
// Count -> scan -> write over 4,096-row tiles: its only scratch is one
// counter per tile, which fits the fixed array of fknn_filter_rows_noalloc.
// The index's fknn_filter_rows / fknn_filter_rows_batch use filter.cu.

constexpr int FC_THREADS = 256;
constexpr int FC_ITEMS = 16;
constexpr int FC_TILE = FC_THREADS * FC_ITEMS;

__device__ __forceinline__ bool row_passes(uint32_t type, int32_t v, float l, float r, float label, float ts) {
  switch (type) {
    case 0: return true;
    case 1: return (int32_t)label == v;
    case 2: return ts >= l && ts <= r;
    default: return (int32_t)label == v && ts >= l && ts <= r;
  }
}

// Pass 1: passing rows per 4096-row tile (warp ballots, coalesced columns).
__global__ void k_filter_count(const float *__restrict__ labels, const float *__restrict__ ts, uint64_t n,
                               float4 m, uint32_t *__restrict__ tile_cnt) {
  __shared__ uint32_t wsum[FC_THREADS / 32];
  const uint32_t type = (uint32_t)m.x;
  const int32_t v = (int32_t)m.y;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint64_t base = (uint64_t)blockIdx.x * FC_TILE;
  uint32_t c = 0;
  for (int i = 0; i < FC_ITEMS; ++i) {
    const uint64_t idx = base + (uint64_t)i * FC_THREADS + threadIdx.x;
    const bool p = idx < n && row_passes(type, v, m.z, m.w, labels[idx], ts[idx]);
    c += __popc(__ballot_sync(0xffffffffu, p));
  }
  if (lane == 0) wsum[w] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t s = 0;
    for (int i = 0; i < FC_THREADS / 32; ++i) s += wsum[i];
    tile_cnt[blockIdx.x] = s;
  }
}

// Pass 2 (after an exclusive scan of tile_cnt): write passing ids in order.
// Each thread keeps its 16 predicates as a bit mask; one block scan over the
// (item, warp) counts gives every ballot its output offset.
__global__ void k_filter_write(const float *__restrict__ labels, const float *__restrict__ ts, uint64_t n, float4 m,
                               const uint32_t *__restrict__ tile_off, uint32_t *__restrict__ out) {
  constexpr int NW = FC_THREADS / 32;
  __shared__ uint32_t cnt[FC_ITEMS * NW + 1];
  const uint32_t type = (uint32_t)m.x;
  const int32_t v = (int32_t)m.y;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint64_t base = (uint64_t)blockIdx.x * FC_TILE;
  uint32_t bits = 0, ballots[FC_ITEMS];
#pragma unroll
  for (int i = 0; i < FC_ITEMS; ++i) {
    const uint64_t idx = base + (uint64_t)i * FC_THREADS + threadIdx.x;
    const bool p = idx < n && row_passes(type, v, m.z, m.w, labels[idx], ts[idx]);
    ballots[i] = __ballot_sync(0xffffffffu, p);
    bits |= (p ? 1u : 0u) << i;
  }
  // counts in output order: item-major, then warp
  if (lane < FC_ITEMS) {
    uint32_t c = 0;
#pragma unroll
    for (int i = 0; i < FC_ITEMS; ++i)
      if (i == lane) c = __popc(ballots[i]);
    cnt[lane * NW + w] = c;
  }
  __syncthreads();
  if (threadIdx.x < 32) {  // exclusive scan of the FC_ITEMS * NW = 128 counts, 4 per lane
    constexpr int PER = FC_ITEMS * NW / 32;
    uint32_t loc[PER], sum = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      loc[j] = cnt[lane * PER + j];
      sum += loc[j];
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    uint32_t run = tile_off[blockIdx.x] + inc - sum;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      cnt[lane * PER + j] = run;
      run += loc[j];
    }
  }
  __syncthreads();
  const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
  for (int i = 0; i < FC_ITEMS; ++i)
    if ((bits >> i) & 1u)
      out[cnt[i * NW + w] + __popc(ballots[i] & lt)] = (uint32_t)(base + (uint64_t)i * FC_THREADS + threadIdx.x);
}

// Exclusive scan of the tile counts in place, one block; *total = their sum.
__global__ void __launch_bounds__(1024) k_exclusive_scan_small(uint32_t *data, uint32_t len, uint32_t *total) {
  __shared__ uint32_t wsum[32];
  __shared__ uint32_t carry;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t base = 0; base < len; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < len ? data[i] : 0u;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    if (w == 0) {
      const uint32_t x = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0u;
      uint32_t y = x;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) y += t;
      }
      wsum[lane] = y - x;  // exclusive sum of the warps before
    }
    __syncthreads();
    const uint32_t c = carry;
    if (i < len) data[i] = c + wsum[w] + inc - v;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = c + wsum[w] + inc;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

__global__ void k_fill_u32(uint32_t *__restrict__ p, uint32_t n, uint32_t v) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = v;
}

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace

// ============================================================== host side

int validate_queries(fknn_index *idx, const float *d_q, const float *d_meta, uint32_t nq, cudaStream_t st) {
  int *flag = idx->d_flag;
  FKNN_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), st));
  unsigned grid = (unsigned)std::min<uint64_t>(((uint64_t)nq * DIM + 255) / 256, 148 * 8);
  if (grid == 0) grid = 1;
  k_validate_queries<<<grid, 256, 0, st>>>(d_q, d_meta, nq, flag);
  g_launches += 1;
  return FKNN_OK;
}

static int check_query_flag(int flag) {
  if (!flag) return FKNN_OK;
  if (flag == ERR_PLAN_BOUND) {
    set_error("fknn_search: the device-built plan met a buffer bound (internal error; no output was written past it)");
    return FKNN_ECUDA;
  }
  std::string m = "fknn_search: ";
  if (flag & ERR_BAD_QUERY_TYPE) m += "query type not in {0,1,2,3}; ";
  if (flag & ERR_BAD_QUERY_VALUE) m += "query category outside int32 or NaN window bound; ";
  if (flag & ERR_BAD_QUERY_VEC) m += "query vector value not finite or above 1e15; ";
  set_error(m);
  return FKNN_EINVAL;
}

int count_matches(fknn_index *idx, const float *d_meta, uint32_t nq, uint32_t *d_counts, cudaStream_t st) {
  if (nq == 0) return FKNN_OK;
  (nq < QP_MANY ? k_count<true> : k_count<false>)<<<query_blocks(nq), QP_THREADS, 0, st>>>(
      d_meta, nq, (uint32_t)idx->n, idx->ord[ORDER_TIME].ts, idx->ord[ORDER_CAT].label, idx->ord[ORDER_CAT].ts, d_counts);
  g_launches += 1;
  FKNN_CUDA(cudaGetLastError());
  return FKNN_OK;
}

// Groups queries into tiles (shape.tq of them) whose slabs overlap (same order and
// predicate class, start bucket, then end), and cuts each tile's union
// range into row chunks.
namespace {

inline int bits_for(uint64_t v) {
  int b = 0;
  while (b < 64 && (v >> b)) ++b;
  return b;
}

// Sorts keys[0..m) of one query class by (bucket, e, s, qi).  The keys
// arrive in increasing qi and the LSD radix sort is stable, so qi needs no
// key bits; bucket, e and s are packed into one 64-bit key at their actual
// widths (under 49 bits at n = 1e6) and sorted with 11-bit digits, passes
// whose digit is constant skipped.  Wider packings use two 64-bit words.
void sort_class(PlanKey *keys, size_t m, Plan::SortScratch &W) {
  if (m < 2) return;
  uint32_t max_e = 0, max_s = 0, max_b = 0;
  for (size_t i = 0; i < m; ++i) {
    max_e = std::max(max_e, keys[i].e);
    max_s = std::max(max_s, keys[i].s);
    max_b = std::max<uint32_t>(max_b, (uint32_t)std::min<uint64_t>(keys[i].bucket, 0xffffffffu));
  }
  const int be = bits_for(max_e), bs = bits_for(max_s), bb = bits_for(max_b);
  const bool one_word = bb + be + bs <= 64;
  auto &hi = W.hi, &lo = W.lo, &hi2 = W.hi2, &lo2 = W.lo2;
  auto &ix = W.ix, &ix2 = W.ix2, &cnt = W.cnt;
  lo.resize(m);
  lo2.resize(m);
  ix.resize(m);
  ix2.resize(m);
  if (!one_word) {
    hi.resize(m);
    hi2.resize(m);
  }
  for (size_t i = 0; i < m; ++i) {
    const PlanKey &k = keys[i];
    if (one_word) {
      lo[i] = ((((uint64_t)k.bucket << be) | k.e) << bs) | k.s;
    } else {
      hi[i] = ((k.bucket & 0xffffffffull) << 32) | k.e;
      lo[i] = k.s;
    }
    ix[i] = (uint32_t)i;
  }
  constexpr int DB = 11, NB = 1 << DB;
  cnt.resize(NB + 1);
  const int words = one_word ? 1 : 2;
  for (int w = 0; w < words; ++w) {
    const int width = w == 0 ? (one_word ? bb + be + bs : 32) : 64;
    for (int shift = 0; shift < width; shift += DB) {
      std::vector<uint64_t> &src = w == 0 ? lo : hi;
      std::vector<uint64_t> &dst = w == 0 ? lo2 : hi2;
      std::fill(cnt.begin(), cnt.end(), 0u);
      for (size_t i = 0; i < m; ++i) ++cnt[((src[i] >> shift) & (NB - 1)) + 1];
      if (cnt[((src[0] >> shift) & (NB - 1)) + 1] == m) continue;  // one digit value: order unchanged
      for (int d = 0; d < NB; ++d) cnt[d + 1] += cnt[d];
      for (size_t i = 0; i < m; ++i) {
        const uint32_t pos = cnt[(src[i] >> shift) & (NB - 1)]++;
        dst[pos] = src[i];
        ix2[pos] = ix[i];
        if (w == 0 && !one_word) hi2[pos] = hi[i];
        if (w == 1) lo2[pos] = lo[i];
      }
      src.swap(dst);
      if (w == 0 && !one_word) hi.swap(hi2);
      if (w == 1) lo.swap(lo2);
      ix.swap(ix2);
    }
  }
  auto &out = W.out;
  out.resize(m);
  for (size_t i = 0; i < m; ++i) out[i] = keys[ix[i]];
  std::copy(out.begin(), out.end(), keys);
}

// Sorts plan keys by (order, cls, bucket, e, s, qi): a stable partition by
// class in (order, cls) order -- classes 0 and 2 on the time order, then 1
// and 3 on the category order -- and the classes' own sorts side by side
// on host threads.  Class 0 (no predicate) needs none: its keys are equal.
void sort_keys(std::vector<PlanKey> &keys, Plan &P) {
  const size_t m = keys.size();
  if (m < 2) return;
  static const int rank_of_cls[4] = {0, 2, 1, 3};  // (order, cls) order of the classes
  size_t start[5] = {0, 0, 0, 0, 0};
  for (const PlanKey &k : keys) ++start[rank_of_cls[k.cls & 3] + 1];
  for (int r = 0; r < 4; ++r) start[r + 1] += start[r];
  auto &part = P.w_keys2;
  part.resize(m);
  size_t fill[4] = {start[0], start[1], start[2], start[3]};
  for (const PlanKey &k : keys) part[fill[rank_of_cls[k.cls & 3]]++] = k;
  keys.swap(part);
  std::vector<std::thread> pool;
  for (int r = 1; r < 4; ++r) {
    const size_t len = start[r + 1] - start[r];
    if (len < 2) continue;
    if (len < 4096 || pool.size() == 2) {
      sort_class(keys.data() + start[r], len, P.w_sort[r]);
    } else {
      pool.emplace_back(sort_class, keys.data() + start[r], len, std::ref(P.w_sort[r]));
    }
  }
  for (auto &t : pool) t.join();
}

}  // namespace

void make_plan(const QueryDesc *desc, const float *meta_host, uint32_t nq, uint64_t n, const PlanShape &shape,
               Plan &P) {
  const int TQ = shape.tq, BLK = shape.blk_rows;
  P.reset();
  std::vector<uint32_t> &big = P.w_big;
  big.clear();
  for (uint32_t i = 0; i < nq; ++i) {
    const uint32_t len = desc[i].e - desc[i].s;
    P.pairs_passing += len;
    if (len <= (uint32_t)shape.small_slab) {
      P.small.push_back(i);
    } else {
      big.push_back(i);
      P.pairs_contraction += len;
    }
  }
  if (big.empty()) return;
  // start buckets: about sqrt(#queries/64) per class so a tile spans little
  const uint64_t nb_all = std::max<uint64_t>(1, (uint64_t)std::sqrt((double)big.size() / 64.0));
  const uint64_t bw = std::max<uint64_t>(BLK, (n + nb_all - 1) / nb_all);
  using Key = PlanKey;
  std::vector<Key> &keys = P.w_keys;
  keys.resize(big.size());
  for (size_t j = 0; j < big.size(); ++j) {
    const uint32_t i = big[j];
    const QueryDesc &d = desc[i];
    Key kk;
    kk.order = (uint32_t)d.order;
    kk.cls = (uint32_t)meta_host[(size_t)i * 4];
    kk.bucket = (kk.cls == 2 || kk.cls == 3) ? d.s / bw : 0;
    kk.s = d.s;
    kk.e = d.e;
    kk.qi = i;
    keys[j] = kk;
  }
  sort_keys(keys, P);
  // greedy tiles
  using TileTmp = PlanTile;
  std::vector<TileTmp> &tt = P.w_tiles;
  tt.clear();
  size_t i = 0;
  while (i < keys.size()) {
    TileTmp t{(uint32_t)i, 1, keys[i].s, keys[i].e, keys[i].order};
    uint32_t maxlen = keys[i].e - keys[i].s;
    size_t j = i + 1;
    while (j < keys.size() && t.count < TQ && keys[j].order == keys[i].order && keys[j].cls == keys[i].cls &&
           keys[j].bucket == keys[i].bucket) {
      const uint32_t S = std::min(t.S, keys[j].s), E = std::max(t.E, keys[j].e);
      const uint32_t ml = std::max(maxlen, keys[j].e - keys[j].s);
      if ((uint64_t)(E - S) > (uint64_t)ml + std::max<uint64_t>(ml / 3, 8192)) break;
      t.S = S;
      t.E = E;
      maxlen = ml;
      ++t.count;
      ++j;
    }
    tt.push_back(t);
    i = j;
  }
  // Row chunks per tile.  Every chunk restarts its candidate bound from the
  // shared one, so fewer, longer chunks mean fewer candidate pushes; a tile
  // is split only as far as needed to give every resident CTA slot several
  // work items (shape.target_items in total), and never below
  // min_chunk_blocks blocks or above max_items_per_tile chunks.
  uint64_t total_blk = 0;
  for (auto &t : tt) total_blk += (t.E + BLK - 1) / BLK - t.S / BLK;
  uint64_t cb = std::max<uint64_t>(1, total_blk / std::max<uint32_t>(1, shape.target_items));
  cb = std::max<uint64_t>(cb, shape.min_chunk_blocks);
  const size_t ntile = tt.size();
  P.tiles.resize(ntile);
  P.lane_q.assign(ntile * TQ, -1);
  P.lane_s.assign(ntile * TQ, 0);
  P.lane_e.assign(ntile * TQ, 0);
  P.big.reserve(big.size());
  P.big_tile.reserve(big.size());
  P.big_lane.reserve(big.size());
  std::vector<WorkItem> &items = P.w_items;
  items.clear();
  for (size_t t = 0; t < ntile; ++t) {
    const TileTmp &T = tt[t];
    for (uint32_t l = 0; l < T.count; ++l) {
      const Key &kk = keys[T.first + l];
      P.lane_q[t * TQ + l] = (int32_t)kk.qi;
      P.lane_s[t * TQ + l] = kk.s;
      P.lane_e[t * TQ + l] = kk.e;
      P.big.push_back(kk.qi);
      P.big_tile.push_back((uint32_t)t);
      P.big_lane.push_back(l);
    }
    const uint32_t b0 = T.S / BLK, b1 = (T.E + BLK - 1) / BLK;
    P.tiles[t].order = (int32_t)T.order;
    P.tiles[t].nq = T.count;
    const uint32_t cbt = std::max<uint32_t>((uint32_t)cb, (b1 - b0 + shape.max_items_per_tile - 1) / shape.max_items_per_tile);
    for (uint32_t b = b0; b < b1; b += cbt) {
      WorkItem w;
      w.tile = (uint32_t)t;
      w.blk0 = b;
      w.blk1 = std::min<uint32_t>(b1, b + cbt);
      w.pad = 0;
      items.push_back(w);
      P.pairs_screened += (uint64_t)(w.blk1 - w.blk0) * BLK * TQ;
    }
  }
  // Launch order: longest items first (the grid drains evenly), equal
  // lengths side by side by row range (L2 reuse of the row blocks).  A
  // tile's items are then spread out; the merge finds them through the
  // per-tile slot table built by the caller.
  std::stable_sort(items.begin(), items.end(), [&](const WorkItem &a, const WorkItem &b) {
    const uint32_t la = a.blk1 - a.blk0, lb = b.blk1 - b.blk0;
    if (la != lb) return la > lb;
    if (P.tiles[a.tile].order != P.tiles[b.tile].order) return P.tiles[a.tile].order < P.tiles[b.tile].order;
    return a.blk0 < b.blk0;
  });
  std::vector<uint32_t> &per_tile = P.w_per_tile;
  per_tile.assign(ntile + 1, 0);
  for (auto &w : items) per_tile[w.tile + 1]++;
  for (size_t t = 0; t < ntile; ++t) per_tile[t + 1] += per_tile[t];
  for (size_t t = 0; t < ntile; ++t) {
    P.tiles[t].item0 = per_tile[t];
    P.tiles[t].item1 = per_tile[t + 1];
  }
  P.items.swap(items);
}

int enqueue_query_prep(fknn_index *idx, const float *d_q, const float *d_meta, uint32_t nq, QueryDesc *d_desc,
                       cudaStream_t st) {
  int rc;
  if ((rc = validate_queries(idx, d_q, d_meta, nq, st))) return rc;
  (nq < QP_MANY ? k_query_prep<true> : k_query_prep<false>)<<<query_blocks(nq), QP_THREADS, 0, st>>>(
      d_q, d_meta, nq, (uint32_t)idx->n, idx->ord[ORDER_TIME].ts, idx->ord[ORDER_CAT].label, idx->ord[ORDER_CAT].ts, d_desc);
  g_launches += 1;
  FKNN_CUDA(cudaGetLastError());
  return FKNN_OK;
}

int check_query_flag_value(int flag) { return check_query_flag(flag); }

int prepare_queries(fknn_index *idx, const float *d_q, const float *d_meta, uint32_t nq, cudaStream_t st,
                    QueryDesc **d_desc_out, QueryDesc **h_desc_out, float **h_meta_out) {
  const uint64_t n = idx->n;
  int rc;
  QueryDesc *d_desc;
  if ((rc = ws_get(idx, 2, (size_t)nq * sizeof(QueryDesc), (void **)&d_desc))) return rc;
  if ((rc = validate_queries(idx, d_q, d_meta, nq, st))) return rc;
  (nq < QP_MANY ? k_query_prep<true> : k_query_prep<false>)<<<query_blocks(nq), QP_THREADS, 0, st>>>(
      d_q, d_meta, nq, (uint32_t)n, idx->ord[ORDER_TIME].ts, idx->ord[ORDER_CAT].label, idx->ord[ORDER_CAT].ts, d_desc);
  g_launches += 1;
  QueryDesc *h_desc;
  float *h_meta;
  int *h_flag;
  if ((rc = hs_get(idx, 0, (size_t)nq * sizeof(QueryDesc), (void **)&h_desc))) return rc;
  if ((rc = hs_get(idx, 1, (size_t)nq * 16, (void **)&h_meta))) return rc;
  if ((rc = hs_get(idx, 2, 64, (void **)&h_flag))) return rc;
  FKNN_CUDA(cudaMemcpyAsync(h_flag, idx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, st));
  FKNN_CUDA(cudaMemcpyAsync(h_desc, d_desc, (size_t)nq * sizeof(QueryDesc), cudaMemcpyDeviceToHost, st));
  FKNN_CUDA(cudaMemcpyAsync(h_meta, d_meta, (size_t)nq * 16, cudaMemcpyDeviceToHost, st));
  FKNN_CUDA(cudaStreamSynchronize(st));
  if ((rc = check_query_flag(*h_flag))) return rc;
  *d_desc_out = d_desc;
  *h_desc_out = h_desc;
  *h_meta_out = h_meta;
  return FKNN_OK;
}

// The queries of list, *d_count of them (d_count NULL: h_count); nmax: about how
// many that may be, 0: as a rule none, and with slabs of any length.
int launch_exact_scan(fknn_index *idx, const uint32_t *list, const uint32_t *d_count, uint32_t h_count, uint32_t nmax,
                      const QueryDesc *desc, const float *q, uint32_t k, uint32_t *ids, float *dists, cudaStream_t st) {
  const OrderData &OT = idx->ord[ORDER_TIME], &OC = idx->ord[ORDER_CAT];
  const bool many = nmax >= SCAN_MANY;
  const uint32_t grid = (uint32_t)idx->num_sms * (nmax ? 8 : 2);
  auto scan = many ? k_exact_scan<256, 2048> : k_exact_scan<512, 4096>;
  scan<<<d_count ? grid : std::min(h_count, grid), many ? 256 : 512, 0, st>>>(
      list, d_count, h_count, desc, q, OT.blocks, OC.blocks, OT.perm, OC.perm, k, ids, dists);
  g_launches += 1;
  FKNN_CUDA(cudaGetLastError());
  return FKNN_OK;
}

// The row-by-row exact scan of every query whose slab has at most
// SMALL_SLAB rows needs only the slabs, so it starts before the host plan,
// on the index's side stream (ordered after everything already on st), and
// runs while the host plans the rest.  Its rows of ids / dists are disjoint
// from the contraction's.  join_small_scans orders st after it.
int launch_small_scans(fknn_index *idx, const QueryDesc *h_desc, const QueryDesc *d_desc, uint32_t nq,
                       const float *d_q, uint32_t k, uint32_t *d_ids, float *d_dists, cudaStream_t st,
                       uint32_t *nsmall) {
  int rc;
  *nsmall = 0;
  uint32_t *h_list, *d_list;
  if ((rc = hs_get(idx, 4, (size_t)nq * 4 + 64, (void **)&h_list))) return rc;
  uint32_t m = 0;
  for (uint32_t i = 0; i < nq; ++i)
    if (h_desc[i].e - h_desc[i].s <= (uint32_t)SMALL_SLAB) h_list[m++] = i;
  *nsmall = m;
  if (!m) return FKNN_OK;
  if ((rc = ws_get(idx, 12, (size_t)m * 4 + 64, (void **)&d_list))) return rc;
  if (!idx->side_stream) FKNN_CUDA(cudaStreamCreateWithFlags(&idx->side_stream, cudaStreamNonBlocking));
  if (!idx->ev_fork) FKNN_CUDA(cudaEventCreateWithFlags(&idx->ev_fork, cudaEventDisableTiming));
  if (!idx->ev_join) FKNN_CUDA(cudaEventCreateWithFlags(&idx->ev_join, cudaEventDisableTiming));
  FKNN_CUDA(cudaEventRecord(idx->ev_fork, st));
  FKNN_CUDA(cudaStreamWaitEvent(idx->side_stream, idx->ev_fork, 0));
  FKNN_CUDA(cudaMemcpyAsync(d_list, h_list, (size_t)m * 4, cudaMemcpyHostToDevice, idx->side_stream));
  if ((rc = launch_exact_scan(idx, d_list, nullptr, m, m, d_desc, d_q, k, d_ids, d_dists, idx->side_stream)))
    return rc;
  FKNN_CUDA(cudaEventRecord(idx->ev_join, idx->side_stream));
  return FKNN_OK;
}

int join_small_scans(fknn_index *idx, cudaStream_t st) {
  if (idx->ev_join) FKNN_CUDA(cudaStreamWaitEvent(st, idx->ev_join, 0));
  return FKNN_OK;
}

int launch_fill_u32(uint32_t *p, uint32_t n, uint32_t v, cudaStream_t st) {
  k_fill_u32<<<std::min<uint32_t>((n + 255) / 256, 1024), 256, 0, st>>>(p, n, v);
  g_launches += 1;
  FKNN_CUDA(cudaGetLastError());
  return FKNN_OK;
}

int search_exact(fknn_index *idx, const float *d_q, const float *d_meta, uint32_t nq, uint32_t k, uint32_t *d_ids,
                 float *d_dists, cudaStream_t st, fknn_search_stats *stats) {
  const uint64_t n = idx->n;
  int rc;
  // 1. validate + resolve slabs
  QueryDesc *d_desc, *h_desc;
  float *h_meta;
  if ((rc = prepare_queries(idx, d_q, d_meta, nq, st, &d_desc, &h_desc, &h_meta))) return rc;
  uint32_t nsmall_early = 0;
  if ((rc = launch_small_scans(idx, h_desc, d_desc, nq, d_q, k, d_ids, d_dists, st, &nsmall_early))) return rc;

  // 2. plan
  auto t0 = std::chrono::steady_clock::now();
  Plan &P = idx->plan;
  PlanShape shape;
  shape.tq = EXACT_TQ;
  shape.blk_rows = EXACT_ROWS;
  shape.small_slab = SMALL_SLAB;
  // without a pilot every item of a tile may fill its list, and the merge holds MERGE_CAP entries
  const uint32_t pstride = idx->tuning[FKNN_MODE_EXACT_FP32].pilot_stride;
  const bool pilot = pstride > 1;
  shape.max_items_per_tile = pilot ? MAX_ITEMS_PER_TILE : MERGE_CAP / EXACT_CAP;
  shape.min_chunk_blocks = (idx->tuning[FKNN_MODE_EXACT_FP32].min_chunk_blocks + 1) / 2;  // (given in 64-row blocks)
  // Several items per SM even out tiles of unequal length; with few queries
  // there are few tiles, cut alike, and every further item only adds its own
  // start and end (100 queries over 1e6 rows: 0.86 ms at one item per SM, 0.99
  // at five; 1e4 queries over 1e5 rows: 3.5 ms at one, 3.2 at four).
  const uint32_t ips = items_per_sm(idx->tuning[FKNN_MODE_EXACT_FP32], FKNN_MODE_EXACT_FP32, nq);
  Candidate *d_out = nullptr, *d_work = nullptr;
  uint32_t *d_ocnt = nullptr, *d_state, sgrid = 0, nitems = 0;
  unsigned char *d_blob;
  if ((rc = ws_get(idx, 5, (size_t)nq * 36 + 64, (void **)&d_state))) return rc;
  // Where the index's HBM budget (or the memory left) does not hold the lists
  // of that many items and a working set for every SM, one item per tile and
  // as many CTAs as fit.
  for (int tight = 0;; ++tight) {
    shape.target_items = tight ? 1u : (uint32_t)idx->num_sms * ips;
    make_plan(h_desc, h_meta, nq, n, shape, P);
    nitems = (uint32_t)P.items.size();
    if (!nitems) break;
    // (the lists last: when tight, they take what is left)
    rc = ws_get(idx, 3, plan_blob_bytes(P), (void **)&d_blob);
    if (!rc) rc = ws_get(idx, 6, (size_t)nitems * EXACT_TQ * EXACT_CAP * sizeof(Candidate), (void **)&d_out);
    if (!rc) rc = ws_get(idx, 7, (size_t)nitems * EXACT_TQ * 4, (void **)&d_ocnt);
    if (!rc)
      for (sgrid = std::min<uint32_t>(nitems, (uint32_t)idx->num_sms);; sgrid = (sgrid + 1) / 2) {
        rc = ws_get(idx, 4, exact_work_bytes(sgrid), (void **)&d_work);
        if (rc != FKNN_ENOMEM || !tight || sgrid == 1) break;
        cudaGetLastError();
      }
    if (!rc) break;
    if (rc != FKNN_ENOMEM || tight) return rc;
    cudaGetLastError();  // (a refused allocation is not this call's error)
    for (int slot : {4, 6, 7, 11}) ws_drop(idx, slot);
  }
  auto t1 = std::chrono::steady_clock::now();
  const uint32_t ntile = (uint32_t)P.tiles.size();
  const uint32_t nbig = (uint32_t)P.big.size(), nsmall = (uint32_t)P.small.size();

  // item slots: the merge reads a tile's lists through tile.item0..item1 of
  // a slot table, the screen writes each item's lists at its launch slot.
  std::vector<uint32_t> &slot_of_tile_item = P.w_slot;
  slot_of_tile_item.resize(nitems);
  {
    std::vector<uint32_t> &fill = P.w_fill;
    fill.resize(ntile);
    for (uint32_t t = 0; t < ntile; ++t) fill[t] = P.tiles[t].item0;
    for (uint32_t s = 0; s < nitems; ++s) slot_of_tile_item[fill[P.items[s].tile]++] = s;
  }

  // 3. upload the plan as one blob
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t o = off;
    off = align_up(off + bytes, 256);
    return o;
  };
  const size_t o_small = take(nsmall * 4), o_big = take(nbig * 4), o_btile = take(nbig * 4),
               o_blane = take(nbig * 4), o_tiles = take(ntile * sizeof(Tile)), o_items = take(nitems * sizeof(WorkItem)),
               o_lq = take((size_t)ntile * EXACT_TQ * 4), o_ls = take((size_t)ntile * EXACT_TQ * 4),
               o_le = take((size_t)ntile * EXACT_TQ * 4), o_slot = take(nitems * 4);
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
  put(o_lq, P.lane_q.data(), (size_t)ntile * EXACT_TQ * 4);
  put(o_ls, P.lane_s.data(), (size_t)ntile * EXACT_TQ * 4);
  put(o_le, P.lane_e.data(), (size_t)ntile * EXACT_TQ * 4);
  put(o_slot, slot_of_tile_item.data(), nitems * 4);
  if (blob) FKNN_CUDA(cudaMemcpyAsync(d_blob, h_blob, blob, cudaMemcpyHostToDevice, st));

  // per-query state: bound, not-screened flag, overflow list; pilot bound
  // and flag; redo flag and list; spill lists of the two merges; then counts
  uint32_t *T_global = d_state, *ovf = d_state + nq, *ovf_list = d_state + 2 * (size_t)nq,
           *T_pilot = d_state + 3 * (size_t)nq, *ovf_p = d_state + 4 * (size_t)nq,
           *redo_skip = d_state + 5 * (size_t)nq, *redo_list = d_state + 6 * (size_t)nq,
           *spill = d_state + 7 * (size_t)nq, *spill2 = d_state + 8 * (size_t)nq, *counts = d_state + 9 * (size_t)nq;
  // counts: exact scans, redos, spills of the two merges, work queues of the three screens
  uint32_t *ovf_count = counts, *redo_count = counts + 1, *spill_count = counts + 2, *spill2_count = counts + 3,
           *queue = counts + 4;

  const OrderData &OT = idx->ord[ORDER_TIME], &OC = idx->ord[ORDER_CAT];
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
  if (stats) {
    for (auto &e : ev) FKNN_CUDA(cudaEventCreate(&e));
  }
  FKNN_CUDA(cudaMemsetAsync(counts, 0, 32, st));
  if (nitems) {
    // bounds start at +inf (as an order-preserving integer image)
    if ((rc = launch_fill_u32(T_global, nq, f32_sortable(INFINITY), st))) return rc;
    FKNN_CUDA(cudaMemsetAsync(ovf, 0, (size_t)nq * 4, st));
    // per device context, so set on every call (cheap)
    using SmallSmem = MergeSmem<MERGE_CAP_SMALL>;
    using LargeSmem = MergeSmem<MERGE_CAP>;
    FKNN_CUDA(cudaFuncSetAttribute(k_merge<MERGE_CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(LargeSmem)));
    if (stats) FKNN_CUDA(cudaEventRecord(ev[0], st));
    ExactScreenArgs A;
    A.items = (const WorkItem *)(d_blob + o_items);
    A.tiles = (const Tile *)(d_blob + o_tiles);
    A.lane_q = (const int32_t *)(d_blob + o_lq);
    A.lane_s = (const uint32_t *)(d_blob + o_ls);
    A.lane_e = (const uint32_t *)(d_blob + o_le);
    A.q = d_q;
    A.desc = d_desc;
    A.blocks_t = OT.blocks;
    A.blocks_c = OC.blocks;
    A.nblk = idx->nblk;
    A.work = d_work;
    A.out = d_out;
    A.out_cnt = d_ocnt;
    A.nitems = nitems;
    A.active = nullptr;
    A.err = idx->d_flag;
    const uint32_t *big_q = (const uint32_t *)(d_blob + o_big), *big_tile = (const uint32_t *)(d_blob + o_btile),
                   *big_lane = (const uint32_t *)(d_blob + o_blane), *item_slot = (const uint32_t *)(d_blob + o_slot);
    if (pilot) {
      // Pilot: the same screen over every pstride-th row block.  A rank in a
      // query's sample that lies a little above where the k-th of all its rows
      // ranks there (exact_seed_rank) seeds its bound; the merge finds the few
      // queries whose seed is below their k-th all the same, and the redo pass
      // below screens them again without one.  A seed admits a few times k
      // rows, a tenth of the pushes that tracking the k-th from nothing makes.
      // (the sample of a short slab is up to twice its nominal share)
      const uint32_t r = exact_seed_rank(k, 2, pstride);
      if ((rc = launch_fill_u32(T_pilot, nq, f32_sortable(INFINITY), st))) return rc;
      FKNN_CUDA(cudaMemsetAsync(ovf_p, 0, (size_t)nq * 4, st));
      FKNN_CUDA(cudaMemsetAsync(redo_skip, 0xff, (size_t)nq * 4, st));
      A.T_global = T_pilot;
      A.ovf = ovf_p;
      A.stride = pstride;
      A.k = r;
      A.queue = queue;
      if ((rc = launch_exact_screen(A, sgrid, st))) return rc;
      if ((rc = launch_exact_seed(big_q, big_tile, big_lane, nbig, A, item_slot, k, T_global, st))) return rc;
    }
    A.T_global = T_global;
    A.ovf = ovf;
    A.stride = 1;
    A.k = k;
    A.queue = queue + 1;
    if ((rc = launch_exact_screen(A, sgrid, st))) return rc;
    if (stats) FKNN_CUDA(cudaEventRecord(ev[1], st));
    ExactMergeArgs G;
    G.big_q = big_q;
    G.big_tile = big_tile;
    G.big_lane = big_lane;
    G.tiles = A.tiles;
    G.item_slot = item_slot;
    G.out = d_out;
    G.out_cnt = d_ocnt;
    G.desc = d_desc;
    G.q = d_q;
    G.vecs = idx->vecs;
    G.perm_t = OT.perm;
    G.perm_c = OC.perm;
    G.T_global = T_global;
    G.ovf = ovf;
    G.ovf_list = ovf_list;
    G.ovf_count = ovf_count;
    G.redo_list = pilot ? redo_list : nullptr;
    G.redo_count = redo_count;
    G.redo_skip = redo_skip;
    G.k = k;
    G.ids = d_ids;
    G.dists = d_dists;
    const unsigned lgrid = std::min<uint32_t>(nbig, (uint32_t)idx->num_sms * 2);
    k_merge<MERGE_CAP_SMALL><<<nbig, MG_THREADS, sizeof(SmallSmem), st>>>(G, nbig, nullptr, nullptr, spill,
                                                                          spill_count);
    k_merge<MERGE_CAP><<<lgrid, MG_THREADS, sizeof(LargeSmem), st>>>(G, 0, spill, spill_count, nullptr, nullptr);
    g_launches += 2;
    if (pilot) {
      // the same plan once more for the queries whose seed was too low, the
      // others (and the items without any such query) skipped
      A.ovf = redo_skip;
      A.active = redo_count;
      A.queue = queue + 2;
      if ((rc = launch_exact_screen(A, sgrid, st))) return rc;
      G.ovf = redo_skip;
      G.redo_list = nullptr;
      k_merge<MERGE_CAP_SMALL><<<lgrid, MG_THREADS, sizeof(SmallSmem), st>>>(G, 0, redo_list, redo_count, spill2,
                                                                             spill2_count);
      k_merge<MERGE_CAP><<<lgrid, MG_THREADS, sizeof(LargeSmem), st>>>(G, 0, spill2, spill2_count, nullptr, nullptr);
      g_launches += 2;
    }
  }
  if (stats) FKNN_CUDA(cudaEventRecord(ev[2], st));
  if (nbig) {
    if ((rc = launch_exact_scan(idx, ovf_list, ovf_count, 0, 0, d_desc, d_q, k, d_ids, d_dists, st))) return rc;
  }
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
    uint32_t h_ovf = 0;
    FKNN_CUDA(cudaMemcpyAsync(&h_ovf, ovf_count, 4, cudaMemcpyDeviceToHost, st));
    FKNN_CUDA(cudaStreamSynchronize(st));
    stats->n_overflow = h_ovf;
  }
  return FKNN_OK;
}

}  // namespace fknn

// ===================================================== no-allocation form
//
// fknn_filter_rows_noalloc: the predicate-compaction kernels above, for
// callers that must not allocate device memory.  Their only scratch (one
// counter per 4096-row tile plus the total) lives in the fixed array below,
// which the module holds on every GPU that loads this library until the
// process exits.

namespace fknn {

constexpr uint32_t NOALLOC_FILTER_MAX_TILES = 1u << 16;  // 65,536 tiles x 4,096 rows = 268,435,456 rows
constexpr uint64_t NOALLOC_FILTER_MAX_ROWS = (uint64_t)NOALLOC_FILTER_MAX_TILES * FC_TILE;
constexpr int NOALLOC_MAX_DEVICES = 64;

static __device__ __align__(256) uint32_t g_noalloc_filter_scratch[NOALLOC_FILTER_MAX_TILES + 1];

static std::mutex g_noalloc_mu;
static uint32_t *g_noalloc_ptr[NOALLOC_MAX_DEVICES];

// Device address of the scratch array on the current device.  The array's
// name in host code is only a host-side handle, so the address is looked up
// once per device (with that device current) and cached.
static int noalloc_scratch(uint32_t **out) {
  int dev = 0;
  FKNN_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
    set_error("fknn_filter_rows_noalloc: device ordinal above 63");
    return FKNN_EINVAL;
  }
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_filter_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_filter_scratch)");
    g_noalloc_ptr[dev] = static_cast<uint32_t *>(p);
  }
  *out = g_noalloc_ptr[dev];
  return FKNN_OK;
}

// True for device memory of device `dev` and for managed memory; false for
// host memory and for another GPU's memory (its kernels would read a peer's
// memory, which faults without peer access).
static bool on_device(const void *p, int dev) { return mem_loc(p, dev) == MemLoc::Here; }

}  // namespace fknn

extern "C" int fknn_filter_rows_noalloc(const float *labels, const float *ts, uint64_t n, const float *meta4,
                                        uint32_t *out_ids, uint64_t *count, void *stream) {
  using namespace fknn;
  g_launches = 0;
  if (!labels || !ts || !meta4 || !out_ids || !count) {
    set_error("fknn_filter_rows_noalloc: NULL argument");
    return FKNN_EINVAL;
  }
  if (n > NOALLOC_FILTER_MAX_ROWS) {
    set_error("fknn_filter_rows_noalloc: n = " + std::to_string(n) + " exceeds the fixed scratch limit of " +
              std::to_string(NOALLOC_FILTER_MAX_ROWS) + " rows (65,536 tiles of 4,096)");
    return FKNN_EINVAL;
  }
  const float t = meta4[0];
  if (!(t == 0.f || t == 1.f || t == 2.f || t == 3.f)) {
    set_error("fknn_filter_rows_noalloc: query type not in {0,1,2,3}");
    return FKNN_EINVAL;
  }
  if ((t == 1.f || t == 3.f) && !(fabsf(meta4[1]) < 2147483648.f)) {
    set_error("fknn_filter_rows_noalloc: category outside int32");
    return FKNN_EINVAL;
  }
  *count = 0;
  if (n == 0) return FKNN_OK;
  int cur = 0;
  FKNN_CUDA(cudaGetDevice(&cur));
  if (!on_device(labels, cur) || !on_device(ts, cur) || !on_device(out_ids, cur)) {
    set_error("fknn_filter_rows_noalloc: labels, ts and out_ids must be device memory of the current device");
    return FKNN_EINVAL;
  }
  uint32_t *tc = nullptr;
  int rc = noalloc_scratch(&tc);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const uint32_t ntiles = (uint32_t)((n + FC_TILE - 1) / FC_TILE);
  const float4 m = make_float4(meta4[0], meta4[1], meta4[2], meta4[3]);
  // every tile counter and the total are rewritten by this call, so nothing
  // left in the array by an earlier call is read
  k_filter_count<<<ntiles, FC_THREADS, 0, st>>>(labels, ts, n, m, tc);
  k_exclusive_scan_small<<<1, 1024, 0, st>>>(tc, ntiles, tc + ntiles);
  k_filter_write<<<ntiles, FC_THREADS, 0, st>>>(labels, ts, n, m, tc, out_ids);
  g_launches += 3;
  FKNN_CUDA(cudaGetLastError());
  uint32_t tot = 0;
  FKNN_CUDA(cudaMemcpyAsync(&tot, tc + ntiles, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  FKNN_CUDA(cudaStreamSynchronize(st));
  *count = tot;
  return FKNN_OK;
}
