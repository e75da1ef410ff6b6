// Batched graph beam search: the B200 form of the pyglass Searcher
// (pyglass/glass/searcher.hpp:162-569) over the reference's saved graphs.
//
// One warp runs one query at a time and replays the reference step for step,
// so on the same graph it returns the same ids:
//   * LinearPool (pyglass/glass/neighbor.hpp:223-283): a sorted array of
//     capacity max(k, ef) plus one overflow slot, zero-initialised; insertion
//     after equal distances (upper bound) with a shift of the tail; bit 31 of
//     the id is the checked flag and `cur` the first unchecked slot.  It
//     lives in shared memory.
//   * Bitset vis / vis1 (neighbor.hpp:41-102): lazily cleared 512-bit blocks;
//     the block flags are in shared memory, the bits in a per-warp global
//     bitmap read through L2.
//   * HNSWInitializer::initialize (HNSWInitializer.hpp:36-58): greedy descent
//     through the upper layers, the scanned list fixed for each pass.
//   * Distances: L2SqrSQ8_sym on the searcher's symmetric SQ8 codes, exact
//     int32.  The neighbours of a node are screened lane-parallel (visited
//     test, edge timestamp, distance) and enter the pool in adjacency order,
//     which is the order the reference inserts them in.
//
// k_graph_beam keeps the pool in two parts, the sorted array and up to 32
// entries not yet merged into it (struct Beam); k_graph_search keeps the
// sorted array alone and serves the calls that read the overflow slot
// (refine = max(k, ef) + 1), which only one-by-one insertion leaves as the
// reference does.
#include <algorithm>
#include <climits>
#include <cstring>
#include <new>
#include <vector>

#include "device_util.cuh"

struct fknn_graph {
  int device = 0;
  uint32_t n = 0, K = 0, upK = 1, nep = 0;
  int32_t ep = -1;
  int32_t *adj = nullptr;     // [n][K] neighbour ids, -1 from a list's end on, -2 for an id listed before
  float *ets = nullptr;       // [n][K] edge timestamps
  int32_t *levels = nullptr;  // [n] upper-layer count per node
  int64_t *up_off = nullptr;  // [n + 1] offsets into up
  int32_t *up = nullptr;      // per node levels * upK ids, level 1 first
  int32_t *eps = nullptr;     // [nep] entry points (graphs without upper layers)
  int8_t *codes = nullptr;    // [n][112] symmetric SQ8 codes, bytes 100..103 the code's squared norm
  float alpha = 0.f;
  // per-call scratch, grown on demand
  float *io = nullptr;        // staged queries, bounds, outputs
  size_t io_cap = 0;
  int8_t *qcodes = nullptr;
  size_t qcodes_cap = 0;
  uint64_t *vis = nullptr;    // per warp slot: two bitmaps of nwords words
  size_t vis_cap = 0;
  int *dflag = nullptr;
};

namespace fknn {
namespace {

constexpr int GS_WARPS = 4;  // warps per block, one query in flight each
constexpr int CODE = 112;    // SQ8 code bytes per point (100 dims aligned to 16)
constexpr int EF_DEFAULT = 32;
constexpr uint32_t CAP_MAX = 4096;
constexpr int GS_OCC_BLOCKS = 8;                 // blocks per SM of the register-capped variant
constexpr int GS_SV_BLOCKS = 5;                  // ... with the visited bits in shared memory,
constexpr int GS_SV_RANGED_BLOCKS = 4;           // ... and a window (few blocks fit; no spills)
constexpr int GS_BASE_BLOCKS = 6;                // ... and of the default one (the registers it needs)
constexpr size_t GS_SMEM_PER_SM = 228 * 1024;    // shared memory of an SM
constexpr size_t VIS_BUDGET = 4ull << 30;  // bytes of visited bitmaps across all warp slots

struct Slot {  // one LinearPool entry; bit 31 of id = checked
  int d;
  int id;
};

struct GParams {
  const int32_t *adj;
  const float *ets;
  const int32_t *levels;
  const int64_t *up_off;
  const int32_t *up;
  const int32_t *eps;
  const int8_t *codes;
  uint32_t n, K, upK, nep;
  int32_t ep;
  float alpha2;
  const int8_t *qcodes;
  uint32_t nq;
  int mode;
  uint32_t cap, refine;
  const float *bounds;
  const int32_t *id_bounds;
  int32_t *out_ids;
  float *out_dists;
  uint64_t *vis;
  uint32_t nwords;  // 64-bit words per bitmap: whole 512-bit blocks
  uint32_t nblkw;   // 32-bit words of block flags per bitmap
  uint32_t nvw;     // 32-bit words of a bitmap in shared memory
  bool v1s;         // vis1 is in shared memory
  int *err;
};

struct Warp {
  Slot *pool;
  uint32_t *chg;   // block flags [2][nblkw]
  int *qw;         // query code as 28 words
  uint64_t *mass;  // bitmaps [2][nwords]
  int qq;
  uint32_t size, cur;
};

__host__ __device__ inline size_t pool_bytes(uint32_t cap) {
  return ((size_t)(cap + 1) * sizeof(Slot) + 15) & ~(size_t)15;
}

__host__ __device__ inline size_t warp_smem_bytes(uint32_t cap, uint32_t nblkw) {
  return pool_bytes(cap) + 2 * (size_t)nblkw * 4 + CODE;
}

__device__ __forceinline__ int gdist(const GParams &P, const Warp &W, uint32_t v) {
  return sq8_dist(W.qw, W.qq, P.codes + (uint64_t)v * CODE);
}

// Bitset::get (neighbor.hpp:88-92) of set b (0 = vis, 1 = vis1).
__device__ __forceinline__ bool vis_get(const GParams &P, const Warp &W, int b, uint32_t v) {
  const uint32_t blk = v >> 9;
  if (!((W.chg[b * P.nblkw + (blk >> 5)] >> (blk & 31)) & 1u)) return false;
  return (__ldcg(reinterpret_cast<const unsigned long long *>(W.mass + (uint64_t)b * P.nwords + (v >> 6))) >>
          (v & 63)) & 1ull;
}

// Bitset::set (neighbor.hpp:80-87) for the lanes with `on`, whole warp: a
// block seen for the first time is cleared, then (after the warp barrier
// that orders the clears) the bits are set.
__device__ __forceinline__ void vis_set(const GParams &P, const Warp &W, int b, uint32_t v, bool on) {
  uint64_t *m = W.mass + (uint64_t)b * P.nwords;
  if (on) {
    const uint32_t blk = v >> 9, bit = 1u << (blk & 31);
    if (!(atomicOr(&W.chg[b * P.nblkw + (blk >> 5)], bit) & bit)) {
#pragma unroll
      for (int w = 0; w < 8; ++w) __stcg(reinterpret_cast<unsigned long long *>(m + (uint64_t)blk * 8 + w), 0ull);
    }
  }
  __syncwarp();
  if (on) atomicOr(reinterpret_cast<unsigned long long *>(m + (v >> 6)), 1ull << (v & 63));
  __syncwarp();
}

// LinearPool::insert (neighbor.hpp:240-255), whole warp, warp-uniform arguments.
__device__ void pool_insert(Warp &W, uint32_t cap, int u, int d) {
  const int lane = threadIdx.x & 31;
  if (W.size == cap && d >= W.pool[W.size - 1].d) return;
  uint32_t lo = 0, hi = W.size;  // first slot whose distance exceeds d
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (W.pool[mid].d > d) hi = mid;
    else lo = mid + 1;
  }
  // move [lo, size) up one slot, top chunk first (slot `size` may be the overflow slot)
  for (int top = (int)W.size - 1; top >= (int)lo; top -= 32) {
    const int idx = top - lane;
    Slot t;
    if (idx >= (int)lo) t = W.pool[idx];
    __syncwarp();
    if (idx >= (int)lo) W.pool[idx + 1] = t;
    __syncwarp();
  }
  if (lane == 0) {
    Slot s;
    s.d = d;
    s.id = u;
    W.pool[lo] = s;
  }
  __syncwarp();
  if (W.size < cap) ++W.size;
  if (lo < W.cur) W.cur = lo;
}

// LinearPool::pop (neighbor.hpp:259-266), whole warp.
__device__ int pool_pop(Warp &W) {
  const int lane = threadIdx.x & 31;
  const uint32_t pre = W.cur;
  const int raw = W.pool[pre].id;
  __syncwarp();
  if (lane == 0) W.pool[pre].id = raw | (int)0x80000000;
  __syncwarp();
  uint32_t c = pre;
  while (c < W.size) {
    const uint32_t idx = c + lane;
    const uint32_t b = __ballot_sync(0xffffffffu, idx < W.size && W.pool[idx].id >= 0);
    if (b) {
      c += __ffs(b) - 1;
      break;
    }
    c = min(c + 32, W.size);
  }
  W.cur = c;
  return raw & 0x7fffffff;
}

// Lanes of one 32-wide chunk of an adjacency list: `valid` for the points the
// reference looks at, each id once (a later copy is already visited when the
// reference reaches it; k_graph_lists leaves only the first).
struct Chunk {
  int v;
  bool valid, end;
};

__device__ __forceinline__ Chunk chunk_of(int v) {
  Chunk c;
  c.v = v;
  c.valid = v >= 0;
  c.end = __any_sync(0xffffffffu, v == -1);
  return c;
}

__device__ __forceinline__ Chunk load_chunk(const int32_t *list, uint32_t len, uint32_t base) {
  const uint32_t i = base + (threadIdx.x & 31);
  return chunk_of(i < len ? list[i] : -1);
}

// At load time, one warp per point: each list -1 from its first -1 on, and -2
// in place of an id that an earlier entry of its 32-entry chunk names.
__global__ void k_graph_lists(int32_t *__restrict__ adj, uint32_t n, uint32_t K) {
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t u = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); u < n; u += warps) {
    int32_t *list = adj + (uint64_t)u * K;
    bool ended = false;
    for (uint32_t base = 0; base < K; base += 32) {
      const uint32_t i = base + lane;
      int v = i < K ? list[i] : -1;
      const uint32_t endb = __ballot_sync(0xffffffffu, v == -1);
      if (ended || (endb && lane >= __ffs(endb) - 1)) v = -1;
      const bool first = (__ffs(__match_any_sync(0xffffffffu, v)) - 1) == lane;
      if (v >= 0 && !first) v = -2;
      if (i < K) list[i] = v;
      ended = ended || endb != 0;
    }
  }
}

// bytes 100..103 of every code: its squared norm (padding in every SQ8 code)
__global__ void k_code_norms(int8_t *__restrict__ codes, uint32_t n) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int *c = reinterpret_cast<int *>(codes + (uint64_t)i * CODE);
    int cc = 0;
    for (int w = 0; w < DIM / 4; ++w) cc = __dp4a(c[w], c[w], cc);
    c[DIM / 4] = cc;
  }
}

// Inserts the lanes of mask m in lane order (the adjacency order).
__device__ __forceinline__ int insert_lanes(const GParams &P, Warp &W, uint32_t m, int v, int d) {
  const int count = __popc(m);
  while (m) {
    const int b = __ffs(m) - 1;
    m &= m - 1;
    pool_insert(W, P.cap, __shfl_sync(0xffffffffu, v, b), __shfl_sync(0xffffffffu, d, b));
  }
  return count;
}

// SearchImpl / SearchFilterImpl / SearchFilterSubTimeImpl (searcher.hpp:172-198,
// 271-299, 386-413): every unvisited neighbour is marked and inserted.
// (SearchFilterImpl's `count1 > count2` exit can never fire: both counts
// grow together.)
__device__ void expand_plain(const GParams &P, Warp &W, uint32_t u) {
  const int32_t *list = P.adj + (uint64_t)u * P.K;
  for (uint32_t base = 0; base < P.K; base += 32) {
    const Chunk c = load_chunk(list, P.K, base);
    const bool fresh = c.valid && !vis_get(P, W, 0, (uint32_t)c.v);
    const int d = fresh ? gdist(P, W, (uint32_t)c.v) : 0;
    vis_set(P, W, 0, (uint32_t)c.v, fresh);
    insert_lanes(P, W, __ballot_sync(0xffffffffu, fresh), c.v, d);
    if (c.end) break;
  }
}

// SearchCategoryRangeImpl (rf = 1, searcher.hpp:320-374) and
// SearchRangeFilter[SubTime]Impl (rf = 2, searcher.hpp:438-491, 516-569): an
// unvisited neighbour is always marked, but inserted only when the edge's
// timestamp lies in [l, r]; while inserts < rf x (unvisited 1-hop
// neighbours), the neighbours' own lists are scanned the same way, stopping
// right after the insert that reaches the bound.
__device__ void expand_filtered(const GParams &P, Warp &W, uint32_t u, float l, float r, int rf) {
  const int lane = threadIdx.x & 31;
  const int32_t *list = P.adj + (uint64_t)u * P.K;
  const float *tlist = P.ets + (uint64_t)u * P.K;
  int count1 = 0, count2 = 0;
  for (uint32_t base = 0; base < P.K; base += 32) {
    const Chunk c = load_chunk(list, P.K, base);
    const bool fresh = c.valid && !vis_get(P, W, 0, (uint32_t)c.v);
    const float t = fresh ? tlist[base + lane] : 0.f;
    const bool pass = fresh && !(t < l || t > r);
    const int d = pass ? gdist(P, W, (uint32_t)c.v) : 0;
    vis_set(P, W, 0, (uint32_t)c.v, fresh);
    count2 += __popc(__ballot_sync(0xffffffffu, fresh));
    count1 += insert_lanes(P, W, __ballot_sync(0xffffffffu, pass), c.v, d);
    if (c.end) break;
  }
  for (uint32_t i = 0; i < P.K; ++i) {
    if (count1 >= rf * count2) break;
    const int nei = list[i];
    if (nei == -1) break;
    if (nei < 0) continue;  // listed before
    if (vis_get(P, W, 1, (uint32_t)nei)) continue;
    vis_set(P, W, 1, (uint32_t)nei, lane == 0);
    const int32_t *list2 = P.adj + (uint64_t)nei * P.K;
    const float *tlist2 = P.ets + (uint64_t)nei * P.K;
    for (uint32_t base = 0; base < P.K; base += 32) {
      const Chunk c = load_chunk(list2, P.K, base);
      const bool fresh = c.valid && !vis_get(P, W, 0, (uint32_t)c.v);
      const float t = fresh ? tlist2[base + lane] : 0.f;
      const bool pass = fresh && !(t < l || t > r);
      const uint32_t passm = __ballot_sync(0xffffffffu, pass);
      // the scan stops after the need-th insert: lanes past it are untouched
      const int need = rf * count2 - count1;
      uint32_t upto = 0xffffffffu;
      bool stop = false;
      if (__popc(passm) >= need) {
        uint32_t mm = passm;
        for (int j = 1; j < need; ++j) mm &= mm - 1;
        const int last = __ffs(mm) - 1;
        upto = last == 31 ? 0xffffffffu : ((2u << last) - 1u);
        stop = true;
      }
      const bool mine = (upto >> lane) & 1u;
      const int d = (pass && mine) ? gdist(P, W, (uint32_t)c.v) : 0;
      vis_set(P, W, 0, (uint32_t)c.v, fresh && mine);
      count1 += insert_lanes(P, W, passm & upto, c.v, d);
      if (stop || c.end) break;
    }
  }
}

// Graph::initialize_search (graph.hpp:90-99): HNSWInitializer::initialize
// when the graph has upper layers (insert the descent's end, then mark it),
// else every entry point inserted, unmarked.
__device__ void initialize_search(const GParams &P, Warp &W) {
  const int lane = threadIdx.x & 31;
  if (P.ep >= 0) {
    int u = P.ep;
    int cur_dist = gdist(P, W, (uint32_t)u);
    for (int level = P.levels[u]; level > 0; --level) {
      bool changed = true;
      while (changed) {
        changed = false;
        const int32_t *list = P.up + P.up_off[u] + (int64_t)(level - 1) * P.upK;
        for (uint32_t base = 0; base < P.upK; base += 32) {
          const uint32_t i = base + lane;
          const int v = i < P.upK ? list[i] : -1;
          const uint32_t endb = __ballot_sync(0xffffffffu, v == -1);
          const bool valid = endb ? lane < __ffs(endb) - 1 : true;
          const int d = valid ? gdist(P, W, (uint32_t)v) : 0;
          uint32_t m = __ballot_sync(0xffffffffu, valid);
          while (m) {  // the reference's sequential scan: a strictly closer point moves u
            const int b = __ffs(m) - 1;
            m &= m - 1;
            const int db = __shfl_sync(0xffffffffu, d, b);
            const int vb = __shfl_sync(0xffffffffu, v, b);
            if (db < cur_dist) {
              cur_dist = db;
              u = vb;
              changed = true;
            }
          }
          if (endb) break;
        }
      }
    }
    pool_insert(W, P.cap, u, cur_dist);
    vis_set(P, W, 0, (uint32_t)u, lane == 0);
  } else {
    for (uint32_t e = 0; e < P.nep; ++e) {
      const int v = P.eps[e];
      pool_insert(W, P.cap, v, gdist(P, W, (uint32_t)v));
    }
  }
}

// Ten evenly spaced seeds of the id range (searcher.hpp:306-313, 421-430,
// 499-508): insert, then mark; a range narrower than ten repeats its start.
__device__ void range_seeds(const GParams &P, Warp &W, int lb, int ub) {
  const int lane = threadIdx.x & 31;
  const int interval = (ub - lb) / 10;
  for (int i = 0; i < 10; ++i) {
    const int point = lb + interval * i;
    pool_insert(W, P.cap, point, gdist(P, W, (uint32_t)point));
    vis_set(P, W, 0, (uint32_t)point, lane == 0);
  }
}

__global__ void __launch_bounds__(GS_WARPS * 32) k_graph_search(GParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  unsigned char *mine = smem_raw + wib * warp_smem_bytes(P.cap, P.nblkw);
  Warp W;
  W.pool = reinterpret_cast<Slot *>(mine);
  W.chg = reinterpret_cast<uint32_t *>(mine + pool_bytes(P.cap));
  W.qw = reinterpret_cast<int *>(W.chg + 2 * P.nblkw);
  const uint32_t slot = blockIdx.x * GS_WARPS + wib;
  W.mass = P.vis + (uint64_t)slot * 2 * P.nwords;
  for (uint32_t qi = slot; qi < P.nq; qi += gridDim.x * GS_WARPS) {
    for (uint32_t i = lane; i <= P.cap; i += 32) {
      Slot z;
      z.d = 0;
      z.id = 0;
      W.pool[i] = z;
    }
    for (uint32_t i = lane; i < 2 * P.nblkw; i += 32) W.chg[i] = 0;
    if (lane < 28) W.qw[lane] = reinterpret_cast<const int *>(P.qcodes + (uint64_t)qi * CODE)[lane];
    __syncwarp();
    int qq = 0;
    for (int w = 0; w < 28; ++w) qq = __dp4a(W.qw[w], W.qw[w], qq);
    W.qq = qq;
    W.size = 0;
    W.cur = 0;
    const bool ranged = P.mode >= FKNN_GRAPH_CATEGORY_RANGE;
    const float l = ranged ? P.bounds[2 * (uint64_t)qi] : 0.f;
    const float r = ranged ? P.bounds[2 * (uint64_t)qi + 1] : 0.f;
    const int lb = ranged ? P.id_bounds[2 * (uint64_t)qi] : 0;
    const int ub = ranged ? P.id_bounds[2 * (uint64_t)qi + 1] : 0;
    // float sel = (float)(ub - lb) / nb; seeds only when sel < 1
    const bool partial = __fdiv_rn((float)(ub - lb), (float)P.n) < 1.f;
    const bool seeded = P.mode == FKNN_GRAPH_CATEGORY_RANGE || (P.mode >= FKNN_GRAPH_RANGE_SUBTIME && partial);
    bool bad = false;
    if (seeded) {  // every seed lb + i * ((ub - lb) / 10), i < 10, must be a point
      const long long last = (long long)lb + 9ll * ((ub - lb) / 10);
      bad = lb < 0 || (uint32_t)lb >= P.n || last < 0 || last >= (long long)P.n;
    }
    if (bad) {
      if (lane == 0) atomicOr(P.err, ERR_BAD_QUERY_VALUE);
      for (uint32_t i = lane; i < P.refine; i += 32) {
        P.out_ids[(uint64_t)qi * P.refine + i] = -1;
        if (P.out_dists) P.out_dists[(uint64_t)qi * P.refine + i] = __int_as_float(0x7fc00000);
      }
      __syncwarp();
      continue;
    }
    if (seeded) range_seeds(P, W, lb, ub);
    else if (P.mode != FKNN_GRAPH_RANGE_SUBTIME) initialize_search(P, W);
    // each pop checks one slot; an expansion inserts each point at most once
    // (vis), besides at most ten seeds and the unmarked entry points, so
    // n + nep + 16 pops is a hard bound
    uint32_t pops = 0;
    while (W.cur < W.size) {
      if (++pops > P.n + P.nep + 16) {
        if (lane == 0) atomicOr(P.err, ERR_WAIT_TIMEOUT);
        break;
      }
      const int u = pool_pop(W);
      if (P.mode == FKNN_GRAPH_CATEGORY_RANGE) expand_filtered(P, W, (uint32_t)u, l, r, 1);
      else if (P.mode >= FKNN_GRAPH_RANGE_SUBTIME) expand_filtered(P, W, (uint32_t)u, l, r, 2);
      else expand_plain(P, W, (uint32_t)u);
    }
    // reorder / reorder_dist (sq8_sym_quant.hpp:76-89): slots 0..refine-1 as
    // they stand, ids unmasked, distances times alpha^2
    for (uint32_t i = lane; i < P.refine; i += 32) {
      const Slot s = W.pool[i];
      P.out_ids[(uint64_t)qi * P.refine + i] = s.id & 0x7fffffff;
      if (P.out_dists) P.out_dists[(uint64_t)qi * P.refine + i] = __fmul_rn((float)s.d, P.alpha2);
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------------
// The beam search with a lazily merged pool.
//
// LinearPool is a priority queue ordered by (distance, insertion), cut at cap
// entries.  Keeping it one sorted array costs a pass over the array per
// expansion: measured at cap 2,500, 9,900 of 13,800 cycles a pop.  Here new
// entries go to a short unsorted buffer in insertion order, a pop takes the
// smallest unchecked entry of both (array entries first among equals: they
// are older), and the buffer is merged when it is full, in one pass for
// about ten pops.  An entry past the cap-th of the union is evicted or
// rejected in the reference and never pops there; here it may sit in the
// buffer until the next merge cuts it off, so a pop checks its rank in the
// union (only more entries can come before it, never fewer).
//
// The second hop of the filtered forms scans list after list: each list, the
// visited bits of its points and the codes of its unvisited points inside the
// window are on their way while the lists before it are handled.

constexpr int BUF = 32;  // unmerged entries

struct Beam {
  Slot *pool;  // sorted array of cap slots
  Slot *buf;   // [BUF] entries since the last merge, in insertion order
  int4 *qw;    // the query's code
  uint32_t *vis, *vis1;  // the two sets: bits in shared memory (vis: SV, vis1: P.v1s), or the block flags of ...
  uint64_t *mass;        // ... bitmaps in global memory [2][nwords]
  int qq, lastd;   // |q|^2; the cap-th distance once the array is full, else INT_MAX
  uint32_t size, cur, nb;
};

__host__ __device__ inline size_t beam_smem_bytes(uint32_t cap, uint32_t vis_words) {
  return (((size_t)(cap + BUF) * sizeof(Slot) + 15) & ~(size_t)15) + CODE + (((size_t)vis_words * 4 + 15) & ~(size_t)15);
}

__device__ __forceinline__ void load_code7(const int8_t *__restrict__ code, int4 (&c)[7]) {
  const int4 *p = reinterpret_cast<const int4 *>(code);
#pragma unroll
  for (int w = 0; w < 7; ++w) c[w] = __ldg(p + w);
}

// |q|^2 + |c|^2 - 2 q.c, |c|^2 from the code's bytes 100..103
__device__ __forceinline__ int dist7(const Beam &W, const int4 (&c)[7]) {
  int a = 0, b = 0;
#pragma unroll
  for (int w = 0; w < 6; ++w) {
    const int4 q = W.qw[w];
    a = __dp4a(q.x, c[w].x, a);
    b = __dp4a(q.y, c[w].y, b);
    a = __dp4a(q.z, c[w].z, a);
    b = __dp4a(q.w, c[w].w, b);
  }
  a = __dp4a(W.qw[6].x, c[6].x, a);
  return W.qq + c[6].y - 2 * (a + b);
}

__device__ __forceinline__ int beam_dist(const GParams &P, const Beam &W, uint32_t v) {
  int4 c[7];
  load_code7(P.codes + (uint64_t)v * CODE, c);
  return dist7(W, c);
}

// Bitset::get / set (neighbor.hpp:80-92): bits in shared memory, or in the
// global bitmap `mass` with the lazily cleared blocks' flags in `flags`
__device__ __forceinline__ bool bit_get(const uint32_t *bits, uint32_t v) { return (bits[v >> 5] >> (v & 31)) & 1u; }
__device__ __forceinline__ uint64_t mass_word(const uint32_t *flags, const uint64_t *mass, uint32_t v) {
  const uint32_t blk = v >> 9;
  if (!((flags[blk >> 5] >> (blk & 31)) & 1u)) return 0;
  return __ldcg(reinterpret_cast<const unsigned long long *>(mass + (v >> 6)));
}
// whole warp, for the lanes with `on`
__device__ __forceinline__ void bit_set(uint32_t *bits, uint32_t v, bool on) {
  if (on) atomicOr(&bits[v >> 5], 1u << (v & 31));
  __syncwarp();
}
__device__ __forceinline__ void mass_set(uint32_t *flags, uint64_t *mass, uint32_t v, bool on) {
  if (on) {
    const uint32_t blk = v >> 9, bit = 1u << (blk & 31);
    if (!(atomicOr(&flags[blk >> 5], bit) & bit)) {
#pragma unroll
      for (int w = 0; w < 8; ++w) __stcg(reinterpret_cast<unsigned long long *>(mass + (uint64_t)blk * 8 + w), 0ull);
    }
  }
  __syncwarp();
  if (on) atomicOr(reinterpret_cast<unsigned long long *>(mass + (v >> 6)), 1ull << (v & 63));
  __syncwarp();
}
// of vis (the points met) ...
template <bool SV>
__device__ __forceinline__ bool beam_get(const Beam &W, uint32_t v) {
  return SV ? bit_get(W.vis, v) : (mass_word(W.vis, W.mass, v) >> (v & 63)) & 1ull;
}
template <bool SV>
__device__ __forceinline__ void beam_set(const Beam &W, uint32_t v, bool on) {
  if (SV) bit_set(W.vis, v, on);
  else mass_set(W.vis, W.mass, v, on);
}
// ... and vis1 (the lists scanned in a second hop)
__device__ __forceinline__ bool beam_get1(const GParams &P, const Beam &W, uint32_t v) {
  return P.v1s ? bit_get(W.vis1, v) : (mass_word(W.vis1, W.mass + P.nwords, v) >> (v & 63)) & 1ull;
}
__device__ __forceinline__ void beam_set1(const GParams &P, const Beam &W, uint32_t v) {  // warp-uniform v
  const bool on = (threadIdx.x & 31) == 0;
  if (P.v1s) bit_set(W.vis1, v, on);
  else mass_set(W.vis1, W.mass + P.nwords, v, on);
}

// array entries with distance <= d among the first hi (32 lanes, each its own d)
__device__ __forceinline__ uint32_t beam_upper(const Slot *pool, uint32_t hi, int d) {
  uint32_t lo = 0;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (pool[mid].d > d) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

// The buffer into the array: sorted by (distance, insertion), every old entry
// moved up by the number of strictly closer new ones (128 read before they
// are written, top first), every new one written at its rank plus
// the old entries not farther; entries past cap fall off.
// (Values in and out, so that the caller's state stays in registers.)
__device__ __noinline__ uint2 beam_merge_parts(Slot *pool, const Slot *buf, uint32_t size, uint32_t first_unchecked,
                                               int n, uint32_t cap) {
  const int lane = threadIdx.x & 31;
  const Slot mine = lane < n ? buf[lane] : Slot{0, 0};
  uint32_t key = lane < n ? ((uint32_t)mine.d << 5) | (uint32_t)lane : 0xffffffffu;
#pragma unroll
  for (int sz = 2; sz <= 32; sz <<= 1)
#pragma unroll
    for (int stride = sz >> 1; stride > 0; stride >>= 1) {
      const uint32_t other = __shfl_xor_sync(0xffffffffu, key, stride);
      const bool asc = (lane & sz) == 0, lower = (lane & stride) == 0;
      key = (lower == asc) ? min(key, other) : max(key, other);
    }
  const int cid = __shfl_sync(0xffffffffu, mine.id, (int)(key & 31));
  const int cd = lane < n ? (int)(key >> 5) : INT_MAX;
  const uint32_t ub = lane < n ? beam_upper(pool, size, cd) : 0xffffffffu;
  const uint32_t first = __shfl_sync(0xffffffffu, ub, 0);  // entries below it do not move
  // An old entry i moves up by the new entries j with ub_j <= i.  The first
  // unchecked one of the array, after its move, and of the buffer:
  uint32_t cur = 0xffffffffu;
  if (first_unchecked < size)
    cur = first_unchecked + __popc(__ballot_sync(0xffffffffu, ub <= first_unchecked));
  const uint32_t bcur = __reduce_min_sync(0xffffffffu, lane < n && cid >= 0 ? ub + (uint32_t)lane : 0xffffffffu);
  for (int top = (int)size; top > (int)first; top -= 128) {
    Slot t[4];
    uint32_t ni[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = top - 1 - c * 32 - lane;
      t[c] = i >= (int)first ? pool[i] : Slot{0, 0};
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      // all of the chunk's entries move alike unless a new one lands among them
      const int hi = top - 1 - c * 32, lo = hi - 31, i = hi - lane;
      const uint32_t below = __ballot_sync(0xffffffffu, (int)ub <= lo && ub != 0xffffffffu);
      uint32_t among = __ballot_sync(0xffffffffu, (int)ub <= hi && ub != 0xffffffffu) & ~below;
      int s = __popc(below);
      while (among) {
        const int j = __ffs(among) - 1;
        among &= among - 1;
        s += (int)__shfl_sync(0xffffffffu, ub, j) <= i ? 1 : 0;
      }
      ni[c] = i >= (int)first ? (uint32_t)(i + s) : cap;
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (ni[c] < cap) pool[ni[c]] = t[c];
    __syncwarp();
  }
  if (lane < n && ub + (uint32_t)lane < cap) pool[ub + lane] = Slot{cd, cid};
  __syncwarp();
  size = min(size + (uint32_t)n, cap);
  return make_uint2(size, min(min(cur, bcur), size));
}
__device__ __forceinline__ void beam_merge(Beam &W, uint32_t cap) {
  if (!W.nb) return;
  const uint2 r = beam_merge_parts(W.pool, W.buf, W.size, W.cur, (int)W.nb, cap);
  W.size = r.x;
  W.cur = r.y;
  W.nb = 0;
  W.lastd = W.size == cap ? W.pool[cap - 1].d : INT_MAX;
}

// The lanes of mask m, in lane order (the adjacency order).
__device__ __forceinline__ void beam_insert(Beam &W, uint32_t cap, uint32_t m, int v, int d) {
  const int lane = threadIdx.x & 31;
  // a full pool rejects what is not closer than its last (LinearPool::insert)
  m &= __ballot_sync(0xffffffffu, d < W.lastd);
  if (!m) return;
  if (W.nb + __popc(m) > BUF) {
    beam_merge(W, cap);
    m &= __ballot_sync(0xffffffffu, d < W.lastd);
  }
  if ((m >> lane) & 1u) W.buf[W.nb + __popc(m & ((1u << lane) - 1u))] = Slot{d, v};
  __syncwarp();
  W.nb += __popc(m);
}

// LinearPool::pop: the closest unchecked entry, checked; -1 when every entry
// of the pool is.
__device__ __forceinline__ int beam_pop(Beam &W, uint32_t cap) {
  const int lane = threadIdx.x & 31;
  const Slot e = (uint32_t)lane < W.nb ? W.buf[lane] : Slot{INT_MAX, -1};
  const int ud = e.id >= 0 ? e.d : INT_MAX;
  const int bmin = __reduce_min_sync(0xffffffffu, ud);
  const bool in_array = W.cur < W.size;
  const Slot a = in_array ? W.pool[W.cur] : Slot{INT_MAX, -1};
  if (!in_array && bmin == INT_MAX) return -1;
  const bool from_array = in_array && a.d <= bmin;
  if (W.size + W.nb > cap) {
    uint32_t rank;
    if (from_array) {
      rank = W.cur + __popc(__ballot_sync(0xffffffffu, e.d < a.d));
    } else {
      const uint32_t eq = __ballot_sync(0xffffffffu, ud == bmin);
      const int l = __ffs(eq) - 1;
      rank = beam_upper(W.pool, W.size, bmin) +
             __popc(__ballot_sync(0xffffffffu, e.d < bmin || (e.d == bmin && lane < l)));
    }
    if (rank >= cap) return -1;
  }
  if (from_array) {
    if (lane == 0) W.pool[W.cur].id = a.id | (int)0x80000000;
    __syncwarp();
    uint32_t c = W.cur + 1;
    while (c < W.size) {
      const uint32_t i = c + lane;
      const uint32_t b = __ballot_sync(0xffffffffu, i < W.size && W.pool[i].id >= 0);
      if (b) {
        c += __ffs(b) - 1;
        break;
      }
      c = min(c + 32, W.size);
    }
    W.cur = c;
    return a.id;
  }
  const int l = __ffs(__ballot_sync(0xffffffffu, ud == bmin)) - 1;
  if (lane == l) W.buf[l].id = e.id | (int)0x80000000;
  __syncwarp();
  return __shfl_sync(0xffffffffu, e.id, l);
}

// As expand_plain; v0 = this lane's neighbour of the first chunk.
template <bool SV>
__device__ __forceinline__ void beam_expand_plain(const GParams &P, Beam &W, const int32_t *list, int v0) {
  const int lane = threadIdx.x & 31;
  for (uint32_t base = 0; base < P.K; base += 32) {
    const int v = base ? (base + lane < P.K ? list[base + lane] : -1) : v0;
    int4 cw[7];
    const bool seen = v < 0 || beam_get<SV>(W, (uint32_t)v);
    if (!seen) load_code7(P.codes + (uint64_t)v * CODE, cw);
    const Chunk c = chunk_of(v);
    const bool fresh = c.valid && !seen;
    beam_set<SV>(W, (uint32_t)v, fresh);
    const uint32_t m = __ballot_sync(0xffffffffu, fresh);
    if (m) beam_insert(W, P.cap, m, v, fresh ? dist7(W, cw) : 0);
    if (c.end) break;
  }
}

// The bitmap word of v, to be looked at later (nothing where the bits are in
// shared memory).
template <bool SV>
__device__ __forceinline__ uint64_t beam_word(const Beam &W, int v) {
  return SV || v < 0 ? 0 : mass_word(W.vis, W.mass, (uint32_t)v);
}

// As expand_filtered; v0, t0 = this lane's neighbour and edge timestamp of
// the first chunk.
template <bool SV>
__device__ __forceinline__ void beam_expand_filtered(const GParams &P, Beam &W, const int32_t *list, const float *tlist,
                                                     int v0, float t0, float l, float r, int rf) {
  const int lane = threadIdx.x & 31;
  auto inside = [&](int v, float t) { return v >= 0 && !(t < l || t > r); };
  int count1 = 0, count2 = 0;
  // The second hop's lists: of the neighbours in v, each scanned once.  Lists
  // n (va), n + 1 (vb), n + 2 (vc): the last on its way.  The first three are
  // asked for before the first hop, whose own loads hide theirs.
  int v = v0, va, vb, vc;
  float ta, tb, tc;
  uint32_t todo = __ballot_sync(0xffffffffu, v >= 0 && !beam_get1(P, W, (uint32_t)v)), ahead = todo;
  auto fetch = [&](int &x, float &t) {
    x = -1;
    t = 0.f;
    if (!ahead) return;
    const int nei = __shfl_sync(0xffffffffu, v, __ffs(ahead) - 1);
    ahead &= ahead - 1;
    if ((uint32_t)lane < P.K) {
      x = P.adj[(uint64_t)nei * P.K + lane];
      t = P.ets[(uint64_t)nei * P.K + lane];
    }
  };
  fetch(va, ta);
  fetch(vb, tb);
  fetch(vc, tc);
  for (uint32_t base = 0; base < P.K; base += 32) {
    const bool in = base + lane < P.K;
    const int v = base ? (in ? list[base + lane] : -1) : v0;
    const float t = base ? (in ? tlist[base + lane] : 0.f) : t0;
    int4 cw[7];
    const bool seen = v < 0 || beam_get<SV>(W, (uint32_t)v);
    if (!seen && inside(v, t)) load_code7(P.codes + (uint64_t)v * CODE, cw);
    const Chunk c = chunk_of(v);
    const bool fresh = c.valid && !seen;
    const bool pass = fresh && inside(v, t);
    const uint32_t passm = __ballot_sync(0xffffffffu, pass);
    beam_set<SV>(W, (uint32_t)v, fresh);
    count2 += __popc(__ballot_sync(0xffffffffu, fresh));
    count1 += __popc(passm);
    if (passm) beam_insert(W, P.cap, passm, v, pass ? dist7(W, cw) : 0);
    if (c.end) break;
  }
  for (uint32_t base = 0; base < P.K; base += 32) {
    if (count1 >= rf * count2) return;
    if (base) {
      v = base + lane < P.K ? list[base + lane] : -1;
      todo = ahead = __ballot_sync(0xffffffffu, v >= 0 && !beam_get1(P, W, (uint32_t)v));
      fetch(va, ta);
      fetch(vb, tb);
      fetch(vc, tc);
    }
    const bool end = __any_sync(0xffffffffu, v == -1);
    bool sa = va < 0 || beam_get<SV>(W, (uint32_t)va);
    uint64_t wb = beam_word<SV>(W, vb);
    int4 cw[7];
    if (SV && !sa && inside(va, ta)) load_code7(P.codes + (uint64_t)va * CODE, cw);
    while (todo) {
      if (count1 >= rf * count2) return;
      const int i = __ffs(todo) - 1;
      todo &= todo - 1;
      const int nei = __shfl_sync(0xffffffffu, v, i);
      // The next list's codes (SV: registers for them leave enough warps; with
      // the bits in global memory more warps hide more), the visited words of
      // the one after, the third one's points
      if (!SV && !sa && inside(va, ta)) load_code7(P.codes + (uint64_t)va * CODE, cw);
      int d0 = 0;
      if (SV && !sa && inside(va, ta)) d0 = dist7(W, cw);
      bool sb = vb < 0 || (SV ? beam_get<SV>(W, (uint32_t)vb) : (wb >> (vb & 63)) & 1ull);
      if (SV && !sb && inside(vb, tb)) load_code7(P.codes + (uint64_t)vb * CODE, cw);
      const uint64_t wc = beam_word<SV>(W, vc);
      int vd;
      float td;
      fetch(vd, td);
      beam_set1(P, W, (uint32_t)nei);
      // this list (its later chunks, out-degrees above 32, are not fetched ahead)
      const Chunk c2 = chunk_of(va);
      bool fresh = c2.valid && !sa;
      uint32_t passm = __ballot_sync(0xffffffffu, fresh && inside(va, ta));
      // the scan stops after the need-th insert: lanes past it are untouched
      auto cut = [&](uint32_t m, bool &stop) -> uint32_t {
        const int need = rf * count2 - count1;
        stop = __popc(m) >= need;
        if (!stop) return 0xffffffffu;
        for (int j = 1; j < need; ++j) m &= m - 1;
        const int last = __ffs(m) - 1;
        return last == 31 ? 0xffffffffu : ((2u << last) - 1u);
      };
      bool stop;
      uint32_t upto = cut(passm, stop);
      const bool mark = fresh && ((upto >> lane) & 1u);
      beam_set<SV>(W, (uint32_t)va, mark);
      count1 += __popc(passm & upto);
      if (!SV && !sa && inside(va, ta)) d0 = dist7(W, cw);
      if (passm & upto) beam_insert(W, P.cap, passm & upto, va, d0);
      // what was just marked is visited in the lists fetched ahead
      uint32_t marked = __ballot_sync(0xffffffffu, mark);
      uint64_t wcx = wc;
      if (!stop && !c2.end && P.K > 32) {
        const int32_t *list2 = P.adj + (uint64_t)nei * P.K;
        const float *tlist2 = P.ets + (uint64_t)nei * P.K;
        for (uint32_t b2 = 32; b2 < P.K; b2 += 32) {
          const bool in = b2 + lane < P.K;
          const int x = in ? list2[b2 + lane] : -1;
          const float t = in ? tlist2[b2 + lane] : 0.f;
          const bool seen = x < 0 || beam_get<SV>(W, (uint32_t)x);
          const Chunk c3 = chunk_of(x);
          fresh = c3.valid && !seen;
          passm = __ballot_sync(0xffffffffu, fresh && inside(x, t));
          upto = cut(passm, stop);
          beam_set<SV>(W, (uint32_t)x, fresh && ((upto >> lane) & 1u));
          count1 += __popc(passm & upto);
          if (passm & upto)
            beam_insert(W, P.cap, passm & upto, x, fresh && inside(x, t) ? beam_dist(P, W, (uint32_t)x) : 0);
          if (stop || c3.end) break;
        }
        // marks beyond the first chunk: the words fetched ahead are asked for again
        if (!SV) {
          sb = vb < 0 || beam_get<SV>(W, (uint32_t)vb);
          wcx = beam_word<SV>(W, vc);
        }
      } else if (!SV) {
        while (marked) {
          const int x = __shfl_sync(0xffffffffu, va, __ffs(marked) - 1);
          marked &= marked - 1;
          sb = sb || vb == x;
          if (vc == x) wcx |= 1ull << (x & 63);
        }
      }
      if (SV) sb = vb < 0 || beam_get<SV>(W, (uint32_t)vb);
      va = vb;
      ta = tb;
      sa = sb;
      vb = vc;
      tb = tc;
      wb = wcx;
      vc = vd;
      tc = td;
    }
    if (end) return;
  }
}

// One entry by the whole warp (warp-uniform arguments), and marked visited
template <bool SV>
__device__ __forceinline__ void beam_seed(const GParams &P, Beam &W, int u, int d, bool mark) {
  beam_insert(W, P.cap, 1u, u, d);
  if (mark) beam_set<SV>(W, (uint32_t)u, (threadIdx.x & 31) == 0);
}

// As initialize_search.
template <bool SV>
__device__ __forceinline__ void beam_initialize(const GParams &P, Beam &W) {
  const int lane = threadIdx.x & 31;
  if (P.ep >= 0) {
    int u = P.ep;
    int cur_dist = beam_dist(P, W, (uint32_t)u);
    for (int level = P.levels[u]; level > 0; --level) {
      bool changed = true;
      while (changed) {
        changed = false;
        const int32_t *list = P.up + P.up_off[u] + (int64_t)(level - 1) * P.upK;
        for (uint32_t base = 0; base < P.upK; base += 32) {
          const uint32_t i = base + lane;
          const int v = i < P.upK ? list[i] : -1;
          const uint32_t endb = __ballot_sync(0xffffffffu, v == -1);
          const bool valid = endb ? lane < __ffs(endb) - 1 : true;
          const int d = valid ? beam_dist(P, W, (uint32_t)v) : INT_MAX;
          // the reference's sequential scan moves u to every strictly closer
          // point: it ends at the first of the closest
          const int m = __reduce_min_sync(0xffffffffu, d);
          if (m < cur_dist) {
            cur_dist = m;
            u = __shfl_sync(0xffffffffu, v, __ffs(__ballot_sync(0xffffffffu, d == m)) - 1);
            changed = true;
          }
          if (endb) break;
        }
      }
    }
    beam_seed<SV>(P, W, u, cur_dist, true);
  } else {
    for (uint32_t e = 0; e < P.nep; ++e) beam_seed<SV>(P, W, P.eps[e], beam_dist(P, W, (uint32_t)P.eps[e]), false);
  }
}

// SV: the visited bits are in shared memory.  MINB: blocks per SM that the
// registers must leave room for.
template <bool SV, bool RANGED, int MINB>
__global__ void __launch_bounds__(GS_WARPS * 32, MINB) k_graph_beam(GParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t words0 = SV ? P.nvw : P.nblkw, vis_words = words0 + (RANGED ? (P.v1s ? P.nvw : P.nblkw) : 0u);
  unsigned char *mine = smem_raw + wib * beam_smem_bytes(P.cap, vis_words);
  Beam W;
  W.pool = reinterpret_cast<Slot *>(mine);
  W.buf = W.pool + P.cap;
  W.qw = reinterpret_cast<int4 *>(mine + (((size_t)(P.cap + BUF) * sizeof(Slot) + 15) & ~(size_t)15));
  W.vis = reinterpret_cast<uint32_t *>(W.qw + CODE / 16);
  W.vis1 = W.vis + words0;
  const uint32_t slot = blockIdx.x * GS_WARPS + wib;
  W.mass = P.vis + (uint64_t)slot * 2 * P.nwords;  // (not looked at where the sets are in shared memory)
  for (uint32_t qi = slot; qi < P.nq; qi += gridDim.x * GS_WARPS) {
    for (uint32_t i = lane; i < P.cap; i += 32) W.pool[i] = Slot{0, 0};
    for (uint32_t i = lane; i < vis_words; i += 32) W.vis[i] = 0;
    if (lane < CODE / 16) W.qw[lane] = reinterpret_cast<const int4 *>(P.qcodes + (uint64_t)qi * CODE)[lane];
    __syncwarp();
    int qq = 0;
#pragma unroll
    for (int w = 0; w < 7; ++w) {
      const int4 x = W.qw[w];
      qq = __dp4a(x.x, x.x, qq);
      qq = __dp4a(x.y, x.y, qq);
      qq = __dp4a(x.z, x.z, qq);
      qq = __dp4a(x.w, x.w, qq);
    }
    W.qq = qq;
    W.size = W.cur = W.nb = 0;
    W.lastd = INT_MAX;
    const float l = RANGED ? P.bounds[2 * (uint64_t)qi] : 0.f;
    const float r = RANGED ? P.bounds[2 * (uint64_t)qi + 1] : 0.f;
    const int lb = RANGED ? P.id_bounds[2 * (uint64_t)qi] : 0;
    const int ub = RANGED ? P.id_bounds[2 * (uint64_t)qi + 1] : 0;
    // float sel = (float)(ub - lb) / nb; seeds only when sel < 1
    const bool partial = __fdiv_rn((float)(ub - lb), (float)P.n) < 1.f;
    const bool seeded = RANGED && (P.mode == FKNN_GRAPH_CATEGORY_RANGE || partial);
    bool bad = false;
    if (seeded) {  // every seed lb + i * ((ub - lb) / 10), i < 10, must be a point
      const long long last = (long long)lb + 9ll * ((ub - lb) / 10);
      bad = lb < 0 || (uint32_t)lb >= P.n || last < 0 || last >= (long long)P.n;
    }
    if (bad) {
      if (lane == 0) atomicOr(P.err, ERR_BAD_QUERY_VALUE);
      for (uint32_t i = lane; i < P.refine; i += 32) {
        P.out_ids[(uint64_t)qi * P.refine + i] = -1;
        if (P.out_dists) P.out_dists[(uint64_t)qi * P.refine + i] = __int_as_float(0x7fc00000);
      }
      __syncwarp();
      continue;
    }
    if (seeded) {  // as range_seeds: the ten distances side by side, then in order
      const int interval = (ub - lb) / 10;
      const int point = lb + interval * min(lane, 9);
      const int d = beam_dist(P, W, (uint32_t)point);
      for (int i = 0; i < 10; ++i)
        beam_seed<SV>(P, W, __shfl_sync(0xffffffffu, point, i), __shfl_sync(0xffffffffu, d, i), true);
    } else if (P.mode != FKNN_GRAPH_RANGE_SUBTIME) {
      beam_initialize<SV>(P, W);
    }
    // each pop checks one entry; an expansion inserts each point at most once
    // (vis), besides at most ten seeds and the unmarked entry points, so
    // n + nep + 16 pops is a hard bound
    uint32_t pops = 0;
    for (;;) {
      const int u = beam_pop(W, P.cap);
      if (u < 0) break;
      if (++pops > P.n + P.nep + 16) {
        if (lane == 0) atomicOr(P.err, ERR_WAIT_TIMEOUT);
        break;
      }
      const int32_t *list = P.adj + (uint64_t)u * P.K;
      const bool in = (uint32_t)lane < P.K;
      const int v0 = in ? list[lane] : -1;
      if (RANGED) {
        const float *tlist = P.ets + (uint64_t)u * P.K;
        const float t0 = in ? tlist[lane] : 0.f;
        if (W.nb > BUF / 2) beam_merge(W, P.cap);  // while the list is on its way
        beam_expand_filtered<SV>(P, W, list, tlist, v0, t0, l, r, P.mode == FKNN_GRAPH_CATEGORY_RANGE ? 1 : 2);
      } else {
        if (W.nb > BUF / 2) beam_merge(W, P.cap);  // while the list is on its way
        beam_expand_plain<SV>(P, W, list, v0);
      }
    }
    beam_merge(W, P.cap);
    // reorder / reorder_dist (sq8_sym_quant.hpp:76-89): slots 0..refine-1 as
    // they stand, ids unmasked, distances times alpha^2
    for (uint32_t i = lane; i < P.refine; i += 32) {
      const Slot s = W.pool[i];
      P.out_ids[(uint64_t)qi * P.refine + i] = s.id & 0x7fffffff;
      if (P.out_dists) P.out_dists[(uint64_t)qi * P.refine + i] = __fmul_rn((float)s.d, P.alpha2);
    }
    __syncwarp();
  }
}

}  // namespace

int graph_codes(const fknn_graph *g, const int8_t **codes, float *alpha, uint32_t *n) {
  *codes = g->codes;
  *alpha = g->alpha;
  *n = g->n;
  return FKNN_OK;
}

namespace {

template <typename T>
int grow(T **p, size_t *cap, size_t want) {
  if (*cap >= want) return FKNN_OK;
  if (*p) cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  FKNN_CUDA(cudaMalloc((void **)p, want * sizeof(T)));
  *cap = want;
  return FKNN_OK;
}

bool on_device(const void *p, int dev) { return mem_loc(p, dev) == MemLoc::Here; }

void free_graph(fknn_graph *g) {
  if (!g) return;
  cudaSetDevice(g->device);
  cudaDeviceSynchronize();
  cudaFree(g->adj);
  cudaFree(g->ets);
  cudaFree(g->levels);
  cudaFree(g->up_off);
  cudaFree(g->up);
  cudaFree(g->eps);
  cudaFree(g->codes);
  cudaFree(g->io);
  cudaFree(g->qcodes);
  cudaFree(g->vis);
  cudaFree(g->dflag);
  delete g;
}

int upload(void **dst, const void *src, size_t bytes) {
  FKNN_CUDA(cudaMalloc(dst, bytes ? bytes : 16));
  if (bytes) FKNN_CUDA(cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice));
  return FKNN_OK;
}

// Parsed Graph::save bytes (graph.hpp:101-115, HNSWInitializer.hpp:73-82).
struct HostGraph {
  std::vector<int32_t> eps, adj, levels, up;
  std::vector<float> ets;
  std::vector<int64_t> up_off;
  int32_t N = 0, K = 0, upK = 0, ep = -1;
};

bool parse_graph(const unsigned char *b, size_t nbytes, HostGraph &h) {
  size_t off = 0;
  auto rd = [&](void *dst, size_t bytes) {
    if (bytes > nbytes - off) return false;
    std::memcpy(dst, b + off, bytes);
    off += bytes;
    return true;
  };
  int32_t nep = 0;
  if (!rd(&nep, 4) || nep < 0 || (size_t)nep > nbytes / 4) return false;
  h.eps.resize(nep);
  if (nep && !rd(h.eps.data(), (size_t)nep * 4)) return false;
  if (!rd(&h.N, 4) || !rd(&h.K, 4) || h.N <= 0 || h.K <= 0 || h.K > 1024) return false;
  const size_t nk = (size_t)h.N * h.K;
  if (nk > (nbytes - off) / 8) return false;
  h.adj.resize(nk);
  h.ets.resize(nk);
  rd(h.adj.data(), nk * 4);
  rd(h.ets.data(), nk * 4);
  for (int32_t v : h.adj)
    if (v < -1 || v >= h.N) return false;
  for (int32_t v : h.eps)
    if (v < 0 || v >= h.N) return false;
  if (off == nbytes) return nep > 0;  // no initializer: the entry points seed the search
  int32_t iN = 0;
  if (!rd(&iN, 4) || !rd(&h.upK, 4) || !rd(&h.ep, 4)) return false;
  if (iN != h.N || h.upK <= 0 || h.upK > 1024 || h.ep < 0 || h.ep >= h.N) return false;
  h.levels.resize(h.N);
  h.up_off.resize((size_t)h.N + 1);
  h.up_off[0] = 0;
  for (int32_t i = 0; i < h.N; ++i) {
    int32_t cur = 0;
    if (!rd(&cur, 4) || cur < 0 || cur % h.upK) return false;
    h.levels[i] = cur / h.upK;
    const size_t at = h.up.size();
    if ((size_t)cur > (nbytes - off) / 4) return false;
    h.up.resize(at + cur);
    if (cur) rd(h.up.data() + at, (size_t)cur * 4);
    h.up_off[i + 1] = (int64_t)h.up.size();
  }
  // a level-L list may only name points that exist at level L (the descent
  // reads the named point's own level-L list next)
  for (int32_t i = 0; i < h.N; ++i)
    for (int64_t j = h.up_off[i]; j < h.up_off[i + 1]; ++j) {
      const int32_t v = h.up[j];
      const int32_t level = (int32_t)((j - h.up_off[i]) / h.upK) + 1;
      if (v < -1 || v >= h.N || (v >= 0 && h.levels[v] < level)) return false;
    }
  return off == nbytes;
}

}  // namespace
}  // namespace fknn

using namespace fknn;

namespace fknn {

// The argument checks of fknn_graph_search; *cap = the pool capacity.
int graph_check_args(const fknn_graph *g, const float *queries, uint32_t nq, int mode, uint32_t k, uint32_t ef,
                     uint32_t refine, const float *bounds, const int32_t *id_bounds, const int32_t *out_ids,
                     uint32_t *cap) {
  (void)nq;
  if (!g || !queries || !out_ids) {
    set_error("fknn_graph_search: NULL argument");
    return FKNN_EINVAL;
  }
  if (mode < FKNN_GRAPH_SEARCH || mode > FKNN_GRAPH_RANGE) {
    set_error("fknn_graph_search: unknown mode");
    return FKNN_EINVAL;
  }
  if (ef == 0) ef = EF_DEFAULT;
  *cap = std::max(k, ef);  // LinearPool(nb, max(k, ef), k)
  if (k == 0 || *cap > CAP_MAX || refine == 0 || refine > *cap + 1) {
    set_error("fknn_graph_search: need 1 <= k, max(k, ef) <= 4096 and 1 <= refine <= max(k, ef) + 1");
    return FKNN_EINVAL;
  }
  if (mode == FKNN_GRAPH_SEARCH && refine != k) {
    set_error("fknn_graph_search: mode 0 (Search) writes k ids; refine must equal k");
    return FKNN_EINVAL;
  }
  if (mode >= FKNN_GRAPH_CATEGORY_RANGE && (!bounds || !id_bounds)) {
    set_error("fknn_graph_search: modes 3-5 need bounds and id_bounds");
    return FKNN_EINVAL;
  }
  return FKNN_OK;
}

// Launch geometry of a search of nq queries at pool capacity cap.
using GraphKernel = void (*)(GParams);

struct GraphGeometry {
  size_t smem = 0, grid = 0;
  uint32_t nwords = 0, nblkw = 0, nvw = 0;
  bool global_vis = true;  // bitmaps in g->vis
  bool v1s = false;        // vis1 in shared memory
  GraphKernel kern = nullptr;
};

static int graph_geometry(const fknn_graph *g, uint32_t nq, uint32_t cap, bool ranged, bool overflow_read,
                          GraphGeometry &G) {
  const uint32_t nblocks512 = (g->n + 511) / 512;
  G.nwords = nblocks512 * 8;
  G.nblkw = (nblocks512 + 31) / 32;
  G.nvw = (g->n + 31) / 32;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device);
  const uint32_t sets = ranged ? 2 : 1;
  // blocks of this many bytes that an SM holds
  auto fits = [](size_t smem) { return GS_SMEM_PER_SM / (smem + 1024); };
  const size_t need = std::max<size_t>(1, ((size_t)nq + (size_t)sms * GS_WARPS - 1) / ((size_t)sms * GS_WARPS));
  if (overflow_read) {
    G.smem = warp_smem_bytes(cap, G.nblkw) * GS_WARPS;
    G.kern = k_graph_search;
  } else {
    // Visited bits in shared memory, or at least those of vis: a test or a
    // mark is then no L2 round trip, and a query runs 2.8 times as fast
    // (windowed form, 100,000 points).  Taken where the SM still holds a block
    // for every query, or a third of the blocks it holds without the bits
    // (SearchFilter, 100,000 points, pool 256, 10,000 queries: 3 blocks against
    // 8, 3.10 against 3.31 ms).
    const size_t f0 = beam_smem_bytes(cap, sets * G.nblkw) * GS_WARPS;
    const size_t s0 = beam_smem_bytes(cap, G.nvw + (sets - 1) * G.nblkw) * GS_WARPS;
    const size_t s1 = beam_smem_bytes(cap, sets * G.nvw) * GS_WARPS;
    const size_t base = std::min<size_t>(fits(f0), ranged ? GS_BASE_BLOCKS : GS_OCC_BLOCKS);
    auto serves = [&](size_t smem) {
      return smem <= 200 * 1024 && fits(smem) >= std::max<size_t>(1, std::min<size_t>(need, (base + 2) / 3));
    };
    if (serves(s1) || (ranged && serves(s0))) {
      G.v1s = ranged && serves(s1);
      G.smem = serves(s1) ? s1 : s0;
      G.global_vis = ranged && !G.v1s;
      G.kern = ranged ? k_graph_beam<true, true, GS_SV_RANGED_BLOCKS> : k_graph_beam<true, false, GS_SV_BLOCKS>;
    } else {
      G.smem = f0;
      G.kern = ranged                           ? k_graph_beam<false, true, GS_BASE_BLOCKS>
               : fits(G.smem) >= GS_OCC_BLOCKS ? k_graph_beam<false, false, GS_OCC_BLOCKS>
                                                : k_graph_beam<false, false, GS_BASE_BLOCKS>;
    }
  }
  if (!overflow_read && G.smem > 200 * 1024) {  // (the plain pool's few bytes less may still fit)
    G.smem = warp_smem_bytes(cap, G.nblkw) * GS_WARPS;
    G.kern = k_graph_search;
  }
  if (G.smem > 200 * 1024) {
    set_error("fknn_graph_search: pool and visited flags exceed shared memory (max(k, ef) or n too large)");
    return FKNN_EINVAL;
  }
  FKNN_CUDA(cudaFuncSetAttribute(G.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G.smem));
  int per_sm = 0;
  FKNN_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, G.kern, GS_WARPS * 32, G.smem));
  size_t gr = (size_t)sms * std::max(per_sm, 1);
  if (G.global_vis) {
    const size_t slot_bytes = (size_t)G.nwords * 16;
    const size_t max_slots = std::max<size_t>(GS_WARPS, VIS_BUDGET / slot_bytes);
    gr = std::min(gr, std::max<size_t>(1, max_slots / GS_WARPS));
  }
  G.grid = std::min(gr, ((size_t)nq + GS_WARPS - 1) / GS_WARPS);
  return FKNN_OK;
}

// Grows the graph's per-call scratch for searches of up to nq queries at
// pool capacity up to cap, so that graph_launch allocates nothing.
int graph_reserve(fknn_graph *g, uint32_t nq, uint32_t cap, bool ranged, bool overflow_read) {
  GraphGeometry G;
  int rc;
  if ((rc = graph_geometry(g, nq, cap, ranged, overflow_read, G))) return rc;
  if ((rc = grow(&g->qcodes, &g->qcodes_cap, (size_t)nq * CODE))) return rc;
  return G.global_vis ? grow(&g->vis, &g->vis_cap, G.grid * GS_WARPS * 2 * (size_t)G.nwords) : FKNN_OK;
}

// Enqueues one search on st (device inputs and outputs, checked arguments);
// the graph's error flag accumulates until graph_flag_reset.
int graph_launch(fknn_graph *g, const float *q_use, uint32_t nq, int mode, uint32_t k, uint32_t cap,
                 uint32_t refine, const float *b_use, const int32_t *ib_use, int32_t *ids_use, float *d_use,
                 cudaStream_t st) {
  int rc;
  if ((rc = grow(&g->qcodes, &g->qcodes_cap, (size_t)nq * CODE))) return rc;
  launch_sq8_encode(q_use, nq, g->alpha, g->qcodes, st);
  const bool ranged = mode >= FKNN_GRAPH_CATEGORY_RANGE;
  GraphGeometry G;
  if ((rc = graph_geometry(g, nq, cap, ranged, refine > cap, G))) return rc;
  if (G.global_vis && (rc = grow(&g->vis, &g->vis_cap, G.grid * GS_WARPS * 2 * (size_t)G.nwords))) return rc;
  GParams P;
  P.adj = g->adj;
  P.ets = g->ets;
  P.levels = g->levels;
  P.up_off = g->up_off;
  P.up = g->up;
  P.eps = g->eps;
  P.codes = g->codes;
  P.n = g->n;
  P.K = g->K;
  P.upK = g->upK;
  P.nep = g->nep;
  P.ep = g->ep;
  P.alpha2 = g->alpha * g->alpha;
  P.qcodes = g->qcodes;
  P.nq = nq;
  P.mode = mode;
  P.cap = cap;
  P.refine = refine;
  P.bounds = ranged ? b_use : nullptr;
  P.id_bounds = ranged ? ib_use : nullptr;
  P.out_ids = ids_use;
  P.out_dists = d_use;
  P.vis = g->vis;
  P.nwords = G.nwords;
  P.nblkw = G.nblkw;
  P.nvw = G.nvw;
  P.v1s = G.v1s;
  P.err = g->dflag;
  G.kern<<<(unsigned)G.grid, GS_WARPS * 32, G.smem, st>>>(P);
  g_launches += 1;
  FKNN_CUDA(cudaGetLastError());
  return FKNN_OK;
}

int graph_flag_reset(fknn_graph *g, cudaStream_t st) {
  FKNN_CUDA(cudaMemsetAsync(g->dflag, 0, 4, st));
  return FKNN_OK;
}

// The searches enqueued since the last reset (call after they finished).
int graph_flag_check(fknn_graph *g) {
  int flag = 0;
  FKNN_CUDA(cudaMemcpy(&flag, g->dflag, 4, cudaMemcpyDeviceToHost));
  if (flag & ERR_BAD_QUERY_VALUE) {
    set_error("fknn_graph_search: id_bounds seed a point outside [0, n)");
    return FKNN_EINVAL;
  }
  if (flag) {
    set_error("fknn_graph_search: a search exceeded its pop bound");
    return FKNN_ETIMEOUT;
  }
  return FKNN_OK;
}

}  // namespace fknn

extern "C" {

int fknn_graph_create(const void *graph_bytes, size_t nbytes, const float *vecs, int device, fknn_graph **out) {
  g_launches = 0;
  if (!graph_bytes || !vecs || !out) {
    set_error("fknn_graph_create: NULL argument");
    return FKNN_EINVAL;
  }
  *out = nullptr;
  HostGraph h;
  if (!parse_graph(static_cast<const unsigned char *>(graph_bytes), nbytes, h)) {
    set_error("fknn_graph_create: malformed graph bytes (expected the Graph::save layout)");
    return FKNN_EINVAL;
  }
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    set_error("fknn_graph_create: no CUDA device");
    return FKNN_ENODEV;
  }
  if (device < 0 || device >= ndev) {
    set_error("fknn_graph_create: bad device ordinal");
    return FKNN_EINVAL;
  }
  FKNN_CUDA(cudaSetDevice(device));
  fknn_graph *g = new (std::nothrow) fknn_graph();
  if (!g) {
    set_error("fknn_graph_create: out of host memory");
    return FKNN_ENOMEM;
  }
  g->device = device;
  g->n = (uint32_t)h.N;
  g->K = (uint32_t)h.K;
  g->nep = (uint32_t)h.eps.size();
  g->ep = h.ep;
  g->upK = h.upK > 0 ? (uint32_t)h.upK : 1u;
  const size_t nk = (size_t)h.N * h.K;
  int rc = upload((void **)&g->adj, h.adj.data(), nk * 4);
  if (!rc) rc = upload((void **)&g->ets, h.ets.data(), nk * 4);
  if (!rc) rc = upload((void **)&g->eps, h.eps.data(), h.eps.size() * 4);
  if (!rc && h.ep >= 0) {
    rc = upload((void **)&g->levels, h.levels.data(), h.levels.size() * 4);
    if (!rc) rc = upload((void **)&g->up_off, h.up_off.data(), h.up_off.size() * 8);
    if (!rc) rc = upload((void **)&g->up, h.up.data(), h.up.size() * 4);
  }
  if (!rc) {
    const cudaError_t e = cudaMalloc((void **)&g->dflag, 64);
    if (e != cudaSuccess) rc = cuda_fail(e, "cudaMalloc");
  }
  if (!rc) {
    const cudaError_t e = cudaMalloc((void **)&g->codes, (size_t)h.N * CODE);
    if (e != cudaSuccess) rc = cuda_fail(e, "cudaMalloc");
  }
  // Searcher::SetData: the searcher's own quantizer, trained on the graph's points
  if (!rc) rc = fknn_sq8_sym_train(vecs, (uint64_t)h.N, &g->alpha, g->codes);
  if (!rc) {
    k_graph_lists<<<148 * 8, 256>>>(g->adj, g->n, g->K);
    k_code_norms<<<148 * 8, 256>>>(g->codes, g->n);
    g_launches += 2;
    const cudaError_t e = cudaStreamSynchronize(0);
    if (e != cudaSuccess) rc = cuda_fail(e, "fknn_graph_create");
  }
  if (rc) {
    free_graph(g);
    return rc;
  }
  *out = g;
  return FKNN_OK;
}

int fknn_graph_destroy(fknn_graph *g) {
  free_graph(g);
  return FKNN_OK;
}

int fknn_graph_info(const fknn_graph *g, uint32_t *n, uint32_t *degree, float *alpha) {
  if (!g) {
    set_error("fknn_graph_info: NULL graph");
    return FKNN_EINVAL;
  }
  if (n) *n = g->n;
  if (degree) *degree = g->K;
  if (alpha) *alpha = g->alpha;
  return FKNN_OK;
}

int fknn_graph_search(fknn_graph *g, const float *queries, uint32_t nq, int mode, uint32_t k, uint32_t ef,
                      uint32_t refine, const float *bounds, const int32_t *id_bounds, int32_t *out_ids,
                      float *out_dists, void *stream) {
  g_launches = 0;
  uint32_t cap = 0;
  int rc;
  if ((rc = fknn::graph_check_args(g, queries, nq, mode, k, ef, refine, bounds, id_bounds, out_ids, &cap))) return rc;
  if (nq == 0) return FKNN_OK;
  FKNN_CUDA(cudaSetDevice(g->device));
  cudaStream_t st = (cudaStream_t)stream;
  const bool ranged = mode >= FKNN_GRAPH_CATEGORY_RANGE;

  // staging: [queries | bounds | id_bounds | ids | dists], 4-byte words
  const size_t qf = (size_t)nq * DIM, bf = ranged ? (size_t)nq * 2 : 0, of = (size_t)nq * refine;
  if ((rc = grow(&g->io, &g->io_cap, qf + 2 * bf + 2 * of))) return rc;
  float *s_q = g->io, *s_b = s_q + qf;
  int32_t *s_ib = reinterpret_cast<int32_t *>(s_b + bf);
  int32_t *s_ids = s_ib + bf;
  float *s_d = reinterpret_cast<float *>(s_ids + of);
  const int dev = g->device;
  if ((rc = fknn::check_local_buffers("fknn_graph_search", dev,
                                      {queries, ranged ? bounds : nullptr, ranged ? id_bounds : nullptr, out_ids,
                                       out_dists})))
    return rc;
  const float *q_use = queries;
  if (!on_device(queries, dev)) {
    FKNN_CUDA(cudaMemcpyAsync(s_q, queries, qf * 4, cudaMemcpyHostToDevice, st));
    q_use = s_q;
  }
  const float *b_use = bounds;
  const int32_t *ib_use = id_bounds;
  if (ranged && !on_device(bounds, dev)) {
    FKNN_CUDA(cudaMemcpyAsync(s_b, bounds, bf * 4, cudaMemcpyHostToDevice, st));
    b_use = s_b;
  }
  if (ranged && !on_device(id_bounds, dev)) {
    FKNN_CUDA(cudaMemcpyAsync(s_ib, id_bounds, bf * 4, cudaMemcpyHostToDevice, st));
    ib_use = s_ib;
  }
  int32_t *ids_use = on_device(out_ids, dev) ? out_ids : s_ids;
  float *d_use = out_dists ? (on_device(out_dists, dev) ? out_dists : s_d) : nullptr;
  FKNN_CUDA(cudaMemsetAsync(g->dflag, 0, 4, st));
  if ((rc = fknn::graph_launch(g, q_use, nq, mode, k, cap, refine, b_use, ib_use, ids_use, d_use, st))) return rc;
  if (ids_use != out_ids) FKNN_CUDA(cudaMemcpyAsync(out_ids, ids_use, of * 4, cudaMemcpyDeviceToHost, st));
  if (out_dists && d_use != out_dists)
    FKNN_CUDA(cudaMemcpyAsync(out_dists, d_use, of * 4, cudaMemcpyDeviceToHost, st));
  FKNN_CUDA(cudaStreamSynchronize(st));
  return fknn::graph_flag_check(g);
}

}  // extern "C"
