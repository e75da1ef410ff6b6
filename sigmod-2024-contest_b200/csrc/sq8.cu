// Symmetric SQ8 (pyglass/glass/quant/sq8_sym_quant.hpp) and the SQ8 slab
// brute force (bruteforce.h:244-289) on the GPU.
//
// bruteforce() returns the reference's maxPQIFCS heap array, which depends
// on the exact insertion history (ties on the int distance are frequent).
// The kernels below reproduce that history (the three steps are described
// above k_sq8_prefix).  Every distance is an exact int32 L2SqrSQ8_sym value:
// |q-c|^2 = |q|^2 + |c|^2 - 2 q.c, from dp4a or from the int8 tensor cores.
#include <climits>

#include "tc_util.cuh"

namespace fknn {

namespace {

constexpr int SQ8_CODE = 112;
constexpr int BF_KMAX = 2048;

__global__ void k_absmax(const float *__restrict__ x, uint64_t count, uint32_t *__restrict__ out) {
  float m = 0.f;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x)
    m = fmaxf(m, fabsf(x[i]));
  for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));  // non-negative floats order as uints
}

// sq8_sym_quant.hpp:63-74: x / alpha (IEEE division), clamp to [-1, 1],
// std::round(x * 127) (half away from zero), dims 100..111 zero.
__global__ void k_sq8_encode(const float *__restrict__ x, uint64_t n, float alpha, int8_t *__restrict__ codes) {
  const uint64_t total = n * SQ8_CODE;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t r = i / SQ8_CODE;
    const int d = (int)(i % SQ8_CODE);
    int8_t c = 0;
    if (d < DIM) {
      float y = __fdiv_rn(x[r * DIM + d], alpha);
      if (y > 1.0f) y = 1.0f;
      if (y < -1.0f) y = -1.0f;
      c = (int8_t)roundf(__fmul_rn(y, 127.0f));
    }
    codes[i] = c;
  }
}

struct HeapNode {
  int d;
  int id;
};

// ------------------------------------------------------------------------
// The slab brute force per batch of queries, over parts of the slab that grow
// by SQ_GROW:
//
//  1. k_sq8_dist and k_sq8_prefix (one warp per query): the distances of the
//     first SQ_PREFIX codes, then their replay -- emplace of the first k, then
//     must_pop_emplace -- with a warp-wide filter in front of the heap steps.
//     The heap root afterwards, T_q, bounds every later root (the root only
//     falls), so a later code can enter only if its distance is below T_q.
//  2. k_sq8_screen (tcgen05, kind::i8): the int32 inner products of a tile of
//     128 queries with the code tiles of one segment of the part, exact in the
//     accumulator; an epilogue thread per query writes every code of the
//     segment with d = |q|^2 + |c|^2 - 2 q.c < T_q, in slab order, to the
//     query's list for that segment.  A list that fills up marks the query.
//  3. k_sq8_tail (one warp per query): the heap so far, the segment lists in
//     order through the same filter and heap steps; then the next part with a
//     lower T_q, or the heap array out.  A marked query scans the part's codes
//     itself instead.
//
// Every distance is the exact int32 L2SqrSQ8_sym value and every code that
// can enter the heap reaches the heap steps in slab order, so the heap array
// is the reference's.
//
// About k (SQ_GROW - 1) codes of a part are below its T_q: 1,800 in all for
// k = 140 and 450,000 codes, where one part after the prefix had 7,700.
constexpr uint32_t SQ_PREFIX = 8192;    // codes replayed before the screen (multiple of 128)
constexpr uint64_t SQ_GROW = 8;         // a part ends at this multiple of its first code
constexpr int SQ_DQ = 32;               // queries of a block of k_sq8_dist
constexpr uint64_t SQ_DIST_BYTES = 192ull << 20;  // prefix distances of a call made all at once, else ...
constexpr uint32_t SQ_REPLAY_WARPS = 32;          // ... for as many queries per SM as k_sq8_prefix has resident
constexpr int SQ_WARPS = 4;             // queries per block of the replay kernels
constexpr int SQ_SCAN = 128;            // codes per warp step of the replay kernels
constexpr uint32_t SQ_TILE = TC_ROWS * 128;  // 128 rows x 128 bytes (112 code bytes, 16 zero)
constexpr int SQ_BS = 4;                // shared-memory stages of code tiles
constexpr int SQ_NB = 2 * SQ_BS;        // ... of their norms, which the epilogue reads up to two tiles later
constexpr int SQ_EPI_WARPS = 4;
constexpr int SQ_THREADS = (2 + SQ_EPI_WARPS) * 32;  // producer, MMA issuer, epilogue
constexpr uint32_t SQ_TMEM_COLS = 2 * TC_ROWS;       // double-buffered accumulator
constexpr int SQ_MMAS = 128 / 32;       // kind::i8: K = 32 bytes per MMA
constexpr int SQ_NCC_PAD = INT_MIN / 2;  // -|c|^2 of rows past the slab: no candidate test passes
constexpr uint32_t SQ_QBATCH = 8192;    // queries per pass (bounds the candidate lists)
// S32 accumulate, signed 8-bit A and B, K-major, N = 128, M = 128
constexpr uint32_t SQ_IDESC =
    (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TC_ROWS >> 3) << 17) | ((uint32_t)(TC_ROWS >> 4) << 24);

// code p (row p of 112 bytes; row 0 when p >= bound) as seven 16-byte words
__device__ __forceinline__ void load_code(const int8_t *__restrict__ codes, uint64_t p, uint64_t bound,
                                          int4 (&c)[7]) {
  const int4 *src = reinterpret_cast<const int4 *>(codes + (p < bound ? p : 0) * SQ8_CODE);
#pragma unroll
  for (int w = 0; w < 7; ++w) c[w] = __ldg(src + w);
}

__device__ __forceinline__ int dot112(const int4 (&c)[7], const int4 (&q)[7]) {
  int s = 0;
#pragma unroll
  for (int w = 0; w < 7; ++w) {
    s = __dp4a(q[w].x, c[w].x, s);
    s = __dp4a(q[w].y, c[w].y, s);
    s = __dp4a(q[w].z, c[w].z, s);
    s = __dp4a(q[w].w, c[w].w, s);
  }
  return s;
}

// Heap steps of maxPQIFCS on a 1-based array, with a hole moved in place of
// the reference's swaps (the same comparisons, so the same array).

// emplace (bruteforce.h:106-113) at position now (1-based, = new size)
__device__ __forceinline__ void heap_emplace(HeapNode *h, int now, HeapNode nd) {
  while (now != 1) {
    const HeapNode p = h[now >> 1];
    if (!(nd.d > p.d)) break;
    h[now] = p;
    now >>= 1;
  }
  h[now] = nd;
}

// The way down from the root always takes the larger child (push_down,
// bruteforce.h:78-87) and does not depend on the new node, only its end does.
// So next[x] keeps every node's larger child (low half) and that child's (high
// half; 0: none), as byte offsets into next: the warp follows two levels per
// load, without a branch, and lane l then moves level l's node.
struct WarpHeap {
  HeapNode *h;      // 1-based, cnt nodes
  uint32_t *next;   // 0 .. cnt (next[0]: none)
  HeapNode *stage;
  int cnt, root;    // root: h[1].d
  int steps;        // loads from the root to any leaf's level
};

// shared memory of one warp's heap, in nodes: the heap (k + 1 nodes), next, the stage
__host__ __device__ __forceinline__ uint32_t sq_heap_nodes(uint32_t k) { return (k + 2u) & ~1u; }
__host__ __device__ __forceinline__ uint32_t sq_next_nodes(uint32_t k) { return (k + 2u) / 2u; }
__host__ __device__ __forceinline__ uint32_t sq_region(uint32_t k) {
  return (sq_heap_nodes(k) + sq_next_nodes(k) + SQ_SCAN + 1u) & ~1u;
}

__device__ __forceinline__ WarpHeap warp_heap(unsigned char *smem, int warp, uint32_t k) {
  WarpHeap w;
  w.h = reinterpret_cast<HeapNode *>(smem) + (size_t)warp * sq_region(k);
  w.next = reinterpret_cast<uint32_t *>(w.h + sq_heap_nodes(k));
  w.stage = w.h + sq_heap_nodes(k) + sq_next_nodes(k);
  w.cnt = (int)k;
  w.steps = (32 - __clz(k)) / 2;  // levels 0 .. floor(log2(k))
  return w;
}

// next and root of a full heap; the whole warp
__device__ __forceinline__ void heap_ready(WarpHeap &w, int lane) {
  __syncwarp();
  for (int x = lane; x <= w.cnt; x += 32) {
    const int c = 2 * x;
    const bool r = x && c < w.cnt && w.h[c + 1].d > w.h[c].d;
    w.next[x] = x && c <= w.cnt ? 4 * (c + (r ? 1 : 0)) : 0;
  }
  __syncwarp();
  for (int x = lane; x <= w.cnt; x += 32) {  // (the low halves stay as they are)
    const uint32_t c = w.next[x] & 0xffffu;
    w.next[x] = c | (w.next[c / 4] & 0xffffu) << 16;
  }
  w.root = w.h[1].d;
  __syncwarp();
}

// must_pop_emplace (bruteforce.h:99-105) behind the root test
// bruteforce.h:258-260 makes, by the whole warp.  A chain of loads and shuffles,
// so bound by latency: 500 cycles a node at k = 140, where lane 0 alone, a level
// at a time with its branch and store, took 1,080.
__device__ __forceinline__ void heap_offer(WarpHeap &w, HeapNode nd, int lane) {
  if (w.root <= nd.d) return;
  const char *const nb = reinterpret_cast<const char *>(w.next);
  // lane l: the node of level l and the one below (offsets; 0 past the leaf)
  uint32_t x = 4, px = lane == 0 ? 4u : 0u, nx = 0;
#pragma unroll 1
  for (int i = 0; i < 2 * w.steps; i += 2) {
    const uint32_t j = *reinterpret_cast<const uint32_t *>(nb + x), j0 = j & 0xffffu;
    x = j >> 16;
    if (lane == i) nx = j0;
    if (lane == i + 1) px = j0, nx = x;
    if (lane == i + 2) px = x;
  }
  // its larger child, and the other one, if there is one, with that one's larger child
  HeapNode c;
  c.d = INT_MIN;
  c.id = 0;
  int sd = INT_MIN;
  uint32_t sn = 0;
  const uint32_t sx = nx ^ 4u;
  if (nx) {
    c = *reinterpret_cast<const HeapNode *>(reinterpret_cast<const char *>(w.h) + 2 * nx);
    if (sx <= 4u * w.cnt) {
      sd = *reinterpret_cast<const int *>(reinterpret_cast<const char *>(w.h) + 2 * sx);
      sn = *reinterpret_cast<const uint32_t *>(nb + sx) & 0xffffu;
    }
  }
  const int cd1 = __shfl_down_sync(0xffffffffu, c.d, 1);
  // the new node's level: the first whose larger child is not larger, or the leaf's
  const int t = __ffs(__ballot_sync(0xffffffffu, px && c.d <= nd.d)) - 1;
  w.root = __shfl_sync(0xffffffffu, t == 0 ? nd.d : c.d, 0);
  // lanes < t: their larger child now (of two equal ones the left)
  const int below = lane + 1 < t ? cd1 : nd.d;
  uint32_t big = nx;
  if (lane < t && ((nx & 4u) ? below <= sd : sd > below)) big = sx;
  const uint32_t big1 = __shfl_down_sync(0xffffffffu, big, 1);
  if (lane <= t) {
    HeapNode v = nd;
    if (lane < t) {
      v = c;
      *reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(w.next) + px) = big | (big == nx ? big1 : sn) << 16;
    }
    *reinterpret_cast<HeapNode *>(reinterpret_cast<char *>(w.h) + 2 * px) = v;
  }
  __syncwarp();
}

// A step of at most SQ_SCAN nodes, (d[i], id[i]) in lane order for i = 0 ..,
// those at the largest distance absent: the ones that can enter are staged in
// order and offered.
__device__ __forceinline__ void offer_step(WarpHeap &w, const int (&d)[SQ_SCAN / 32], const int (&id)[SQ_SCAN / 32],
                                           int lane) {
  const uint32_t below = (1u << lane) - 1u;
  int off = 0;
#pragma unroll
  for (int i = 0; i < SQ_SCAN / 32; ++i) {
    const uint32_t m = __ballot_sync(0xffffffffu, d[i] < w.root);
    if ((m >> lane) & 1u) {
      HeapNode nd;
      nd.d = d[i];
      nd.id = id[i];
      w.stage[off + __popc(m & below)] = nd;
    }
    off += __popc(m);
  }
  if (off == 0) return;
  __syncwarp();
  HeapNode nd = w.stage[0];
#pragma unroll 1
  for (int j = 1; j <= off; ++j) {
    const HeapNode nn = w.stage[min(j, off - 1)];
    heap_offer(w, nd, lane);
    nd = nn;
  }
  __syncwarp();
}

// Codes [p0, p1) of the slab (heap full) through one query's heap, in order;
// the warp scores SQ_SCAN codes per step.  |c_p|^2 = -ncc[p].
__device__ __forceinline__ void scan_codes(WarpHeap &w, const int4 (&qv)[7], int qq, const int8_t *__restrict__ codes,
                                           const int *__restrict__ ncc, uint64_t p0, uint64_t p1, int lane) {
  for (uint64_t base = p0; base < p1; base += SQ_SCAN) {
    int d[SQ_SCAN / 32], id[SQ_SCAN / 32];
    int4 c[SQ_SCAN / 32][7];
#pragma unroll
    for (int i = 0; i < SQ_SCAN / 32; ++i) load_code(codes, base + 32 * i + lane, p1, c[i]);
#pragma unroll
    for (int i = 0; i < SQ_SCAN / 32; ++i) {
      const uint64_t p = base + 32 * i + lane;
      d[i] = p < p1 ? qq - ncc[p] - 2 * dot112(c[i], qv) : INT_MAX;
      id[i] = (int)p;
    }
    offer_step(w, d, id, lane);
  }
}

__device__ __forceinline__ void load_query(const int8_t *__restrict__ queries, uint32_t q, int4 (&qv)[7], int &qq) {
  const int4 *src = reinterpret_cast<const int4 *>(queries + (uint64_t)q * SQ8_CODE);
#pragma unroll
  for (int w = 0; w < 7; ++w) qv[w] = __ldg(src + w);
  qq = dot112(qv, qv);
}

// closest_points[k - l - 1] = data_[l + 1].id (bruteforce.h:262-264), and for
// bruteforce_subgraph distances[k - l - 1] = data_[l + 1].dist * alpha^2
__device__ __forceinline__ void write_heap(const HeapNode *heap, uint32_t k, uint64_t q, int *__restrict__ closest,
                                           float *__restrict__ dists, float alpha, int lane) {
  for (uint32_t l = lane; l < k; l += 32) {
    closest[q * k + (k - l - 1)] = heap[l + 1].id;
    if (dists) dists[q * k + (k - l - 1)] = (float)heap[l + 1].d * alpha * alpha;
  }
}

// The screen's accumulator carries most of -|c|^2/2: bytes 112..127 of a
// row (zero padding in every SQ8 code, so the dot product is unchanged) hold
// base-127 digits of f = min(ceil(|c|^2 / 2), SQ_FOLD_MAX) on the code side --
// fifteen digits of weight 127 and one of weight 1 -- and the multipliers
// -127 / -1 on the query side, so the MMA returns z = q.c - f.
constexpr int SQ_FOLD_MAX = 127 * (15 * 127) + 126;

__host__ __device__ __forceinline__ int sq_fold(int cc) { return min((cc + 1) >> 1, SQ_FOLD_MAX); }

// Rows [row0, row0 + 128 * ntiles) of n rows of 112 bytes as 128-row
// core-matrix tiles of 128 bytes per row (rows past n zero), bytes 112..127
// the fold digits (side 0, codes) or multipliers (side 1, queries), and
// ncc[r] = -|row r|^2 (SQ_NCC_PAD past n).  One block per tile.
__global__ void __launch_bounds__(256) k_sq8_tiles(const int8_t *__restrict__ rows, uint64_t n, uint64_t row0,
                                                   int side, unsigned char *__restrict__ tiles,
                                                   int *__restrict__ ncc) {
  const uint64_t t = blockIdx.x;
  unsigned char *o = tiles + t * SQ_TILE;
  for (uint32_t c = threadIdx.x; c < TC_ROWS * 8; c += blockDim.x) {
    const uint32_t r = c >> 3, kc = c & 7;
    const uint64_t p = row0 + t * TC_ROWS + r;
    int4 v = make_int4(0, 0, 0, 0);
    if (p < n) {
      if (kc < 7) {
        v = __ldg(reinterpret_cast<const int4 *>(rows + p * SQ8_CODE) + kc);
      } else {
        int4 cw[7];
        load_code(rows, p, n, cw);
        const int cc = dot112(cw, cw);
        ncc[t * TC_ROWS + r] = -cc;
        int8_t b[16];
        if (side == 0) {
          const int f = sq_fold(cc);
          int e = f / 127;
          for (int i = 0; i < 15; ++i) {
            const int di = e > 127 ? 127 : e;
            b[i] = (int8_t)di;
            e -= di;
          }
          b[15] = (int8_t)(f % 127);
        } else {
          for (int i = 0; i < 15; ++i) b[i] = (int8_t)-127;
          b[15] = (int8_t)-1;
        }
        memcpy(&v, b, 16);
      }
    } else if (kc == 7) {
      ncc[t * TC_ROWS + r] = SQ_NCC_PAD;
    }
    *reinterpret_cast<int4 *>(o + cm_byte(r, kc * 16)) = v;
  }
}

// Distances of the first n codes (rows of stride n padded to SQ_SCAN in dist):
// a thread per code, SQ_DQ queries of a block from shared memory.  Bound by the
// dot products: 28 per pair, |q|^2 and |c|^2 taken once a block (2,048 queries
// over 8,192 codes, k = 140, whole call: 407 us with |q|^2 for every pair, 389
// us now).
__global__ void __launch_bounds__(SQ_SCAN)
    k_sq8_dist(const int8_t *__restrict__ codes, uint64_t n, uint64_t stride, const int8_t *__restrict__ queries,
               uint32_t nq, int *__restrict__ dist) {
  __shared__ int4 qs[SQ_DQ][7];
  __shared__ int qq[SQ_DQ];
  const uint32_t q0 = blockIdx.y * SQ_DQ, m = min((uint32_t)SQ_DQ, nq - q0);
  for (uint32_t i = threadIdx.x; i < m * 7; i += SQ_SCAN)
    qs[i / 7][i % 7] = __ldg(reinterpret_cast<const int4 *>(queries + (uint64_t)q0 * SQ8_CODE) + i);
  const uint64_t p = (uint64_t)blockIdx.x * SQ_SCAN + threadIdx.x;
  int4 c[7];
  load_code(codes, p, n, c);
  const int cc = dot112(c, c);
  __syncthreads();
  if (threadIdx.x < m) qq[threadIdx.x] = dot112(qs[threadIdx.x], qs[threadIdx.x]);
  __syncthreads();
  for (uint32_t j = 0; j < m; ++j) {
    int4 qv[7];
#pragma unroll
    for (int w = 0; w < 7; ++w) qv[w] = qs[j][w];
    dist[(uint64_t)(q0 + j) * stride + p] = p < n ? qq[j] + cc - 2 * dot112(c, qv) : INT_MAX;
  }
}

// Step 1.  With final set (the whole slab is the prefix) it writes the
// answer; else the heap and its root T_q.  dist: the prefix's distances.
__global__ void __launch_bounds__(SQ_WARPS * 32, 4)
    k_sq8_prefix(const int *__restrict__ dist, uint64_t prefix, uint64_t stride, uint32_t nq, uint32_t k, int final,
                 HeapNode *__restrict__ heaps, int *__restrict__ T, int *__restrict__ closest,
                 float *__restrict__ dists, float alpha) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t q = blockIdx.x * SQ_WARPS + warp;
  if (q >= nq) return;  // warp-uniform; the kernel has no block barrier
  WarpHeap w = warp_heap(smem_raw, warp, k);
  const int *row = dist + (uint64_t)q * stride;
  // emplace of the first k
  for (uint64_t base = 0; base < k; base += SQ_SCAN) {
    const int n = (int)min((uint64_t)SQ_SCAN, k - base);
    for (int i = lane; i < n; i += 32) {
      HeapNode nd;
      nd.d = row[base + i];
      nd.id = (int)(base + i);
      w.stage[i] = nd;
    }
    __syncwarp();
    if (lane == 0)
      for (int j = 0; j < n; ++j) heap_emplace(w.h, (int)base + j + 1, w.stage[j]);
    __syncwarp();
  }
  heap_ready(w, lane);
  // the rest, a step's distances loaded while the one before is offered
  const uint64_t b0 = k / SQ_SCAN * SQ_SCAN;
  int nx[SQ_SCAN / 32];
  auto fetch = [&](uint64_t base) {
#pragma unroll
    for (int i = 0; i < SQ_SCAN / 32; ++i) {
      const uint64_t p = base + 32 * i + lane;
      nx[i] = base < prefix && p >= k ? row[p] : INT_MAX;
    }
  };
  fetch(b0);
#pragma unroll 1
  for (uint64_t base = b0; base < prefix; base += SQ_SCAN) {
    int d[SQ_SCAN / 32], id[SQ_SCAN / 32];
#pragma unroll
    for (int i = 0; i < SQ_SCAN / 32; ++i) {
      d[i] = nx[i];
      id[i] = (int)(base + 32 * i + lane);
    }
    fetch(base + SQ_SCAN);
    offer_step(w, d, id, lane);
  }
  if (final) {
    write_heap(w.h, k, q, closest, dists, alpha, lane);
  } else {
    for (uint32_t l = lane; l <= k; l += 32) heaps[(uint64_t)q * (k + 1) + l] = w.h[l];
    if (lane == 0) T[q] = w.root;
  }
}

constexpr int SQ_STAGE_ROW = 36;  // ints per lane row of the candidate staging area

struct SqScreenSmem {
  unsigned char a[SQ_TILE];
  unsigned char b[SQ_BS][SQ_TILE];
  // per epilogue lane, the 32 values y of a chunk that holds candidates
  // (rows padded to 36 ints: conflict-free 16-byte stores)
  int stage[SQ_EPI_WARPS][32 * SQ_STAGE_ROW];
  int ncc[SQ_NB][TC_ROWS];  // -|c|^2 of the tiles' rows
  uint64_t full[SQ_BS], empty[SQ_BS], accfull[2], accempty[2], abar;
  uint32_t tmem_base;
};
static_assert(sizeof(SqScreenSmem) <= 113 * 1024, "two screen CTAs per SM");

__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(SQ_IDESC), "r"(accumulate));
}

// Step 2.  Block (query tile, segment); the segment is code tiles
// [seg * tps, min(nct, (seg + 1) * tps)) of the part, whose tile t
// holds slab rows row0 + 128 t ...  The list of query q for segment seg is
// cand[(q * nseg + seg) * cap ...], its length counts[q * nseg + seg].
__global__ void __launch_bounds__(SQ_THREADS, 2)
    k_sq8_screen(const unsigned char *__restrict__ qtiles, const int *__restrict__ qncc, uint32_t nq,
                 const unsigned char *__restrict__ ctiles, const int *__restrict__ cncc, uint32_t nct, uint32_t tps,
                 uint32_t nseg, uint32_t row0, uint64_t npoints, const int *__restrict__ T, int2 *__restrict__ cand,
                 uint32_t cap, uint32_t *__restrict__ counts, uint32_t *__restrict__ mark, int *err) {
  extern __shared__ __align__(1024) unsigned char screen_smem[];
  SqScreenSmem &sm = *reinterpret_cast<SqScreenSmem *>(screen_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t qt = blockIdx.x, seg = blockIdx.y;
  const uint32_t t0 = seg * tps;
  const uint32_t ntile = t0 < nct ? min(tps, nct - t0) : 0u;

  if (tid == 0) {
    for (int s = 0; s < SQ_BS; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&sm.accfull[a], 1);
      mbar_init(&sm.accempty[a], SQ_EPI_WARPS);
    }
    mbar_init(&sm.abar, 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(SQ_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  if (warp == 0) {
    // ------------------------------------------------ producer
    if (lane == 0) {
      mbar_arrive_expect_tx(&sm.abar, SQ_TILE);
      bulk_g2s(sm.a, qtiles + (uint64_t)qt * SQ_TILE, SQ_TILE, &sm.abar);
      uint32_t issued = 0;
      for (uint32_t sub = 0; sub < ntile; ++sub) {
        const int st = sub % SQ_BS;
        if (sub >= SQ_BS && !mbar_wait_bounded(&sm.empty[st], ((sub / SQ_BS) - 1) & 1, err)) break;
        mbar_arrive_expect_tx(&sm.full[st], SQ_TILE + TC_ROWS * 4);
        bulk_g2s(sm.b[st], ctiles + (uint64_t)(t0 + sub) * SQ_TILE, SQ_TILE, &sm.full[st]);
        // (tile sub - SQ_NB's are done with: its accumulator was released
        // before the MMAs of tile sub - SQ_BS were issued)
        bulk_g2s(sm.ncc[sub % SQ_NB], cncc + (uint64_t)(t0 + sub) * TC_ROWS, TC_ROWS * 4, &sm.full[st]);
        ++issued;
      }
      // no copy may still be landing when the block exits
      mbar_wait_bounded(&sm.abar, 0, err);
      for (uint32_t i = issued > SQ_BS ? issued - SQ_BS : 0; i < issued; ++i)
        mbar_wait_bounded(&sm.full[i % SQ_BS], (i / SQ_BS) & 1, err);
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer
    if (lane == 0) {
      uint32_t done = 0;
      if (mbar_wait_bounded(&sm.abar, 0, err)) {
        const uint32_t a0 = smem_u32(sm.a);
        for (uint32_t sub = 0; sub < ntile; ++sub) {
          const int st = sub % SQ_BS, ab = sub & 1;
          if (!mbar_wait_bounded(&sm.full[st], (sub / SQ_BS) & 1, err)) break;
          if (sub >= 2 && !mbar_wait_bounded(&sm.accempty[ab], ((sub >> 1) - 1) & 1, err)) break;
          tc_fence_after();
          const uint32_t b0 = smem_u32(sm.b[st]);
#pragma unroll
          for (int kk = 0; kk < SQ_MMAS; ++kk) {
            const uint64_t da = umma_desc(a0 + kk * 2 * (TC_ROWS / 8) * 128, (TC_ROWS / 8) * 128, 128);
            const uint64_t db = umma_desc(b0 + kk * 2 * (TC_ROWS / 8) * 128, (TC_ROWS / 8) * 128, 128);
            umma_i8(tmem + ab * TC_ROWS, da, db, kk > 0);
          }
          umma_commit(&sm.empty[st]);
          umma_commit(&sm.accfull[ab]);
          ++done;
        }
      }
      // no MMA may be in flight when TMEM is released
      if (done) mbar_wait_bounded(&sm.accfull[(done - 1) & 1], ((done - 1) >> 1) & 1, err);
    }
  } else {
    // ------------------------------------------------ epilogue: thread = query
    const int wg = warp & 3;  // TMEM lanes 32*wg .. 32*wg+31 are reachable from this warp
    const uint32_t q = qt * TC_ROWS + wg * 32 + lane;
    const bool valid = q < nq;
    // The accumulator is z = q.c - f with f = sq_fold(|c|^2) <= (|c|^2 + 1) / 2,
    // so d = qq + |c|^2 - 2 q.c < T implies 2 z > qq - T - 1: the test
    // z > floor((qq - T - 1) / 2) keeps every code that can enter the heap
    // (and a few more), and d = qq + cc - 2 (z + f) is exact.
    const int qq = valid ? -qncc[q] : 0;
    const int thr = valid ? ((qq - T[q] - 1) >> 1) : INT_MAX;
    int2 *list = cand + ((uint64_t)(valid ? q : 0) * nseg + seg) * cap;
    int *row = &sm.stage[wg][lane * SQ_STAGE_ROW];
    uint32_t cnt = 0;
    bool ok = true;
    for (uint32_t sub = 0; sub < ntile; ++sub) {
      const int ab = sub & 1;
      // warp-uniform: the lanes' timers may disagree at the deadline
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(&sm.accfull[ab], (sub >> 1) & 1, err))) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t tile = t0 + sub;
      const int *nc = sm.ncc[sub % SQ_NB];
      const int id0 = (int)(row0 + tile * TC_ROWS);
      const int ncols = (int)min((uint64_t)TC_ROWS, npoints - (uint64_t)id0);  // the slab's last tile is short
#pragma unroll 1
      for (int c2 = 0; c2 < TC_ROWS; c2 += 64) {
        float v[64];
        tmem_ld64(tmem + ((uint32_t)(wg * 32) << 16) + ab * TC_ROWS + c2, v);
#pragma unroll
        for (int h = 0; h < 64; h += 32) {
          // candidate bits of 32 columns, four independent chains
          uint32_t mk[4] = {0u, 0u, 0u, 0u};
#pragma unroll
          for (int j = 0; j < 32; ++j) mk[j & 3] |= (__float_as_int(v[h + j]) > thr ? 1u : 0u) << j;
          uint32_t mask = (mk[0] | mk[1]) | (mk[2] | mk[3]);
          const int lim = ncols - (c2 + h);
          if (lim < 32) mask &= lim > 0 ? (1u << lim) - 1u : 0u;
          if (mask) {
            // the lane's candidates in column order, z read back from its
            // staging row (the loop runs once per candidate)
#pragma unroll
            for (int j = 0; j < 32; j += 4)
              *reinterpret_cast<int4 *>(row + j) =
                  make_int4(__float_as_int(v[h + j]), __float_as_int(v[h + j + 1]), __float_as_int(v[h + j + 2]),
                            __float_as_int(v[h + j + 3]));
            do {
              const int j = __ffs(mask) - 1;
              mask &= mask - 1;
              const int cc = -nc[c2 + h + j];
              if (cnt < cap) list[cnt] = make_int2(qq + cc - 2 * (row[j] + sq_fold(cc)), id0 + c2 + h + j);
              ++cnt;
            } while (mask);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive1(&sm.accempty[ab]);
    }
    if (valid) {
      counts[(uint64_t)q * nseg + seg] = min(cnt, cap);
      if (!ok || cnt > cap) mark[q] = 1u;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(SQ_TMEM_COLS));
  }
}

// Step 3, the part [r0, r1); last: the answer, else the heap and T_q go on.
// The lists of 32 segments are read as one: a lane finds its entry's segment
// among their running counts, and the next step's entries load while one is
// offered.  (A segment at a time cost a query on its own, whose part has 592
// of them, two memory latencies each.)
__global__ void __launch_bounds__(SQ_WARPS * 32, 4)
    k_sq8_tail(const int8_t *__restrict__ codes, const int *__restrict__ ncc, uint64_t r0, uint64_t r1, int last,
               const int8_t *__restrict__ queries, uint32_t nq, uint32_t k, HeapNode *__restrict__ heaps,
               int *__restrict__ T, const int2 *__restrict__ cand, uint32_t cap, const uint32_t *__restrict__ counts,
               uint32_t nseg, const uint32_t *__restrict__ mark, int *__restrict__ closest, float *__restrict__ dists,
               float alpha) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t q = blockIdx.x * SQ_WARPS + warp;
  if (q >= nq) return;  // warp-uniform; the kernel has no block barrier
  WarpHeap w = warp_heap(smem_raw, warp, k);
  for (uint32_t l = lane; l <= k; l += 32) w.h[l] = heaps[(uint64_t)q * (k + 1) + l];
  heap_ready(w, lane);
  if (mark[q]) {
    int4 qv[7];
    int qq;
    load_query(queries, q, qv, qq);
    scan_codes(w, qv, qq, codes, ncc, r0, r1, lane);
  } else {
    const uint32_t *cn = counts + (uint64_t)q * nseg;
    uint32_t c = lane < nseg ? cn[lane] : 0u;
#pragma unroll 1
    for (uint32_t s0 = 0; s0 < nseg; s0 += 32) {
      uint32_t inc = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      const uint32_t total = __shfl_sync(0xffffffffu, inc, 31), first = inc - c;
      c = s0 + 32 + lane < nseg ? cn[s0 + 32 + lane] : 0u;
      const int2 *lists = cand + ((uint64_t)q * nseg + s0) * cap;
      int2 nx[SQ_SCAN / 32];
      auto fetch = [&](uint32_t j0) {
#pragma unroll
        for (int i = 0; i < SQ_SCAN / 32; ++i) {
          const uint32_t j = j0 + 32 * i + lane;
          int seg = 0;  // the lists that end at or before j
#pragma unroll
          for (int o = 16; o; o >>= 1)
            if (__shfl_sync(0xffffffffu, inc, seg + o - 1) <= j) seg += o;
          const uint32_t f = __shfl_sync(0xffffffffu, first, seg & 31);
          nx[i] = j < total ? lists[(uint64_t)seg * cap + (j - f)] : make_int2(INT_MAX, 0);
        }
      };
      if (total) fetch(0);
#pragma unroll 1
      for (uint32_t j0 = 0; j0 < total; j0 += SQ_SCAN) {
        int d[SQ_SCAN / 32], id[SQ_SCAN / 32];
#pragma unroll
        for (int i = 0; i < SQ_SCAN / 32; ++i) {
          d[i] = nx[i].x;
          id[i] = nx[i].y;
        }
        if (j0 + SQ_SCAN < total) fetch(j0 + SQ_SCAN);
        offer_step(w, d, id, lane);
      }
    }
  }
  __syncwarp();
  if (last) {
    write_heap(w.h, k, q, closest, dists, alpha, lane);
  } else {
    for (uint32_t l = lane; l <= k; l += 32) heaps[(uint64_t)q * (k + 1) + l] = w.h[l];
    if (lane == 0) T[q] = w.root;
  }
}

// Device memory of the current device (or managed memory).
bool is_dev(const void *p) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return mem_loc(p, dev) == MemLoc::Here;
}

struct Scoped {
  void *p = nullptr;
  ~Scoped() {
    if (p) cudaFree(p);
  }
};

// Device copy of a host buffer (or the pointer itself when it is already a
// 16-byte aligned device pointer; the code rows are read as int4).
int stage_in(const void *src, size_t bytes, Scoped &s, const void **out, cudaStream_t st) {
  if (is_dev(src) && ((uintptr_t)src & 15) == 0) {
    *out = src;
    return FKNN_OK;
  }
  FKNN_CUDA(cudaMalloc(&s.p, bytes ? bytes : 16));
  FKNN_CUDA(cudaMemcpyAsync(s.p, src, bytes, cudaMemcpyDefault, st));
  *out = s.p;
  return FKNN_OK;
}

int stage_out(void *dst, size_t bytes, Scoped &s, void **out) {
  if (is_dev(dst)) {
    *out = dst;
    return FKNN_OK;
  }
  FKNN_CUDA(cudaMalloc(&s.p, bytes ? bytes : 16));
  *out = s.p;
  return FKNN_OK;
}

int ensure_device() {
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    set_error("no CUDA device");
    return FKNN_ENODEV;
  }
  return FKNN_OK;
}

int sq8_encode_impl(const float *vecs, uint64_t n, float alpha, int8_t *codes, bool train, float *alpha_out) {
  if (!vecs || !codes || n == 0) {
    set_error("fknn_sq8: bad arguments");
    return FKNN_EINVAL;
  }
  int rc = ensure_device();
  if (rc) return rc;
  int dev = 0;
  FKNN_CUDA(cudaGetDevice(&dev));
  if ((rc = check_local_buffers("fknn_sq8", dev, {vecs, codes}))) return rc;
  cudaStream_t st = 0;
  Scoped sin, sout, sa;
  const float *d_x;
  int8_t *d_c;
  if ((rc = stage_in(vecs, n * DIM * 4, sin, (const void **)&d_x, st))) return rc;
  if ((rc = stage_out(codes, n * SQ8_CODE, sout, (void **)&d_c))) return rc;
  if (train) {
    FKNN_CUDA(cudaMalloc(&sa.p, 4));
    FKNN_CUDA(cudaMemsetAsync(sa.p, 0, 4, st));
    k_absmax<<<148 * 4, 256, 0, st>>>(d_x, n * DIM, (uint32_t *)sa.p);
    g_launches += 1;
    uint32_t bits = 0;
    FKNN_CUDA(cudaMemcpyAsync(&bits, sa.p, 4, cudaMemcpyDeviceToHost, st));
    FKNN_CUDA(cudaStreamSynchronize(st));
    alpha = bits_f32(bits);
    if (alpha_out) *alpha_out = alpha;
  }
  if (!(alpha > 0.f) || !(alpha <= 3.0e38f)) {
    set_error("fknn_sq8: alpha must be positive and finite (all-zero or non-finite training data?)");
    return FKNN_EINVAL;
  }
  k_sq8_encode<<<148 * 8, 256, 0, st>>>(d_x, n, alpha, d_c);
  g_launches += 1;
  FKNN_CUDA(cudaGetLastError());
  if (d_c != codes) FKNN_CUDA(cudaMemcpyAsync(codes, d_c, n * SQ8_CODE, cudaMemcpyDeviceToHost, st));
  FKNN_CUDA(cudaStreamSynchronize(st));
  return FKNN_OK;
}

// Device scratch of the slab brute force: one per calling host thread, with
// its own non-blocking stream, kept between calls (it only grows).  The
// reference calls bruteforce() from concurrent OpenMP workers
// (hybrid_graph.cpp:168,380); with a scratch and a stream each, their calls
// run side by side on the GPU, and after the first call of a thread at a
// given size none of them allocates (cudaFree would wait for the device).
struct Sq8Scratch {
  void *p = nullptr;
  size_t bytes = 0;
  cudaStream_t st = nullptr;
  cudaEvent_t ev = nullptr;  // orders the call after the legacy default stream
  int device = -1;
  int num_sms = 0;
  void release() {
    if (p) cudaFree(p);
    if (ev) cudaEventDestroy(ev);
    if (st) cudaStreamDestroy(st);
    p = nullptr;
    ev = nullptr;
    st = nullptr;
    bytes = 0;
    device = -1;
  }
  ~Sq8Scratch() { release(); }
};

Sq8Scratch &sq8_scratch() {
  thread_local Sq8Scratch s;
  return s;
}

size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

// Segments and list capacity of one part [r0, r1) for a pass of nqb queries.
struct Sq8Part {
  uint64_t r0, r1;
  uint32_t nct, tps, nseg, cap;
};

Sq8Part sq8_part(uint64_t r0, uint64_t npoints, uint32_t nqt, size_t k, int num_sms) {
  Sq8Part p{};
  p.r0 = r0;
  p.r1 = std::min(npoints, r0 * SQ_GROW);
  p.nct = (uint32_t)((p.r1 - p.r0 + TC_ROWS - 1) / TC_ROWS);
  // about four screen CTAs per SM (two resident, two waves)
  const uint32_t nseg = std::max(1u, std::min(p.nct, (uint32_t)((4u * num_sms + nqt - 1) / nqt)));
  p.tps = (p.nct + nseg - 1) / nseg;
  p.nseg = (p.nct + p.tps - 1) / p.tps;
  // a code of the part is a candidate iff it is below the k-th smallest of
  // the r0 before it: about k / r0 of them; the lists hold twice that, and a
  // query whose list fills up takes the exact scan
  const double expect = (double)p.tps * TC_ROWS * (double)k / (double)r0;
  p.cap = (uint32_t)std::min<double>((double)p.tps * TC_ROWS, ((uint32_t)(2.0 * expect) + 64 + 31) & ~31u);
  return p;
}

// Scratch of a pass of nqb queries: query tiles, norms, heaps, bounds, the
// prefix's distances (over before the lists begin) or the lists, counts, marks.
struct Sq8Pass {
  uint32_t nqt;
  size_t lists, counts, bytes;
};

// The prefix's distances: entries of a query, and the queries at a time.  A
// call of many queries makes them for as many as are replayed together, which
// bounds the scratch: 155 MB in place of 268 for 8,192 queries and codes, at
// 1,187 us as before (k = 140).
size_t sq8_dist_stride(uint64_t prefix) { return (size_t)((prefix + SQ_SCAN - 1) / SQ_SCAN * SQ_SCAN); }
uint32_t sq8_dist_queries(uint32_t nqb, uint64_t prefix, int num_sms) {
  return nqb * sq8_dist_stride(prefix) * 4 <= SQ_DIST_BYTES ? nqb : std::min(nqb, (uint32_t)num_sms * SQ_REPLAY_WARPS);
}

Sq8Pass sq8_pass(uint32_t nqb, uint64_t npoints, uint64_t prefix, size_t k, int num_sms) {
  Sq8Pass p{};
  p.nqt = (nqb + TC_ROWS - 1) / TC_ROWS;
  p.lists = sq8_dist_queries(nqb, prefix, num_sms) * sq8_dist_stride(prefix) * 4;
  for (uint64_t r0 = prefix; r0 < npoints;) {
    const Sq8Part a = sq8_part(r0, npoints, p.nqt, k, num_sms);
    p.lists = std::max(p.lists, (size_t)nqb * a.nseg * a.cap * sizeof(int2));
    p.counts = std::max(p.counts, (size_t)nqb * a.nseg * 4);
    r0 = a.r1;
  }
  p.bytes = al256((size_t)p.nqt * SQ_TILE) + al256((size_t)p.nqt * TC_ROWS * 4) +
            al256((size_t)nqb * (k + 1) * sizeof(HeapNode)) + al256((size_t)nqb * 4) + al256(p.lists) +
            al256(p.counts) + al256((size_t)nqb * 4) + 256;
  return p;
}

int sq8_bf_impl(size_t k, int *closest, float *dists, size_t npoints, const char *codes_in, float alpha,
                size_t nqueries, const int8_t *queries_in) {
  if (!closest || !codes_in || !queries_in || k == 0 || k > npoints || k > (size_t)BF_KMAX || nqueries == 0 ||
      npoints >= (1ull << 31) || nqueries >= (1ull << 31)) {
    set_error("fknn_sq8_bruteforce: need 1 <= k <= npoints, k <= 2048, 1 <= nqueries < 2^31, npoints < 2^31");
    return FKNN_EINVAL;
  }
  int rc = ensure_device();
  if (rc) return rc;
  int dev = 0;
  FKNN_CUDA(cudaGetDevice(&dev));
  if ((rc = check_local_buffers("fknn_sq8_bruteforce", dev, {closest, dists, codes_in, queries_in}))) return rc;
  Sq8Scratch &scr = sq8_scratch();
  if (scr.device != dev) {
    // once per thread and device: stream, event, SM count, and the kernels'
    // dynamic shared-memory limits at their largest (k = BF_KMAX)
    scr.release();
    FKNN_CUDA(cudaStreamCreateWithFlags(&scr.st, cudaStreamNonBlocking));
    FKNN_CUDA(cudaEventCreateWithFlags(&scr.ev, cudaEventDisableTiming));
    FKNN_CUDA(cudaDeviceGetAttribute(&scr.num_sms, cudaDevAttrMultiProcessorCount, dev));
    const int rmax = (int)((size_t)SQ_WARPS * sq_region(BF_KMAX) * sizeof(HeapNode));
    FKNN_CUDA(cudaFuncSetAttribute(k_sq8_prefix, cudaFuncAttributeMaxDynamicSharedMemorySize, rmax));
    FKNN_CUDA(cudaFuncSetAttribute(k_sq8_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, rmax));
    FKNN_CUDA(cudaFuncSetAttribute(k_sq8_screen, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(SqScreenSmem)));
    scr.device = dev;
  }
  const int num_sms = scr.num_sms;
  const uint32_t nq = (uint32_t)nqueries, K = (uint32_t)k;
  const bool screened = npoints > SQ_PREFIX;
  const uint64_t prefix = screened ? SQ_PREFIX : npoints;
  const uint32_t nct_all = (uint32_t)((npoints + TC_ROWS - 1) / TC_ROWS);
  const uint32_t qbatch = std::min(nq, SQ_QBATCH);
  const uint32_t qlast = nq - (nq - 1) / qbatch * qbatch;
  const Sq8Pass pa = sq8_pass(qbatch, npoints, prefix, k, num_sms);
  const Sq8Pass pb = sq8_pass(qlast, npoints, prefix, k, num_sms);

  // inputs already on the device (16-byte aligned) are used in place, the
  // rest staged through the scratch, as are outputs that live on the host
  const bool codes_dev = is_dev(codes_in) && ((uintptr_t)codes_in & 15) == 0;
  const bool q_dev = is_dev(queries_in) && ((uintptr_t)queries_in & 15) == 0;
  const bool ids_dev = is_dev(closest);
  const bool d_dev = dists && is_dev(dists);
  const size_t b_codes = codes_dev ? 0 : al256(npoints * SQ8_CODE);
  const size_t b_q = q_dev ? 0 : al256(nqueries * SQ8_CODE);
  const size_t b_ids = ids_dev ? 0 : al256(nqueries * k * 4);
  const size_t b_d = (!dists || d_dev) ? 0 : al256(nqueries * k * 4);
  const size_t codes_bytes = screened ? al256((size_t)nct_all * SQ_TILE) + al256((size_t)nct_all * TC_ROWS * 4) : 0;
  const size_t need = b_codes + b_q + b_ids + b_d + codes_bytes + std::max(pa.bytes, pb.bytes) + 256;

  if (scr.bytes < need) {
    if (scr.p) cudaFree(scr.p);
    scr.p = nullptr;
    scr.bytes = 0;
    FKNN_CUDA(cudaMalloc(&scr.p, need));
    scr.bytes = need;
  }
  const cudaStream_t st = scr.st;
  // device inputs are read in place: whatever the legacy default stream (and
  // the blocking streams it orders) has queued so far comes first
  FKNN_CUDA(cudaEventRecord(scr.ev, 0));
  FKNN_CUDA(cudaStreamWaitEvent(st, scr.ev, 0));
  unsigned char *base = static_cast<unsigned char *>(scr.p);
  const int8_t *d_codes = codes_dev ? reinterpret_cast<const int8_t *>(codes_in) : reinterpret_cast<int8_t *>(base);
  base += b_codes;
  const int8_t *d_q = q_dev ? queries_in : reinterpret_cast<int8_t *>(base);
  base += b_q;
  int *d_ids = ids_dev ? closest : reinterpret_cast<int *>(base);
  base += b_ids;
  float *d_d = !dists ? nullptr : d_dev ? dists : reinterpret_cast<float *>(base);
  base += b_d;
  if (!codes_dev)
    FKNN_CUDA(cudaMemcpyAsync(const_cast<int8_t *>(d_codes), codes_in, npoints * SQ8_CODE, cudaMemcpyDefault, st));
  if (!q_dev)
    FKNN_CUDA(cudaMemcpyAsync(const_cast<int8_t *>(d_q), queries_in, nqueries * SQ8_CODE, cudaMemcpyDefault, st));
  unsigned char *ctiles = base;
  int *cncc = reinterpret_cast<int *>(base + al256((size_t)nct_all * SQ_TILE));
  unsigned char *pass_base = base + codes_bytes;
  int *d_err = reinterpret_cast<int *>(base + codes_bytes + std::max(pa.bytes, pb.bytes));

  const size_t rsmem = (size_t)SQ_WARPS * sq_region(K) * sizeof(HeapNode);
  if (screened) {
    FKNN_CUDA(cudaMemsetAsync(d_err, 0, sizeof(int), st));
    // |c|^2 of every code (the tail uses it too) and the tiles.  A slab that is
    // replayed whole needs neither, nor an error flag (2,048 queries over 2,000
    // codes, k = 140: 256 us with them, 240 without)
    k_sq8_tiles<<<nct_all, 256, 0, st>>>(d_codes, npoints, 0, 0, ctiles, cncc);
    g_launches += 1;
  }
  for (uint32_t q0 = 0; q0 < nq; q0 += qbatch) {
    const uint32_t nqb = std::min(qbatch, nq - q0);
    const Sq8Pass ps = sq8_pass(nqb, npoints, prefix, k, num_sms);
    size_t off = 0;
    auto take = [&](size_t b) {
      unsigned char *p = pass_base + off;
      off += al256(b);
      return p;
    };
    unsigned char *qtiles = take((size_t)ps.nqt * SQ_TILE);
    int *qncc = reinterpret_cast<int *>(take((size_t)ps.nqt * TC_ROWS * 4));
    HeapNode *heaps = reinterpret_cast<HeapNode *>(take((size_t)nqb * (k + 1) * sizeof(HeapNode)));
    int *T = reinterpret_cast<int *>(take((size_t)nqb * 4));
    void *lists = take(ps.lists);
    int2 *cand = static_cast<int2 *>(lists);
    uint32_t *counts = reinterpret_cast<uint32_t *>(take(ps.counts));
    uint32_t *mark = reinterpret_cast<uint32_t *>(take((size_t)nqb * 4));
    const int8_t *qs = d_q + (uint64_t)q0 * SQ8_CODE;
    int *ids = d_ids + (uint64_t)q0 * k;
    float *dd = d_d ? d_d + (uint64_t)q0 * k : nullptr;
    const unsigned rblocks = (nqb + SQ_WARPS - 1) / SQ_WARPS;
    int *dist = static_cast<int *>(lists);
    const size_t stride = sq8_dist_stride(prefix);
    const uint32_t dq = sq8_dist_queries(nqb, prefix, num_sms);
    for (uint32_t c0 = 0; c0 < nqb; c0 += dq) {
      const uint32_t m = std::min(nqb - c0, dq);
      k_sq8_dist<<<dim3((unsigned)(stride / SQ_SCAN), (m + SQ_DQ - 1) / SQ_DQ), SQ_SCAN, 0, st>>>(
          d_codes, prefix, stride, qs + (uint64_t)c0 * SQ8_CODE, m, dist);
      k_sq8_prefix<<<(m + SQ_WARPS - 1) / SQ_WARPS, SQ_WARPS * 32, rsmem, st>>>(
          dist, prefix, stride, m, K, screened ? 0 : 1, heaps + (uint64_t)c0 * (k + 1), T + c0, ids + (uint64_t)c0 * k,
          dd ? dd + (uint64_t)c0 * k : nullptr, alpha);
      g_launches += 2;
    }
    if (screened) {
      k_sq8_tiles<<<ps.nqt, 256, 0, st>>>(qs, nqb, 0, 1, qtiles, qncc);
      g_launches += 1;
    }
    for (uint64_t r0 = prefix; r0 < npoints;) {
      const Sq8Part a = sq8_part(r0, npoints, ps.nqt, k, num_sms);
      FKNN_CUDA(cudaMemsetAsync(mark, 0, (size_t)nqb * 4, st));
      k_sq8_screen<<<dim3(ps.nqt, a.nseg), SQ_THREADS, sizeof(SqScreenSmem), st>>>(
          qtiles, qncc, nqb, ctiles + (size_t)(r0 / TC_ROWS) * SQ_TILE, cncc + r0, a.nct, a.tps, a.nseg, (uint32_t)r0,
          a.r1, T, cand, a.cap, counts, mark, d_err);
      k_sq8_tail<<<rblocks, SQ_WARPS * 32, rsmem, st>>>(d_codes, cncc, r0, a.r1, a.r1 == npoints, qs, nqb, K, heaps, T,
                                                        cand, a.cap, counts, a.nseg, mark, ids, dd, alpha);
      g_launches += 2;
      r0 = a.r1;
    }
    FKNN_CUDA(cudaGetLastError());
  }
  // the kernels finish before any copy to (pageable) host memory is queued,
  // so those copies do not wait on the GPU inside the driver's copy path,
  // where concurrent callers' copies would queue behind them
  FKNN_CUDA(cudaStreamSynchronize(st));
  if (!ids_dev) FKNN_CUDA(cudaMemcpyAsync(closest, d_ids, nqueries * k * 4, cudaMemcpyDeviceToHost, st));
  if (dists && !d_dev) FKNN_CUDA(cudaMemcpyAsync(dists, d_d, nqueries * k * 4, cudaMemcpyDeviceToHost, st));
  int err = 0;
  if (screened) FKNN_CUDA(cudaMemcpyAsync(&err, d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
  FKNN_CUDA(cudaStreamSynchronize(st));
  if (err & ERR_WAIT_TIMEOUT) {
    // outputs are complete (the affected queries took the exact scan)
    set_error("fknn_sq8_bruteforce: a bounded device wait gave up; affected queries were answered by the exact scan");
    return FKNN_ETIMEOUT;
  }
  return FKNN_OK;
}

}  // namespace

void launch_sq8_encode(const float *d_x, uint64_t n, float alpha, int8_t *d_codes, cudaStream_t st) {
  k_sq8_encode<<<148 * 8, 256, 0, st>>>(d_x, n, alpha, d_codes);
  g_launches += 1;
}

}  // namespace fknn

using namespace fknn;

extern "C" {

int fknn_sq8_sym_train(const float *vecs, uint64_t n, float *alpha, int8_t *codes) {
  g_launches = 0;
  if (!alpha) {
    set_error("fknn_sq8_sym_train: alpha is NULL");
    return FKNN_EINVAL;
  }
  return sq8_encode_impl(vecs, n, 0.f, codes, true, alpha);
}

int fknn_sq8_sym_encode(const float *vecs, uint64_t n, float alpha, int8_t *codes) {
  g_launches = 0;
  return sq8_encode_impl(vecs, n, alpha, codes, false, nullptr);
}

int fknn_sq8_bruteforce(size_t dim, size_t k, int *closest_points, size_t npoints, const char *codes_in, float alpha,
                        size_t nqueries, const int8_t *queries_in) {
  (void)dim;
  g_launches = 0;
  return sq8_bf_impl(k, closest_points, nullptr, npoints, codes_in, alpha, nqueries, queries_in);
}

int fknn_sq8_bruteforce_subgraph(size_t dim, size_t k, int *closest_points, float *distances, size_t npoints,
                                 const char *codes_in, float alpha, size_t nqueries, const int8_t *queries_in) {
  (void)dim;
  g_launches = 0;
  if (!distances) {
    set_error("fknn_sq8_bruteforce_subgraph: distances is NULL");
    return FKNN_EINVAL;
  }
  return sq8_bf_impl(k, closest_points, distances, npoints, codes_in, alpha, nqueries, queries_in);
}

int fknn_sq8_release_thread_scratch(void) {
  // the thread's stream has no work left: every SQ8 call waits for it
  sq8_scratch().release();
  return FKNN_OK;
}

}  // extern "C"
