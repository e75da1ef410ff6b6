// Screen of the exact FP32 search on the tensor cores.
//
// Rows and queries are scaled by powers of two taken from their norms (so
// that every element is below 2^14 and the smallest error an fp16 pair makes
// is 2^-38 of the norm) and split into two fp16 pieces, x = h + l with h the
// nearest fp16 and l the nearest fp16 of the rest: 22 bits and a sign, |x - h
// - l| <= 2^-22 |x|.  q.x is qh.xl + ql.xh + qh.xh, accumulated in FP32 by
// tcgen05.mma with the small products first, so that only the last seven MMA
// steps add at full magnitude, where the FMA chain adds 100 times; the
// epilogue takes the scales back (exactly) and adds -|x|^2/2.
//
// Error: the pieces and the dropped ql.xl are within 3 * 2^-22 |q||x|; with
// each step's 17 addends cut at the 24th bit below the largest, the seven
// full-size steps are within 7.1e-6 |q||x|.  ds = |q|^2 + |x|^2 - 2 q.x is
// then inside screen_eps's bound five times over, and measured against 64 bits
// its error is no larger than an FMA chain's (4.3e-8 rms, 3.1e-7 at most,
// relative to (|x| + |q|)^2; the chain 5.5e-8 and 3.5e-7).  The candidates it keeps are
// re-scored in FP32 (k_merge), so results do not depend on it.
#include <algorithm>
#include <cfloat>
#include <climits>

#include <cuda_fp16.h>

#include "screen_util.cuh"

namespace fknn {

namespace {

constexpr int XQ = EXACT_TQ;                  // queries per tile: two halves of 128 = MMA M = TMEM lanes
constexpr int XM = XQ / 2;
constexpr int XR = EXACT_ROWS;                // rows per sub-tile = MMA N: two 64-row layout blocks
constexpr int XK = 112;                       // 100 dims, zero padding
constexpr uint32_t X_PIECE = (uint32_t)XR * XK * 2;  // one fp16 piece of a sub-tile
constexpr int X_MMAS = XK / 16;               // kind::f16: K = 16 per MMA
constexpr int X_ST = 2;                       // split sub-tiles in shared memory
constexpr int X_FB = 3;                       // ... and 64-row blocks as they come from memory
constexpr int X_NORMS = 8;                    // sub-tiles whose norms are kept (the epilogue is less than 5 behind)
constexpr int X_GROUPS = 2;                   // accumulators, each with a group of epilogue warps
constexpr int X_EPI_WARPS = 4;                // warps of a group: TMEM lanes 32 w ..
constexpr int X_EPI = X_GROUPS * X_EPI_WARPS; // warps 0 .. 7
static_assert(X_EPI * 32 == XQ, "an epilogue thread per query of a tile");
constexpr int X_CONV_WARPS = 6;               // warps 8 .. 13
constexpr int X_UNITS = (BLK / 32) * 13;      // converter units of a block: 32 rows x 8 dims
constexpr int X_LOAD_WARP = X_EPI + X_CONV_WARPS;
constexpr int X_MMA_WARP = X_LOAD_WARP + 1;
constexpr int X_THREADS = (X_MMA_WARP + 1) * 32;
constexpr uint32_t X_TMEM_COLS = 512;
constexpr uint32_t X_A = XK;                  // TMEM columns of a half's query pieces (two of XK / 2)
constexpr uint32_t X_ACC = 256;               // accumulators: columns 256.. and 384..; the query pieces below
constexpr int X_LIST = 384;                   // entries of an epilogue thread's working list
constexpr int X_NPL = X_LIST / 32;
constexpr int X_SLACK = 24;                   // entries past the k-th that a trim may keep
constexpr int X_NO_FOLD = INT_MAX;
constexpr int X_FOLD_SPAN = 36;               // query scales of one item whose norm slots all fit fp16's powers of two
constexpr int X_SLOTS = 8;                    // candidate rows an epilogue warp stages at a time
constexpr uint32_t X_REFRESH = 16;            // sub-tiles between reads of the shared bound
// F32 accumulate, FP16 A and B, K-major, N = XR, M = XM
constexpr uint32_t X_IDESC = (1u << 4) | ((uint32_t)(XR >> 3) << 17) | ((uint32_t)(XM >> 4) << 24);

using XWarp = ScreenWarp<X_SLOTS>;

struct XSmem {
  unsigned char b[X_ST][2][X_PIECE];  // split row sub-tiles
  float f[X_FB][BLK_FLOATS];          // row blocks
  XWarp w[X_EPI];
  float nh[X_NORMS][XR];              // -|x|^2 / 2 per row
  float rs[X_NORMS][XR];              // 1 / scale per row
  float crs[X_NORMS][XR / 32];        // 32 rows' 1 / scale: where they agree and -|x|^2/2 is in the MMA; negative
                                      // where they agree only; 0 where they differ
  float thr[XQ];                      // per epilogue thread: current upper bound T on the k-th distance
  int cnt[XQ];
  float qn[XQ];
  int32_t lq[XQ];
  uint64_t ffull[X_FB], fempty[X_FB], bfull[X_ST], bempty[X_ST], accfull[X_GROUPS], accempty[X_GROUPS], afull;
  uint32_t tmem_base;
  int hmin[2], hmax[2];  // by item parity: smallest and largest 14 - scale_exp of the item's queries
  uint32_t next[2];  // the next work item, by item parity
};
static_assert(sizeof(XSmem) <= 227 * 1024, "one screen CTA per SM");

// D[tmem] (+)= A[tmem] * B[smem]: A is the query side, lane = query, two K
// elements per 32-bit column
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(db), "r"(X_IDESC), "r"(accumulate));
}

// Exponent of the scale of a vector with squared norm n2: |x_i| 2^e < 2^14
// (1 + 1e-5).  Any float n2 >= 0, a zero or subnormal one included.
__device__ __forceinline__ int scale_exp(float n2) {
  const int eb = (int)(__float_as_uint(n2) >> 23) - 127;  // n2 < 2^(eb + 1)
  return 14 - ((eb + 2) >> 1);
}
__device__ __forceinline__ float pow2f(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }

// (a, b) -> packed fp16 pieces, a in the low half; the difference is exact
__device__ __forceinline__ void split2(float a, float b, uint32_t &h, uint32_t &l) {
  const __half2 hh = __floats2half2_rn(a, b);
  const float2 f = __half22float2(hh);
  const __half2 ll = __floats2half2_rn(a - f.x, b - f.y);
  memcpy(&h, &hh, 4);
  memcpy(&l, &ll, 4);
}

// The scale exponent of an item's norm slots: one above its queries' smallest
// 14 - scale_exp, so that the queries' side, 2^(scale_exp + fold), lies in
// [2^-21, 2^15].
__device__ __forceinline__ int fold_exp(const XSmem &sm, uint32_t par) {
  const int lo = sm.hmin[par], hi = sm.hmax[par];
  return lo <= hi && hi - lo <= X_FOLD_SPAN ? lo + 1 : X_NO_FOLD;
}

// The entries of up to two lists (32 NPL entries at most, n in all, element i
// of the concatenation given by at(i)) bounded and written to dst: the k-th
// screening distance, or one a little above, bounds the k-th reference
// distance from above (screen_hi), and rows whose lower bound (screen_lo)
// exceeds the bound go.  Without `select` only the bound at hand is applied.
// Whole warp; returns the number kept, which may exceed what the caller can
// hold (then nothing past dst_cap is written).
template <int NPL, class At>
__device__ __forceinline__ int x_bound(At at, int n, bool select, uint32_t k, float qn, float &T, uint32_t *T_q,
                                       uint32_t *hist, Candidate *dst_list, int dst_cap) {
  const int lane = threadIdx.x & 31;
  const float Tg = sortable_f32(ld_volatile_u32(T_q));
  uint32_t key[NPL], pos[NPL];
#pragma unroll
  for (int j = 0; j < NPL; ++j) {
    const int i = j * 32 + lane;
    uint2 c = make_uint2(0xffffffffu, 0u);
    if (i < n) c = at(i);
    key[j] = i < n ? f32_sortable(__uint_as_float(c.x)) : 0xffffffffu;
    pos[j] = c.y;
  }
  if (select && n >= (int)k)
    T = fminf(T, screen_hi(sortable_f32(warp_kth_upper<NPL>(key, n, (int)k, X_SLACK, hist)), qn));
  if (Tg < T) T = Tg;
  if (lane == 0 && T < Tg) atomicMin(T_q, f32_sortable(T));
  // (the bound on ds itself, one compare per entry: rows past it have screen_lo > T)
  const float lim = screen_push_limit(T, qn);
  int kept = 0;
  const uint32_t lt = (1u << lane) - 1u;
  uint2 *dst = reinterpret_cast<uint2 *>(dst_list);
  __syncwarp();
#pragma unroll
  for (int j = 0; j < NPL; ++j) {
    if (j * 32 >= n) break;
    const float ds = sortable_f32(key[j]);
    const bool keep = j * 32 + lane < n && (T == INFINITY || ds <= lim);
    const uint32_t b = __ballot_sync(0xffffffffu, keep);
    const int o = kept + __popc(b & lt);
    if (keep && o < dst_cap) dst[o] = make_uint2(__float_as_uint(ds), pos[j]);
    kept += __popc(b);
  }
  __syncwarp();
  return kept;
}

// Trim of one working list that could overflow in its next sub-tile.
__device__ __noinline__ void x_trim(Candidate *list, XSmem &sm, int L, uint32_t k, uint32_t *T_global, uint32_t *ovf) {
  const int n = sm.cnt[L];
  const int32_t qi = sm.lq[L];
  float T = sm.thr[L];
  const uint2 *src = reinterpret_cast<const uint2 *>(list);
  const int kept = x_bound<X_NPL>([&](int i) { return src[i]; }, n, true, k, sm.qn[L], T, T_global + qi,
                                  sm.w[threadIdx.x >> 5].hist, list, X_LIST);
  if ((threadIdx.x & 31) == 0) {
    if (kept > X_LIST - XR) {
      ovf[qi] = 1u;  // more near-ties than the list can hold: the exact scan answers the query
      sm.cnt[L] = 0;
      sm.thr[L] = -INFINITY;
    } else {
      sm.cnt[L] = kept;
      sm.thr[L] = T;
    }
  }
  __syncwarp();
}

// The item's result for one query: its working list (or two, one of each
// group: L1 >= 0), at most EXACT_CAP entries.
template <int NPL>
__device__ __noinline__ void x_finish(const Candidate *work, XSmem &sm, int L, int L1, uint32_t k, uint32_t *T_global,
                                      uint32_t *ovf, Candidate *out, uint32_t *out_cnt) {
  const int n0 = sm.cnt[L], n = n0 + (L1 >= 0 ? sm.cnt[L1] : 0);
  const int32_t qi = sm.lq[L];
  float T = L1 >= 0 ? fminf(sm.thr[L], sm.thr[L1]) : sm.thr[L];
  if (n == 0 || T == -INFINITY) {  // nothing, or marked: the exact scan answers it (and the mark is no bound)
    if ((threadIdx.x & 31) == 0) *out_cnt = 0;
    return;
  }
  const uint2 *s0 = reinterpret_cast<const uint2 *>(work + (uint64_t)L * X_LIST);
  const uint2 *s1 = reinterpret_cast<const uint2 *>(work + (uint64_t)(L1 >= 0 ? L1 : 0) * X_LIST);
  int kept = x_bound<NPL>([&](int i) { return i < n0 ? s0[i] : s1[i - n0]; }, n, n > EXACT_CAP, k, sm.qn[L], T,
                          T_global + qi, sm.w[threadIdx.x >> 5].hist, out, EXACT_CAP);
  if (kept > EXACT_CAP) {
    if ((threadIdx.x & 31) == 0) ovf[qi] = 1u;
    kept = 0;
  }
  if ((threadIdx.x & 31) == 0) *out_cnt = (uint32_t)kept;
}

// A converter warp's loop over an item's sub-tiles: units cw, cw + 6, ... of
// each of their two 64-row blocks (unit u: rows 32 (u % 2) .., dims 8 (u / 2)
// ..).  The blocks come through shared memory as bulk copies, so the loop
// body is short and holds nothing in flight in registers: with loads from
// global memory in it (72 registers of them, the units unrolled) its code
// and the epilogue's did not fit the instruction caches together and both ran
// at half speed.  g0: the sub-tiles of this CTA's earlier items.
//
// The last unit of a row (dims 96..103) also hands on its norm: as slots 100
// .. 102 of the high piece, -|x|^2/2 2^(14 - H - fold) in three fp16 pieces
// against the queries' 2^(14 - Hq + fold), where the 32 rows of the unit share
// the scale 2^(14 - H) and the slot stays in range (fold - 8 <= H <= fold + 2);
// else the slots are zero and the epilogue adds it.
__device__ __forceinline__ bool convert_rows(XSmem &sm, uint32_t nblk, uint32_t blk0, uint32_t stride, uint32_t nsub,
                                             uint32_t g0, int cw, int fold, int *err) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (uint32_t sub = 0; sub < nsub; ++sub) {
    const uint32_t gs = g0 + sub;
    const uint32_t st = gs % X_ST, rd = gs / X_ST;
    // warp-uniform: the lanes' timers may disagree at the deadline
    if (rd > 0 && !__all_sync(0xffffffffu, mbar_wait_bounded(&sm.bempty[st], (rd - 1) & 1, err))) return false;
#pragma unroll 1
    for (uint32_t hb = 0; hb < XR / BLK; ++hb) {
      const uint32_t fi = gs * (XR / BLK) + hb;
      const uint32_t fs = fi % X_FB, fr = fi / X_FB;
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(&sm.ffull[fs], fr & 1, err))) return false;
      const bool on = (blk0 + sub * stride) * (XR / BLK) + hb < nblk;  // the base's last 64-row block may be absent
#pragma unroll 1
      for (int u = cw; u < X_UNITS; u += X_CONV_WARPS) {
        const int rb = (u & 1) * 32 + lane, r = (int)hb * BLK + rb, grp = u >> 1;
        const float *x = sm.f[fs] + grp * 8 * BLK + rb;
        const float xn = on ? sm.f[fs][DIM * BLK + rb] : 0.f;
        const int ex = scale_exp(xn);
        const float sc = pow2f(ex);
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = on && (e < 4 || grp < 12) ? x[e * BLK] * sc : 0.f;
        uint32_t h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split2(v[2 * e], v[2 * e + 1], h[e], l[e]);
        if (grp == 12) {
          const uint32_t slot = gs % X_NORMS;
          const float inv = pow2f(-ex), nh = -0.5f * xn;
          const int H = 14 - ex;
          const bool same = __all_sync(0xffffffffu, ex == __shfl_sync(0xffffffffu, ex, 0));
          const bool folded = same && fold != X_NO_FOLD && H >= fold - 8 && H <= fold + 2;
          if (folded) {
            const float w = nh * pow2f(ex - fold);
            const float n1 = __half2float(__float2half_rn(w)), n2 = __half2float(__float2half_rn(w - n1));
            const __half2 a = __floats2half2_rn(n1, n2), b = __floats2half2_rn(w - n1 - n2, 0.f);
            memcpy(&h[2], &a, 4);
            memcpy(&h[3], &b, 4);
          }
          sm.nh[slot][r] = nh;
          sm.rs[slot][r] = inv;
          if (lane == 0) sm.crs[slot][r >> 5] = !same ? 0.f : folded ? inv : -inv;
        }
        const uint32_t o = cm_byte((uint32_t)r, (uint32_t)grp * 16);
        *reinterpret_cast<uint4 *>(sm.b[st][0] + o) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4 *>(sm.b[st][1] + o) = make_uint4(l[0], l[1], l[2], l[3]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive1(&sm.fempty[fs]);  // this warp is done with the block
    }
    fence_proxy_async();  // the MMAs read these bytes through the async proxy
    __syncwarp();
    if (lane == 0) mbar_arrive1(&sm.bfull[st]);
  }
  return true;
}

// acc -> q.x - |x|^2/2 of 32 columns whose norms are not in the accumulator
__device__ __forceinline__ void x_values(uint32_t (&r)[32], const XSmem &sm, uint32_t slot, int c, float cr, float iq) {
  const float4 *nh = reinterpret_cast<const float4 *>(&sm.nh[slot][c]);
  const float4 *rs = reinterpret_cast<const float4 *>(&sm.rs[slot][c]);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float4 v = nh[j];
    const float4 s = cr != 0.f ? make_float4(-cr, -cr, -cr, -cr) : rs[j];
    r[4 * j] = __float_as_uint(fmaf(__uint_as_float(r[4 * j]) * s.x, iq, v.x));
    r[4 * j + 1] = __float_as_uint(fmaf(__uint_as_float(r[4 * j + 1]) * s.y, iq, v.y));
    r[4 * j + 2] = __float_as_uint(fmaf(__uint_as_float(r[4 * j + 2]) * s.z, iq, v.z));
    r[4 * j + 3] = __float_as_uint(fmaf(__uint_as_float(r[4 * j + 3]) * s.w, iq, v.w));
  }
}

// A sub-tile in which some norms are not in the accumulator (rows whose
// scales differ, or are far from the queries'): one chunk, every lane
// appending from its own registers.
__device__ __noinline__ int x_push_norms(uint32_t taddr, const XSmem &sm, uint32_t slot, int c, float iq, float bound,
                                         float qn, int r0, int r1, uint32_t pos, Candidate *list, int cnt) {
  uint32_t r[32];
  tmem_ld32_issue(taddr, r);
  tmem_wait_ld(r);
  const float cr = sm.crs[slot][c >> 5];
  if (cr > 0.f) {
    const float f = cr * iq;
#pragma unroll
    for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * f);
  } else {
    x_values(r, sm, slot, c, cr, iq);
  }
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    const float v = __uint_as_float(r[j]);
    if (v >= bound && j >= r0 && j < r1) {
      Candidate cd;
      cd.ds = fmaf(-2.f, v, qn);
      cd.pos = pos + j;
      list[cnt++] = cd;
    }
  }
  return cnt;
}

// Persistent, one CTA per SM (the split sub-tiles fill the shared memory),
// pulling work items (longest first) from a queue: warp 14 copies row blocks
// in, warps 8-13 convert them, warp 15 issues MMAs, warps 0-3 screen accumulator 0 and warps 4-7 accumulator 1.
// The query pieces stay in TMEM for the whole item, so the MMAs read only the
// row side from shared memory.  A tile of more than 128 queries multiplies
// every sub-tile with both halves of its queries, one accumulator each, so a
// conversion and its loads serve 256 queries and the MMAs of one half run
// while the other half is screened; a smaller tile has one half, and the
// accumulators (and epilogue groups) take its sub-tiles in turn.
// Bound by the tensor cores on long slabs (42 MMAs of 91 cycles a sub-tile of
// 256 queries, 60 % busy over a whole call) and by the candidates on short
// ones.  Screens of a call, pilot included, before (FP32 cores) and now: 16
// queries over 1e6 rows 2.99 and 0.33 ms, 100,000 over 1e6 225 and 26.4 ms,
// 10,000 over 1e5 18.7 and 1.55 ms.
// Barrier phases run on across items: g counts the sub-tiles of this CTA's
// earlier items, nrun those items themselves, u0 / u1 the uses of the accumulators.
__global__ void __launch_bounds__(X_THREADS, 1) k_exact_screen(ExactScreenArgs A) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  XSmem &sm = *reinterpret_cast<XSmem *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (A.active && *A.active == 0) return;  // (uniform: before any barrier or TMEM use)

  if (tid == 0) {
    for (int s = 0; s < X_ST; ++s) {
      mbar_init(&sm.bfull[s], X_CONV_WARPS);
      mbar_init(&sm.bempty[s], 1);
    }
    for (int s = 0; s < X_FB; ++s) {
      mbar_init(&sm.ffull[s], 1);
      mbar_init(&sm.fempty[s], X_CONV_WARPS);
    }
    for (int a = 0; a < X_GROUPS; ++a) {
      mbar_init(&sm.accfull[a], 1);
      mbar_init(&sm.accempty[a], X_EPI_WARPS);
    }
    mbar_init(&sm.afull, X_EPI);
    sm.hmin[0] = INT_MAX;
    sm.hmax[0] = INT_MIN;
    fence_mbar_init();
  }
  if (warp == X_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(X_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  // the last 16 bytes of K (dims 104..111) are zero for good (written by
  // converter threads, whose fence precedes every hand-over to the MMAs)
  if (warp >= X_EPI && warp < X_LOAD_WARP)
    for (int c = tid - X_EPI * 32; c < X_ST * 2 * XR; c += X_CONV_WARPS * 32)
      *reinterpret_cast<uint4 *>(sm.b[c / XR / 2][c / XR % 2] + cm_byte(c % XR, (XK / 8 - 1) * 16)) =
          make_uint4(0, 0, 0, 0);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  uint32_t g = 0, iter = 0, nrun = 0, u0 = 0, u1 = 0;
  // a bounded wait gave up: the CTA's later items only mark their queries
  // (combined over the block at each item's closing barrier, so uniform)
  bool aborted = false;
  for (uint32_t item_id = blockIdx.x; item_id < A.nitems; ++iter) {
    const WorkItem it = A.items[item_id];
    const Tile tl = A.tiles[it.tile];
    const float *blocks = tl.order == ORDER_TIME ? A.blocks_t : A.blocks_c;
    const bool both = tl.nq > (uint32_t)XM;
    // every stride-th row block of the item (stride 1: all of them)
    uint32_t nsub = (it.blk1 - it.blk0 + A.stride - 1) / A.stride;
    bool gave_up = false;

    if (warp >= X_EPI && warp < X_LOAD_WARP) {
      // ------------------------------------------------ converters
      if (!__syncthreads_or(0)) nsub = 0;  // the item's opening barrier
      if (!aborted)
        gave_up = !convert_rows(sm, A.nblk, it.blk0, A.stride, nsub, g, warp - X_EPI, fold_exp(sm, iter & 1), A.err);
    } else if (warp == X_LOAD_WARP) {
      // ------------------------------------------------ producer
      if (!__syncthreads_or(0)) nsub = 0;  // the item's opening barrier
      if (lane == 0 && !aborted) {
        const uint32_t f0 = g * (XR / BLK), nf = nsub * (XR / BLK);
        uint32_t done = 0;
#pragma unroll 1
        for (; done < nf; ++done) {
          const uint32_t fi = f0 + done, fs = fi % X_FB, fr = fi / X_FB;
          if (fr > 0 && !mbar_wait_bounded(&sm.fempty[fs], (fr - 1) & 1, A.err)) break;
          const uint32_t b = (it.blk0 + (done / (XR / BLK)) * A.stride) * (XR / BLK) + done % (XR / BLK);
          if (b < A.nblk) {
            mbar_arrive_expect_tx(&sm.ffull[fs], BLK_BYTES);
            bulk_g2s(sm.f[fs], blocks + (uint64_t)b * BLK_FLOATS, BLK_BYTES, &sm.ffull[fs]);
          } else {
            mbar_arrive1(&sm.ffull[fs]);
          }
        }
        // every issued copy has landed before the item ends
        bool ok = done == nf;
#pragma unroll 1
        for (uint32_t i = done > X_FB ? done - X_FB : 0; i < done; ++i)
          ok = mbar_wait_bounded(&sm.ffull[(f0 + i) % X_FB], ((f0 + i) / X_FB) & 1, A.err) && ok;
        if (!ok) gave_up = true;
      }
      __syncwarp();
    } else if (warp == X_MMA_WARP) {
      // ------------------------------------------------ MMA issuer
      if (!__syncthreads_or(0)) nsub = 0;  // the item's opening barrier
      if (lane == 0 && !aborted && nsub) {
        uint32_t done = 0, ua[X_GROUPS] = {u0, u1};
        bool ok = mbar_wait_bounded(&sm.afull, nrun & 1, A.err);
#pragma unroll 1
        for (uint32_t sub = 0; sub < nsub && ok; ++sub) {
          const uint32_t st = (g + sub) % X_ST, rd = (g + sub) / X_ST;
          if (!mbar_wait_bounded(&sm.bfull[st], rd & 1, A.err)) break;
          const uint32_t b0 = smem_u32(sm.b[st][0]);
#pragma unroll 1
          for (int half = 0; half < (both ? X_GROUPS : 1); ++half) {
            const int a = both ? half : (int)(sub & 1);  // the accumulator
            const uint32_t u = a ? ua[1] : ua[0];
            if (u > 0 && !mbar_wait_bounded(&sm.accempty[a], (u - 1) & 1, A.err)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t d = tmem + X_ACC + a * XR, q = tmem + half * X_A;
            // (query piece, row piece), small products first
            constexpr int PA[3] = {0, 1, 0}, PB[3] = {1, 0, 0};
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
              for (int kk = 0; kk < X_MMAS; ++kk) {
                const uint64_t db = umma_desc(b0 + PB[p] * X_PIECE + kk * 2 * (XR / 8) * 128, (XR / 8) * 128, 128);
                umma_ts(d, q + PA[p] * (XK / 2) + kk * 8, db, p > 0 || kk > 0);
              }
            umma_commit(&sm.accfull[a]);  // the accumulator is ready for the epilogue
            if (a) ++ua[1];
            else ++ua[0];
          }
          if (!ok) break;
          umma_commit(&sm.bempty[st]);  // the pieces may be overwritten once these MMAs finish
          ++done;
        }
        // no MMA of this item is in flight when the next item (or the dealloc) comes
        for (int a = 0; a < X_GROUPS; ++a)
          if (ua[a] > (a ? u1 : u0)) mbar_wait_bounded(&sm.accfull[a], (ua[a] - 1) & 1, A.err);
        if (done != nsub) gave_up = true;
      }
      __syncwarp();
    } else {
      // ------------------------------------------------ epilogue: thread = query = TMEM lane
      const int grp = warp / X_EPI_WARPS;
      const int L = both ? tid : tid & (XM - 1);  // its query's place in the tile
      const int32_t qi = A.lane_q[it.tile * XQ + L];
      uint32_t s = 0, e = 0;
      float qn = 0.f, T = -INFINITY;
      if (qi >= 0) {
        s = A.lane_s[it.tile * XQ + L];
        e = A.lane_e[it.tile * XQ + L];
        qn = A.desc[qi].qn;
        T = sortable_f32(ld_volatile_u32(A.T_global + qi));
        if (ld_volatile_u32(A.ovf + qi)) T = -INFINITY;
      }
      const int qex = scale_exp(qn);
      const float iq = pow2f(-qex);
      const int hlo = __reduce_min_sync(0xffffffffu, qi >= 0 ? 14 - qex : INT_MAX);
      const int hhi = __reduce_max_sync(0xffffffffu, qi >= 0 ? 14 - qex : INT_MIN);
      if (lane == 0) {
        atomicMin(&sm.hmin[iter & 1], hlo);
        atomicMax(&sm.hmax[iter & 1], hhi);
      }
      sm.cnt[tid] = 0;
      sm.thr[tid] = T;
      sm.lq[tid] = qi;
      sm.qn[tid] = qn;
      // the query's pieces into TMEM, 16 dims (8 columns of each piece) at a
      // time; the groups share a single half's work
      const uint32_t tq = tmem + ((uint32_t)((warp & 3) * 32) << 16);
      const uint32_t ta = tq + (both ? grp * X_A : 0u);
      const float *qp = A.q + (uint64_t)(qi >= 0 ? qi : 0) * DIM;
      const float qs = pow2f(qex);
      // an item whose queries are all answered (or marked) is skipped
      if (!__syncthreads_or(T != -INFINITY)) nsub = 0;  // the item's opening barrier
      if (nsub) {
        const int fold = fold_exp(sm, iter & 1);
        const float fold_side = fold != X_NO_FOLD ? pow2f(qex + fold) : 0.f;
        double q2 = 0.0;
#pragma unroll 1
        for (int c = 0; c < X_MMAS; ++c) {
          uint32_t h[8], l[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int d = c * 16 + 2 * j;
            const bool on = qi >= 0 && d < DIM;
            const float a = on ? qp[d] : 0.f, b = on ? qp[d + 1] : 0.f;
            q2 += (double)a * (double)a + (double)b * (double)b;
            split2(a * qs, b * qs, h[j], l[j]);
          }
          if (!both && (c & 1) != grp) continue;
          if (c == X_MMAS - 1 && qi >= 0) {  // slots 100, 101, 102
            const __half2 a = __floats2half2_rn(fold_side, fold_side), b = __floats2half2_rn(fold_side, 0.f);
            memcpy(&h[2], &a, 4);
            memcpy(&h[3], &b, 4);
          }
          tmem_st8(ta + c * 8, h);
          tmem_st8(ta + XK / 2 + c * 8, l);
        }
        // ds is taken from |q|^2 rounded once; the error bound's argument (screen_eps) is the FMA chain's qn
        // everywhere, so that bounds computed here and in the merge agree
        const float qd = (float)q2;
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive1(&sm.afull);

        Candidate *work = A.work + (uint64_t)blockIdx.x * XQ * X_LIST;
        Candidate *lists = work + (uint64_t)(warp * 32) * X_LIST, *list = lists + lane * X_LIST;
        XWarp &wsm = sm.w[warp];
        // a pilot over a slab of many sampled rows keeps the best of every XR
        // or 32 of them: the few that matter lie apart as a rule, so the seed's
        // rank in these is little above its rank in all (and never below it)
        const uint32_t sampled = (e - s) / A.stride;
        const int sample = A.stride == 1 ? 0 : sampled / XR >= 2 * A.k ? XR : sampled / 32 >= 2 * A.k ? 32 : 0;
        int cnt = 0;
        bool ok = !aborted;
        // keep iff qn - 2 v <= push limit, as one compare on v = q.x - |x|^2/2
        // (the limit's own slack covers this rounding); no bound yet: every row
        auto acc_bound = [&](float t) {
          return t == -INFINITY ? INFINITY : t == INFINITY ? -FLT_MAX : 0.5f * (qd - screen_push_limit(t, qn));
        };
        float cq = acc_bound(T);
        float cs = cq * qs;
        uint32_t until_refresh = X_REFRESH, u = grp ? u1 : u0;
#pragma unroll 1
        for (uint32_t sub = both ? 0u : (uint32_t)grp; sub < nsub && ok; sub += both ? 1u : X_GROUPS, ++u) {
          const uint32_t slot = (g + sub) % X_NORMS;
          if (!__all_sync(0xffffffffu, mbar_wait_bounded(&sm.accfull[grp], u & 1, A.err))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t p0 = (it.blk0 + sub * A.stride) * XR;
          const int r0 = (int)min(max(s, p0), p0 + XR) - (int)p0;
          const int r1 = (int)min(max(e, p0), p0 + XR) - (int)p0;
          const uint32_t tb = tq + X_ACC + grp * XR;
          const float4 cr4 = *reinterpret_cast<const float4 *>(sm.crs[slot]);
          if (cr4.x > 0.f && cr4.x == cr4.y && cr4.x == cr4.z && cr4.x == cr4.w) {  // (block-uniform)
            // the rows' scale 2^ex = 1 / cr: v >= cq iff acc >= cs 2^ex (-inf would admit masked columns)
            ScreenQuery q;
            q.bound = r0 < r1 ? fmaxf(cs * pow2f(127 - (int)(__float_as_uint(cr4.x) >> 23)), -FLT_MAX) : INFINITY;
            q.f2 = -2.f * (cr4.x * iq);
            q.qn = qd;
            q.range = (r0 << 16) | r1;
            // 32-column chunks, two at a time: one whose maximum reaches the
            // bound holds a candidate, or a row outside the slab that raises it.
            // One that passes on its own, as in most chunks, is the maximum, and
            // its lane appends it; the rest are staged (x_flush looks closer).  A
            // pilot over a long slab keeps the maxima themselves.
            uint32_t hits = 0;
            float best = -INFINITY;
#pragma unroll 1
            for (int c = 0; c < XR; c += 64) {
              uint32_t ra[32], rb[32];
              float ga[4], gb[4];
              tmem_ld32_issue(tb + c, ra);
              tmem_ld32_issue(tb + c + 32, rb);
              tmem_wait_ld(ra);
              tmem_wait_ld(rb);
              const float ma = max32(ra, ga), mb = max32(rb, gb);
              best = fmax3(best, ma, mb);
              uint32_t h = (ma >= q.bound ? 1u : 0u) | (mb >= q.bound ? 2u : 0u);
              if (!__any_sync(0xffffffffu, h != 0)) continue;
              if (sample) {
                if (sample == 32) {
                  if ((h & 1u) && c >= r0 && c + 32 <= r1) list[cnt++] = {fmaf(q.f2, ma, qd), p0 + c};
                  if ((h & 2u) && c + 32 >= r0 && c + 64 <= r1) list[cnt++] = {fmaf(q.f2, mb, qd), p0 + c + 32};
                }
                h = 0;
              }
              if (h & 1u) {
                const uint32_t all = ge_mask32(ra, ga, q.bound), in = all & range_mask(r0 - c, r1 - c);
                if (in == 0 || (all & (all - 1)) == 0) h ^= 1u;
                if (in && !(h & 1u)) list[cnt++] = {fmaf(q.f2, ma, qd), p0 + c + __ffs(in) - 1};
              }
              if (h & 2u) {
                const uint32_t all = ge_mask32(rb, gb, q.bound), in = all & range_mask(r0 - c - 32, r1 - c - 32);
                if (in == 0 || (all & (all - 1)) == 0) h ^= 2u;
                if (in && !(h & 2u)) list[cnt++] = {fmaf(q.f2, mb, qd), p0 + c + 31 + __ffs(in)};
              }
              hits |= h << (c / 32);
              __syncwarp();  // (the next TMEM loads are the whole warp's)
            }
            if (sample == XR && best >= q.bound && r1 - r0 == XR) list[cnt++] = {fmaf(q.f2, best, qd), p0};
            int ns = 0;
            if (__any_sync(0xffffffffu, hits != 0)) {
#pragma unroll 1
              for (int c = 0; c < XR / 32; ++c) {
                const uint32_t fm = __ballot_sync(0xffffffffu, (hits >> c) & 1u);
                if (fm) {
                  const int cn = x_stage(tb, 32 * c, fm, q, p0, wsm, ns, lists, X_LIST, cnt);
                  ns = cn & 0xff;
                  cnt = cn >> 8;
                }
              }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive1(&sm.accempty[grp]);
            if (ns) cnt = x_flush(wsm, ns, p0, lists, X_LIST, cnt);
          } else {
#pragma unroll 1
            for (int o = 0; o < XR; o += 32)
              cnt = x_push_norms(tb + o, sm, slot, o, iq, cq, qd, r0 - o, r1 - o, p0 + o, list, cnt);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive1(&sm.accempty[grp]);
          }
          // lists that could overflow in the next sub-tile are bounded and trimmed
          uint32_t msk = __ballot_sync(0xffffffffu, cnt > X_LIST - XR);
          if (msk) {
            sm.cnt[tid] = cnt;
            __syncwarp();
            while (msk) {
              const int Lb = warp * 32 + __ffs(msk) - 1;
              msk &= msk - 1;
              x_trim(work + (uint64_t)Lb * X_LIST, sm, Lb, A.k, A.T_global, A.ovf);
            }
            cnt = sm.cnt[tid];
            T = sm.thr[tid];
            cq = acc_bound(T);
            cs = cq * qs;
          }
          // other items of the query (and the other group) tighten the bound meanwhile
          if (--until_refresh == 0) {
            until_refresh = X_REFRESH;
            if (qi >= 0) {
              const float Tg = sortable_f32(ld_volatile_u32(A.T_global + qi));
              if (Tg < T) {
                T = Tg;
                sm.thr[tid] = T;
                cq = acc_bound(T);
                cs = cq * qs;
              }
            }
          }
        }
        if (!ok) {
          // a wait gave up: this item's queries are answered by the exact scan
          if (qi >= 0) A.ovf[qi] = 1u;
          cnt = 0;
          gave_up = true;
        }
        sm.cnt[tid] = cnt;
        // every list of the item is complete (and visible)
        asm volatile("bar.sync 1, %0;" ::"n"(X_EPI * 32) : "memory");
        const int per = both ? XQ / X_EPI : XM / X_EPI;
#pragma unroll 1
        for (int b = 0; b < per; ++b) {
          const int Lb = warp * per + b;
          const uint64_t o = (uint64_t)item_id * XQ + Lb;
          if (both) x_finish<X_NPL>(work, sm, Lb, -1, A.k, A.T_global, A.ovf, A.out + o * EXACT_CAP, A.out_cnt + o);
          else
            x_finish<X_GROUPS * X_NPL>(work, sm, Lb, XM + Lb, A.k, A.T_global, A.ovf, A.out + o * EXACT_CAP,
                                       A.out_cnt + o);
        }
      } else {
        A.out_cnt[(uint64_t)item_id * XQ + tid] = 0;  // read all the same: by the seeds, which know no marks
      }
    }
    g += nsub;
    nrun += nsub != 0;
    u0 += both ? nsub : (nsub + 1) / 2;
    u1 += both ? nsub : nsub / 2;
    // double-buffered by item parity: a slow thread may still read the slot
    // of this barrier while thread 0 writes the one after
    if (tid == 0) {
      sm.next[iter & 1] = atomicAdd(A.queue, 1u) + gridDim.x;
      sm.hmin[(iter + 1) & 1] = INT_MAX;
      sm.hmax[(iter + 1) & 1] = INT_MIN;
    }
    tc_fence_before();
    // the item's shared state (query pieces, counts, bounds) is reused by the next
    aborted = __syncthreads_or(aborted || gave_up) != 0;
    tc_fence_after();
    item_id = sm.next[iter & 1];
  }
  if (warp == X_MMA_WARP)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(X_TMEM_COLS));
}

}  // namespace

size_t exact_work_bytes(uint32_t grid) { return (size_t)grid * XQ * X_LIST * sizeof(Candidate); }

int launch_exact_screen(const ExactScreenArgs &A, uint32_t grid, cudaStream_t st) {
  // per device context, so set on every call (cheap)
  FKNN_CUDA(cudaFuncSetAttribute(k_exact_screen, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(XSmem)));
  k_exact_screen<<<grid, X_THREADS, sizeof(XSmem), st>>>(A);
  g_launches += 1;
  FKNN_CUDA(cudaGetLastError());
  return FKNN_OK;
}

namespace {
struct ExactSeedBound {
  __device__ float operator()(float ds, const QueryDesc &dq) const { return screen_hi(ds, dq.qn); }
};
}  // namespace

int launch_exact_seed(const uint32_t *big_q, const uint32_t *big_tile, const uint32_t *big_lane, uint32_t nbig,
                      const ExactScreenArgs &A, const uint32_t *item_slot, uint32_t k, uint32_t *T_global,
                      cudaStream_t st) {
  SeedArgs S;
  S.big_q = big_q;
  S.big_tile = big_tile;
  S.big_lane = big_lane;
  S.nbig = nbig;
  S.nbig_d = nullptr;
  S.tiles = A.tiles;
  S.items = A.items;
  S.item_slot = item_slot;
  S.out = A.out;
  S.out_cnt = A.out_cnt;
  S.tq = XQ;
  S.list_cap = EXACT_CAP;
  S.blk_rows = XR;
  S.desc = A.desc;
  S.stride = A.stride;
  S.k = k;
  S.T_global = T_global;
  S.seeded = nullptr;
  launch_screen_seed(S, nbig, ExactSeedBound(), st);
  FKNN_CUDA(cudaGetLastError());
  return FKNN_OK;
}

}  // namespace fknn
