// CLUE 2D on GB300: the four serial stages of
// src/serial/plugin-CLUEClusterizer/CLUEAlgoKernels.h re-designed for the GPU.
//
// Pipeline of one batch (events concatenated in CSR order):
//   k_init         the batch's counters, tickets and flags
//   k_count        points per (event, layer), warp-aggregated atomics; also
//                  notes whether every event is already grouped by layer
//   k_layer_scan   per-event exclusive scan -> first position of each layer
//                  (and, for batches of a few layers per CTA, layer sizes)
//   k_order        those batches only: layers in descending size
//   k_scatter      group points by (event, layer) when the input is not
//   k_layers       persistent CTAs over the (event, layer) queue (one wide
//                  pass for a single event, else one or two classes of layer
//                  size); the next layer's inputs prefetched into L2.  Per layer,
//                  on-chip: counting sort into the reference's 5 cm tiles
//                  (column-major, index order inside a tile), density,
//                  nearest-higher, seed/outlier flags (and the seeds as bits
//                  of each event-aligned chunk of 4096 points) and the walk
//                  to each point's root
//   k_seed_chunk_scan / k_seed_rank
//                  event-wide seed numbering in index order
//   k_label        clusterIndex = cluster of the root seed, -1 when the
//                  chain ends at an outlier
//
// Bit-exactness with the serial backend:
//  * candidates of a query are enumerated xBin-outer, yBin-inner, index order
//    inside a tile (CLUEAlgoKernels.h:35-44,76-85); a column-major sort key
//    makes each column's rows one contiguous range of the sorted layer;
//  * rho is a sequential float sum in that order, (i==j ? 1 : 0.5) * w_j,
//    with __fmul_rn/__fadd_rn (no contraction; the file is built --fmad=false);
//  * "sqrtf(dx*dx+dy*dy) <= d" is evaluated as "dx*dx+dy*dy <= t" with t the
//    largest float whose correctly rounded square root is <= d, which is the
//    same predicate because sqrt_rn is monotone;
//  * nearest-higher keeps the reference's strict "dist < delta" on the
//    square-rooted distance (first candidate wins a tie); the squared
//    distance only filters candidates that cannot win;
//  * seeds are numbered by rank in point-index order over the whole event
//    (CLUEAlgoKernels.h:114-131) and labels follow nearestHigher chains
//    exactly where the reference's follower stack walks (:133-152).
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>

#include <algorithm>

#include "clue_internal.h"
#include "clue_pdl.cuh"

namespace clue {

namespace {

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ int warp_id() { return threadIdx.x >> 5; }

// LayerTilesSerial::getXBin / getYBin (src/serial/DataFormats/LayerTilesSerial.h:24-40):
// (v - (-250)) * 0.2 in float, truncated toward zero (saturating), clamped to
// [0, 99]; a NaN lands in bin 0 (the conversion gives 0 or INT_MIN, both
// clamped to 0), as (int)NaN does on the aarch64 host.
__device__ __forceinline__ int tile_bin(float v) {
  const int b = __float2int_rz(__fmul_rn(__fsub_rn(v, -250.f), 0.2f));
  return min(max(b, 0), kGridCols - 1);
}

// Event of a chunk: the last e with chunk_start[e] <= c (empty events own no chunk).
__device__ __forceinline__ int chunk_event(const int32_t* chunk_start, int n_events, int c) {
  int lo = 0, hi = n_events;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (chunk_start[mid] <= c) lo = mid; else hi = mid;
  }
  return lo;
}

// Event of a chunk: from the host-built table when the batch has one.
__device__ __forceinline__ int event_of_chunk(const Batch2D& b, int c) {
  return b.chunk_ev ? b.chunk_ev[c] : chunk_event(b.chunk_start, b.n_events, c);
}

template <int NT>
__device__ __forceinline__ int block_inclusive_scan(int v, int* s_ws, int* total) {
  constexpr int NW = NT / 32;
  const int lane = lane_id(), warp = warp_id();
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += t;
  }
  if (lane == 31) s_ws[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int wv = lane < NW ? s_ws[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, wv, o);
      if (lane >= o) wv += t;
    }
    if (lane < NW) s_ws[lane] = wv;
  }
  __syncthreads();
  const int res = x + (warp > 0 ? s_ws[warp - 1] : 0);
  *total = s_ws[NW - 1];
  __syncthreads();
  return res;
}

// Exclusive scan of tbl[0..n) in place, tbl[n] = total (32-bit counts, HBM tables).
template <int NT>
__device__ void block_scan_table(int32_t* tbl, int n, int* s_ws) {
  const int per = (n + NT - 1) / NT;
  const int beg = min((int)threadIdx.x * per, n);
  const int end = min(beg + per, n);
  int sum = 0;
  for (int i = beg; i < end; ++i) sum += tbl[i];
  int total;
  const int incl = block_inclusive_scan<NT>(sum, s_ws, &total);
  int run = incl - sum;
  for (int i = beg; i < end; ++i) {
    const int c = tbl[i];
    tbl[i] = run;
    run += c;
  }
  if (threadIdx.x == 0) tbl[n] = total;
  __syncthreads();
}

// The same for the on-chip 16-bit table: each thread scans whole 16-byte
// groups of 8 counts (kTiles = 10000 is a multiple of 8).  Two counts are
// added per 32-bit word: a layer there has fewer than 65536 points, so no half
// carries into the other (5.4 -> 4.7 % of the kernel's time on the 4096-event
// batch against counts added one by one).
template <int NT>
__device__ void block_scan_table(uint16_t* tbl, int n, int* s_ws) {
  const int groups = n / 8;
  const int per = (groups + NT - 1) / NT;
  const int beg = min((int)threadIdx.x * per, groups);
  const int end = min(beg + per, groups);
  uint4* t4 = reinterpret_cast<uint4*>(tbl);
  unsigned sum2 = 0;
  for (int g = beg; g < end; ++g) {
    const uint4 v = t4[g];
    sum2 += (v.x + v.y) + (v.z + v.w);
  }
  const int sum = (int)(sum2 & 0xffffu) + (int)(sum2 >> 16);
  int total;
  const int incl = block_inclusive_scan<NT>(sum, s_ws, &total);
  unsigned run2 = (unsigned)(incl - sum) * 0x10001u;  // the running total, in both halves
  // (a, b) -> (run, run + a); then run += a + b, which is the upper half of (a, b) * 0x10001
  auto word = [&](unsigned w) {
    const unsigned out = run2 + (w << 16);
    run2 += __byte_perm(w * 0x10001u, 0u, 0x3232);
    return out;
  };
  for (int g = beg; g < end; ++g) {
    uint4 v = t4[g];
    v.x = word(v.x);
    v.y = word(v.y);
    v.z = word(v.z);
    v.w = word(v.w);
    t4[g] = v;
  }
  if (threadIdx.x == 0) tbl[n] = (uint16_t)total;
  __syncthreads();
}

// Histogram increment returning the previous count.  The on-chip table holds
// 16-bit counts (a layer there has < 65536 points), two per 32-bit word.
__device__ __forceinline__ int hist_add(uint16_t* t, int key, int n) {
  unsigned* w = reinterpret_cast<unsigned*>(t) + (key >> 1);
  const int sh = (key & 1) * 16;
  return (int)((atomicAdd(w, (unsigned)n << sh) >> sh) & 0xffffu);
}
__device__ __forceinline__ int hist_add(int32_t* t, int key, int n) { return atomicAdd(t + key, n); }

// Squared distance dx*dx + dy*dy with the reference's rounding: two
// correctly rounded differences, two correctly rounded squares (computed as
// one packed f32x2 pair each) and one correctly rounded sum.
__device__ __forceinline__ float dist2(float2 a, float2 b) {
  float sx, sy;
  asm("{\n\t.reg .b64 pa, pb, pd;\n\t"
      "mov.b64 pa, {%2, %3};\n\t"
      "mov.b64 pb, {%4, %5};\n\t"
      "sub.rn.f32x2 pd, pa, pb;\n\t"
      "mul.rn.f32x2 pd, pd, pd;\n\t"
      "mov.b64 {%0, %1}, pd;\n\t}"
      : "=f"(sx), "=f"(sy)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return __fadd_rn(sx, sy);
}

// Order-preserving map of a non-NaN float to 32 bits (rho is never -0: it
// starts at +0 and only adds terms).  NaN maps to 0, below every number.
__device__ __forceinline__ unsigned float_ord(float f) {
  const unsigned u = __float_as_uint(f);
  if (f != f) return 0u;
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord_float(unsigned o) {
  if (o == 0u) return __uint_as_float(0x7fffffffu);  // NaN
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// Per-layer working set, sorted by tile: on-chip for layers up to the tuned
// capacity (16-bit table and query order), in HBM scratch beyond it (32-bit).
// One 16-byte record per point, so a candidate is a single 128-bit load:
//   {x, y, gid, aux}: aux = 0.5f*w (bits) during the density search and
//   float_ord(rho) during the nearest-higher search, when the upper 8 bytes
//   read as one 64-bit key (float_ord(rho) << 32) | gid.
// 22 bytes per point on chip plus the 20 KB table.
template <class TT, class QT>
struct LayerStore {
  uint4* rec;
  int32_t* nh;  // own weight (bits), then float_ord(rho), then the parent pointer
  QT* qord;     // query order of the current search
  TT* tbl;      // kTableInts: exclusive scan over key = xBin*100 + yBin
};

struct LayerIO {
  const float* x;
  const float* y;
  const float* w;
  const int32_t* gid;  // nullptr: gid = gid_base + p
  int32_t gid_base;
  int64_t ev_start;
  int32_t chunk0;  // first seed-count chunk of the event
};

__device__ __forceinline__ float2 rec_xy(const uint4& r) { return make_float2(__uint_as_float(r.x), __uint_as_float(r.y)); }
__device__ __forceinline__ unsigned long long rec_key(const uint4& r) {
  return ((unsigned long long)r.w << 32) | r.z;
}

template <class TT>
__device__ __forceinline__ int candidate_count(const TT* tbl, int bx0, int bx1, int by0, int by1) {
  int cnt = 0;
  for (int c = bx0; c <= bx1; ++c) cnt += max(0, (int)tbl[c * kGridCols + by1 + 1] - (int)tbl[c * kGridCols + by0]);
  return cnt;
}

// Query order of a search phase: queries bucketed by their candidate count,
// heaviest first; warps then take chunks of 32 in that order, so the lanes
// of a warp run loops of similar length.  Which thread runs which query never
// changes a result.  The bucket is computed twice instead of being stored.
template <int NT, class TT, class QT>
__device__ void order_queries(const LayerStore<TT, QT>& S, const int m, const float d, int* s_bins) {
  constexpr int NB = 64;
  const int tid = threadIdx.x;
  auto bucket = [&](int q) {
    const float2 p = rec_xy(S.rec[q]);
    const int bx0 = tile_bin(__fsub_rn(p.x, d)), bx1 = tile_bin(__fadd_rn(p.x, d));
    const int by0 = tile_bin(__fsub_rn(p.y, d)), by1 = tile_bin(__fadd_rn(p.y, d));
    // 2 candidates per bucket; 8 for boxes of three columns and more, which would
    // crowd the first bucket (the same event: 58.9 -> 57.2 us)
    return NB - 1 - min(candidate_count(S.tbl, bx0, bx1, by0, by1) >> (d > 5.f ? 3 : 1), NB - 1);
  };
  for (int i = tid; i < NB; i += NT) s_bins[i] = 0;
  __syncthreads();
  for (int q = tid; q < m; q += NT) atomicAdd(&s_bins[bucket(q)], 1);
  __syncthreads();
  if (tid < 32) {
    const int a = s_bins[2 * tid], c = s_bins[2 * tid + 1];
    int x = a + c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, x, o);
      if (tid >= o) x += t;
    }
    const int ex = x - a - c;
    s_bins[2 * tid] = ex;
    s_bins[2 * tid + 1] = ex + a;
  }
  __syncthreads();
  for (int q = tid; q < m; q += NT) S.qord[atomicAdd(&s_bins[bucket(q)], 1)] = (QT)q;
  __syncthreads();
}

// Candidate sequence of a search box spanning one to three tile columns:
// segment j is column bx0+j, rows [by0, by1], i.e. sorted positions
// [s_j, s_j + l_j).  at(t) maps the t-th candidate of the concatenation to
// its sorted position with compares and selects only.
struct SegIndex {
  int b1 = 0, b2 = 0, total = 0, d0 = 0, d1 = 0, d2 = 0;
  template <class TT>
  __device__ __forceinline__ void init(const TT* tbl, int bx0, int nseg, int by0, int by1) {
    int s[3] = {0, 0, 0}, l[3] = {0, 0, 0};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      if (j < nseg) {
        const int c = (bx0 + j) * kGridCols;
        s[j] = (int)tbl[c + by0];
        l[j] = max(0, (int)tbl[c + by1 + 1] - s[j]);
      }
    }
    b1 = l[0];
    b2 = l[0] + l[1];
    total = b2 + l[2];
    d0 = s[0];
    d1 = s[1] - b1;
    d2 = s[2] - b2;
  }
  __device__ __forceinline__ int at(int t) const { return t + (t < b1 ? d0 : (t < b2 ? d1 : d2)); }
};

// Visits the candidates of a search box in the reference order: the
// branchless flattened form for boxes of up to three columns, otherwise a
// general column loop.  Both flattened loops are unrolled four times
// (4096-event batch: two-column loop unrolled 2/4/8 times 21.72/21.46/22.62
// ms, three-column loop 2/4 times 21.46/21.38 ms).
template <class TT, class F>
__device__ __forceinline__ void for_candidates(const TT* tbl, int bx0, int bx1, int by0, int by1, F&& visit) {
  const int nseg = bx1 - bx0 + 1;
  // the widest box among the active lanes picks the loop form for the warp,
  // so that lanes never split between two loops
  const unsigned act = __activemask();
  const bool any3 = __any_sync(act, nseg == 3);
  const bool anywide = __any_sync(act, nseg > 3);
  if (!any3 && !anywide) {
    // one or two columns (every density box when dc < 2.5 cm): one compare
    // and one select per candidate
    int b1 = 0, total = 0, d0 = 0, d1 = 0;
    if (nseg >= 1) {
      const int s0 = (int)tbl[bx0 * kGridCols + by0];
      const int l0 = max(0, (int)tbl[bx0 * kGridCols + by1 + 1] - s0);
      int s1 = 0, l1 = 0;
      if (nseg == 2) {
        s1 = (int)tbl[(bx0 + 1) * kGridCols + by0];
        l1 = max(0, (int)tbl[(bx0 + 1) * kGridCols + by1 + 1] - s1);
      }
      b1 = l0;
      total = l0 + l1;
      d0 = s0;
      d1 = s1 - l0;
    }
#pragma unroll 4
    for (int t = 0; t < total; ++t) visit(t + (t < b1 ? d0 : d1));
  } else if (!anywide) {
    SegIndex sg;
    sg.init(tbl, bx0, nseg, by0, by1);
#pragma unroll 4
    for (int t = 0; t < sg.total; ++t) visit(sg.at(t));
  } else {
    // the next column's run is read while this one is walked (one toy event with
    // dc 20 cm: 60.1 -> 58.9 us)
    int k = (int)tbl[bx0 * kGridCols + by0], e = (int)tbl[bx0 * kGridCols + by1 + 1];
    for (int c = bx0; c <= bx1; ++c) {
      const int cn = min(c + 1, bx1) * kGridCols;
      const int kn = (int)tbl[cn + by0], en = (int)tbl[cn + by1 + 1];
      for (; k < e; ++k) visit(k);
      k = kn;
      e = en;
    }
  }
}

// Next chunk of 32 queries for this warp (dynamic, in query order).
__device__ __forceinline__ int next_chunk(int* s_next) {
  int base = 0;
  if ((threadIdx.x & 31) == 0) base = atomicAdd(s_next, 32);
  return __shfl_sync(0xffffffffu, base, 0);
}

// Running nearest higher over candidates in visiting order: the first
// smallest d2 and, in `prev`, the smallest d2 before it.  The reference
// compares sqrt_rn(d2) strictly, so the winner is the first candidate with the
// smallest rounded square root: the one kept here unless a candidate visited
// before it has a larger d2 with the same root.  Then `prev` is within the
// margin of `d2`, near() is true and the query is decided again on square
// roots.  A later candidate with an equal or larger d2 never replaces the
// first.  Three moves under one predicate per candidate: a margin test on
// each candidate instead (a product, a compare and the flag's logic) made
// the search the larger part of the kernel (4096-event batch: 22.8 -> 20.5
// ms, 200 HGCAL events: 6.30 -> 5.55 ms).
struct NhBest {
  float d2, prev;
  int k = -1;
  __device__ __forceinline__ explicit NhBest(float limit) : d2(limit), prev(limit) {}
  __device__ __forceinline__ void visit(float2 pq, unsigned long long kq, const uint4& rk, int pos) {
    const float d = dist2(pq, rec_xy(rk));
    if (rec_key(rk) > kq && d < d2) {
      prev = d2;
      d2 = d;
      k = pos;
    }
  }
  __device__ __forceinline__ bool near() const { return near(d2, prev); }
  // sqrt_rn(a) < sqrt_rn(b) whenever a * 1.00002f < b
  static __device__ __forceinline__ bool near(float d2, float prev) { return !(__fmul_rn(d2, 1.00002f) < prev); }
};

// One (event, layer) item through every stage.  next_item: in thread 0, the
// item this CTA takes next (-1 when none), whose inputs are prefetched.
template <int NT, class TT, class QT>
__device__ void process_layer(const Params2D& P, const LayerStore<TT, QT>& S, const int m, const LayerIO& in,
                              const Batch2D& b, int* s_ws, int* s_bins, int* s_next, int next_item) {
  const int tid = threadIdx.x, lane = tid & 31;
  QT* kkey = S.qord;                                     // sort key, later final slot
  int32_t* kprov = S.nh;                                 // provisional slot in tile
  int32_t* slot_p = reinterpret_cast<int32_t*>(S.rec);  // input position at provisional slot
  int32_t* slot_g = slot_p + m;                          // gid at provisional slot

  // -- counting sort into tiles (kernel_compute_histogram, CLUEAlgoKernels.h:18-23)
  {
    constexpr int kTableBytes = ((kTableInts * (int)sizeof(TT) + 15) / 16) * 16;
    uint4* t4 = reinterpret_cast<uint4*>(S.tbl);
    for (int i = tid; i < kTableBytes / 16; i += NT) t4[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  __syncthreads();
  {
    const unsigned lt = (1u << lane) - 1u;
    // gid = gid_base + p ascends with p (layer-ordered input); otherwise the
    // gids come from the layer-grouping gather in arbitrary order
    const bool mono = in.gid == nullptr;
    int32_t* lead_p = slot_p + 2 * m;  // by point: size of the group it leads, else 0
    int32_t* lead_q = slot_p + 3 * m;  // the same by provisional slot
    // the loads of the next pass are issued before this pass's atomics (6.4 ->
    // 5.2 % of the kernel's time on the 4096-event batch)
    float nx_x = tid < m ? in.x[tid] : 0.f, nx_y = tid < m ? in.y[tid] : 0.f;
    for (int base = 0; base < m; base += NT) {
      const int p = base + tid;
      const int key = p < m ? tile_bin(nx_x) * kGridCols + tile_bin(nx_y) : -1;
      if (p + NT < m) {
        nx_x = in.x[p + NT];
        nx_y = in.y[p + NT];
      }
      const unsigned grp = __match_any_sync(0xffffffffu, key);
      const int leader = __ffs(grp) - 1;
      int old = 0;
      if (key >= 0 && lane == leader) old = hist_add(S.tbl, key, __popc(grp));
      old = __shfl_sync(0xffffffffu, old, leader);
      if (key >= 0) {
        kkey[p] = (QT)key;
        kprov[p] = old + __popc(grp & lt);
        if (mono) lead_p[p] = lane == leader ? __popc(grp) : 0;
      }
    }
    __syncthreads();
    block_scan_table<NT>(S.tbl, kTiles, s_ws);
    for (int p = tid; p < m; p += NT) {
      const int q = (int)S.tbl[kkey[p]] + kprov[p];
      slot_g[q] = in.gid ? in.gid[p] : in.gid_base + p;
      slot_p[q] = p;
      if (mono) lead_q[q] = lead_p[p];
    }
    __syncthreads();
    // Atomics gave an arbitrary order inside a tile; the reference appends in
    // index order, so place each point at its gid rank within the tile.  With
    // layer-ordered input a tile's slots are groups (one atomic each) of lanes
    // of one warp pass over 32 consecutive points: gids ascend inside a group
    // and different groups cover disjoint gid ranges, so the rank is the sizes
    // of the groups that start below g plus g's place in its own group -- a
    // walk over the tile's groups instead of its points.
    for (int q = tid; q < m; q += NT) {
      const int p = slot_p[q];
      const int key = (int)kkey[p];
      const int s = (int)S.tbl[key], e = (int)S.tbl[key + 1];
      const int g = slot_g[q];
      int rank = 0;
      if (mono) {
        for (int t = s; t < e;) {
          const int c = max(lead_q[t], 1);
          if (q >= t && q < t + c) rank += q - t;
          else if (slot_g[t] < g) rank += c;
          t += c;
        }
      } else {
        for (int t = s; t < e; ++t) rank += (slot_g[t] < g);
      }
      kkey[p] = (QT)(s + rank);
    }
    __syncthreads();
  }
  for (int p = tid; p < m; p += NT) {
    const int f = (int)kkey[p];
    const float wv = in.w[p];
    const unsigned g = (unsigned)(in.gid ? in.gid[p] : in.gid_base + p);
    S.rec[f] = make_uint4(__float_as_uint(in.x[p]), __float_as_uint(in.y[p]), g, __float_as_uint(__fmul_rn(0.5f, wv)));
    S.nh[f] = __float_as_int(wv);
  }
  __syncthreads();

  // the next layer's inputs (the ticket taken while this layer started) into
  // L2 while this one is searched: its histogram and records then read L2
  if (tid < 32) {
    const int nx = __shfl_sync(0xffffffffu, next_item, 0);
    if (nx >= 0) {
      const int nm = b.lcnt[nx];
      const int ns = b.lstart[nx];
      const bool gr = b.flags[kFlagGrouped] != 0;
      const float* ax = (gr ? b.x : b.gx) + ns;
      const float* ay = (gr ? b.y : b.gy) + ns;
      const float* aw = (gr ? b.w : b.gw) + ns;
      for (int o = lane * 32; o < nm; o += 32 * 32) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(ax + o));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(ay + o));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(aw + o));
      }
    }
  }

  // One query order for both searches, by the nearest-higher box (the
  // larger box and the more expensive search).  Layers of up to 256 points
  // keep the input order: there the ordering costs more than it saves
  // (4096-event batch: k_layers 21.58 -> 21.46 ms; 21.59 ms with the
  // threshold at 512).  So do layers in HBM scratch, in the tiles' order:
  // neighbouring queries read the same lines, which the order by count scatters
  // (one event of 200,000 points, 43,000 on a layer, dc 5.5 cm: 3.27 -> 2.28 ms,
  // and 2.96 with finer buckets; 600,000 points, 6,000 to a layer: 152 -> 134 us),
  // unless the boxes hold one tile or four (two events, 47,000 points on a layer
  // each, boxes of 1.8 cm: 3.58 ms, 3.84 without the order).
  if (m > 256 && (sizeof(TT) == 2 || P.dm < 2.5f)) {
    order_queries<NT>(S, m, P.dm, s_bins);
  } else {
    for (int i = tid; i < m; i += NT) S.qord[i] = (QT)i;
    __syncthreads();
  }

  // -- local density (kernel_calculate_density, CLUEAlgoKernels.h:25-55)
  if (tid == 0) *s_next = 0;
  __syncthreads();
  for (;;) {
    const int base = next_chunk(s_next);
    if (base >= m) break;
    const int i = base + lane;
    if (i < m) {
      const int q = (int)S.qord[i];
      const uint4 rq = S.rec[q];
      const float2 pq = rec_xy(rq);
      const float wq = __int_as_float(S.nh[q]);
      const int bx0 = tile_bin(__fsub_rn(pq.x, P.dc)), bx1 = tile_bin(__fadd_rn(pq.x, P.dc));
      const int by0 = tile_bin(__fsub_rn(pq.y, P.dc)), by1 = tile_bin(__fadd_rn(pq.y, P.dc));
      float r = 0.f;
      for_candidates(S.tbl, bx0, bx1, by0, by1, [&](int k) {
        const uint4 rk = S.rec[k];
        const float h = (k == q) ? wq : __uint_as_float(rk.w);  // the i == j term is w, not 0.5 w
        if (dist2(pq, rec_xy(rk)) <= P.t_dc) r = __fadd_rn(r, h);
      });
      b.rho[in.ev_start + rq.z] = r;
      S.nh[q] = (int)float_ord(r);  // nobody reads nh[q] during this search but this thread
    }
  }
  __syncthreads();
  for (int q = tid; q < m; q += NT) S.rec[q].w = (unsigned)S.nh[q];
  __syncthreads();

  // -- distance to the nearest higher (kernel_calculate_distanceToHigher, :57-106)
  // "higher" (rho_j > rho_i, or equal rho and j > i) is key_j > key_i; a NaN
  // rho is higher than nothing and nothing is higher than it, as in the
  // reference.  The winner is the first candidate with the smallest
  // correctly rounded sqrt(d2), found on d2 (NhBest).
  if (tid == 0) *s_next = 0;
  __syncthreads();
  int32_t* par = S.nh;  // parent: nearest higher for followers, -2 seed root, -3 other root
  for (;;) {
    const int base = next_chunk(s_next);
    if (base >= m) break;
    const int i = base + lane;
    if (i < m) {
      const int q = (int)S.qord[i];
      const uint4 rq = S.rec[q];
      const float2 pq = rec_xy(rq);
      const unsigned long long ks = rec_key(rq);
      const unsigned long long kq = rq.w == 0u ? ~0ull : ks;
      const int bx0 = tile_bin(__fsub_rn(pq.x, P.dm)), bx1 = tile_bin(__fadd_rn(pq.x, P.dm));
      const int by0 = tile_bin(__fsub_rn(pq.y, P.dm)), by1 = tile_bin(__fadd_rn(pq.y, P.dm));
      NhBest nb(P.t_dm_next);  // d2 < t_dm_next <=> d2 <= t_dm
      for_candidates(S.tbl, bx0, bx1, by0, by1, [&](int k) { nb.visit(pq, kq, S.rec[k], k); });
      int best = nb.k;
      float best_s = best >= 0 ? __fsqrt_rn(nb.d2) : FLT_MAX;
      if (best >= 0 && nb.near()) {
        // an earlier candidate's root may equal the winner's: decide this
        // query again with the reference's comparison on sqrt'd distances
        best_s = FLT_MAX;
        best = -1;
        for_candidates(S.tbl, bx0, bx1, by0, by1, [&](int k) {
          const uint4 rk = S.rec[k];
          const float d2 = dist2(pq, rec_xy(rk));
          if (rec_key(rk) > kq && d2 <= P.t_dm) {
            const float sd = __fsqrt_rn(d2);
            if (sd < best_s) {
              best_s = sd;
              best = k;
            }
          }
        });
      }
      // -- seeds, outliers, outputs (kernel_findAndAssign_clusters, :108-136)
      const float r = ord_float(rq.w);
      const bool seed = (best_s > P.dc) && (r >= P.rhoc);
      const bool outlier = (best_s > P.dm) && (r < P.rhoc);
      const int64_t o = in.ev_start + rq.z;
      b.delta[o] = best_s;
      b.nh[o] = best >= 0 ? (int)S.rec[best].z : -1;
      b.seed[o] = seed ? 1 : 0;
      // the seeds of each event-aligned chunk of 4096 points as bits, for the seed ranks
      if (seed && b.seed_bits) atomicOr(&b.seed_bits[(int64_t)in.chunk0 * kChunkWords + (rq.z >> 5)], 1u << (rq.z & 31));
      par[q] = (!seed && !outlier && best >= 0) ? best : (seed ? -2 : -3);
    }
  }
  __syncthreads();
  // -- roots of the nearestHigher chains (replaces the follower stack,
  // :138-152): each point walks its chain to the root and labels itself.  A
  // walk of 64 steps without a root leaves the parent pointer at the farthest
  // point reached (every ancestor is a valid parent; the words are read and
  // written whole) and is taken up again in another pass, which finds the
  // chains 64 times shorter.  (Roots first and labels after a barrier, with a
  // root array: 8.0 against 6.6 % of the kernel's time.)
  for (;;) {
    int unresolved = 0;
    for (int q = tid; q < m; q += NT) {
      int r = q, p = par[q];
      for (int step = 0; p >= 0 && step < 64; ++step) {
        r = p;
        p = par[r];
      }
      // a chain ending at a seed carries -(seed's event-local index + 2) until
      // k_seed_rank (seeds) and k_label (the others) put the seed's rank there
      if (p < 0) {
        b.ci[in.ev_start + S.rec[q].z] = p == -2 ? -((int)S.rec[r].z + 2) : -1;
      } else {
        par[q] = r;
        unresolved = 1;
      }
    }
    if (!__syncthreads_or(unresolved)) break;
  }
}

// -- small layers ------------------------------------------------------------

// A layer of fewer than kTiny points takes one warp and no tile table: its
// points are ranked by (tile, index) and every query looks at all of them in that
// order, which is the reference's order for those in its search box; a candidate
// that passes the distance test is then tested against the box.  A whole CTA per
// layer waits at a dozen barriers and clears and scans a table of 10,000 tiles for
// a few dozen points (5.4 us per layer and CTA with one point in it); the warps of
// an SM have 32 such layers in flight.  The cost is the candidates outside the box:
// with 128 points and four queries per lane 300 events of 12,600 points took
// 0.70 ms, 0.61 with the table.
constexpr int kTiny = 64;  // a whole number of size classes and of points per lane
constexpr int kTinyBytes = kTiny * (16 + 4 + 2);  // records, weights / parents, tiles

// Search box (or a point's tile, twice) in bytes: columns, rows.
__device__ __forceinline__ unsigned pack_box(float x, float y, float d) {
  return (unsigned)tile_bin(__fsub_rn(x, d)) | (unsigned)tile_bin(__fadd_rn(x, d)) << 8 |
         (unsigned)tile_bin(__fsub_rn(y, d)) << 16 | (unsigned)tile_bin(__fadd_rn(y, d)) << 24;
}
__device__ __forceinline__ bool in_box(unsigned box, unsigned tile) {  // tile: column | row << 8
  const unsigned c = tile & 255u, r = tile >> 8;
  return c >= (box & 255u) && c <= ((box >> 8) & 255u) && r >= ((box >> 16) & 255u) && r <= (box >> 24);
}

__device__ __forceinline__ void tiny_layer(const Params2D& P, unsigned char* ws, const int m, const LayerIO& in,
                                        const Batch2D& b) {
  constexpr int NJ = kTiny / 32;  // queries per lane
  const int lane = lane_id();
  uint4* rec = reinterpret_cast<uint4*>(ws);
  int32_t* nh = reinterpret_cast<int32_t*>(rec + kTiny);
  uint16_t* tile = reinterpret_cast<uint16_t*>(nh + kTiny);
  {
    unsigned long long* sk = reinterpret_cast<unsigned long long*>(ws);
    unsigned long long key[NJ];
    float x[NJ], y[NJ], w[NJ];
    int rank[NJ];
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int p = lane + 32 * j;
      rank[j] = 0;
      key[j] = 0;
      if (p < m) {
        x[j] = in.x[p];
        y[j] = in.y[p];
        w[j] = in.w[p];
        const unsigned g = (unsigned)(in.gid ? in.gid[p] : in.gid_base + p);
        key[j] = (unsigned long long)(unsigned)(tile_bin(x[j]) << 8 | tile_bin(y[j])) << 32 | g;
        sk[p] = key[j];
      }
    }
    __syncwarp();
    for (int t = 0; t < m; ++t) {
      const unsigned long long k = sk[t];
#pragma unroll
      for (int j = 0; j < NJ; ++j) rank[j] += k < key[j] ? 1 : 0;
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      if (lane + 32 * j < m) {
        rec[rank[j]] = make_uint4(__float_as_uint(x[j]), __float_as_uint(y[j]), (unsigned)key[j],
                                  __float_as_uint(__fmul_rn(0.5f, w[j])));
        nh[rank[j]] = __float_as_int(w[j]);
        const unsigned t = (unsigned)(key[j] >> 32);
        tile[rank[j]] = (uint16_t)(t >> 8 | (t & 255u) << 8);
      }
    }
    __syncwarp();
  }
  float2 pq[NJ];
  unsigned gq[NJ], box[NJ];
  float r[NJ], wq[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int q = lane + 32 * j;
    const uint4 rq = q < m ? rec[q] : make_uint4(0u, 0u, 0u, 0u);
    pq[j] = rec_xy(rq);
    gq[j] = rq.z;
    wq[j] = q < m ? __int_as_float(nh[q]) : 0.f;
    box[j] = pack_box(pq[j].x, pq[j].y, P.dc);
    r[j] = 0.f;
  }
  for (int k = 0; k < m; ++k) {
    const uint4 rk = rec[k];
    const unsigned tk = tile[k];
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      if (dist2(pq[j], rec_xy(rk)) <= P.t_dc && in_box(box[j], tk))
        r[j] = __fadd_rn(r[j], k == lane + 32 * j ? wq[j] : __uint_as_float(rk.w));
    }
  }
  __syncwarp();
  unsigned long long kq[NJ];
  float d2[NJ], prev[NJ];
  int best[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int q = lane + 32 * j;
    const unsigned o = float_ord(r[j]);
    if (q < m) {
      b.rho[in.ev_start + gq[j]] = r[j];
      rec[q].w = o;
    }
    kq[j] = o == 0u ? ~0ull : ((unsigned long long)o << 32 | gq[j]);
    box[j] = pack_box(pq[j].x, pq[j].y, P.dm);
    d2[j] = prev[j] = P.t_dm_next;
    best[j] = -1;
  }
  __syncwarp();
  for (int k = 0; k < m; ++k) {
    const uint4 rk = rec[k];
    const unsigned tk = tile[k];
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const float d = dist2(pq[j], rec_xy(rk));
      if (rec_key(rk) > kq[j] && d < d2[j] && in_box(box[j], tk)) {  // as NhBest
        prev[j] = d2[j];
        d2[j] = d;
        best[j] = k;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int q = lane + 32 * j;
    if (q >= m) continue;
    float best_s = best[j] >= 0 ? __fsqrt_rn(d2[j]) : FLT_MAX;
    if (best[j] >= 0 && NhBest::near(d2[j], prev[j])) {
      best_s = FLT_MAX;
      best[j] = -1;
      for (int k = 0; k < m; ++k) {
        const uint4 rk = rec[k];
        const float d = dist2(pq[j], rec_xy(rk));
        if (rec_key(rk) > kq[j] && d <= P.t_dm && in_box(box[j], tile[k])) {
          const float sd = __fsqrt_rn(d);
          if (sd < best_s) {
            best_s = sd;
            best[j] = k;
          }
        }
      }
    }
    const bool seed = (best_s > P.dc) && (r[j] >= P.rhoc);
    const bool outlier = (best_s > P.dm) && (r[j] < P.rhoc);
    const int64_t o = in.ev_start + gq[j];
    b.delta[o] = best_s;
    b.nh[o] = best[j] >= 0 ? (int)rec[best[j]].z : -1;
    b.seed[o] = seed ? 1 : 0;
    if (seed && b.seed_bits) atomicOr(&b.seed_bits[(int64_t)in.chunk0 * kChunkWords + (gq[j] >> 5)], 1u << (gq[j] & 31));
    nh[q] = (!seed && !outlier && best[j] >= 0) ? best[j] : (seed ? -2 : -3);
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int q = lane + 32 * j;
    if (q >= m) continue;
    int e = q, p = nh[q];
    while (p >= 0) {
      e = p;
      p = nh[e];
    }
    b.ci[in.ev_start + gq[j]] = p == -2 ? -((int)rec[e].z + 2) : -1;
  }
  __syncwarp();
}

// ------------------------------------------------------------------ kernels

// Per-batch counters to their start values: layer counts, seed bits and size
// classes to 0, the tickets and pass counters to 0, "grouped"
// to 1 (k_count clears it on the first layer decrease), and the error word to
// 0 unless it accumulates over several batches (clear_error = 0).  It also
// brings the batch's offset and chunk tables over from the host's page-locked
// staging, so that a batch queues no copies and no memsets of its own: each of
// those was a stream operation of 2-3 us, in a graph as well.
__global__ void k_init(Batch2D b, int64_t n_lcnt) {
  pdl_trigger();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < b.n_table_words) b.table_dst[i] = b.table_src[i];
  if (i < b.n_in16) b.in_dst[i] = b.host_in[i];
  if (i < n_lcnt) b.lcnt[i] = 0;
  if (b.seed_bits && i < (int64_t)b.n_chunks * (kChunkWords / 4))
    reinterpret_cast<uint4*>(b.seed_bits)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (b.use_order && i < 2 * kSizeBuckets) b.size_hist[i] = 0;
  if (i < kFlagCount && i != kFlagError) b.flags[i] = i == kFlagGrouped ? 1 : 0;
  if (i == kFlagError && b.clear_error) b.flags[kFlagError] = 0;
}

__global__ void __launch_bounds__(kChunkThreads) k_count(Batch2D b) {
  const int c = blockIdx.x;
  __shared__ int s_e;
  __shared__ int s_cnt[kLayers];
  for (int l = threadIdx.x; l < kLayers; l += kChunkThreads) s_cnt[l] = 0;
  pdl_begin();
  if (threadIdx.x == 0) s_e = event_of_chunk(b, c);
  __syncthreads();
  const int e = s_e;
  const int64_t es = b.offsets[e], ee = b.offsets[e + 1];
  const int64_t i0 = es + (int64_t)(c - b.chunk_start[e]) * kChunk;
  const int64_t i1 = min(i0 + (int64_t)kChunk, ee);
  const int lane = lane_id();
  bool ungrouped = false;
  // Four consecutive points per load and lane, from the 16-byte boundary at or
  // below the chunk's first point when the array has one (all loads first, so
  // that they are in flight together; the last round is the boundary's remainder);
  // single points otherwise (4096-event batch: 0.42 ms with one point per load and
  // a vote per 32 points, 0.255 ms).
  constexpr int PER = kChunk / kChunkThreads / 4 + 1;
  const bool vec = (reinterpret_cast<uintptr_t>(b.layer) & 15) == 0;
  const int64_t a0 = vec ? i0 & ~int64_t(3) : i0;
  int4 lv[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int64_t i = a0 + 4 * (threadIdx.x + j * (int64_t)kChunkThreads);
    lv[j] = make_int4(0, 0, 0, 0);
    if (i >= i1) continue;
    if (vec && i + 4 <= b.n_points) {
      lv[j] = *reinterpret_cast<const int4*>(b.layer + i);
    } else {
      lv[j].x = b.layer[i];
      if (i + 1 < i1) lv[j].y = b.layer[i + 1];
      if (i + 2 < i1) lv[j].z = b.layer[i + 2];
      if (i + 3 < i1) lv[j].w = b.layer[i + 3];
    }
  }
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int64_t i = a0 + 4 * (threadIdx.x + j * (int64_t)kChunkThreads);
    if (__all_sync(0xffffffffu, i >= i1)) break;
    const int v[4] = {lv[j].x, lv[j].y, lv[j].z, lv[j].w};
    const int prev = __shfl_up_sync(0xffffffffu, v[3], 1);
    // a warp whose 128 points hold one layer (most warps of grouped input): one increment
    const bool inside = i >= i0 && i + 4 <= i1;
    const int k0 = __shfl_sync(0xffffffffu, v[0], 0);
    const bool same = inside && v[0] == k0 && v[1] == k0 && v[2] == k0 && v[3] == k0;
    if (__all_sync(0xffffffffu, same) && k0 >= 0 && k0 < kLayers) {
      if (lane == 0) {
        atomicAdd(&s_cnt[k0], 128);
        // grouped input: a point's layer is not below its predecessor's
        if (i > es && k0 < b.layer[i - 1]) ungrouped = true;
      }
      continue;
    }
    // the others: one increment per run of a lane's points
    int run = 0, key = -1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i + k < i0 || i + k >= i1) continue;
      const int l = v[k];
      if (l < 0 || l >= kLayers) {
        atomicExch(&b.flags[kFlagError], 1);
        ungrouped = true;
        continue;
      }
      if (i + k > es) {
        const int pl = k ? v[k - 1] : (lane && i > i0 ? prev : b.layer[i - 1]);
        if (l < pl) ungrouped = true;
      }
      if (l != key) {
        if (run) atomicAdd(&s_cnt[key], run);
        key = l;
        run = 0;
      }
      ++run;
    }
    if (run) atomicAdd(&s_cnt[key], run);
  }
  if (__syncthreads_or(ungrouped) && threadIdx.x == 0) b.flags[kFlagGrouped] = 0;
  for (int l = threadIdx.x; l < kLayers; l += kChunkThreads)
    if (s_cnt[l]) atomicAdd(&b.lcnt[e * kLayers + l], s_cnt[l]);
}

// Ordered batches up to this size take their layers by size alone.  Larger
// ones that are not grouped by layer go event by event in each pass: a layer's
// outputs are then single words spread over its whole event, and with the
// layers of all events in turn their sectors leave L2 before the event's other
// layers complete them (15.4M points in 300 shuffled events: 155 + 144 B/point of
// DRAM traffic in k_layers; batch 3.16 -> 2.00 ms; 32M points in 100 HGCAL
// events 7.25 -> 4.11 ms).  Smaller batches stay in L2 and lose the even end that
// the size order gives: 10.8M points 1.44 against 1.48 ms, 1.7M 0.27 against 0.30.
constexpr int64_t kOrderBySize = 12 << 20;

// Size class of a non-empty layer: 0 for the largest.
__device__ __forceinline__ int size_bucket(int m) { return kSizeBuckets - 1 - min(m >> 4, kSizeBuckets - 1); }

// Place class of event e's layer of m points in the ordered batch: its size
// class, or, in a large batch that is not grouped by layer, the event's part
// of the classes of the pass that takes it.
__device__ __forceinline__ int order_class(const Batch2D& b, bool by_event, int e, int m) {
  const int c = size_bucket(m);
  if (!by_event) return c;
  const int lo = c < b.order_big ? 0 : b.order_big, n = (c < b.order_big ? b.order_big : kSizeBuckets) - lo;
  return lo + (int)((int64_t)e * n / b.n_events);
}

// One warp per event: layers 4*lane .. 4*lane+3.  Also counts the non-empty
// layers per place class for k_order.
__global__ void k_layer_scan(Batch2D b) {
  pdl_begin();
  const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (e >= b.n_events) return;
  const int lane = lane_id();
  const bool by_event = b.n_points > kOrderBySize && !b.flags[kFlagGrouped];
  int c[4];
  int sum = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int l = lane * 4 + j;
    c[j] = l < kLayers ? b.lcnt[e * kLayers + l] : 0;
    sum += c[j];
  }
  int x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += t;
  }
  int run = (int)b.offsets[e] + x - sum;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int l = lane * 4 + j;
    if (l < kLayers) {
      b.lstart[e * kLayers + l] = run;
      b.cursor[e * kLayers + l] = run;
    }
    run += c[j];
    if (!b.use_order) continue;
    const int key = c[j] > 0 ? order_class(b, by_event, e, c[j]) : -1;
    const unsigned grp = __match_any_sync(0xffffffffu, key);
    if (key >= 0 && lane == __ffs(grp) - 1) atomicAdd(&b.size_hist[key], __popc(grp));
  }
}

// The non-empty (event, layer) items in descending size class (a counting
// sort over the classes; the order inside a class is arbitrary).  The layer
// kernel takes its tickets in this order, so each pass ends on its smallest
// layers instead of on whichever layer came last.  Which CTA runs which
// layer never changes a result.  One warp per event; 256 threads per block,
// one per size class for the scan.
__global__ void __launch_bounds__(kSizeBuckets) k_order(Batch2D b) {
  static_assert(kSizeBuckets == 256, "one thread per size class");
  __shared__ int s_base[kSizeBuckets];
  __shared__ int s_ws[33];
  const int tid = threadIdx.x;
  pdl_begin();
  const int v = b.size_hist[tid];
  int total;
  const int inc = block_inclusive_scan<kSizeBuckets>(v, s_ws, &total);
  s_base[tid] = inc - v;
  __syncthreads();
  if (blockIdx.x == 0 && tid == 0) {
    // the large layers come first in the order: the large-layer pass takes
    // those, the other pass's tickets start behind them
    const int big = b.order_big > 0 ? s_base[b.order_big] : 0;
    // (size order: without the layers that k_layers takes by the warp)
    const bool by_size = b.n_points <= kOrderBySize || b.flags[kFlagGrouped];
    b.flags[kFlagOrdered] = b.small_layers && by_size ? s_base[size_bucket(kTiny - 1)] : total;
    b.flags[kFlagBigCount] = big;
    b.flags[kFlagTicket] = big;
  }
  const int e = (blockIdx.x * blockDim.x + tid) >> 5;
  if (e >= b.n_events) return;
  const int lane = lane_id();
  const bool by_event = b.n_points > kOrderBySize && !b.flags[kFlagGrouped];
  const unsigned lt = (1u << lane) - 1u;
  for (int l0 = 0; l0 < kLayers; l0 += 32) {
    const int l = l0 + lane;
    const int m = l < kLayers ? b.lcnt[e * kLayers + l] : 0;
    const int key = m > 0 ? order_class(b, by_event, e, m) : -1;
    const unsigned grp = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(grp) - 1;
    int pos = 0;
    if (key >= 0 && lane == leader) pos = atomicAdd(&b.size_hist[kSizeBuckets + key], __popc(grp));
    pos = __shfl_sync(0xffffffffu, pos, leader);
    if (key >= 0) b.order[s_base[key] + pos + __popc(grp & lt)] = e * kLayers + l;
  }
}

// Each chunk's points to their layers' grouped positions: counted per layer in
// shared memory first, so that a block reserves its places with one global
// atomic per layer (the order inside a layer is arbitrary: k_layers restores
// the index order).  With a global atomic per warp group of every pass the
// passes ran one after another at its round trip: 57 -> 21 us on one shuffled
// HGCAL event of 323k points.
// The chunk is put into layer order in shared memory and stored from there, so
// that a warp stores runs of a layer's points (some forty of a chunk's) and not 32
// words in 32 sectors of each array, which bound the kernel (15.4M shuffled points:
// 0.455 ms, the batch 2.02 -> 1.76 ms; 32M points in 100 HGCAL events 4.15 -> 3.55;
// 40 registers instead of 64 for three blocks per SM: the same).
// kSlices blocks per chunk where the chunks are fewer than the SMs (the kernel
// then waits on each block's chain of rank, reservation and stores): a shuffled
// HGCAL event as a host call 275 -> 270 us with four, 265 with the stores in
// runs; with more chunks one block each, which reserves and adds less.
template <int kSlices>
constexpr size_t kScatterSmem = 17 * (size_t)(kChunk / kSlices);  // a record and a layer per point

template <int kSlices>
__global__ void __launch_bounds__(kChunkThreads) k_scatter(Batch2D b) {
  extern __shared__ __align__(16) unsigned char dsm[];
  uint4* s_rec = reinterpret_cast<uint4*>(dsm);
  uint8_t* s_layer = reinterpret_cast<uint8_t*>(s_rec + kChunk / kSlices);
  __shared__ int s_e;
  __shared__ int s_cnt[kLayers];   // the slice's points per layer
  __shared__ int s_at[kLayers];    // their first slot here
  __shared__ int s_base[kLayers];  // their first position
  __shared__ int s_total;
  __shared__ int s_it;
  const int lane = lane_id();
  const unsigned lt = (1u << lane) - 1u;
  pdl_begin();
  if (b.flags[kFlagGrouped]) return;  // input already grouped by layer
  // a resident block's next slices from a ticket, taken while one is done
  const bool ticket = b.n_chunks * kSlices > 2 * (int)gridDim.x;
  for (int it = blockIdx.x; it < b.n_chunks * kSlices;) {
    const int c = it / kSlices;
    if (ticket && threadIdx.x == kChunkThreads - 1) s_it = (int)gridDim.x + atomicAdd(&b.flags[kFlagTicketScatter], 1);
    for (int l = threadIdx.x; l < kLayers; l += kChunkThreads) s_cnt[l] = 0;
    if (threadIdx.x == 0) s_e = event_of_chunk(b, c);
    __syncthreads();
    const int e = s_e;
    const int64_t es = b.offsets[e], ee = b.offsets[e + 1];
    const int64_t i0 = es + (int64_t)(c - b.chunk_start[e]) * kChunk + it % kSlices * (kChunk / kSlices);
    const int64_t i1 = min(i0 + kChunk / kSlices, ee);
    constexpr int PER = kChunk / kSlices / kChunkThreads;
    int lv[PER], rank[PER];
    float px[PER], py[PER], pw[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int64_t i = i0 + threadIdx.x + (int64_t)j * kChunkThreads;
      lv[j] = -1;
      if (i < i1) {
        lv[j] = b.layer[i];
        px[j] = b.x[i];
        py[j] = b.y[i];
        pw[j] = b.w[i];
        if (lv[j] >= kLayers) lv[j] = -1;
      }
    }
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const unsigned mask = __match_any_sync(0xffffffffu, lv[j]);
      const int leader = __ffs(mask) - 1;
      int old = 0;
      if (lv[j] >= 0 && lane == leader) old = atomicAdd(&s_cnt[lv[j]], __popc(mask));
      rank[j] = __shfl_sync(0xffffffffu, old, leader) + __popc(mask & lt);
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // slots of the layers, four per lane
      int n[4], sum = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        n[k] = 4 * lane + k < kLayers ? s_cnt[4 * lane + k] : 0;
        sum += n[k];
      }
      int x = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += t;
      }
      if (lane == 31) s_total = x;
      x -= sum;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (4 * lane + k < kLayers) s_at[4 * lane + k] = x;
        x += n[k];
      }
    } else if (threadIdx.x < 32 + kLayers) {
      const int l = threadIdx.x - 32;
      s_base[l] = s_cnt[l] ? atomicAdd(&b.cursor[e * kLayers + l], s_cnt[l]) : 0;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      if (lv[j] >= 0) {
        const int slot = s_at[lv[j]] + rank[j];
        const int64_t i = i0 + threadIdx.x + (int64_t)j * kChunkThreads;
        s_rec[slot] = make_uint4(__float_as_uint(px[j]), __float_as_uint(py[j]), __float_as_uint(pw[j]), (unsigned)(i - es));
        s_layer[slot] = (uint8_t)lv[j];
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int slot = threadIdx.x + j * kChunkThreads;
      if (slot < s_total) {
        const int l = s_layer[slot];
        const int pos = s_base[l] + slot - s_at[l];
        const uint4 r = s_rec[slot];
        b.gx[pos] = __uint_as_float(r.x);
        b.gy[pos] = __uint_as_float(r.y);
        b.gw[pos] = __uint_as_float(r.z);
        b.gid[pos] = (int32_t)r.w;
      }
    }
    it = ticket ? s_it : it + (int)gridDim.x;
    __syncthreads();  // the shared arrays of the next slice
  }
}

__device__ __forceinline__ LayerIO layer_io(const Batch2D& b, int item, bool grouped) {
  const int e = item / kLayers;
  const int64_t es = b.offsets[e];
  const int start = b.lstart[item];
  LayerIO io;
  io.ev_start = es;
  io.chunk0 = b.chunk_start[e];
  if (grouped) {
    io.x = b.x + start;
    io.y = b.y + start;
    io.w = b.w + start;
    io.gid = nullptr;
    io.gid_base = (int32_t)(start - es);
  } else {
    io.x = b.gx + start;
    io.y = b.gy + start;
    io.w = b.gw + start;
    io.gid = b.gid + start;
    io.gid_base = 0;
  }
  return io;
}

// Persistent CTAs over the (event, layer) queue, in event order or, when
// launched with use_order, largest layers first (k_order).  Two classes of layers: the
// first pass (big_pass = 0) takes every item from an atomic ticket and
// handles layers of at most max_m points on chip with `cap` points of shared
// memory (several CTAs per SM); larger layers are appended to a list that the
// second pass (big_pass = 1, launched with a large `cap` and fewer CTAs per
// SM) drains.  Layers above `cap` in either pass use HBM scratch.  In an
// ordered batch both lists are known beforehand (the order's two ends), and the
// passes run beside one another, see launch_clue2d.
template <int NT, bool kSmall>
__global__ void __launch_bounds__(NT, 1024 / NT) k_layers(Batch2D b, Params2D P, int cap, int max_m, int big_pass) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ int s_item;
  __shared__ int s_next;
  __shared__ int s_ws[33];
  __shared__ int s_bins[64];
  pdl_begin();
  const int n_items = b.use_order ? b.flags[kFlagOrdered] : b.n_events * kLayers;
  const bool grouped = b.flags[kFlagGrouped] != 0;
  LayerStore<uint16_t, uint16_t> sm;
  sm.tbl = reinterpret_cast<uint16_t*>(dsm);
  sm.rec = reinterpret_cast<uint4*>(dsm + kSmemTableBytes);
  sm.nh = reinterpret_cast<int32_t*>(sm.rec + cap);
  sm.qord = reinterpret_cast<uint16_t*>(sm.nh + cap);
  int32_t* big_list = b.cursor;  // k_scatter's cursors are dead by now
  if constexpr (kSmall) {  // small layers first, a warp each, in turn over all warps of the grid
    static_assert(NT / 32 * kTinyBytes <= kSmemTableBytes, "a warp's layer");
    unsigned char* ws = dsm + warp_id() * kTinyBytes;
    for (int item = blockIdx.x + gridDim.x * warp_id(); item < b.n_events * kLayers; item += gridDim.x * (NT / 32)) {
      const int m = b.lcnt[item];
      if (m > 0 && m < kTiny) tiny_layer(P, ws, m, layer_io(b, item, grouped), b);
    }
    __syncthreads();
  }
  // The next ticket is taken as soon as the current item is known and only
  // published at the next iteration, so the atomic's round trip overlaps the
  // current layer instead of holding the whole CTA at a barrier.
  auto fetch = [&]() {
    if (!big_pass) {
      const int t = atomicAdd(&b.flags[kFlagTicket], 1);
      if (t >= n_items) return -1;
      return b.use_order ? b.order[t] : t;
    }
    const int t = atomicAdd(&b.flags[kFlagTicket2], 1);
    return t < b.flags[kFlagBigCount] ? big_list[t] : -1;
  };
  int next = threadIdx.x == 0 ? fetch() : -1;
  for (;;) {
    if (threadIdx.x == 0) s_item = next;
    __syncthreads();
    const int item = s_item;
    __syncthreads();
    if (item < 0) break;
    if (threadIdx.x == 0) next = fetch();
    const int m = b.lcnt[item];
    if (m == 0) continue;
    if constexpr (kSmall) {
      if (m < kTiny) continue;
    }
    if (m > max_m) {  // first pass: leave it to the large-capacity pass
      if (threadIdx.x == 0) big_list[atomicAdd(&b.flags[kFlagBigCount], 1)] = item;
      continue;
    }
    // (layer_io() written out: with the call 60 HGCAL events took 1.669 ms against 1.657)
    const int e = item / kLayers;
    const int64_t es = b.offsets[e];
    const int start = b.lstart[item];
    LayerIO io;
    io.ev_start = es;
    io.chunk0 = b.chunk_start[e];
    if (grouped) {
      io.x = b.x + start;
      io.y = b.y + start;
      io.w = b.w + start;
      io.gid = nullptr;
      io.gid_base = (int32_t)(start - es);
    } else {
      io.x = b.gx + start;
      io.y = b.gy + start;
      io.w = b.gw + start;
      io.gid = b.gid + start;
      io.gid_base = 0;
    }
    if (m <= cap) {
      process_layer<NT>(P, sm, m, io, b, s_ws, s_bins, &s_next, next);
    } else {
      // spill: the same stages on HBM scratch at this layer's grouped position
      LayerStore<int32_t, int32_t> g;
      g.rec = reinterpret_cast<uint4*>(b.sp[0]) + start;
      g.nh = reinterpret_cast<int32_t*>(b.sp[4]) + start;
      g.qord = reinterpret_cast<int32_t*>(b.sp[5]) + start;
      g.tbl = b.sp_tbl + (size_t)blockIdx.x * kTableStride;
      if (threadIdx.x == 0) atomicAdd(&b.flags[kFlagSpilled], 1);
      process_layer<NT>(P, g, m, io, b, s_ws, s_bins, &s_next, next);
    }
  }
}
// The seeds of a lane's 128 points of event e's chunk c, four words: of the
// chunk's bits (kBits), or, where the run has no memory for those, built from its
// flags.  (One kernel that asks which: a toy event 33.3 -> 34.0 us.)
template <bool kBits>
__device__ __forceinline__ uint4 seed_words(const Batch2D& b, int e, int c) {
  const int lane = lane_id();
  if constexpr (kBits) return reinterpret_cast<const uint4*>(b.seed_bits + (int64_t)c * kChunkWords)[lane];
  const int64_t i0 = b.offsets[e] + (int64_t)(c - b.chunk_start[e]) * kChunk, i1 = b.offsets[e + 1];
  unsigned w[4] = {0u, 0u, 0u, 0u};
#pragma unroll 4
  for (int k = 0; k < kChunkWords; ++k) {
    const int64_t i = i0 + 32 * k + lane;
    const unsigned v = __ballot_sync(0xffffffffu, i < i1 && b.seed[i] == 1);
    if (lane == k >> 2) w[k & 3] = v;
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// One block per event: exclusive scan of its chunks' seed counts, which are
// counted from the bits by a warp per chunk.  The bits of large events come
// through one SM, so their blocks are as wide as they go (see launch_clue2d).
template <bool kBits, int NT>
__global__ void __launch_bounds__(NT) k_seed_chunk_scan(Batch2D b) {
  __shared__ int s_n[NT];
  __shared__ int s_ws[33];
  pdl_begin();
  const int e = blockIdx.x;
  const int c0 = b.chunk_start[e], c1 = b.chunk_start[e + 1];
  int run = 0;
  for (int base = c0; base < c1; base += NT) {
#pragma unroll 4
    for (int k = warp_id(); k < min(NT, c1 - base); k += NT / 32) {
      const uint4 w = seed_words<kBits>(b, e, base + k);
      const int n = (int)__reduce_add_sync(0xffffffffu, (unsigned)(__popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w)));
      if (lane_id() == 0) s_n[k] = n;
    }
    __syncthreads();
    const int c = base + threadIdx.x;
    const int v = c < c1 ? s_n[threadIdx.x] : 0;
    int total;
    const int x = block_inclusive_scan<NT>(v, s_ws, &total);
    if (c < c1) b.chunk_base[c] = run + x - v;
    run += total;
  }
}

// Cluster id of each seed = its rank among the event's seeds in index order.
// One warp per chunk, from the seeds' bits (512 bytes of a chunk; reading its
// 16 KB of seed flags took 0.325 ms on the 4096-event batch, this 0.121 ms).
template <bool kBits>
__global__ void __launch_bounds__(256) k_seed_rank(Batch2D b) {
  pdl_begin();
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= b.n_chunks) return;
  const int lane = lane_id();
  const uint4 w4 = seed_words<kBits>(b, kBits ? 0 : event_of_chunk(b, c), c);
  const unsigned w[4] = {w4.x, w4.y, w4.z, w4.w};
  const int n = __popc(w[0]) + __popc(w[1]) + __popc(w[2]) + __popc(w[3]);
  int x = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += t;
  }
  const int e = event_of_chunk(b, c);
  const int64_t i0 = b.offsets[e] + (int64_t)(c - b.chunk_start[e]) * kChunk + lane * 128;
  int run = b.chunk_base[c] + x - n;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    for (unsigned m = w[k]; m; m &= m - 1) b.ci[i0 + 32 * k + __ffs((int)m) - 1] = run++;
}

// kHostOut: a small host run, whose outputs also go to the page-locked staging
// (an instantiation of its own: the branch cost the others 0.1 ms per 65M points).
// There a chunk is cut into slices of a block each: a block's stores to host
// memory complete a few at a time, and a 5,000-point event is two chunks (one
// host call of 5,000 points: 67 -> 58 us; this kernel 21.8 -> 5.6 us).
constexpr int kHostSlices = 8;
template <bool kHostOut>
__global__ void __launch_bounds__(kChunkThreads) k_label(Batch2D b) {
  constexpr int kSlices = kHostOut ? kHostSlices : 1;
  const int c = blockIdx.x / kSlices;
  __shared__ int s_e;
  pdl_wait();
  // the run's status words, final by now, to the host's page-locked copy
  if (blockIdx.x == 0 && threadIdx.x < kFlagCount && b.host_flags) b.host_flags[threadIdx.x] = b.flags[threadIdx.x];
  if (threadIdx.x == 0) s_e = event_of_chunk(b, c);
  __syncthreads();
  const int e = s_e;
  const int64_t es = b.offsets[e], ee = b.offsets[e + 1];
  const int64_t i0 = es + (int64_t)(c - b.chunk_start[e]) * kChunk + blockIdx.x % kSlices * (kChunk / kSlices);
  const int64_t i1 = min(i0 + kChunk / kSlices, ee);
  const int64_t n_ev = ee - es;
  // ci holds a seed's rank (>= 0, from k_seed_rank), -1 (no cluster), or
  // -(root + 2) for a point whose chain ends at the seed `root` (event-local
  // index); only the last kind is rewritten, with the root's rank.  Points
  // with an invalid layer were never written, so the root is range-checked.
  // The roots are seeds, which this kernel never writes; the gathers of one
  // thread's points are issued together.
  constexpr int PER = kChunk / kSlices / kChunkThreads;
  int v[PER], r[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int64_t i = i0 + threadIdx.x + (int64_t)j * kChunkThreads;
    v[j] = i < i1 ? b.ci[i] : -1;
  }
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int64_t root = -(int64_t)v[j] - 2;
    r[j] = (v[j] <= -2 && root < n_ev) ? b.ci[es + root] : -1;
  }
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int64_t i = i0 + threadIdx.x + (int64_t)j * kChunkThreads;
    if (i < i1 && v[j] <= -2) b.ci[i] = r[j];
  }
  if constexpr (kHostOut) {
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int64_t i = i0 + threadIdx.x + (int64_t)j * kChunkThreads;
      if (i < i1) {
        float* o = b.host_out + i;
        o[0] = b.rho[i];
        o[b.n_points] = b.delta[i];
        o[2 * b.n_points] = __int_as_float(b.nh[i]);
        o[3 * b.n_points] = __int_as_float(b.seed[i]);
        o[4 * b.n_points] = __int_as_float(v[j] <= -2 ? r[j] : v[j]);
      }
    }
  }
}

// Beside event dependencies a kernel is launched the ordinary way (its
// pdl_wait() then has nothing to wait for).
enum LaunchKind { kDependent, kOrdinary };

template <int NT, bool kSmall = false>
cudaError_t launch_layers(const Batch2D& b, const Params2D& p, int cap, int max_m, int big_pass, int grid,
                          cudaStream_t s, LaunchKind kind) {
  Tuning2D t;
  t.layer_capacity = cap;
  if (kind == kOrdinary) {
    k_layers<NT, kSmall><<<grid, NT, layer_smem_bytes(t), s>>>(b, p, cap, max_m, big_pass);
    return cudaGetLastError();
  }
  return launch_pdl(k_layers<NT, kSmall>, grid, NT, layer_smem_bytes(t), s, b, p, cap, max_m, big_pass);
}

cudaError_t launch_layers_any(int threads, const Batch2D& b, const Params2D& p, int cap, int max_m, int big_pass,
                              int grid, cudaStream_t s, LaunchKind kind) {
  switch (threads) {
    case 128: return launch_layers<128>(b, p, cap, max_m, big_pass, grid, s, kind);
    case 256:
      if (b.small_layers && !big_pass) return launch_layers<256, true>(b, p, cap, max_m, big_pass, grid, s, kind);
      return launch_layers<256>(b, p, cap, max_m, big_pass, grid, s, kind);
    case 1024: return launch_layers<1024>(b, p, cap, max_m, big_pass, grid, s, kind);
    default: return launch_layers<512>(b, p, cap, max_m, big_pass, grid, s, kind);
  }
}

template <int NT, bool kSmall = false>
cudaError_t allow_max_smem(int optin) {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, k_layers<NT, kSmall>);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_layers<NT, kSmall>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              optin - (int)a.sharedSizeBytes);
}

}  // namespace

cudaError_t prepare_clue2d_kernels(int device) {
  int optin = 0;
  cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  if (e != cudaSuccess) return e;
  if ((e = allow_max_smem<128>(optin)) != cudaSuccess) return e;
  if ((e = allow_max_smem<256>(optin)) != cudaSuccess) return e;
  if ((e = allow_max_smem<256, true>(optin)) != cudaSuccess) return e;
  if ((e = allow_max_smem<512>(optin)) != cudaSuccess) return e;
  if ((e = allow_max_smem<1024>(optin)) != cudaSuccess) return e;
  // Asking for a kernel's attributes loads its code on this device (the
  // runtime loads kernels lazily, at first use, by default), so that no
  // later launch of the pipeline has code to load.
  const void* rest[] = {reinterpret_cast<const void*>(k_init), reinterpret_cast<const void*>(k_count),
                        reinterpret_cast<const void*>(k_layer_scan), reinterpret_cast<const void*>(k_order),
                        reinterpret_cast<const void*>(k_scatter<1>), reinterpret_cast<const void*>(k_scatter<4>),
                        reinterpret_cast<const void*>(k_seed_chunk_scan<true, 256>),
                        reinterpret_cast<const void*>(k_seed_chunk_scan<true, 1024>),
                        reinterpret_cast<const void*>(k_seed_chunk_scan<false, 1024>),
                        reinterpret_cast<const void*>(k_seed_rank<true>),
                        reinterpret_cast<const void*>(k_seed_rank<false>), reinterpret_cast<const void*>(k_label<false>),
                        reinterpret_cast<const void*>(k_label<true>)};
  if ((e = cudaFuncSetAttribute(k_scatter<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScatterSmem<1>)) !=
      cudaSuccess)
    return e;
  for (const void* f : rest) {
    cudaFuncAttributes a;
    if ((e = cudaFuncGetAttributes(&a, f)) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

float sqrt_le_threshold(float d) {
  // P(t) = sqrtf(t) <= d is monotone over t >= 0; binary search over the
  // ordered bit patterns of non-negative finite floats.
  if (!(sqrtf(0.f) <= d)) return -1.f;
  uint32_t lo = 0, hi = 0x7f7fffffu;  // P(lo) holds
  auto val = [](uint32_t u) {
    float f;
    memcpy(&f, &u, 4);
    return f;
  };
  if (sqrtf(val(hi)) <= d) return val(hi);
  while (hi - lo > 1) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (sqrtf(val(mid)) <= d) lo = mid; else hi = mid;
  }
  return val(lo);
}

Params2D make_params2d(float dc, float rhoc, float odf) {
  Params2D p;
  p.dc = dc;
  p.rhoc = rhoc;
  p.odf = odf;
  volatile float a = odf, c = dc;
  p.dm = a * c;
  p.t_dc = sqrt_le_threshold(dc);
  p.t_dm = sqrt_le_threshold(p.dm);
  // the next float above t_dm (d2 < t_dm_next <=> d2 <= t_dm); -1 stays -1
  p.t_dm_next = p.t_dm < 0.f ? p.t_dm : nextafterf(p.t_dm, INFINITY);
  return p;
}

size_t layer_smem_bytes(const Tuning2D& t) {
  // 16-bit tile table, then 22 bytes per point (see LayerStore)
  return (size_t)kSmemTableBytes + (size_t)t.layer_capacity * 22;
}

int layer_grid_max(const Tuning2D& t, int n_items) {
  int g = layer_grid(t, n_items);
  if (t.big_threads > 0 && t.big_capacity > t.layer_capacity) {
    Tuning2D big;
    big.threads = t.big_threads;
    big.layer_capacity = t.big_capacity;
    const int g2 = layer_grid(big, n_items);
    g = g2 > g ? g2 : g;
  }
  return g;
}

int layer_grid(const Tuning2D& t, int n_items) {
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int per_sm = t.ctas_per_sm;
  if (per_sm <= 0) {
    // resident CTAs per SM as the hardware sees them (registers, shared memory, threads)
    const size_t smem = layer_smem_bytes(t);
    cudaError_t e = cudaErrorInvalidValue;
    switch (t.threads) {
      case 128: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_layers<128, false>, 128, smem); break;
      case 256: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_layers<256, false>, 256, smem); break;
      case 512: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_layers<512, false>, 512, smem); break;
      case 1024: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_layers<1024, false>, 1024, smem); break;
      default: break;
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      per_sm = 1;
    }
    per_sm = per_sm < 1 ? 1 : per_sm;
  }
  int g = sms * per_sm;
  if (g > n_items) g = n_items;  // never more CTAs than (event, layer) items: see launch_clue2d
  return g < 1 ? 1 : g;
}

// Largest layers first only where a pass ends on a visible tail: a few
// layers per CTA (a sub-batch, a served batch).  With one layer per CTA or
// less (a single event) every layer starts at once, and with hundreds per
// CTA the tail is negligible and the event order measured faster.
bool layers_ordered(const Tuning2D& t, int n_items) {
  const int g = layer_grid(t, n_items);
  return n_items > g && n_items <= 64 * g;
}

cudaError_t launch_clue2d(const Batch2D& batch, const Params2D& p, const Tuning2D& t, cudaStream_t s,
                          cudaEvent_t* ev, int64_t* kernels, const SideStream* side) {
  if (batch.n_events <= 0 || batch.n_points <= 0) return cudaSuccess;
  Batch2D b = batch;
  const int n_items = b.n_events * kLayers;
  // No more layers than SMs (a single event): one pass of the widest CTA per
  // layer, so that each layer's phases spread over 32 warps and large layers
  // stay on chip.  Measured per producer call: 0.177 -> 0.131 ms on events of
  // 150k-200k points, 0.136 -> 0.117 ms on 50k-150k, 0.113 -> 0.101 ms on 5k-20k.
  Tuning2D tt = t;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (n_items <= sms) {
    tt.threads = 1024;
    tt.layer_capacity = std::max(std::max(t.layer_capacity, t.big_capacity), 4096);
    tt.ctas_per_sm = 0;
    tt.big_threads = tt.big_capacity = 0;
  }
  const bool two_class = tt.big_threads > 0 && tt.big_capacity > tt.layer_capacity;
  b.use_order = layers_ordered(t, n_items) ? 1 : 0;
  // the size classes that may hold a layer above the first capacity; all of
  // their layers fit the second one, or its HBM scratch
  b.order_big = two_class ? kSizeBuckets - std::min(tt.layer_capacity >> 4, kSizeBuckets - 1) : 0;
  // Batches whose layers hold 80 points and fewer on average take theirs of
  // fewer than kTiny points by the warp (500 events of 6,300 points: 0.80 -> 0.63 ms, of
  // 6,700: 0.81 -> 0.67, 2,000 events of 100 points: 1.79 -> 0.28; with few small
  // layers the others lose: 48 events of 5,000 to 200,000 points 1 %).  A
  // single event has warps to spare for each layer and stays with whole CTAs (5,000
  // points as a host call: 58 us, 67 with a warp per layer).
  b.small_layers = n_items > layer_grid(tt, n_items) && b.n_points <= (int64_t)80 * n_items && tt.threads == 256 &&
                   tt.layer_capacity >= 2 * kTiny;
  cudaError_t err;
  auto mark = [&](int i) {
    if (ev) cudaEventRecord(ev[i], s);
  };
  const int nc = b.n_chunks;
  {
    // counters, tickets and flags of this batch
    const int64_t n_lcnt = (int64_t)b.n_events * kLayers;
    const int64_t n_init = std::max({n_lcnt, (int64_t)nc * (kChunkWords / 4), b.n_table_words, b.n_in16, (int64_t)2 * kSizeBuckets});
    NvtxRange r("clue2d/init");
    k_init<<<(unsigned)((n_init + 255) / 256), 256, 0, s>>>(b, n_lcnt);
    if ((err = cudaGetLastError()) != cudaSuccess) return err;
  }
  const int warps_grid = (b.n_events * 32 + 255) / 256;
  mark(0);
  {
    NvtxRange r("clue2d/count");
    if ((err = launch_pdl(k_count, nc, kChunkThreads, 0, s, b)) != cudaSuccess) return err;
  }
  mark(1);
  {
    NvtxRange r("clue2d/layer_scan");
    if ((err = launch_pdl(k_layer_scan, warps_grid, 256, 0, s, b)) != cudaSuccess) return err;
    if (b.use_order && (err = launch_pdl(k_order, warps_grid, kSizeBuckets, 0, s, b)) != cudaSuccess) return err;
  }
  mark(2);
  {
    NvtxRange r("clue2d/scatter");
    // A resident grid, two blocks of 64 registers a thread per SM: grouped input
    // has nothing to do here (57 -> 4 us on the 4096-event batch against a block
    // per chunk), and of three per SM every third block started with as many
    // chunks to go as the others when those were done (15.3M shuffled points 0.198
    // -> 0.160 ms, 32.5M 0.407 -> 0.323).  Up to five chunks per SM leave
    // two and a few threes to a block of two per SM, and take three (2.5M points 244
    // us in all, 247).
    err = nc <= sms ? launch_pdl(k_scatter<4>, nc * 4, kChunkThreads, kScatterSmem<4>, s, b)
                    : launch_pdl(k_scatter<1>, std::min(nc, sms * (nc <= 5 * sms ? 3 : 2)), kChunkThreads, kScatterSmem<1>, s, b);
    if (err != cudaSuccess) return err;
  }
  mark(3);
  // Invariant: every layer-kernel grid is at most n_items = n_events * kLayers
  // (layer_grid caps it there).  The per-CTA HBM tile tables of the spill
  // path are sized on it: one table per (event, layer) at most, e.g. 100 for
  // a single event, which the allocation-free entry point relies on.
  {
    NvtxRange r("clue2d/layers");
    const int grid = layer_grid(tt, n_items);
    const int max_m = two_class ? tt.layer_capacity : INT_MAX;
    Tuning2D big;
    big.threads = tt.big_threads;
    big.layer_capacity = tt.big_capacity;
    if (two_class && b.use_order) {
      // The large layers first, so that they do not start last.  In a captured
      // run the others go beside them, from the same point on the side stream: their
      // CTAs start as the large pass runs out of layers, instead of after its last
      // one has ended (48 uneven events replayed 289 -> 264 us, 380: 1.95 -> 1.91 ms).
      // With up to three layers per CTA one after the other: side by side their few
      // long layers share SMs to the end (8 events 154 against 120 us, 12: 159 / 132,
      // 16: 142 / 134; but 24: 178 / 210).  Direct launches go one after the other
      // as well: there the side stream's pass often took the SMs first and the large
      // layers came last (48 events 342 against 299 us; 65 of which two layers hold a
      // third 2.46 against 1.36 ms; 380 even ones 1.94 against 1.95).
      if (side) {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        if ((err = cudaStreamIsCapturing(s, &capture)) != cudaSuccess) return err;
        if (capture == cudaStreamCaptureStatusNone || n_items <= 3 * grid) side = nullptr;
      }
      const LaunchKind kind = side ? kOrdinary : kDependent;
      Batch2D large = b;
      large.cursor = b.order;  // the list that the large-layer pass drains
      cudaStream_t s2 = side ? side->stream : s;
      if (side && (err = cudaEventRecord(side->fork, s)) != cudaSuccess) return err;
      err = launch_layers_any(big.threads, large, p, big.layer_capacity, INT_MAX, 1, layer_grid(big, n_items), s,
                              kind);
      if (err == cudaSuccess && side) err = cudaStreamWaitEvent(s2, side->fork, 0);
      if (err == cudaSuccess) err = launch_layers_any(tt.threads, b, p, tt.layer_capacity, max_m, 0, grid, s2, kind);
      if (err == cudaSuccess && side) err = cudaEventRecord(side->join, s2);
      if (err == cudaSuccess && side) err = cudaStreamWaitEvent(s, side->join, 0);
    } else {
      side = nullptr;
      err = launch_layers_any(tt.threads, b, p, tt.layer_capacity, max_m, 0, grid, s, kDependent);
      if (err == cudaSuccess && two_class)
        err = launch_layers_any(big.threads, b, p, big.layer_capacity, INT_MAX, 1, layer_grid(big, n_items), s, kDependent);
    }
  }
  if (err != cudaSuccess) return err;
  mark(4);
  {
    NvtxRange r("clue2d/seed_chunk_scan");
    // from 24 chunks per event on (100,000 points; fewer are done in the same time
    // by narrow blocks, which more events share an SM with): one event of 9M points
    // 109 -> 33 us, 200 of 325,000 10 -> 8
    const bool wide = !b.seed_bits || nc >= 24 * (int64_t)b.n_events;
    auto* k = !b.seed_bits ? k_seed_chunk_scan<false, 1024> : wide ? k_seed_chunk_scan<true, 1024> : k_seed_chunk_scan<true, 256>;
    const int threads = wide ? 1024 : 256;
    if (side) {  // behind the join of the two passes
      k<<<b.n_events, threads, 0, s>>>(b);
      err = cudaGetLastError();
    } else {
      err = launch_pdl(k, b.n_events, threads, 0, s, b);
    }
    if (err != cudaSuccess) return err;
  }
  mark(5);
  {
    NvtxRange r("clue2d/seed_rank");
    if ((err = launch_pdl(b.seed_bits ? k_seed_rank<true> : k_seed_rank<false>, (nc + 7) / 8, 256, 0, s, b)) != cudaSuccess) return err;
  }
  mark(6);
  {
    NvtxRange r("clue2d/label");
    err = b.host_out ? launch_pdl(k_label<true>, nc * kHostSlices, kChunkThreads, 0, s, b)
                     : launch_pdl(k_label<false>, nc, kChunkThreads, 0, s, b);
    if (err != cudaSuccess) return err;
  }
  mark(7);
  if (kernels) *kernels += 8 + (b.use_order ? 1 : 0) + (two_class ? 1 : 0);
  return cudaSuccess;
}

}  // namespace clue

namespace clue {
namespace {

// Order-sensitive 64-bit digest of a word array: sum of w[i] * (2i+1) * K.
__global__ void k_digest(const uint32_t* a, int64_t n, unsigned long long* out) {
  unsigned long long acc = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    acc += (unsigned long long)a[i] * (2ull * (unsigned long long)i + 1ull) * 0x9E3779B97F4A7C15ull;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, acc);
}

}  // namespace

cudaError_t launch_digest(const void* words, int64_t n_words, unsigned long long* d_out, cudaStream_t s) {
  if (n_words <= 0) return cudaSuccess;
  int blocks = (int)((n_words + 255) / 256);
  if (blocks > 4096) blocks = 4096;
  k_digest<<<blocks, 256, 0, s>>>(static_cast<const uint32_t*>(words), n_words, d_out);
  return cudaGetLastError();
}

}  // namespace clue
