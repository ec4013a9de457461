// CLUE3D on GB300: the SoA tracksterizer stages of
// src/serial/plugin-CLUETracksterizer/CLUE3DAlgoKernels.h re-designed for
// batches of events.
//
// Layout: per event, the layer clusters are counting-sorted by their flat
// tile key  key = layer*4284 + phiBin + 126*etaBin  (the reference's tiles
// are one contiguous array over layers, so an eta row of 34 lands in the next
// layer's row 0, and phiBin may be 126; both are reproduced).  A "row" is
// key/126 (one (layer, eta) line of 126 phi bins); inside a row entries are
// ordered by (phi bin, index), which is the reference's visiting order for
// a phi window that does not wrap.  A wrapping window is visited as its two
// arcs in the reference's order.
//
// Stages (one launch each, flattened over all events of the batch):
//   k3_init       counters and masks to zero, tables over from the host
//   k3_key        flat key per cluster; clusters per (event, row) and each
//                 cluster's arrival slot in its row
//   k3_row_scan   per event: first position of each row
//   k3_scatter    place clusters into their rows (arrival order) with their
//                 candidate and query records; row occupancy and repeat masks
//   k3_row_sort   order each row by (phi bin, index): a counting sort by
//                 column through the mask, or a count where a column repeats
//   k3_search<true>   KernelCalculateDensitySoA (:26-150), one block per
//                     (event, slab of layers) with the slab's rows staged
//   k3_search<false>  KernelComputeDistanceToHigherSoA (:286-392), likewise,
//                     then seeds, outliers and parent pointers (:509-560)
//   k3_rank, k3_label   trackster ids by seed rank, walks along
//                 nearestHigher, labels (:564-577)
// Float arithmetic uses explicit _rn intrinsics in the reference's operation
// order; phiBin's product is in double, as in TICLLayerTile.h:28-34.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdint>

#include "clue_internal.h"
#include "clue_pdl.cuh"

namespace clue {
namespace {

constexpr int kEtaBins = 34;
constexpr int kPhiBins = 126;
constexpr int kBins = kEtaBins * kPhiBins;

// Event of cluster i: from the event of its 256-cluster block's first
// cluster, forward past the events that end at or before i.
__device__ __forceinline__ int event_of_blk(const Batch3D& b, int64_t i) {
  int e = b.blk_ev[i >> 8];
  while (b.offsets[e + 1] <= i) ++e;
  return e;
}


// reco::reduceRange for float (src/serial/DataFormats/Math/deltaPhi.h:16-23)
__device__ __forceinline__ float reduce_range(float x, const Params3D& P) {
  if (fabsf(x) <= P.pi_f) return x;
  const float n = roundf(__fmul_rn(x, P.o2pi));
  return __fsub_rn(x, __fmul_rn(n, P.twopi_f));
}

// TICLLayerTileT::etaBin (src/serial/DataFormats/TICLLayerTile.h:19-26)
__device__ __forceinline__ int eta_bin(float eta, const Params3D& P) {
  const int b = __float2int_rz(__fmul_rn(__fsub_rn(fabsf(eta), 1.5f), P.eta_r));
  return min(max(b, 0), kEtaBins - 1);
}

// TICLLayerTileT::phiBin (TICLLayerTile.h:28-34): (normPhi + M_PI) * r in double.
// A NaN (phi NaN or +-inf, which reduce to NaN) takes bin 0: the reference's
// int conversion is undefined there, 0 on the aarch64 host, and the device's
// conversion would give INT_MIN.
__device__ __noinline__ int phi_bin_double(float norm, float phi_r) {
  if (norm != norm) return 0;
  return __double2int_rz(__dmul_rn(__dadd_rn((double)norm, 3.14159265358979323846), (double)phi_r));
}

// The same bin from the single-precision product where that cannot lie on the
// other side of a bin edge: the sum is off by at most 3.3e-7 (the float pi, one
// rounding below 6.3), times 20.05 bins per radian, plus half an ulp of 126:
// 1.1e-5, so values 1e-4 and more from an edge truncate alike; the others
// (one in 5,000) call the double form.
__device__ __forceinline__ int phi_bin(float phi, const Params3D& P) {
  const float norm = reduce_range(phi, P);
  const float t = __fmul_rn(__fadd_rn(norm, P.pi_f), P.phi_r);
  const float f = t - truncf(t);
  if (t > 0.f && t < 127.f && f > 1e-4f && f < 1.f - 1e-4f) return __float2int_rz(t);
  return phi_bin_double(norm, P.phi_r);
}

// The reference's layer window (CLUE3DAlgoKernels.h:49-58 density, :308-317
// nearest higher; the upper side starts one layer later there).
__device__ __forceinline__ void layer_window(int layer, int sib, int n_layers, int upper_shift, int* lo, int* hi) {
  const int last = n_layers / 2;
  int mx = 2 * last - 1, mn = 0;
  if (layer < last) {
    mn = max(layer - sib, mn);
    mx = min(layer + sib, last - 1);
  } else {
    mn = max(layer - sib, last + upper_shift);
    mx = min(layer + sib, mx);
  }
  *lo = mn;
  *hi = mx;
}

// Row of a flat key; clusters rejected by k3_key (key -1) go to the
// event's last row, which no search visits.
__device__ __forceinline__ int row_of(int k, int n_rows) { return k >= 0 ? k / kPhiBins : n_rows - 1; }

// A placed cluster is one 32-byte record, a whole memory sector written by one
// store: as a candidate {roa, phi, energy, rho} (rho added by the density
// search), as a query {z, event-local index, density threshold, bins}.  Records
// go to scattered places; in pieces (two 16-byte records, the index and the
// column in arrays of their own) half the sectors reached DRAM partly written
// and were read back to be completed.
__device__ __forceinline__ void store_record(float4* rec, int64_t at, float roa, float phi, float energy, float z, int idx,
                                             float thr, int bins) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(rec + 2 * at), "r"(__float_as_int(roa)),
               "r"(__float_as_int(phi)), "r"(__float_as_int(energy)), "r"(0), "r"(__float_as_int(z)), "r"(idx),
               "r"(__float_as_int(thr)), "r"(bins)
               : "memory");
}

// bins: layer | etaBin << 11 | phiBin << 17 | isSilicon << 24, or -1 for a
// cluster rejected by the binning (its row is never searched).
__device__ __forceinline__ int pack_bins(int l, int eb, int pb, bool sil) {
  return l | (eb << 11) | (pb << 17) | ((sil ? 1 : 0) << 24);
}
__device__ __forceinline__ int bins_key(int bins) {
  return (bins & 0x7ff) * kBins + ((bins >> 17) & 0x7f) + ((bins >> 11) & 0x3f) * kPhiBins;
}
// Phi column in the row: phi bin 126 is column 0 of the next row.
__device__ __forceinline__ int bins_col(int bins) {
  const int pb = (bins >> 17) & 0x7f;
  return pb < kPhiBins ? pb : 0;
}

// Row counts, row masks and status words to zero, the offset and block tables
// (and a small host run's inputs) over from the host's page-locked staging: a
// run queues kernels only.
__global__ void k3_init(Batch3D b) {
  pdl_trigger();
  const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = i0; i < b.n_table_words; i += step) b.table_dst[i] = b.table_src[i];
  for (int64_t i = i0; i < b.n_in16; i += step) b.in_dst[i] = b.host_in[i];
  const int64_t rows = (int64_t)b.n_events * b.n_rows;
  uint4* m = reinterpret_cast<uint4*>(b.row_mask);
  uint4* r = reinterpret_cast<uint4*>(b.row_rep);
  for (int64_t i = i0; i < rows; i += step) {
    b.row_cnt[i] = 0;
    m[i] = make_uint4(0u, 0u, 0u, 0u);
    r[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  if (i0 < kFlagCount) b.flags[i0] = 0;
}

__global__ void k3_key(Batch3D b, Params3D P) {
  pdl_begin();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int row = -1, e = 0;
  if (i < b.n_points) {
    e = event_of_blk(b, i);
    const int l = b.layer[i];
    const int pb = phi_bin(b.phi[i], P);
    int k = -1;
    if (l < 0 || l >= P.n_layers) {
      atomicExch(&b.flags[kFlagError], 1);
    } else if (pb < 0 || pb > kPhiBins) {
      atomicExch(&b.flags[kFlagError], 2);
    } else {
      k = l * kBins + pb + eta_bin(b.eta[i], P) * kPhiBins;
    }
    b.key[i] = k;
    if (k < 0) b.seed[i] = -1;  // not searched: k3_rank makes it a root of its own
    row = row_of(k, b.n_rows);
  }
  const int gkey = row >= 0 ? e * b.n_rows + row : -1;
  const unsigned mask = __match_any_sync(0xffffffffu, gkey);
  const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
  int old = 0;
  if (gkey >= 0 && lane == leader) old = atomicAdd(&b.row_cnt[gkey], __popc(mask));
  old = __shfl_sync(0xffffffffu, old, leader);
  if (gkey >= 0) b.arr[i] = old + __popc(mask & ((1u << lane) - 1u));
}

// Entries of a row whose phi column lies in [a, c] (0 <= a <= c <= 125) are
// one run of the row (entries are sorted by column): its first position and
// length, from the column-occupancy mask, when no column repeats.
__device__ __forceinline__ int bits_below(unsigned long long m0, unsigned long long m1, int p) {
  // set bits of columns < p (0 <= p <= 126)
  if (p <= 0) return 0;
  if (p < 64) return __popcll(m0 & ((1ull << p) - 1));
  return __popcll(m0) + __popcll(m1 & ((1ull << (p - 64)) - 1));
}

// One block per event: exclusive scan of its rows.
__global__ void __launch_bounds__(256) k3_row_scan(Batch3D b) {
  pdl_begin();
  const int e = blockIdx.x;
  const int R = b.n_rows;
  const int per = (R + 255) / 256;
  const int beg = min((int)threadIdx.x * per, R), end = min(beg + per, R);
  const int32_t* cnt = b.row_cnt + (int64_t)e * R;
  int sum = 0;
  for (int r = beg; r < end; ++r) sum += cnt[r];
  __shared__ int s_w[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += t;
  }
  if (lane == 31) s_w[warp] = x;
  __syncthreads();
  int before = 0;
  for (int w = 0; w < warp; ++w) before += s_w[w];
  int run = (int)b.offsets[e] + before + x - sum;
  for (int r = beg; r < end; ++r) {
    b.row_start[(int64_t)e * R + r] = run;
    run += cnt[r];
  }
  if (e == b.n_events - 1 && threadIdx.x == 255) b.row_start[(int64_t)b.n_events * R] = (int)b.offsets[b.n_events];
}

// Each cluster's record, read here in input order (coalesced), to its arrival
// slot in its row.  The cluster also goes into its row's 128-bit phi-column
// occupancy mask; bit 127 marks a column held twice.
__global__ void k3_scatter(Batch3D b, Params3D P) {
  pdl_begin();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= b.n_points) return;
  const int e = event_of_blk(b, i);
  const int k = b.key[i];
  const int row = row_of(k, b.n_rows);
  const int64_t r = (int64_t)e * b.n_rows + row;
  const int pos = b.row_start[r] + b.arr[i];
  const int idx = (int)(i - b.offsets[e]);
  if (k < 0) {  // the last row's entries are never queried
    store_record(b.trec, pos, 0.f, 0.f, 0.f, 0.f, idx, 0.f, -1);
    return;
  }
  // the phi bin from the key (key = layer * 4284 + phiBin + 126 * etaBin,
  // phiBin up to 126)
  const int li = b.layer[i], eb = eta_bin(b.eta[i], P);
  const bool sil = b.sil[i];
  const float radius = b.radius[i];
  store_record(b.trec, pos, b.roa[i], b.phi[i], b.energy[i], b.z[i], idx, sil ? P.dens_thr : __fmul_rn(radius, radius),
               pack_bins(li, eb, k - li * kBins - eb * kPhiBins, sil));
  const int col = k % kPhiBins;
  unsigned long long* m = b.row_mask + 2 * r;
  const unsigned long long bit = 1ull << (col & 63);
  if (atomicOr(m + (col >> 6), bit) & bit) {
    atomicOr(m + 1, 1ull << 63);
    // a second entry in the column: the column's bit in the repeat mask; a
    // third: bit 127 of the repeat mask
    unsigned long long* rp = b.row_rep + 2 * r;
    if (atomicOr(rp + (col >> 6), bit) & bit) atomicOr(rp + 1, 1ull << 63);
  }
}

// Each entry's rank inside its row by (column, index) gives its final slot:
// a counting sort by column through the occupancy mask (the entries in lower
// columns are the mask's set bits below the entry's column) when no column
// repeats, a count over the row otherwise.  One thread per scattered entry;
// its record moves within the row's range.
__global__ void k3_row_sort(Batch3D b) {
  pdl_begin();
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= b.n_points) return;
  const float4 c = b.trec[2 * p], d = b.trec[2 * p + 1];
  const int bins = __float_as_int(d.w), idx = __float_as_int(d.y);
  if (bins < 0) return;
  const int e = event_of_blk(b, p);
  const int col = bins_col(bins);
  const int64_t r = (int64_t)e * b.n_rows + bins_key(bins) / kPhiBins;
  const int s = b.row_start[r];
  const ulonglong2 m = reinterpret_cast<const ulonglong2*>(b.row_mask)[r];
  int rank;
  if (!(m.y >> 63)) {
    rank = bits_below(m.x, m.y, col);
  } else {
    const int t = b.row_start[r + 1];
    rank = 0;
    for (int q = s; q < t; ++q) {
      const float4 o = b.trec[2 * (int64_t)q + 1];
      const int c2 = bins_col(__float_as_int(o.w)), i2 = __float_as_int(o.y);
      rank += (c2 < col) || (c2 == col && i2 < idx);
    }
  }
  store_record(b.rec, s + rank, c.x, c.y, c.z, d.x, idx, d.z, bins);
}

// The rows of one event as the searches see them: the whole event in global
// memory, or a staged copy of a range of rows in shared memory.  Positions
// are sorted positions (global, or relative to the first staged entry).
struct RowsGlobal {
  const unsigned long long* mask;  // 2 words per row of the event
  const int32_t* rstart;           // first sorted position of each row of the event
  const float4* recs;              // 2 per entry
  __device__ __forceinline__ unsigned long long m0(int r) const { return mask[2 * r]; }
  __device__ __forceinline__ unsigned long long m1(int r) const { return mask[2 * r + 1]; }
  __device__ __forceinline__ int start(int r) const { return rstart[r]; }
  __device__ __forceinline__ float4 rec(int q) const { return recs[2 * (int64_t)q]; }
  __device__ __forceinline__ int col(int q) const { return bins_col(__float_as_int(recs[2 * (int64_t)q + 1].w)); }
};

// A staged row: its 126 column-occupancy bits as four 32-bit words; its entries
// in the columns before each word, a byte per word (at most two entries per
// column there); and its start, relative to the first staged entry, with a slot
// of second-entry words where a column holds two (few rows do) and two flags.
// Rows with a third entry in a column, or beyond the slots, are searched by
// their entries' columns, staged as bytes for up to kSlabWalks rows of a slab
// and read from the records in global memory for others.  (The layer clusters of
// an HGCAL event: a good half lies below eta 1.5, in the first eta row, so that
// row holds some thirty entries and often three in a column; 1.24M such clusters
// of 200 events: columns counted from global memory 0.67 ms, from the bytes by a
// binary search 0.43.  Both ends of a window are searched for: with the entries
// counted on from its first one, 20,000 clusters on a line of phi, some hundred to
// a column, took 1.23 ms, 0.65 now.)
constexpr int kRowStartBits = 12, kRowSlotBits = 8;
constexpr int kRowRepeat = 1 << 30;  // a column holds two entries
constexpr int kRowWalk = 1 << 29;    // counted by its entries' columns
constexpr int kRowCols = 1 << 28;    // those staged; the slot field then counts words of them
struct RowsStaged {
  const uint32_t* mask;    // 4 words per staged row
  const uint32_t* rep;     // 4 words per slot
  const int32_t* rstart;
  const uint32_t* before;
  const float4* cand;
  const uint8_t* cols;     // columns of the rows with kRowCols
  const float4* recs;      // the first staged entry's record in global memory
  int row_lo;              // first staged row
  __device__ __forceinline__ unsigned long long m0(int r) const { return word64(r, 0); }
  __device__ __forceinline__ unsigned long long m1(int r) const {
    return word64(r, 2) | ((rstart[r - row_lo] & kRowRepeat) ? 1ull << 63 : 0ull);
  }
  __device__ __forceinline__ unsigned long long word64(int r, int w) const {
    const uint32_t* p = mask + 4 * (r - row_lo) + w;
    return ((unsigned long long)p[1] << 32) | p[0];
  }
  __device__ __forceinline__ int start(int r) const { return rstart[r - row_lo] & ((1 << kRowStartBits) - 1); }
  __device__ __forceinline__ float4 rec(int q) const { return cand[q]; }
  __device__ __forceinline__ int col(int q) const { return bins_col(__float_as_int(recs[2 * (int64_t)q + 1].w)); }
};

// First of the positions [s, t), which are in column order, whose column is at
// or above a.
template <class F>
__device__ __forceinline__ int first_at(int s, int t, int a, F&& col) {
  int len = t - s;
  while (len > 0) {
    const int h = len >> 1;
    const bool below = col(s + h) < a;
    s = below ? s + h + 1 : s;
    len = below ? len - h - 1 : h;
  }
  return s;
}

// Visits the entries of rows [s, t) whose phi column lies in the window
// [p0, p1] (p0 may be negative, p1 may exceed 125), in the reference's
// order: iphi_it = p0..p1 mapped modulo 126.
// The first column is found by a binary search: slabs beyond the staging area
// walk their rows in global memory (10 events of 100,000 clusters, 31 to a row:
// 8.9 ms counting from each row's start, 2.3 ms).
template <class V, class F>
__device__ __forceinline__ void visit_row(const V& v, int s, int t, int p0, int p1, F&& f) {
  const bool wraps = p0 < 0 || p1 >= kPhiBins;
  const int a0 = p0 < 0 ? p0 + kPhiBins : p0;  // first arc [a0, a1], then [0, c1] when the window wraps
  const int a1 = wraps ? kPhiBins - 1 : p1;
  for (int q = first_at(s, t, a0, [&](int k) { return v.col(k); }); q < t && v.col(q) <= a1; ++q) f(q);
  if (!wraps) return;
  const int c1 = p0 < 0 ? p1 : p1 - kPhiBins;
  for (int q = s; q < t && v.col(q) <= c1; ++q) f(q);
}

// Phi columns of the window [pb - d, pb + d] modulo 126 as a 126-bit mask
// (the reference's iphi = iphi_it mod nPhiBins, CLUE3DAlgoKernels.h:80-84).
struct ColMask {
  unsigned long long w0 = 0, w1 = 0;
  // columns [lo, lo + n), 0 <= n <= 5, lo + n <= 126
  __device__ __forceinline__ void run(int lo, int n) {
    const unsigned long long r = (1ull << n) - 1;
    if (lo >= 64) {
      w1 |= r << (lo - 64);
    } else {
      w0 |= r << lo;
      if (lo + n > 64) w1 |= r >> (64 - lo);
    }
  }
  __device__ __forceinline__ ColMask(int pb, int d) {  // 0 <= pb <= 126, d <= 2
    const int a = pb - d, c = pb + d;
    if (a < 0) {
      run(a + kPhiBins, -a);
      run(0, c + 1);
    } else if (c >= kPhiBins) {
      run(a, kPhiBins - a);
      run(0, c - kPhiBins + 1);
    } else {
      run(a, 2 * d + 1);
    }
  }
};

// visit_row() for row r through its occupancy mask: a row with no entry in
// the window's columns is skipped on the mask alone, the row start is read
// only when the window holds an entry, and the row is not scanned.
template <class V, class F>
__device__ __forceinline__ void visit_row_masked(const V& v, int r, const ColMask& wm, int p0, int p1, F&& f) {
  const unsigned long long m0 = v.m0(r), m1 = v.m1(r);
  // bit 127 of m1 marks a repeated column; the window never holds column 127
  if (((m0 & wm.w0) | (m1 & wm.w1)) == 0) return;
  if (m1 >> 63) {  // a column holds several entries: walk the row
    visit_row(v, v.start(r), v.start(r + 1), p0, p1, f);
    return;
  }
  int a0, c0, a1 = 0, c1 = -1;  // first run [a0, c0], then [a1, c1] (wrapping windows)
  if (p0 >= 0 && p1 < kPhiBins) {
    a0 = p0; c0 = p1;
  } else if (p0 < 0) {
    a0 = p0 + kPhiBins; c0 = kPhiBins - 1; a1 = 0; c1 = p1;
  } else {
    a0 = p0; c0 = kPhiBins - 1; a1 = 0; c1 = p1 - kPhiBins;
  }
  const int lo0 = bits_below(m0, m1, a0), n0 = bits_below(m0, m1, c0 + 1) - lo0;
  const int n1 = c1 >= a1 ? bits_below(m0, m1, c1 + 1) : 0;  // the second run starts at column 0
  if (n0 + n1 == 0) return;
  const int s = v.start(r);
  for (int q = s + lo0; q < s + lo0 + n0; ++q) f(q);
  for (int q = s; q < s + n1; ++q) f(q);
}

// A query's phi window of n = 2 d + 1 columns as visited: a0, a0 + 1, ...,
// modulo 126.  A row's occupancy of the window is a field of n bits in that
// order: the columns from a0 up to 125 (arc A), then, when the window wraps,
// those from 0 (arc B).
struct PhiField {
  int word, sh, wrap;    // a0 = 32 * word + sh; columns of arc A (n or more: no wrap)
  unsigned in_a, all;    // the field's bits of arc A; all its bits
  __device__ __forceinline__ PhiField(int pb, int d) {  // 0 <= pb <= 126, d <= 2
    const int p0 = pb - d, a0 = p0 < 0 ? p0 + kPhiBins : p0;
    word = a0 >> 5;
    sh = a0 & 31;
    wrap = kPhiBins - a0;
    all = (1u << (2 * d + 1)) - 1u;
    in_a = all & ((1u << min(wrap, 5)) - 1u);
  }
  // Arc A of a row's words (the word after a row's last one is read but holds
  // no column of arc A).
  __device__ __forceinline__ unsigned arc_a(const uint32_t* w) const {
    return __funnelshift_r(w[word], w[word + 1], sh) & in_a;
  }
  __device__ __forceinline__ unsigned arc_b(const uint32_t* w) const { return (w[0] << wrap) & all & ~in_a; }
  __device__ __forceinline__ bool wraps() const { return in_a != all; }
};

// Rows of a query's window that hold an entry in its phi columns, as bits
// (cl - lo) * 8 + (ie - e0) of a 64-bit word: ascending bit order is the
// reference's visiting order (layers outer, eta rows inner).  Reading every
// row's mask in one uniform pass and then visiting only the rows whose bit is
// set keeps the lanes of a warp together: otherwise each of the ~25 rows would
// send the few lanes with an entry down the visit while the others wait.
// Windows of more than 8 layers or 5 eta rows return false (the caller loops
// directly).
__device__ __forceinline__ bool live_rows(const RowsStaged& v, int lo, int hi, int skip, int e0, int e1,
                                          const PhiField& f, unsigned long long* live) {
  if (hi - lo >= 8 || e1 - e0 >= 5) return false;
  unsigned long long m = 0;
  const int ne = e1 - e0;
  for (int cl = lo; cl <= hi; ++cl) {
    if (cl == skip) continue;
    const uint32_t* w = v.mask + 4 * (cl * kEtaBins + e0 - v.row_lo);
    unsigned bits = 0;
#pragma unroll
    for (int de = 0; de < 5; ++de) {
      if (de <= ne) {
        unsigned x = f.arc_a(w + 4 * de);
        if (f.wraps()) x |= f.arc_b(w + 4 * de);
        bits |= (x != 0 ? 1u : 0u) << de;
      }
    }
    m |= (unsigned long long)bits << ((cl - lo) * 8);
  }
  *live = m;
  return true;
}

// What a search needs of its query cluster.
struct Query3 {
  float phi, z, r0, aux;  // aux: density threshold (density), rho (nearest higher)
  int li, eb, pb, self;   // self: the cluster's own position in the view
  float energy;
  bool sil;
};

// One density term (KernelCalculateDensitySoA, :26-150): candidate q of a
// row of layer cl, in the reference's operation order.
template <class V>
__device__ __forceinline__ void density_term(const V& v, const Params3D& P, const Query3& Q, float coef, int q,
                                             float& rho) {
  const float4 cj = v.rec(q);  // {roa, phi, energy, -}; q == self is the cluster itself
  const float r1 = __fmul_rn(cj.x, Q.z);
  const float dphi = reduce_range(__fsub_rn(Q.phi, cj.y), P);
  const float d0 = __fsub_rn(Q.r0, r1);
  const float a = __fmul_rn(d0, d0);
  const float c = __fmul_rn(__fmul_rn(__fmul_rn(r1, r1), dphi), dphi);
  if (__fadd_rn(a, c) < Q.aux) rho = __fadd_rn(rho, __fmul_rn((q == Q.self) ? 1.f : coef, cj.z));
}

__device__ __forceinline__ float density_coef(const Params3D& P, const Query3& Q, int cl) {
  return __fmul_rn(P.kdf, (cl == Q.li && !P.dens_same) ? 0.f : 1.f);
}

// Density terms of one row of a query's window: the clusters of the row in
// the window's phi columns, in order.
template <class V>
__device__ __forceinline__ void density_row(const V& v, const Params3D& P, const Query3& Q, const ColMask& wm, int cl,
                                            int ie, float& rho) {
  const float coef = density_coef(P, Q, cl);
  visit_row_masked(v, cl * kEtaBins + ie, wm, Q.pb - 2, Q.pb + 2,
                   [&](int q) { density_term(v, P, Q, coef, q, rho); });
}

// One cluster's nearest higher (KernelComputeDistanceToHigherSoA, :286-392)
// over the rows in `v`: best squared distance (FLT_MAX: none), its sqrt, the
// layer distance, the layer and the position in `v`.
struct Nh3 {
  float best = FLT_MAX, best_t = FLT_MAX;
  int best_l = INT_MAX, nl = -1, nq = -1;
};

template <class V>
__device__ __forceinline__ void nh_term(const V& v, const Params3D& P, const Query3& Q, int cl, int q, Nh3& o) {
  const float4 cj = v.rec(q);  // {roa, phi, energy, rho}
  const float r1 = __fmul_rn(cj.x, Q.z);
  const float dphi = reduce_range(__fsub_rn(Q.phi, cj.y), P);
  const float d0 = __fsub_rn(Q.r0, r1);
  const float d = __fadd_rn(__fmul_rn(d0, d0), __fmul_rn(__fmul_rn(__fmul_rn(r1, r1), dphi), dphi));
  if (cj.w > Q.aux && d <= o.best) {  // "<=": the last candidate wins a tie
    o.best = d;
    o.best_t = __fsqrt_rn(d);
    o.best_l = abs(cl - Q.li);
    o.nl = cl;
    o.nq = q;
  }
}

template <class V>
__device__ __forceinline__ void nh_row(const V& v, const Params3D& P, const Query3& Q, const ColMask& wm, int cl, int ie,
                                       Nh3& o) {
  visit_row_masked(v, cl * kEtaBins + ie, wm, Q.pb - 1, Q.pb + 1, [&](int q) { nh_term(v, P, Q, cl, q, o); });
}

// A live row's entries in the window, in the reference's order: the run of
// arc A, [qa, qa + na), then the run of arc B, [s, s + nb) (the row's start).
// The counts come from popcounts of the row's words, where a column holds two
// entries also of its second-entry words; only a row with three or more entries
// in one column is counted entry by entry (rows are short).  Popcounts issue
// at a quarter of the rate of other instructions: three per row here, against
// 24 with 128-bit masks of the window and of the columns below it (1,000
// events: density search 1.07 -> 0.87 ms, nearest higher 0.72 -> 0.64 ms).
struct RowRuns {
  int qa, na, s, nb;
};

__device__ __forceinline__ RowRuns row_runs(const RowsStaged& v, int r, const PhiField& f) {
  const int i = r - v.row_lo;
  const uint32_t* w = v.mask + 4 * i;
  const int rs = v.rstart[i];
  const unsigned below = (1u << f.sh) - 1u;
  RowRuns o;
  o.s = rs & ((1 << kRowStartBits) - 1);
  o.na = __popc(f.arc_a(w));
  o.nb = f.wraps() ? __popc(f.arc_b(w)) : 0;
  o.qa = o.s + (int)((v.before[i] >> (8 * f.word)) & 0xffu) + __popc(w[f.word] & below);
  if (rs & kRowRepeat) {
    if (rs & kRowWalk) {
      const int t = v.start(r + 1);
      const int a0 = 32 * f.word + f.sh, a1 = a0 + (f.all == 31u ? 5 : (f.all == 7u ? 3 : 1));
      const uint8_t* cs = v.cols + 4 * ((rs >> kRowStartBits) & ((1 << kRowSlotBits) - 1)) - o.s;
      auto col = [&](int q) { return (rs & kRowCols) ? (int)cs[q] : v.col(q); };
      o.qa = first_at(o.s, t, a0, col);
      o.na = first_at(o.qa, t, a1, col) - o.qa;
      o.nb = f.wraps() ? first_at(o.s, o.qa, a1 - kPhiBins, col) - o.s : 0;
    } else {
      const uint32_t* p = v.rep + 4 * ((rs >> kRowStartBits) & ((1 << kRowSlotBits) - 1));
      o.na += __popc(f.arc_a(p));
      o.nb += f.wraps() ? __popc(f.arc_b(p)) : 0;
      o.qa += __popc(p[f.word] & below);
    }
  }
  return o;
}

// The window of a query: layers [lo, hi] (without `skip`), eta rows
// [e0, e1], phi columns pb +- d.
struct Window3 {
  int lo, hi, e0, e1, skip;
};

__device__ __forceinline__ Window3 window_of(const Params3D& P, const Query3& Q, bool density) {
  Window3 w;
  const int de = density ? 2 : 1;
  layer_window(Q.li, density ? P.dens_sib : P.nh_sib, P.n_layers, density ? 0 : 1, &w.lo, &w.hi);
  w.e0 = max(Q.eb - de, 0);
  w.e1 = min(Q.eb + de, kEtaBins);
  w.skip = (density || P.nh_same) ? -1 : Q.li;
  return w;
}

// A whole search over the rows of `v`, every window row in order (the rows
// whose mask shows no entry return at once).
template <bool kDensity, class V, class R>
__device__ __forceinline__ void search_all(const V& v, const Params3D& P, const Query3& Q, R& res) {
  const Window3 w = window_of(P, Q, kDensity);
  const ColMask wm(Q.pb, kDensity ? 2 : 1);
  for (int cl = w.lo; cl <= w.hi; ++cl) {
    if (cl == w.skip) continue;
    for (int ie = w.e0; ie <= w.e1; ++ie) {
      if constexpr (kDensity) density_row(v, P, Q, wm, cl, ie, res);
      else nh_row(v, P, Q, wm, cl, ie, res);
    }
  }
}

// The same search over the rows named by a live_rows() mask.
template <bool kDensity, class R>
__device__ __forceinline__ void search_live(const RowsStaged& v, const Params3D& P, const Query3& Q,
                                            unsigned long long live, R& res) {
  const Window3 w = window_of(P, Q, kDensity);
  const PhiField f(Q.pb, kDensity ? 2 : 1);
  // One candidate per iteration: the lanes of a warp step through their own
  // candidate sequences together, and a lane moves to its next run (arc B of
  // the row, or the next live row) only when its current run is done.
  int q = 0, qe = 0, qb = 0, qbe = 0, cl = 0;
  float coef = 0.f;
  bool more = true;
  for (;;) {
    while (q >= qe) {
      if (qb < qbe) {
        q = qb;
        qe = qbe;
        qb = qbe = 0;
      } else if (live) {
        const int k = __ffsll((long long)live) - 1;
        live &= live - 1;
        cl = w.lo + (k >> 3);
        if constexpr (kDensity) coef = density_coef(P, Q, cl);
        const RowRuns rr = row_runs(v, cl * kEtaBins + w.e0 + (k & 7), f);
        q = rr.qa;
        qe = rr.qa + rr.na;
        qb = rr.s;
        qbe = rr.s + rr.nb;
      } else {
        more = false;
        break;
      }
    }
    if (!more) break;
    if constexpr (kDensity) density_term(v, P, Q, coef, q, res);
    else nh_term(v, P, Q, cl, q, res);
    ++q;
  }
}

// Staging of the searches: one block per (event, slab of kSlabLayers
// layers).  The block copies the rows of the slab's layers and of the
// sibling layers around them (occupancy words, row starts and the 16-byte
// candidate halves of the records) into shared memory once, then runs the
// searches of the slab's clusters from there (5 blocks of 256 threads per SM,
// since the searches wait on latency: 4 blocks, with second-entry words for every
// row and the columns staged as well, 0.86 + 0.64 ms against 0.80 + 0.60;
// slabs of 2, 6 and 8 layers measured slower or the same).  A cluster whose window leaves
// the staged rows (the phi bin 126 quirk can move a cluster into the next
// layer's first row) and a slab larger than the staging area read the global
// arrays instead; either way the visiting order and arithmetic are the
// reference's.
constexpr int kSlabLayers = 4;
constexpr int kSlabThreads = 256;
constexpr int kSlabMaxRows = 384;  // 10 layers of rows and one more: sibling windows up to +-3 layers
constexpr int kSlabMaxCand = 2048;
constexpr int kSlabSlots = 128;
constexpr int kSlabWalks = 32;       // rows whose columns are staged
constexpr int kSlabColWords = 256;   // room for those, four entries each
static_assert(kSlabColWords <= 1 << kRowSlotBits, "packed row starts");
static_assert(kSlabMaxCand < 1 << kRowStartBits && kSlabSlots <= 1 << kRowSlotBits, "packed row starts");
// candidate records, row words, second-entry words, row starts and counts
constexpr size_t kSlabSmem = 16 * (size_t)kSlabMaxCand + 16 * (size_t)kSlabMaxRows + 16 * (size_t)kSlabSlots +
                             8 * (size_t)(kSlabMaxRows + 1) + 4 * (size_t)kSlabColWords;

// How a launch takes its slabs: each in one part, or in halves or single layers
// where its staging does not fit, or all from global memory (see launch_clue3d).
enum SlabMode { kWhole, kInParts, kGlobal };

template <bool kDensity, SlabMode kMode>
__global__ void __launch_bounds__(kSlabThreads, 5) k3_search(Batch3D b, Params3D P, int n_slabs) {
  constexpr bool kParts = kMode == kInParts;
  extern __shared__ __align__(16) unsigned char sm3[];
  float4* s_cand = reinterpret_cast<float4*>(sm3);
  uint32_t* s_mask = reinterpret_cast<uint32_t*>(s_cand + kSlabMaxCand);
  uint32_t* s_rep = s_mask + 4 * kSlabMaxRows;
  int32_t* s_rs = reinterpret_cast<int32_t*>(s_rep + 4 * kSlabSlots);
  uint32_t* s_before = reinterpret_cast<uint32_t*>(s_rs + kSlabMaxRows + 1);
  uint8_t* s_col = reinterpret_cast<uint8_t*>(s_before + kSlabMaxRows + 1);
  __shared__ int s_slots, s_walks, s_words;  // taken so far
  __shared__ int s_walk[kSlabWalks];         // the rows with staged columns
  if (threadIdx.x == 0) s_slots = s_walks = s_words = 0;
  pdl_begin();
  const int e = blockIdx.x / n_slabs;
  const int L0 = (blockIdx.x % n_slabs) * kSlabLayers;
  const int L1 = min(L0 + kSlabLayers, P.n_layers);
  const int sib = kDensity ? P.dens_sib : P.nh_sib;
  const int R = b.n_rows;
  const int64_t rbase = (int64_t)e * R;
  const int32_t* rs = b.row_start + rbase;
  // the last layer's clusters end with the row behind it, which holds those of
  // phi bin 126 in its last eta row
  auto layers_end = [&](int l) { return rs[l * kEtaBins + (l == P.n_layers ? 1 : 0)]; };
  if (rs[L0 * kEtaBins] >= layers_end(L1)) return;
  for (int La = L0, Lb; La < L1; La = kParts ? Lb : L1) {
    // rows of layers [La - sib, Lb + sib) and the first row after them (the
    // reference's eta window reaches row 34 of a layer, the next layer's row 0)
    int row_lo, row_hi, nrows, pos_lo, pos_hi;  // row_hi inclusive, <= R - 2
    bool staged;
    for (Lb = L1;;) {
      row_lo = max(La - max(sib, 0), 0) * kEtaBins;
      row_hi = min(Lb + max(sib, 0), P.n_layers) * kEtaBins;
      nrows = row_hi - row_lo + 1;
      pos_lo = rs[row_lo];
      pos_hi = rs[row_hi + 1];
      staged = kMode != kGlobal && nrows <= kSlabMaxRows && pos_hi - pos_lo <= kSlabMaxCand;
      if (staged || !kParts) break;
      if (Lb - La == 1) {  // not even one layer's: from global memory, together
        Lb = L1;
        break;
      }
      Lb = La + (Lb - La + 1) / 2;
    }
    const int q_lo = rs[La * kEtaBins], q_hi = layers_end(Lb);
    if (kParts && La > L0) {
      __syncthreads();  // the searches of the part before
      if (threadIdx.x == 0) s_slots = s_walks = s_words = 0;
    }
    if (staged) {
      __syncthreads();  // s_slots
      const uint4* gm = reinterpret_cast<const uint4*>(b.row_mask + 2 * (rbase + row_lo));
      const uint4* gr = reinterpret_cast<const uint4*>(b.row_rep + 2 * (rbase + row_lo));
      for (int i = threadIdx.x; i <= nrows; i += kSlabThreads) {
        int st = rs[row_lo + i] - pos_lo;
        if (i < nrows) {
          uint4 m = gm[i], p = make_uint4(0u, 0u, 0u, 0u);
          if (m.w >> 31) {  // bit 127 of the row's masks: a column repeats / holds a third entry
            p = gr[i];
            const int slot = p.w >> 31 ? kSlabSlots : atomicAdd(&s_slots, 1);
            p.w &= 0x3fffffffu;
            if (slot < kSlabSlots) {
              st |= kRowRepeat | (slot << kRowStartBits);
              reinterpret_cast<uint4*>(s_rep)[slot] = p;
            } else {
              const int words = (rs[row_lo + i + 1] - rs[row_lo + i] + 3) >> 2;
              const int at = atomicAdd(&s_words, words), k = at + words <= kSlabColWords ? atomicAdd(&s_walks, 1) : kSlabWalks;
              if (k < kSlabWalks) s_walk[k] = i;
              st |= kRowRepeat | kRowWalk | (k < kSlabWalks ? kRowCols | (at << kRowStartBits) : 0);
            }
          }
          m.w &= 0x3fffffffu;
          reinterpret_cast<uint4*>(s_mask)[i] = m;
          const unsigned c0 = __popc(m.x) + __popc(p.x), c1 = c0 + __popc(m.y) + __popc(p.y),
                         c2 = c1 + __popc(m.z) + __popc(p.z);
          s_before[i] = (c0 << 8) | (c1 << 16) | (c2 << 24);
        }
        s_rs[i] = st;
      }
      for (int i = threadIdx.x; i < pos_hi - pos_lo; i += kSlabThreads) {
        s_cand[i] = b.rec[2 * (int64_t)(pos_lo + i)];
      }
      __syncthreads();
      if (s_walks > 0) {
        constexpr int kStart = (1 << kRowStartBits) - 1;
        for (int k = threadIdx.x >> 5; k < min(s_walks, kSlabWalks); k += kSlabThreads / 32) {
          const int st = s_rs[s_walk[k]], a = st & kStart, z = s_rs[s_walk[k] + 1] & kStart;
          uint8_t* c = s_col + 4 * ((st >> kRowStartBits) & ((1 << kRowSlotBits) - 1)) - a;
          for (int q = a + (threadIdx.x & 31); q < z; q += 32)
            c[q] = (uint8_t)bins_col(__float_as_int(b.rec[2 * (int64_t)(pos_lo + q) + 1].w));
        }
        __syncthreads();
      }
    }
    RowsStaged sv{s_mask, s_rep, s_rs, s_before, s_cand, s_col, b.rec + 2 * (int64_t)pos_lo, row_lo};
    RowsGlobal gv{b.row_mask + 2 * rbase, rs, b.rec};
    const int64_t es = b.offsets[e];
    const int tid = threadIdx.x;
    // the query rows hold only accepted clusters (rejected ones are in the
    // event's last row); a query's own data is read in sorted order
    auto query = [&](int p, bool* inside, int* idx) {
      const float4 qr = b.rec[2 * (int64_t)p + 1];
      const float4 cr = staged ? s_cand[p - pos_lo] : b.rec[2 * (int64_t)p];
      *idx = __float_as_int(qr.y);
      const int bins = __float_as_int(qr.w);
      Query3 Q;
      Q.li = bins & 0x7ff;
      Q.eb = (bins >> 11) & 0x3f;
      Q.pb = (bins >> 17) & 0x7f;
      Q.sil = (bins >> 24) & 1;
      Q.energy = cr.z;
      Q.phi = cr.y;
      Q.z = qr.x;
      Q.r0 = __fmul_rn(cr.x, qr.x);
      Q.aux = kDensity ? qr.z : cr.w;
      int lo, hi;
      layer_window(Q.li, sib, P.n_layers, kDensity ? 0 : 1, &lo, &hi);
      *inside = staged && lo * kEtaBins >= row_lo && hi * kEtaBins + kEtaBins <= row_hi;
      Q.self = *inside ? p - pos_lo : p;
      return Q;
    };
    for (int p = q_lo + tid; p < q_hi; p += kSlabThreads) {
      bool inside;
      int idx;
      const Query3 Q = query(p, &inside, &idx);
      const int64_t gi = es + idx;
      // staged windows: the rows holding an entry first, in one uniform pass
      unsigned long long live = 0;
      bool by_live = false;
      if (inside) {
        const Window3 w = window_of(P, Q, kDensity);
        by_live = live_rows(sv, w.lo, w.hi, w.skip, w.e0, w.e1, PhiField(Q.pb, kDensity ? 2 : 1), &live);
      }
      if constexpr (kDensity) {
        float rho = 0.f;
        if (by_live) search_live<true>(sv, P, Q, live, rho);
        else if (inside) search_all<true>(sv, P, Q, rho);
        else search_all<true>(gv, P, Q, rho);
        b.rho[gi] = rho;
        reinterpret_cast<float*>(b.rec)[8 * (int64_t)p + 3] = rho;
      } else {
        Nh3 o;
        if (by_live) search_live<false>(sv, P, Q, live, o);
        else if (inside) search_all<false>(sv, P, Q, o);
        else search_all<false>(gv, P, Q, o);
        if (o.nq >= 0 && inside) o.nq += pos_lo;
        const bool found = o.best != FLT_MAX;
        const float dt = found ? o.best_t : FLT_MAX;
        const int dl = found ? o.best_l : INT_MAX, nl = found ? o.nl : -1;
        const int ni = found ? __float_as_int(b.rec[2 * (int64_t)o.nq + 1].y) : -1;
        b.delta_t[gi] = dt;
        b.delta_l[gi] = dl;
        b.nh_l[gi] = nl;
        b.nh_i[gi] = ni;
        // seeds and outliers (CLUE3DAlgoKernels.h:521-560); par: the nearest
        // higher for followers, -2 for seeds, -3 for other roots
        const float r = Q.aux;
        const float dxy = Q.sil ? P.crit_xy : b.radius[gi];
        const bool seed = (dt > dxy || __int2float_rn(dl) > P.crit_z) && (r >= P.crit_rho) &&
                          (__fdiv_rn(Q.energy, r) > P.crit_self);
        const bool outlier = (dt > P.out_thr) && (r < P.crit_rho);
        b.seed[gi] = seed ? 1 : 0;
        b.par[gi] = seed ? -2 : ((!outlier && nl >= 0) ? ni : -3);
      }
    }
  }
}


// One block per event: trackster ids by seed rank in index order, eight
// clusters per thread and scan round; clusters without a place in the rows
// become roots of their own.
constexpr int kRankThreads = 512;
constexpr int kRankPer = 8;

__global__ void __launch_bounds__(kRankThreads) k3_rank(Batch3D b) {
  pdl_begin();
  const int e = blockIdx.x;
  const int64_t es = b.offsets[e];
  const int n = (int)(b.offsets[e + 1] - es);
  int32_t* ti = b.ti + es;
  int32_t* seed = b.seed + es;
  __shared__ int s_w[kRankThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int base_rank = 0;
  for (int base = 0; base < n; base += kRankThreads * kRankPer) {
    const int i0 = base + threadIdx.x * kRankPer;
    int f[kRankPer], sum = 0;
#pragma unroll
    for (int j = 0; j < kRankPer; ++j) f[j] = i0 + j < n ? seed[i0 + j] : 0;
#pragma unroll
    for (int j = 0; j < kRankPer; ++j) {
      if (f[j] < 0) {
        f[j] = 0;
        seed[i0 + j] = 0;
        b.par[es + i0 + j] = -3;
      }
      sum += f[j];
    }
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += t;
    }
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kRankThreads / 32; ++w) {
      if (w < warp) before += s_w[w];
      total += s_w[w];
    }
    int rank = base_rank + before + x - sum;
#pragma unroll
    for (int j = 0; j < kRankPer; ++j)
      if (f[j]) ti[i0 + j] = rank++;
    base_rank += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    b.ev_seeds[e] = base_rank;
    if (b.host_nt) b.host_nt[e] = base_rank;
  }
}

// Each cluster's walk along nearestHigher to its root, and its label (replaces
// the LIFO propagation); par holds event-local indices.  Every 64 steps a walk
// leaves its own pointer at the farthest cluster reached, so that walks that
// come through it later skip those steps (every ancestor is a valid parent).
// The walks of a batch run side by side in as many blocks as it has clusters
// for: rounds of pointer jumping by one block per event took 20 us on one
// event of 5,000 clusters and 0.153 ms on 1,000 events; ranks and walks as two
// kernels 8 + 9 us and 0.055 + 0.085 ms.
__global__ void k3_label(Batch3D b) {
  pdl_wait();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < kFlagCount && b.host_flags) b.host_flags[i] = b.flags[i];
  if (i >= b.n_points) return;
  int t;
  int p = b.par[i];
  if (p == -2) {
    t = b.ti[i];  // a seed
  } else {
    int32_t* par = b.par + b.offsets[event_of_blk(b, i)];
    int32_t* ti = b.ti + (par - b.par);
    int r = -1;
    for (int step = 1; p >= 0; ++step) {
      r = p;
      if ((step & 63) == 0) b.par[i] = r;
      p = par[r];
    }
    t = p == -2 ? ti[r] : -1;
    b.ti[i] = t;
  }
  if (b.host_out) {  // a small host run's outputs, array after array
    float* o = b.host_out + i;
    const int64_t N = b.n_points;
    o[0] = b.rho[i];
    o[N] = b.delta_t[i];
    o[2 * N] = __int_as_float(b.delta_l[i]);
    o[3 * N] = __int_as_float(b.nh_l[i]);
    o[4 * N] = __int_as_float(b.nh_i[i]);
    o[5 * N] = __int_as_float(b.seed[i]);
    o[6 * N] = __int_as_float(t);
  }
}

}  // namespace

cudaError_t prepare_clue3d_kernels() {
  // also loads the kernels' code, so that no launch has any to load (the staging
  // itself, 44 KB, is within what a kernel may use without asking)
  for (auto* k : {k3_search<true, kWhole>, k3_search<true, kInParts>, k3_search<true, kGlobal>, k3_search<false, kWhole>,
                  k3_search<false, kInParts>, k3_search<false, kGlobal>}) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSlabSmem);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_clue3d(const Batch3D& b, const Params3D& p, cudaStream_t s) {
  if (b.n_events <= 0 || b.n_points <= 0) return cudaSuccess;
  cudaError_t err;
  const int T = 256;
  const int grid = (int)((b.n_points + T - 1) / T);
  {
    NvtxRange r("clue3d/init");
    const int64_t work = std::max({(int64_t)b.n_events * b.n_rows, b.n_table_words, b.n_in16});
    k3_init<<<(unsigned)std::min<int64_t>((work + T - 1) / T, 8192), T, 0, s>>>(b);
    if ((err = cudaGetLastError()) != cudaSuccess) return err;
  }
  {
    NvtxRange r("clue3d/key");
    if ((err = launch_pdl(k3_key, grid, T, 0, s, b, p)) != cudaSuccess) return err;
  }
  {
    NvtxRange r("clue3d/row_scan");
    if ((err = launch_pdl(k3_row_scan, b.n_events, 256, 0, s, b)) != cudaSuccess) return err;
  }
  {
    NvtxRange r("clue3d/scatter");
    if ((err = launch_pdl(k3_scatter, grid, T, 0, s, b, p)) != cudaSuccess) return err;
  }
  {
    NvtxRange r("clue3d/row_sort");
    if ((err = launch_pdl(k3_row_sort, grid, T, 0, s, b)) != cudaSuccess) return err;
  }
  const int n_slabs = (p.n_layers + kSlabLayers - 1) / kSlabLayers;
  const int64_t slab_blocks = (int64_t)b.n_events * n_slabs;
  if (slab_blocks > INT32_MAX) return cudaErrorInvalidValue;
  // Slabs may have to be searched in parts where the batch's largest event, its
  // clusters spread evenly over the layers, would fill seven eighths of the
  // staging area (1,792 candidates to a slab: six standard deviations below its
  // 2,048; 100 events of 20,000 clusters with three sibling layers, 2,130
  // candidates to a slab: 1.42 ms from global memory, 0.59 in two parts).
  // Other batches keep the form without the loop (1,000 events of up to 20,000 with
  // two: 2.07 ms, 2.10 with it); a slab that is crowded all the same then reads
  // global memory.  Where the rows of a slab exceed the area (four sibling layers
  // and more) none is staged, and the memory is left to the L1 cache (50
  // events of 10,000 with six: 0.577 ms beside an unused area, 0.466; with four:
  // 0.366 in halves, 0.351, and with half the clusters in one eta row 0.454 and
  // 0.356; with five, which takes single layers, 0.650 and 0.408).
  auto mode = [&](int sib) {
    const int64_t window = kSlabLayers + 2 * (int64_t)std::clamp(sib, 0, p.n_layers);
    if (std::min<int64_t>(window, p.n_layers) * kEtaBins + 1 > kSlabMaxRows) return kGlobal;
    return b.max_event * window > (int64_t)p.n_layers * (kSlabMaxCand / 8 * 7) ? kInParts : kWhole;
  };
  // More slabs than SMs, all resident at once (five to an SM): such a search
  // takes as long as its fullest SM.  As a dependent launch its blocks fill the SMs
  // that the kernel before leaves first; launched when that one has ended they
  // spread evenly (123 events of 4,671 clusters on 20 layers, 615 slabs, 0.947 -> 0.851
  // ms; 480 slabs of spread clusters 101 -> 92 us).  Larger launches keep the 3 us
  // that a dependent launch saves (1,200 slabs 169 against 175 us).
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const bool even = slab_blocks > sms && slab_blocks <= 5 * (int64_t)sms;
  auto search = [&](auto* whole, auto* parts, auto* global, int sib) {
    const SlabMode m = mode(sib);
    auto* k = m == kWhole ? whole : m == kInParts ? parts : global;
    const size_t smem = m == kGlobal ? 0 : kSlabSmem;
    if (even) {
      k<<<(unsigned)slab_blocks, kSlabThreads, smem, s>>>(b, p, n_slabs);
      return cudaGetLastError();
    }
    return launch_pdl(k, (unsigned)slab_blocks, kSlabThreads, smem, s, b, p, n_slabs);
  };
  {
    NvtxRange r("clue3d/density");
    err = search(k3_search<true, kWhole>, k3_search<true, kInParts>, k3_search<true, kGlobal>, p.dens_sib);
    if (err != cudaSuccess) return err;
  }
  {
    NvtxRange r("clue3d/nearest_higher");
    err = search(k3_search<false, kWhole>, k3_search<false, kInParts>, k3_search<false, kGlobal>, p.nh_sib);
    if (err != cudaSuccess) return err;
  }
  {
    NvtxRange r("clue3d/finish");
    if ((err = launch_pdl(k3_rank, b.n_events, kRankThreads, 0, s, b)) != cudaSuccess) return err;
    if ((err = launch_pdl(k3_label, grid, T, 0, s, b)) != cudaSuccess) return err;
  }
  return cudaSuccess;
}

}  // namespace clue
