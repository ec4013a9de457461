// 2D -> 3D bridge: the layer clusters of a clustered 2D batch, built on the
// device as CLUE3D input (a ClusterCollection per event,
// src/serial/DataFormats/ClusterCollection.h:6-19).  The reference has no such
// step (its CLUE3D reads raw3D files, src/serial/bin/Source.cc:43-60), so the
// definition is this file's:
//
//   * layer cluster c of event e = the 2D points with clusterIndex == c; the
//     clusters of an event keep the 2D ids' order (seed rank in index order);
//   * energy = sum of the weights, position = weight-weighted mean of x, y.
//     The sums are exact fixed-point integers (weights in units of 2^-24,
//     weight * coordinate in units of 2^-16, both rounded to nearest), so
//     they do not depend on the order of accumulation and the GPU result is
//     deterministic; the division and conversions are IEEE double;
//   * layer = the seed's layer, z = layer_z[layer], r = |(x, y)|,
//     r_over_absz = r / |z|, eta = asinh(z / max(r, 1e-9)), phi = atan2(y, x),
//     radius and isSilicon constant.  Clusters with zero total weight take the
//     seed's position.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "clue_runtime.h"

namespace clue {
namespace {

constexpr double kWScale = 16777216.0;  // 2^24
constexpr double kPScale = 65536.0;     // 2^16

enum BridgeSlot {
  B_TABLES,  // event offsets | cluster offsets | layer z | event of each chunk, as in the pinned staging
  B_COUNT,
  B_SUMS,    // sums | seed of each cluster | status words: zero at the start of a build
  B_SLOTS
};

// Points per block of the point kernels: each block finds the event of its
// first point once and then follows event boundaries forwards.
constexpr int kBridgeChunk = 4096;
constexpr int kBridgeThreads = 256;

int chunks_for(int64_t n) { return (int)((n + kBridgeChunk - 1) / kBridgeChunk); }

// The double formula, for values outside the fixed-point forms' ranges.  Not
// inlined: the compiler otherwise computes it for every point beside the
// other form, and the FP64 pipe bounds the kernel.
__device__ __noinline__ unsigned long long fx_double(float w, float v, double scale) {
  return (unsigned long long)__double2ll_rn((double)w * (double)v * scale);
}

// Fixed-point weight, round(w * 2^24) to nearest even: the scaled float is
// exact, so one conversion rounds as the double formula does.  NaN, infinities
// and weights of 64 and more take the double formula.
__device__ __forceinline__ unsigned long long fx_weight(float w) {
  const float v = __fmul_rn(w, (float)kWScale);
  if (fabsf(v) < 1073741824.f) return (unsigned long long)(long long)__float2int_rn(v);
  return fx_double(w, 1.f, kWScale);
}

// Fixed-point weighted coordinate, round(w * v * 2^16) to nearest even, as
// the double formula gives it (the double product of two floats is exact),
// without FP64, which is slow on this GPU: the product as a float p and its
// exact rest e (one fused multiply-add), both scaled.  p rounds to an integer
// r; e is at most half a unit of p, so it counts only where p has no fraction
// (then its own rounding is added) or where p is half way between two
// integers (then its sign decides; without a rest the tie went to even).
// Infinities, NaN and products of 2^14 and more take the double formula.
// The 64-bit shifts of the same arithmetic on integer significands took three
// times the instructions (with FP64 kept out of line, k_bridge_accumulate
// on 200 HGCAL events: 0.635 -> 0.283 ms).
__device__ __forceinline__ unsigned long long fx_pos(float w, float v) {
  const float p = __fmul_rn(w, v);
  const float ps = __fmul_rn(p, (float)kPScale);
  if (!(fabsf(ps) < 1073741824.f)) return fx_double(w, v, kPScale);
  const float es = __fmul_rn(__fmaf_rn(w, v, -p), (float)kPScale);
  int r = __float2int_rn(ps);
  const float d = __fsub_rn(ps, __int2float_rn(r));
  if (fabsf(d) == 0.5f) r += (d > 0.f ? (es > 0.f ? 1 : 0) : (es < 0.f ? -1 : 0));
  r += __float_as_int(__fadd_rn(es, 12582912.f)) - 0x4B400000;  // es to the nearest even integer
  return (unsigned long long)(long long)r;
}

// Points of a thread per round (loads of a round are issued together).
constexpr int kBridgePer = 8;
constexpr int kBridgeRounds = kBridgeChunk / (kBridgeThreads * kBridgePer);
static_assert(kBridgeRounds * kBridgeThreads * kBridgePer == kBridgeChunk, "chunk layout");

// Seeds per event: each block counts its chunk's seeds per event in shared
// memory (a chunk touches few events) and adds each count once; seeds of
// events beyond the first kBlockEvents of the chunk go to global memory.
constexpr int kBlockEvents = 32;

__global__ void __launch_bounds__(kBridgeThreads) k_bridge_count(int64_t N, const int64_t* __restrict__ off,
                                                                   const int32_t* __restrict__ chunk_ev,
                                                                   const int32_t* __restrict__ seed,
                                                                   int32_t* __restrict__ counts) {
  __shared__ int32_t s_cnt[kBlockEvents];
  if (threadIdx.x < kBlockEvents) s_cnt[threadIdx.x] = 0;
  const int64_t c0 = (int64_t)blockIdx.x * kBridgeChunk;
  const int32_t e0 = chunk_ev[blockIdx.x];
  int32_t e = e0;
  int64_t next = off[e + 1];  // first point after event e
  __syncthreads();
  for (int rd = 0; rd < kBridgeRounds; ++rd) {
    const int64_t i0 = c0 + (int64_t)rd * kBridgeThreads * kBridgePer + threadIdx.x;
    int32_t sv[kBridgePer];
#pragma unroll
    for (int j = 0; j < kBridgePer; ++j) {
      const int64_t i = i0 + (int64_t)j * kBridgeThreads;
      sv[j] = i < N ? seed[i] : 0;
    }
#pragma unroll
    for (int j = 0; j < kBridgePer; ++j) {
      const int64_t i = i0 + (int64_t)j * kBridgeThreads;
      if (i < N && sv[j]) {
        while (next <= i) next = off[++e + 1];  // i grows with (rd, j)
        if (e - e0 < kBlockEvents) atomicAdd(&s_cnt[e - e0], 1);
        else atomicAdd(&counts[e], 1);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < kBlockEvents && s_cnt[threadIdx.x]) atomicAdd(&counts[e0 + threadIdx.x], s_cnt[threadIdx.x]);
}

// The sums of a cluster are exact integers, so they may be added in any
// grouping: each thread takes kRun consecutive points (read 8 at a time with
// 32-byte loads), keeps running sums while the cluster stays the same (a
// cluster's points are mostly consecutive), and makes the three atomic
// additions once per run.
constexpr int kRun = kBridgeChunk / kBridgeThreads;  // 16 points per thread
static_assert(kRun % 8 == 0, "vector loads");

// Eight consecutive words: one 32-byte load, or two of 16 bytes.
template <class T>
__device__ __forceinline__ void load8(const T* p, bool wide, T* v) {
  static_assert(sizeof(T) == 4, "words");
  unsigned u[8];
  if (wide) {
    asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "l"(p));
  } else {
    const uint4 a = *reinterpret_cast<const uint4*>(p), b = *reinterpret_cast<const uint4*>(p + 4);
    u[0] = a.x, u[1] = a.y, u[2] = a.z, u[3] = a.w, u[4] = b.x, u[5] = b.y, u[6] = b.z, u[7] = b.w;
  }
  memcpy(v, u, 32);
}

__global__ void __launch_bounds__(kBridgeThreads) k_bridge_accumulate(
    int64_t N, const int64_t* __restrict__ off, const int32_t* __restrict__ chunk_ev,
    const int64_t* __restrict__ coff, const float* __restrict__ x, const float* __restrict__ y,
    const float* __restrict__ w, const int32_t* __restrict__ seed, const int32_t* __restrict__ ci,
    unsigned long long* __restrict__ acc, int32_t* __restrict__ seed_of, int32_t* __restrict__ flags) {
  const int64_t i0 = (int64_t)blockIdx.x * kBridgeChunk + (int64_t)threadIdx.x * kRun;
  if (i0 >= N) return;
  int32_t e = chunk_ev[blockIdx.x];
  int64_t next = off[e + 1];  // first point after event e
  while (next <= i0) next = off[++e + 1];
  int64_t cbase = coff[e];
  int32_t ccount = (int32_t)(coff[e + 1] - cbase);
  int32_t cur = -1;   // clusterIndex of the run
  bool live = false;  // it is a cluster of event e
  unsigned long long s0 = 0, s1 = 0, s2 = 0;
  auto flush = [&]() {
    if (live) {
      unsigned long long* a = acc + 3 * (cbase + cur);
      atomicAdd(a, s0);
      atomicAdd(a + 1, s1);
      atomicAdd(a + 2, s2);
    }
  };
  auto point = [&](int32_t c, int32_t sd, float wv, float xv, float yv, int64_t i) {
    if (c != cur) {
      flush();
      cur = c;
      live = c >= 0 && c < ccount;
      if (c >= ccount) atomicExch(&flags[kFlagError], 1);
      s0 = s1 = s2 = 0;
    }
    if (live) {
      s0 += fx_weight(wv);
      s1 += fx_pos(wv, xv);
      s2 += fx_pos(wv, yv);
      if (sd) seed_of[cbase + c] = (int32_t)i;
    }
  };
  // wide loads when the run is whole, in one event and every array is 16-byte
  // aligned (i0 is a multiple of 16 points); otherwise points are read one by
  // one.  A thread's run is 64 bytes of each array, so a 16-byte load uses half
  // of each sector it touches; with 32-byte loads, in groups of eight that are
  // not unrolled (72 registers when they are), the bridge on 200 HGCAL events
  // takes 0.49 ms against 0.525.  Arrays on a 16-byte boundary only: 0.515.
  const uintptr_t at = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) |
                       reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(seed) |
                       reinterpret_cast<uintptr_t>(ci);
  if (i0 + kRun <= next && (at & 15) == 0) {
    const bool wide = (at & 31) == 0;
#pragma unroll 1
    for (int k0 = 0; k0 < kRun; k0 += 8) {
      int32_t c8[8], s8[8];
      float w8[8], x8[8], y8[8];
      load8(ci + i0 + k0, wide, c8);
      load8(seed + i0 + k0, wide, s8);
      load8(w + i0 + k0, wide, w8);
      load8(x + i0 + k0, wide, x8);
      load8(y + i0 + k0, wide, y8);
#pragma unroll
      for (int k = 0; k < 8; ++k) point(c8[k], s8[k], w8[k], x8[k], y8[k], i0 + k0 + k);
    }
  } else {
#pragma unroll 1
    for (int64_t i = i0; i < min(i0 + (int64_t)kRun, N); ++i) {
      if (next <= i) {
        flush();
        live = false;
        cur = -1;
        while (next <= i) next = off[++e + 1];
        cbase = coff[e];
        ccount = (int32_t)(coff[e + 1] - cbase);
      }
      point(ci[i], seed[i], w[i], x[i], y[i], i);
    }
  }
  flush();
}

// What a cluster's sums give.
struct ClusterFields {
  float x, y, r_over_absz, eta, phi, energy;
};

// The definition, in double.  Not inlined: few clusters come here.
__device__ __noinline__ ClusterFields cluster_double(long long sw, long long swx, long long swy, const float* seed_x,
                                                     const float* seed_y, float z) {
  ClusterFields o;
  if (sw != 0) {
    const double den = (double)sw;
    o.x = __double2float_rn((double)swx * (kWScale / kPScale) / den);
    o.y = __double2float_rn((double)swy * (kWScale / kPScale) / den);
  } else {
    o.x = *seed_x;
    o.y = *seed_y;
  }
  const double xd = o.x, yd = o.y;
  const double r = sqrt(xd * xd + yd * yd);
  o.r_over_absz = __double2float_rn(r / fabs((double)z));
  o.eta = __double2float_rn(asinh((double)z / fmax(r, 1e-9)));
  o.phi = __double2float_rn(atan2(yd, xd));
  o.energy = __double2float_rn((double)sw / kWScale);
  return o;
}

// Sums of two floats (Dekker 1971, Knuth 2: error-free sum and product, the
// quotient and the square root with one correction), 45 bits and more.
struct Ff {
  float h, l;
};
__device__ __forceinline__ Ff ff_fast(float a, float b) {  // |a| >= |b|, or a == 0
  const float s = __fadd_rn(a, b);
  return Ff{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ Ff ff_sum(float a, float b) {
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return Ff{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ Ff ff_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return Ff{p, __fmaf_rn(a, b, -p)};
}
__device__ __forceinline__ Ff ff_add(Ff a, Ff b) {
  Ff s = ff_sum(a.h, b.h);
  const Ff t = ff_sum(a.l, b.l);
  s = ff_fast(s.h, __fadd_rn(s.l, t.h));
  return ff_fast(s.h, __fadd_rn(s.l, t.l));
}
__device__ __forceinline__ Ff ff_mul(Ff a, Ff b) {
  const Ff p = ff_prod(a.h, b.h);
  return ff_fast(p.h, __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, p.l)));
}
__device__ __forceinline__ Ff ff_div(Ff a, Ff b) {
  const float q = __fdiv_rn(a.h, b.h);
  // a.h - q * b.h is exact; the rest of the remainder is small beside it
  const float r = __fadd_rn(__fmaf_rn(-q, b.h, a.h), __fmaf_rn(-q, b.l, a.l));
  return ff_fast(q, __fdiv_rn(r, b.h));
}
__device__ __forceinline__ Ff ff_sqrt(Ff a) {
  const float x = __fsqrt_rn(a.h);
  return ff_fast(x, __fdiv_rn(__fadd_rn(__fmaf_rn(-x, x, a.h), a.l), __fmul_rn(2.f, x)));
}
// Whether rounding h + l to float is in doubt: |l| within 2^-13 of half an
// ulp of h, or h (whose lower neighbour is nearer) a power of two.
__device__ __forceinline__ bool ff_doubt(Ff a) {
  const unsigned u = __float_as_uint(a.h);
  const float half = __fmul_rn(__uint_as_float(u & 0x7f800000u), 5.9604644775390625e-08f);  // 2^-24
  return !(fabsf(a.l) < __fmul_rn(half, 0.9998779296875f)) || (u & 0x7fffffu) == 0;
}
// ln of w >= 1 (w.h below 2^60), by the series of atanh((m - 1) / (m + 1)) on
// the mantissa; relative error below 2^-40.
__device__ __forceinline__ Ff ff_log(Ff w) {
  int k = (int)(__float_as_uint(w.h) >> 23) - 127;
  if ((__float_as_uint(w.h) & 0x7fffffu) > 0x3504f3u) ++k;  // mantissa above sqrt(2): m in [0.707, 1.414]
  const float sc = __uint_as_float((unsigned)(127 - k) << 23);
  const Ff m{__fmul_rn(w.h, sc), __fmul_rn(w.l, sc)};
  const Ff one{1.f, 0.f};
  const Ff s = ff_div(ff_add(m, Ff{-1.f, 0.f}), ff_add(m, one));
  const Ff s2 = ff_mul(s, s);
  // ln m = 2 s (1 + s2 / 3 + s2^2 (1 / 5 + s2 (1 / 7 + ...)))
  const float t = s2.h;
  float q = __fmaf_rn(t, 0.05882353f, 0.06666667f);
  q = __fmaf_rn(t, q, 0.07692308f);
  q = __fmaf_rn(t, q, 0.09090909f);
  q = __fmaf_rn(t, q, 0.11111111f);
  q = __fmaf_rn(t, q, 0.14285715f);
  const Ff fifth{0.2f, -2.98023224e-09f}, third{0.333333343f, -9.93410776e-09f};
  const Ff u = ff_fast(fifth.h, __fmaf_rn(t, q, fifth.l));
  const Ff b = ff_add(ff_mul(s2, third), ff_mul(ff_mul(s2, s2), u));
  const Ff r = ff_add(s, ff_mul(s, b));
  const Ff kl = ff_mul(Ff{(float)k, 0.f}, Ff{0.693147182f, -1.90465421e-09f});
  return ff_add(kl, Ff{__fmul_rn(2.f, r.h), __fmul_rn(2.f, r.l)});
}
// atan(j / 8) as a sum of two floats.
__constant__ float kAtan[9][2] = {{0.f, 0.f},
                                  {0x1.fd5baap-4f, -0x1.54f424p-30f},
                                  {0x1.f5b760p-3f, -0x1.b4dfc8p-29f},
                                  {0x1.6f6194p-2f, 0x1.e4def0p-30f},
                                  {0x1.dac670p-2f, 0x1.586ed4p-28f},
                                  {0x1.1e00bap-1f, 0x1.7bdfd6p-26f},
                                  {0x1.4978fap-1f, 0x1.934f70p-28f},
                                  {0x1.700a7cp-1f, 0x1.5e118cp-27f},
                                  {0x1.921fb6p-1f, -0x1.777a5cp-26f}};

// atan of q in (0, 1], by atan q = atan c + atan((q - c) / (1 + q c)) for the
// nearest c = j / 8 and the series of the rest; relative error below 2^-40.
__device__ __forceinline__ Ff ff_atan(Ff q) {
  const int j = (int)__fadd_rn(__fmul_rn(q.h, 8.f), 0.5f);
  const float c = __fmul_rn((float)j, 0.125f);
  const Ff cq = ff_mul(q, Ff{c, 0.f});
  const Ff u = ff_div(ff_add(q, Ff{-c, 0.f}), ff_add(Ff{1.f, 0.f}, cq));
  const Ff u2 = ff_mul(u, u);
  // atan u = u - u (u2 / 3 - u2^2 (1 / 5 - u2 (1 / 7 - u2 / 9)))
  const float t = u2.h;
  const float p = __fmaf_rn(-t, __fmaf_rn(-t, 0.11111111f, 0.14285715f), 0.2f);
  const Ff third{0.333333343f, -9.93410776e-09f};
  const Ff b = ff_add(ff_mul(u2, third), Ff{-__fmul_rn(__fmul_rn(t, t), p), 0.f});
  const Ff ub = ff_mul(u, b);
  const Ff r = ff_add(u, Ff{-ub.h, -ub.l});
  return ff_add(Ff{kAtan[j][0], kAtan[j][1]}, r);
}

// The same fields without FP64 (which this GPU issues at a sixty-fourth of the
// single-precision rate: the double form bounded the kernel, 200 HGCAL events
// 0.271 ms, this 0.041 ms).  Sums of two floats give each field to 2^-40 and
// better; where that leaves its rounding to float in doubt (one cluster in
// some 1,600) or a value is out of the forms' range, returns false and the
// double form decides, so the results are the double form's.
__device__ __forceinline__ bool cluster_fast(long long sw, long long swx, long long swy, float z, ClusterFields* o) {
  constexpr long long kMost = 1ll << 46;
  const float az = fabsf(z);
  if (!(sw > 0 && sw < kMost && llabs(swx) < kMost && llabs(swy) < kMost && az > 1e-3f && az < 1e6f)) return false;
  // 48-bit integers as two exact floats
  auto exact = [](long long v) { return ff_sum(__fmul_rn((float)(int)(v >> 24), 16777216.f), (float)(int)(v & 0xffffff)); };
  const Ff w = exact(sw);
  const Ff qx = ff_div(exact(swx), w), qy = ff_div(exact(swy), w);
  if (ff_doubt(qx) || ff_doubt(qy)) return false;
  const float x = __fmul_rn(qx.h, (float)(kWScale / kPScale)), y = __fmul_rn(qy.h, (float)(kWScale / kPScale));
  const float ax = fabsf(x), ay = fabsf(y), big = fmaxf(ax, ay), small = fminf(ax, ay);
  if (!(small > 1e-6f && big < 1e6f)) return false;
  const Ff r2 = ff_add(ff_prod(x, x), ff_prod(y, y)), r = ff_sqrt(r2);
  if (!(__fmul_rn(4.f, az) > r.h)) return false;  // asinh of little: the logarithm below would cancel
  const Ff roa = ff_div(r, Ff{az, 0.f});
  // asinh(az / r) = ln((az + sqrt(az^2 + r^2)) / r)
  const Ff eta = ff_log(ff_div(ff_add(ff_sqrt(ff_add(ff_prod(az, az), r2)), Ff{az, 0.f}), r));
  Ff phi = ff_atan(ff_div(Ff{small, 0.f}, Ff{big, 0.f}));
  if (ay > ax) phi = ff_add(Ff{1.57079637f, -4.37113883e-08f}, Ff{-phi.h, -phi.l});
  if (x < 0.f) phi = ff_add(Ff{3.14159274f, -8.74227766e-08f}, Ff{-phi.h, -phi.l});
  if (ff_doubt(roa) || ff_doubt(eta) || ff_doubt(phi)) return false;
  o->x = x;
  o->y = y;
  o->r_over_absz = roa.h;
  o->eta = z < 0.f ? -eta.h : eta.h;
  o->phi = y < 0.f ? -phi.h : phi.h;
  o->energy = __fmul_rn(w.h, 1.f / 16777216.f);
  return true;
}

__global__ void k_bridge_finalize(int64_t C, const unsigned long long* __restrict__ acc,
                                  const int32_t* __restrict__ seed_of, const float* __restrict__ x,
                                  const float* __restrict__ y, const int32_t* __restrict__ layer,
                                  const float* __restrict__ layer_z, int32_t n_layers, float radius, int32_t sil,
                                  clue_layer_clusters o, int32_t* __restrict__ flags) {
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < C; g += (int64_t)gridDim.x * blockDim.x) {
    const int32_t s = seed_of[g];
    int32_t L = layer[s];
    if (L < 0 || L >= n_layers) {
      atomicExch(&flags[kFlagError], 2);
      L = 0;
    }
    const long long sw = (long long)acc[3 * g], swx = (long long)acc[3 * g + 1], swy = (long long)acc[3 * g + 2];
    const float z = layer_z[L];
    ClusterFields f;
    if (!cluster_fast(sw, swx, swy, z, &f)) f = cluster_double(sw, swx, swy, x + s, y + s, z);
    o.x[g] = f.x;
    o.y[g] = f.y;
    o.z[g] = z;
    o.r_over_absz[g] = f.r_over_absz;
    o.eta[g] = f.eta;
    o.phi[g] = f.phi;
    o.radius[g] = radius;
    o.layer[g] = L;
    o.energy[g] = f.energy;
    o.isSilicon[g] = sil;
  }
}

int check_offsets(int32_t E, const int64_t* off, const char* what) {
  if (E < 0) return set_error(CLUE_EINVAL, "n_events < 0");
  if (E == 0) return CLUE_OK;
  if (!off) return set_error(CLUE_EINVAL, "%s is NULL", what);
  if (off[0] != 0) return set_error(CLUE_EINVAL, "%s[0] must be 0", what);
  for (int32_t e = 0; e < E; ++e)
    if (off[e + 1] < off[e]) return set_error(CLUE_EINVAL, "%s must be non-decreasing", what);
  if (off[E] > INT32_MAX) return set_error(CLUE_EINVAL, "more than 2^31-1 entries in %s", what);
  return CLUE_OK;
}

// Event of the first point of each chunk of kBridgeChunk points (empty
// events own no point; the event of a point is the last e with off[e] <= i).
void chunk_events(int32_t E, const int64_t* off, int nch, int32_t* cev) {
  int c = 0;
  for (int32_t e = 0; e < E; ++e) {
    const int end = e + 1 < E ? (int)std::min<int64_t>(chunks_for(off[e + 1]), nch) : nch;
    for (; c < end; ++c) cev[c] = e;
  }
}

int grid_for(int64_t n, int device) {
  int sms = 1;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, sms * 16));
}

}  // namespace
}  // namespace clue

using clue::Handle;
using clue::cuda_error;
using clue::set_error;

extern "C" {

int clue_bridge_count(clue_handle* hh, int32_t E, const int64_t* off, const int32_t* isSeed,
                      int64_t* cluster_offsets) {
  return clue::guarded([&]() -> int {
    if (!hh || !cluster_offsets) return set_error(CLUE_EINVAL, "NULL argument");
    int rc = clue::check_offsets(E, off, "event_offsets");
    if (rc) return rc;
    cluster_offsets[0] = 0;
    if (E == 0) return CLUE_OK;
    const int64_t N = off[E];
    if (N > 0 && !isSeed) return set_error(CLUE_EINVAL, "isSeed is NULL");
    Handle* h = reinterpret_cast<Handle*>(hh);
    cudaError_t e = cudaSetDevice(h->device);
    if (e != cudaSuccess) return cuda_error(e, "cudaSetDevice");
    if ((rc = h->wait_previous())) return rc;
    std::vector<size_t> need(clue::B_SLOTS, 0);
    const int nch = clue::chunks_for(N);
    const size_t table_bytes = 8 * (size_t)(E + 1) + 4 * (size_t)nch;
    need[clue::B_TABLES] = table_bytes;
    need[clue::B_COUNT] = 4 * (size_t)E;
    if ((rc = h->reserve_beside(h->arena_bridge, need, {&h->arena, &h->arena3d}))) return rc;
    if ((rc = h->stage.reserve(table_bytes))) return rc;
    if ((rc = h->nt_host.reserve(4 * (size_t)E))) return rc;
    auto P = [&](int s) { return h->arena_bridge.ptr(s); };
    cudaStream_t s = h->stream;
    memcpy(h->stage.p, off, 8 * (size_t)(E + 1));
    int32_t* cev = reinterpret_cast<int32_t*>(static_cast<char*>(h->stage.p) + 8 * (size_t)(E + 1));
    clue::chunk_events(E, off, nch, cev);
    if ((e = cudaMemcpyAsync(P(clue::B_TABLES), h->stage.p, table_bytes, cudaMemcpyHostToDevice, s)) ||
        (e = cudaMemsetAsync(P(clue::B_COUNT), 0, 4 * (size_t)E, s)))
      return cuda_error(e, "bridge set-up");
    const int64_t* d_off = static_cast<const int64_t*>(P(clue::B_TABLES));
    if (N > 0)
      clue::k_bridge_count<<<nch, clue::kBridgeThreads, 0, s>>>(N, d_off,
                                                                  reinterpret_cast<const int32_t*>(d_off + (E + 1)),
                                                                  isSeed, static_cast<int32_t*>(P(clue::B_COUNT)));
    if ((e = cudaGetLastError())) return cuda_error(e, "k_bridge_count");
    const int32_t* counts = static_cast<const int32_t*>(h->nt_host.p);
    if ((e = cudaMemcpyAsync(h->nt_host.p, P(clue::B_COUNT), 4 * (size_t)E, cudaMemcpyDeviceToHost, s)) ||
        (e = cudaStreamSynchronize(s)))
      return cuda_error(e, "bridge counts");
    for (int32_t i = 0; i < E; ++i) cluster_offsets[i + 1] = cluster_offsets[i] + counts[i];
    return CLUE_OK;
  });
}

int clue_bridge_build(clue_handle* hh, const clue_bridge_params* p, int32_t E, const int64_t* off, const float* x,
                      const float* y, const int32_t* layer, const float* weight, const int32_t* isSeed,
                      const int32_t* clusterIndex, const int64_t* coff, const clue_layer_clusters* out) {
  return clue::guarded([&]() -> int {
    if (!hh || !p || !out) return set_error(CLUE_EINVAL, "NULL argument");
    int rc = clue::check_offsets(E, off, "event_offsets");
    if (rc) return rc;
    if ((rc = clue::check_offsets(E, coff, "cluster_offsets"))) return rc;
    if (p->n_layers < 1 || !p->layer_z) return set_error(CLUE_EINVAL, "bridge needs n_layers >= 1 and a z table");
    if (E == 0) return CLUE_OK;
    const int64_t N = off[E], C = coff[E];
    if (N > 0 && (!x || !y || !layer || !weight || !isSeed || !clusterIndex))
      return set_error(CLUE_EINVAL, "NULL input array");
    const void* outs[10] = {out->x, out->y, out->z, out->eta, out->phi, out->r_over_absz, out->radius,
                            out->layer, out->energy, out->isSilicon};
    if (C > 0)
      for (auto q : outs)
        if (!q) return set_error(CLUE_EINVAL, "NULL output array");
    Handle* h = reinterpret_cast<Handle*>(hh);
    cudaError_t e = cudaSetDevice(h->device);
    if (e != cudaSuccess) return cuda_error(e, "cudaSetDevice");
    if ((rc = h->wait_previous())) return rc;
    std::vector<size_t> need(clue::B_SLOTS, 0);
    const int nch = clue::chunks_for(N);
    const size_t table_bytes = 16 * (size_t)(E + 1) + 4 * (size_t)p->n_layers + 4 * (size_t)nch;
    const size_t sum_bytes = 28 * (size_t)C + 4 * clue::kFlagCount;
    need[clue::B_TABLES] = table_bytes;
    need[clue::B_COUNT] = 4 * (size_t)E;
    need[clue::B_SUMS] = sum_bytes;
    if ((rc = h->reserve_beside(h->arena_bridge, need, {&h->arena, &h->arena3d}))) return rc;
    if ((rc = h->stage.reserve(table_bytes))) return rc;
    if ((rc = h->flags_host.reserve(4 * clue::kFlagCount))) return rc;
    auto P = [&](int s) { return h->arena_bridge.ptr(s); };
    char* st = static_cast<char*>(h->stage.p);
    memcpy(st, off, 8 * (size_t)(E + 1));
    memcpy(st + 8 * (size_t)(E + 1), coff, 8 * (size_t)(E + 1));
    memcpy(st + 16 * (size_t)(E + 1), p->layer_z, 4 * (size_t)p->n_layers);
    int32_t* cev = reinterpret_cast<int32_t*>(st + 16 * (size_t)(E + 1) + 4 * (size_t)p->n_layers);
    clue::chunk_events(E, off, nch, cev);
    cudaStream_t s = h->stream;
    if ((e = cudaMemcpyAsync(P(clue::B_TABLES), st, table_bytes, cudaMemcpyHostToDevice, s)) ||
        (e = cudaMemsetAsync(P(clue::B_SUMS), 0, sum_bytes, s)))
      return cuda_error(e, "bridge set-up");
    const int64_t* d_off = static_cast<const int64_t*>(P(clue::B_TABLES));
    const int64_t* d_coff = d_off + (E + 1);
    const float* d_lz = reinterpret_cast<const float*>(d_coff + (E + 1));
    const int32_t* d_cev = reinterpret_cast<const int32_t*>(d_lz + p->n_layers);
    auto* acc = static_cast<unsigned long long*>(P(clue::B_SUMS));
    auto* seed_of = reinterpret_cast<int32_t*>(acc + 3 * C);
    int32_t* flags = seed_of + C;
    if (N > 0)
      clue::k_bridge_accumulate<<<nch, clue::kBridgeThreads, 0, s>>>(N, d_off, d_cev, d_coff, x, y, weight, isSeed,
                                                                     clusterIndex, acc, seed_of, flags);
    if ((e = cudaGetLastError())) return cuda_error(e, "k_bridge_accumulate");
    if (C > 0)
      clue::k_bridge_finalize<<<clue::grid_for(C, h->device), 256, 0, s>>>(C, acc, seed_of, x, y, layer,
                                                                 d_lz, p->n_layers, p->radius, p->isSilicon, *out, flags);
    if ((e = cudaGetLastError())) return cuda_error(e, "k_bridge_finalize");
    if ((e = cudaMemcpyAsync(h->flags_host.p, flags, 4 * clue::kFlagCount, cudaMemcpyDeviceToHost, s)) ||
        (e = cudaStreamSynchronize(s)))
      return cuda_error(e, "bridge");
    int32_t* fh = static_cast<int32_t*>(h->flags_host.p);
    const int32_t err = fh[clue::kFlagError];
    fh[clue::kFlagError] = 0;
    if (err == 1) return set_error(CLUE_EINVAL, "a clusterIndex is not below its event's cluster count");
    if (err == 2) return set_error(CLUE_EINVAL, "a layer cluster's layer is outside [0, %d)", p->n_layers);
    return CLUE_OK;
  });
}

}  // extern "C"
