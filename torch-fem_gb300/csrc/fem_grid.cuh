// Grid-wide scalars and barriers of the persistent cooperative kernels.
#pragma once

#include "fem_common.cuh"

namespace tfg {

// Sums of K doubles per lane on the integer pipe, the same values in every
// lane: each is aligned to its largest exponent as a 58-bit integer (five
// bits below an FP64 mantissa, rounded to nearest), added exactly in three
// redux words and rounded to FP64 once.  The error is at most 32 half units
// of 2^-58 of the largest value plus that rounding, no more than five FP64
// additions leave.  Exponents at either end of the range (and NaN,
// infinities) take the FP64 tree.
template <int K>
__device__ __forceinline__ void sum_fixed(double (&v)[K]) {
  int ex[K], e[K];
  bool plain = true;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    ex[k] = (__double2hiint(v[k]) >> 20) & 0x7ff;
    e[k] = (int)__reduce_max_sync(0xffffffffu, (unsigned)ex[k]);
    plain = plain && e[k] >= 128 && e[k] <= 1990;
  }
  if (!plain) {
#pragma unroll
    for (int k = 0; k < K; ++k)
      v[k] = __any_sync(0xffffffffu, (__double_as_longlong(v[k]) << 1) != 0) ? warp_sum(v[k]) : 0.0;
    return;
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const long long bits = __double_as_longlong(v[k]);
    const int sh = min(e[k] - ex[k], 62);
    unsigned long long m = ((unsigned long long)(bits & 0xfffffffffffffLL) | (1ull << 52)) << 5;
    m = ex[k] == 0 ? 0ull : (m + ((1ull << sh) >> 1)) >> sh;
    const long long f = bits < 0 ? -(long long)m : (long long)m;
    const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)f & 0x3fffffu);
    const unsigned mid = __reduce_add_sync(0xffffffffu, (unsigned)(f >> 22) & 0x3fffffu);
    const int hi = __reduce_add_sync(0xffffffffu, (int)(f >> 44));
    const long long t = ((long long)hi << 44) + ((long long)mid << 22) + (long long)lo;
    v[k] = t == 0 ? 0.0 : __longlong_as_double(__double_as_longlong((double)t) + ((long long)(e[k] - 1080) << 52));
  }
}

// Kept out of line: an iteration calls them several times, and straight-line code
// that runs once an iteration is fetched more slowly than it executes.
static __device__ __noinline__ double warp_sum_fixed(double a) {
  double v[1] = {a};
  sum_fixed<1>(v);
  return v[0];
}
static __device__ __noinline__ double2 warp_sum_fixed2(double a, double b) {
  double v[2] = {a, b};
  sum_fixed<2>(v);
  return make_double2(v[0], v[1]);
}

// Block-level sum as block_sum, by warp_sum_fixed: FP64 additions in a tree
// cost a warp 64 cycles of its sub-partition's pipe each.  Valid in warp 0.
__device__ __forceinline__ double block_sum_fixed(double v, double* smem32) {
  v = warp_sum_fixed(v);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) smem32[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (wid == 0) t = warp_sum_fixed(lane < (int)(blockDim.x >> 5) ? smem32[lane] : 0.0);
  __syncthreads();
  return t;
}

// isfinite and == 0 by the bits: a comparison costs an FP64 instruction.
__device__ __forceinline__ bool finite_bits(double v) { return ((__double2hiint(v) >> 20) & 0x7ff) != 0x7ff; }
__device__ __forceinline__ bool zero_bits(double v) { return (__double_as_longlong(v) << 1) == 0; }

// Grid-wide sums and barriers of the persistent kernels, with bounded waits.
//
// grid_barrier: one counter, a release reduction and acquire polls (2,500
// cycles on 152 CTAs); it orders the CTA's writes before the other CTAs'
// reads after it.
//
// grid_sum: the sum of NK doubles per CTA in one hop, by the counter itself.
// Each value is added as a 144-bit fixed-point number in four words, 36 bits to
// a word above an 18-bit count of arrivals, so the word that a CTA polls for the
// last arrival already holds the sum: no release, no second trip for the
// values, no additions by the reader (1,700 cycles for the hop; 4,500 with
// per-CTA partials behind a counter; polling every CTA's own slot, 3,400,
// since 152 pollers queue at the slots' L2 lines).  Integer additions commute:
// the sum does not depend on the order of arrival.  The fixed point's scale
// comes from the last sum of the same quantity, known to all: 2^-97 of it is
// the unit, and a share up to 2^40 times as large fits.  A share beyond that
// or not finite is marked in the words (nine bits above the count).  A sum below
// 2^-35 of the last one has lost bits: every share was cut to the unit, 500 of them
// by less than 2^-53 of a sum that large.  In either case, which every CTA sees in the
// same words, and for a first sum without a scale, the doubles themselves go
// round (grid_sum_plain).  The words only ever grow and are read as differences; two
// sets alternate, since a CTA that adds to one again has seen every CTA in the
// other, hence every CTA has read the first.
constexpr int kSumWords = 4, kSumBits = 36, kSumFall = 35;
constexpr int kSumLine = 16;                                   // 8-byte words from one to the next
constexpr int kSumHead = kSumLine * (1 + 2 * 2 * kSumWords);   // the counter, 2 sets of 2 values; plain slots follow
struct GridSync {
  unsigned long long* mem;      // zeroed before the launch
  unsigned long long prev0, prev1;  // warp 0: this lane's word of either set at its last sum
  unsigned long long barriers;  // barriers passed (thread 0)
  uint32_t sums, plain;         // sums so far, those of them by plain doubles
};
__device__ __forceinline__ void grid_sync_init(GridSync& g, unsigned long long* mem) {
  g.mem = mem;
  g.prev0 = g.prev1 = g.barriers = 0;
  g.sums = g.plain = 0;
}

__device__ __forceinline__ bool grid_barrier(int* error, long long spin_limit, GridSync& g) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    g.barriers += gridDim.x;
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(g.mem) : "memory");
    const long long t0 = clock64();
    bool good = true;
    while (true) {
      unsigned long long now;
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(g.mem) : "memory");
      if (now >= g.barriers) break;
      if (clock64() - t0 > spin_limit) {
        good = false;
        break;
      }
    }
    if (!good) atomicExch(error, 1);
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// The sum of the doubles themselves, each to its CTA's slot as two words of half
// a value and a sequence number; warp 0 of every CTA.
struct PlainSum {
  double x, y;
  int good;
};
template <int NK>
static __device__ __noinline__ PlainSum grid_sum_plain(unsigned long long* mem, uint32_t seq, long long spin_limit, double x,
                                                double y) {
  const int lane = threadIdx.x & 31, NC = gridDim.x;
  ulonglong2* buf = reinterpret_cast<ulonglong2*>(mem + kSumHead) + (size_t)(seq & 1) * NC * 2;
  if (lane < NK) {
    const unsigned long long w = (unsigned long long)__double_as_longlong(lane ? y : x);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(buf + (size_t)blockIdx.x * 2 + lane),
                 "l"((w << 32) | seq), "l"((w & 0xffffffff00000000ull) | seq)
                 : "memory");
  }
  bool good = true;
  double sums[NK];
  const long long t0 = clock64();
#pragma unroll
  for (int j = 0; j < NK; ++j) {
    sums[j] = 0.0;
    for (int i = lane; i < NC; i += 32) {
      unsigned long long a, b;
      while (true) {
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                     : "=l"(a), "=l"(b)
                     : "l"(buf + (size_t)i * 2 + j)
                     : "memory");
        if ((uint32_t)a == seq && (uint32_t)b == seq) break;
        if (clock64() - t0 > spin_limit) {
          good = false;
          break;
        }
      }
      sums[j] += __longlong_as_double((long long)((a >> 32) | (b & 0xffffffff00000000ull)));
    }
  }
  PlainSum t;
  t.good = __all_sync(0xffffffffu, good);
  t.x = warp_sum_fixed(sums[0]);
  t.y = NK > 1 ? warp_sum_fixed(sums[NK - 1]) : 0.0;
  return t;
}

// mine: this CTA's values, on every lane of warp 0.  ref: the scale of this
// quantity (of lane j: of value j / 4), 0 at first.  on_sums runs in thread 0,
// with the same sums on every CTA.  False (on every thread) if the wait ran
// out; the kernel then stops, and so, by their own limits, do the other CTAs.
// kData orders the CTA's writes before the other CTAs' reads after the sum, as
// grid_barrier does (the caller has synchronised its threads since it wrote).
template <int NK, bool kData = false, typename F>
__device__ __forceinline__ bool grid_sum(int* error, long long spin_limit, GridSync& g, const double (&mine)[NK],
                                         int& ref, F&& on_sums) {
  __shared__ int ok;
  if (threadIdx.x < 32) {
    if constexpr (kData) asm volatile("fence.acq_rel.gpu;" ::: "memory");
    const int lane = threadIdx.x, word = lane & (kSumWords - 1);
    const bool part = lane < NK * kSumWords;
    const uint32_t set = ++g.sums & 1;
    bool good = true, plain = __any_sync(0xffffffffu, part && ref == 0);
    double v[NK];
#pragma unroll
    for (int j = 0; j < NK; ++j) v[j] = mine[j];
    if (!plain) {
      unsigned long long delta = 0;
      if (part) {
        const long long bits = __double_as_longlong(lane < kSumWords ? mine[0] : mine[NK - 1]);
        const int ex = (int)((bits >> 52) & 0x7ff);
        const unsigned long long m = ex == 0 ? 0ull : (unsigned long long)(bits & 0xfffffffffffffLL) | (1ull << 52);
        const bool off = ex - ref > 40;  // includes the exponent of infinities and NaN
        const int sh = ex - ref + 45 - kSumBits * word;
        unsigned long long q = off || sh <= -53 || sh >= kSumBits ? 0ull : sh < 0 ? m >> -sh : m << sh;
        q &= (1ull << kSumBits) - 1;
        if (bits < 0) q = 0ull - q;
        unsigned long long* at = g.mem + kSumLine * (1 + (int)set * 2 * kSumWords + lane);
        asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(at), "l"((q << 18) + (off ? 513ull : 1ull))
                     : "memory");
        const long long t0 = clock64();
        const unsigned long long before = set ? g.prev1 : g.prev0;
        unsigned long long now;
        while (true) {
          asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(at) : "memory");
          delta = now - before;
          if ((delta & 511) == gridDim.x) break;
          if (clock64() - t0 > spin_limit) {
            good = false;
            break;
          }
        }
        if (set) g.prev1 = now;
        else g.prev0 = now;
      }
      __syncwarp();
      good = __all_sync(0xffffffffu, good);
      const long long sum = (long long)delta >> 18;
      double d = sum == 0 ? 0.0
                          : __longlong_as_double(__double_as_longlong((double)sum) +
                                                 ((long long)(kSumBits * word + ref - 1120) << 52));
      d += __shfl_xor_sync(0xffffffffu, d, 1);
      d += __shfl_xor_sync(0xffffffffu, d, 2);
      const bool fell = ((__double2hiint(d) >> 20) & 0x7ff) < ref - kSumFall;
      plain = __any_sync(0xffffffffu, part && (fell || ((delta >> 9) & 511) != 0));
#pragma unroll
      for (int j = 0; j < NK; ++j) v[j] = __shfl_sync(0xffffffffu, d, j * kSumWords);
    }
    if (plain && good) {
      const PlainSum t = grid_sum_plain<NK>(g.mem, ++g.plain, spin_limit, mine[0], mine[NK - 1]);
      v[0] = t.x;
      if constexpr (NK > 1) v[1] = t.y;
      good = t.good;
    }
    if constexpr (kData) asm volatile("fence.acq_rel.gpu;" ::: "memory");
    const int e = (__double2hiint(lane < kSumWords ? v[0] : v[NK - 1]) >> 20) & 0x7ff;
    ref = e >= 256 && e <= 1900 ? e : 0;
    if (lane == 0) {
      if (!good) atomicExch(error, 1);
      ok = good;
      on_sums(v);
    }
  }
  __syncthreads();
  return ok != 0;
}

// GridSync memory of a grid: its counters and, per CTA, two buffers of two
// 16-byte plain slots.
inline size_t sync_bytes(int64_t grid) { return sizeof(unsigned long long) * (kSumHead + 8 * (size_t)grid); }

}  // namespace tfg
