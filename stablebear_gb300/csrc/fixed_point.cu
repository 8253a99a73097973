// Pairwise integrals of float64 PCFs in 64-bit fixed point (sm_103a).
//
// The FP64 pipe of this GPU retires about two lanes per SM and clock, 1/64 of
// the FP32 rate, and the merge of pair_kernels.cu needs three to four FP64
// operations per rectangle: 58 to 78 SM cycles per warp-step, all spent on
// that pipe.  Here the merge runs on the integer pipe.  Times become integers
// T = rint(t 2^s) below 2^62, values integers too, and
//   sum over rectangles of (T_right - T_left) * op(F, G)
// is an exact integer sum: it does not depend on the order of the pair, the
// processing order, window ends or the launch shape.  FP64 appears once per
// pair, where the sum becomes a double.
//
// Values come in two forms, chosen on the device from the data:
//   counts   every value a multiple of one power of two with at most 13 bits
//            (26 for L1), as the ranks and Betti numbers of persistence
//            summaries are.  op(F, G) is an exact 32-bit integer; a rectangle
//            costs two 32 x 32 -> 64 multiply-adds (times are kept as two
//            31-bit limbs whose differences need no carry).
//   general  |F| < 2^62 (products: 2^63); op(F, G) is the top 64 bits of the
//            product, times the 62-bit width into a 128-bit sum.
//
// Error.  A time of at least 2^52 units is a whole number of them, as is a
// value of at least 2^52; a smaller one may be off by half a unit.  Each PCF
// carries what that can move (Shape), and from two of those follows a bound of
// the pair's error, whatever the order of its breakpoints and wherever its
// windows end; op drops at most a unit per unit of time.
// A pair whose usual error may be above 2^-51 of the sum of |terms|, or its
// worst above 2^-47, is walked again in double precision,
// as is every pair of a call whose data fits no form (NaN or infinite values,
// times out of order, extreme exponents or outliers): then pairs_kernel or
// the hybrid kernel runs instead, gated by the same device-side record.
#include "sbg_internal.hpp"

#include "fixed_point.cuh"

#include <cfloat>

namespace sbg
{
  namespace
  {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int U = 8;                                  // steps per block
    constexpr uint64_t T_END = (1ull << 62) - 1;          // after every breakpoint
    constexpr int MAX_EXP = 300;                          // larger exponents go the direct way
    constexpr uint32_t LOW_BIAS = 4096;

    // ---- the record of the data ---------------------------------------------------

    __device__ __forceinline__ int exponent(double x)  // of a finite x > 0: 2^e <= x < 2^(e + 1)
    {
      const uint64_t b = (uint64_t)__double_as_longlong(x);
      const int e = (int)(b >> 52) & 0x7ff;
      return e ? e - 1023 : 63 - __clzll((long long)(b & 0xfffffffffffffull)) - 1074;
    }
    __device__ __forceinline__ int low_exponent(double x)  // of the lowest set bit of a finite x != 0
    {
      const uint64_t b = (uint64_t)__double_as_longlong(x) & 0x7fffffffffffffffull;
      const int e = (int)(b >> 52);
      const uint64_t m = (b & 0xfffffffffffffull) | (e ? 1ull << 52 : 0ull);
      return (e ? e : 1) - 1075 + __ffsll((long long)m) - 1;
    }
    // Whether x 2^e is a whole number (x finite).
    __device__ __forceinline__ bool whole(double x, int e)
    {
      const uint64_t b = (uint64_t)__double_as_longlong(x) & 0x7fffffffffffffffull;
      const int field = (int)(b >> 52), low = field - 1075 + e;  // of the mantissa's last bit, scaled
      if (b == 0 || (field && low >= 0)) return true;
      if (field == 0 || low < -52) return false;
      return (((b & 0xfffffffffffffull) | 1ull << 52) & ((1ull << -low) - 1)) == 0;
    }
    __device__ __forceinline__ double pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }

    // What the record says: the form and its scales.
    struct Form
    {
      int kind;   // 0 direct, 1 counts, 2 general
      int s;      // T = rint(t 2^s)
      int r;      // F = rint(v 2^r)
      bool sign;  // some value is negative
    };

    __device__ Form form_of(const FixedRecord& d, int opk)
    {
      Form f{0, 0, 0, d.negative != 0};
      if (d.bad) return f;
      const double tmax = __longlong_as_double((long long)d.tmax_bits);
      const double vmax = __longlong_as_double((long long)d.vmax_bits);
      int te = 0, ve = 0, low = 0;
      if (tmax > 0) te = exponent(tmax);
      if (vmax > 0)
      {
        ve = exponent(vmax);
        low = (int)LOW_BIAS - (int)d.low;
      }
      if (te > MAX_EXP || te < -MAX_EXP || ve > MAX_EXP || low < -MAX_EXP) return f;
      f.s = 61 - te;
      if (ve - low < (opk == OPK_L1 ? 26 : 13))
      {
        f.kind = 1;
        f.r = -low;
        return f;
      }
      // Outliers push the other values down to the general form's last
      // bits, and its pairs to the direct walk: such data goes there at once.
      const double mean = d.vsum / (double)(d.points ? d.points : 1);
      if (mean < vmax * (opk == OPK_L1 ? 0x1p-11 : 0x1p-6)) return f;
      f.kind = 2;
      f.r = (opk == OPK_INNER ? 62 : 61) - ve;
      return f;
    }

    // ---- the error bound ------------------------------------------------------------
    //
    // With f' for f as rounded,
    //   sum of |f' - f| over time <= f.tv / 2 + f.ev / 2   (times, then values),
    // and op(f', g') - op(f, g) is at most
    //   L1        |f' - f| + |g' - g|
    //   products  |f' - f| max |g| + |g' - g| max |f|
    //   squares   (|f' - f| + |g' - g|) 2 max |f - g|.
    // Times that round lie below 2^52 units, so their share has the maxima of
    // what starts there, for squares that of the two ranges' distance: PCFs that
    // start alike are as close there as they are large elsewhere.
    // (0.501 for a half: the floats here round.)  Roundings of times in both
    // directions even out: usually a third of the root of the sum of squares
    // stands for half the sum.  A pair is taken if its usual error is at most
    // 2^-51 of its sum of |terms| (4.4e-16; the direct walk's is 3e-16), for
    // squares 2^-50, which the root halves, and its worst at most 2^-47, the
    // worst of the direct walk's naive blocks of 64.  Values count with their
    // worst both times.
    struct Bound
    {
      float worst, usual;
      __device__ __forceinline__ bool within(int opk, float total) const
      {
        if (worst <= total * 0x1p-51f) return true;  // most pairs
        return worst <= total * 0x1p-47f && usual <= total * (opk == OPK_L2DIST ? 0x1p-50f : 0x1p-51f);
      }
    };
    // Times, in integer values (general: over 2^32, squares and products over 2^64).
    __device__ __forceinline__ Bound counts_bound(int opk, const Shape& f, const Shape& g)
    {
      float worst, a = f.rv, b = g.rv, scale = 1.0f;
      if (opk == OPK_INNER)
      {
        const float mf = fmaxf(fabsf(f.lo), fabsf(f.hi)), mg = fmaxf(fabsf(g.lo), fabsf(g.hi));
        worst = 0.501f * (f.tv * mg + g.tv * mf);
        a *= 0x1p-20f * (mg * 0x1p-20f);  // general products are beyond a float when squared
        b *= 0x1p-20f * (mf * 0x1p-20f);
        scale = 0x1p40f;
      }
      else if (opk == OPK_L2DIST)
      {
        // (the ranges' own rounding to floats included)
        const float far = fmaxf(f.hi - g.lo, g.hi - f.lo) +
                          0x1p-22f * (fabsf(f.lo) + fabsf(f.hi) + fabsf(g.lo) + fabsf(g.hi));
        worst = 1.002f * (f.tv + g.tv) * far;
        scale = 2.0f * far;
      }
      else worst = 0.501f * (f.tv + g.tv);
      return Bound{worst, 0.289f * sqrtf(fmaf(a, a, b * b)) * scale};
    }
    // And values, whose times count over all of the PCF; products and squares
    // drop up to one unit up to the time T from which they are 0.
    __device__ __forceinline__ Bound general_bound(int opk, const Shape& f, const Shape& g, float T)
    {
      const Bound t = counts_bound(opk, f, g);
      if (opk == OPK_L1)
      {
        const float v = 0.501f * (f.ev + g.ev);
        return Bound{fmaf(t.worst, 0x1p32f, v), fmaf(t.usual, 0x1p32f, v)};
      }
      const float v = opk == OPK_INNER ? 0.501f * (f.ev * g.vmax + g.ev * f.vmax)
                                       : 1.002f * (f.ev + g.ev) * (f.vmax + g.vmax);
      return Bound{fmaf(v, 0x1p-32f, t.worst) + T, fmaf(v, 0x1p-32f, t.usual) + T};
    }

    // x 2^e as a float for estimates: cut off, not rounded, and 0 below 2^-126
    // (without the FP64 pipe, which is the slow one).
    __device__ __forceinline__ float scaled(double x, int e)
    {
      const int hi = __double2hiint(x), field = (hi >> 20 & 0x7ff) + e - 896;
      if ((hi >> 20 & 0x7ff) == 0 || field < 1) return 0.0f;
      return __uint_as_float((uint32_t)(hi & 0x80000000) | (uint32_t)min(field, 254) << 23 |
                             (uint32_t)(hi & 0xfffff) << 3 | (uint32_t)__double2loint(x) >> 29);
    }

    // Whether the call had better go to the direct kernels at once: where most
    // pairs would be refused, every pair would be walked twice.  A PCF is
    // risky if a pair of it and one like it would be (fixed_pack_kernel);
    // distances are refused where both sides are, products where one is.
    // N = 1000, L = 256, one PCF ending 1000 times later, L1 / L2 / L2 kernel:
    // 1.89 / 2.50 / 1.89 ms, 9.42 / 10.1 / 9.74 with every pair walked twice.
    __device__ __forceinline__ bool mostly_refused(const FixedRecord& d, int opk)
    {
      return 10ull * d.risky > (opk == OPK_INNER ? 2ull : 7ull) * d.packed;
    }

    // One warp per PCF.  Times count from the second breakpoint on (the walk
    // starts at 0 whatever the first says).  A PCF longer than `longest`, which
    // the host sized the call's buffers for, sends it to the direct kernels,
    // which check lengths for themselves.
    __global__ void __launch_bounds__(256) fixed_record_kernel(const double* __restrict__ pts,
                                                               const uint64_t* __restrict__ off, uint64_t n,
                                                               uint64_t cap, uint32_t longest, FixedRecord* rec)
    {
      const int lane = threadIdx.x & 31;
      const uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
      const uint64_t nw = (gridDim.x * (uint64_t)blockDim.x) >> 5;
      // the largest time and |value| as bit patterns; NaN and inf order above every finite one
      uint64_t tmax = 0, vmax = 0;
      uint32_t low = 0, neg = 0, bad = 0;
      float vsum = 0.0f;
      uint64_t points = 0;
      constexpr uint64_t INF = 0x7ff0000000000000ull;
      for (uint64_t i = w; i < n; i += nw)
      {
        const uint64_t o = off[i], e = off[i + 1];
        if (e <= o || e > cap || e - o > longest) { bad = 1; continue; }
        const uint64_t len = e - o;
        points += lane == 0 ? len : 0;
        for (uint64_t k = lane; k < len; k += 32)
        {
          const double t = pts[2 * (o + k)], v = pts[2 * (o + k) + 1];  // 8-byte aligned, no more
          if (k > 0)
          {
            const uint64_t tb = (uint64_t)__double_as_longlong(t);
            // times >= 0 order as their bit patterns; a set sign bit is above them all
            const uint64_t before = k > 1 ? (uint64_t)__double_as_longlong(pts[2 * (o + k - 1)]) : 0;
            bad |= tb < before || tb >= INF ? 1u : 0u;
            if (v != pts[2 * (o + k) - 1]) tmax = tb > tmax ? tb : tmax;  // no breakpoint of the function otherwise
          }
          const uint64_t vb = (uint64_t)__double_as_longlong(v) & 0x7fffffffffffffffull;
          if (vb)
          {
            vmax = vb > vmax ? vb : vmax;
            neg |= __double_as_longlong(v) < 0 ? 1u : 0u;
            const uint32_t l = (uint32_t)((int)LOW_BIAS - low_exponent(v));
            low = l > low ? l : low;
            vsum += fabsf((float)v);
          }
        }
      }
      if (vmax >= INF) bad = 1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
      {
        const uint64_t a = __shfl_xor_sync(FULL, tmax, o), b = __shfl_xor_sync(FULL, vmax, o);
        tmax = a > tmax ? a : tmax;
        vmax = b > vmax ? b : vmax;
        vsum += __shfl_xor_sync(FULL, vsum, o);
      }
      low = __reduce_max_sync(FULL, low);
      neg = __reduce_or_sync(FULL, neg);
      bad = __reduce_or_sync(FULL, bad);
      if (lane == 0)
      {
        if (bad) atomicOr(&rec->bad, 1u);
        if (neg) atomicOr(&rec->negative, 1u);
        atomicMax(&rec->low, low);
        atomicMax(reinterpret_cast<unsigned long long*>(&rec->tmax_bits), (unsigned long long)tmax);
        atomicMax(reinterpret_cast<unsigned long long*>(&rec->vmax_bits), (unsigned long long)vmax);
        atomicAdd(&rec->vsum, (double)vsum);
        atomicAdd(reinterpret_cast<unsigned long long*>(&rec->points), (unsigned long long)points);
      }
    }

    // The (v, t) elements that the hybrid kernel reads, by a warp.
    __device__ __forceinline__ void write_elements(const double* pts, uint64_t o, uint64_t len, Elem<double>* packed,
                                                   int lane)
    {
      for (uint64_t k = lane; k < len; k += 32)
        packed[o + k] = Elem<double>{pts[2 * (o + k) + 1],
                                     k + 1 == len ? tmax_of<double>() : fmin(pts[2 * (o + k + 1)], tmax_of<double>())};
    }

    // The times of a PCF's elements (an element ends where the value next
    // changes, the last at T_END) and their values, at the CSR's own offsets,
    // and how many there are: neighbours of equal value are one element (a
    // rank that has reached 0 and stays there, say), which changes no exact
    // sum.  Where the record says direct, the (v, t) elements the hybrid
    // kernel reads, in the same buffer, all of them.  One warp per PCF.
    __global__ void __launch_bounds__(256) fixed_pack_kernel(const double* __restrict__ pts,
                                                             const uint64_t* __restrict__ off, uint64_t n,
                                                             uint64_t cap, FixedRecord* rec, int opk,
                                                             void* __restrict__ packed, Shape* __restrict__ shapes,
                                                             uint32_t* __restrict__ lens, bool elements,
                                                             unsigned* __restrict__ gate)
    {
      const Form f = form_of(*rec, opk);
      if (blockIdx.x == 0 && threadIdx.x == 0) *gate = f.kind == 0 ? 0u : 1u;  // closes the direct kernels
      const int lane = threadIdx.x & 31;
      const uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
      const uint64_t nw = (gridDim.x * (uint64_t)blockDim.x) >> 5;
      uint64_t* times = static_cast<uint64_t*>(packed);
      void* values = times + cap;
      const int unit_exp = f.kind == 1 ? f.r : f.r - 32;
      const double ts = pow2(f.s), vs = pow2(f.r), unit = pow2(unit_exp);
      uint32_t risky = 0, seen = 0;
      for (uint64_t i = w; i < n; i += nw)
      {
        const uint64_t o = off[i], e = off[i + 1];
        if (e <= o || e > cap)  // never write past the packed buffer
        {
          if (lane == 0) lens[i] = 0;
          continue;
        }
        const uint64_t len = e - o;
        if (f.kind == 0)
        {
          if (lane == 0) lens[i] = (uint32_t)len;
          if (elements) write_elements(pts, o, len, static_cast<Elem<double>*>(packed), lane);
          continue;
        }
        float tv = 0.0f, qv = 0.0f, ev = 0.0f, vm = 0.0f, area = 0.0f, end = 0.0f, lo = FLT_MAX, hi = -FLT_MAX;
        uint64_t count = 0;  // elements before this chunk
        for (uint64_t k0 = 0; k0 < len; k0 += 32)
        {
          const uint64_t k = k0 + lane;
          double t = 0.0, v = 0.0, before = 0.0;
          if (k < len)
          {
            t = pts[2 * (o + k)];
            v = pts[2 * (o + k) + 1];
            if (k > 0)
            {
              before = pts[2 * (o + k) - 1];
              if (f.kind == 2 && !whole(before, f.r)) ev += (float)((t - (k > 1 ? pts[2 * (o + k) - 2] : 0.0)) * ts);
            }
          }
          const bool starts = k < len && (k == 0 || v != before);
          const unsigned mask = __ballot_sync(FULL, starts);
          if (starts)
          {
            const uint64_t at = o + count + __popc(mask & ((1u << lane) - 1u));  // <= o + k
            const long long F = __double2ll_rn(v * vs);
            const float value = (float)F * (f.kind == 1 ? 1.0f : 0x1p-32f);
            if (k > 0)
            {
              if (!whole(t, f.s))
              {
                const float c = fabsf((float)((v - before) * unit));
                tv += c;
                qv = fmaf(c, c, qv);
              }
              const float x = scaled(before, unit_exp), y = scaled(v, unit_exp);
              end = scaled(t, f.s);
              area = fmaf(opk == OPK_L1 ? fabsf(x) - fabsf(y) : (x - y) * (x + y), end, area);
            }
            if (k == 0 || end < 0x1p52f)  // (cut off, so right at the border)
            {
              lo = fminf(lo, value);
              hi = fmaxf(hi, value);
            }
            vm = fmaxf(vm, fabsf(value));
            if (f.kind == 1)
              static_cast<uint32_t*>(values)[at] = (uint32_t)(int32_t)F;
            else
              // the product needs magnitudes and signs, differences need two's complement
              static_cast<uint64_t*>(values)[at] =
                  opk == OPK_INNER ? (uint64_t)(F < 0 ? -F : F) | (F < 0 ? 1ull << 63 : 0ull) : (uint64_t)F;
            if (k > 0)  // ends the element before
            {
              const uint64_t T = (uint64_t)__double2ll_rn(t * ts);
              times[at - 1] = f.kind == 1 ? ((T >> 31) << 32) | (T & 0x7fffffffull) : T;
            }
          }
          count += (uint64_t)__popc(mask);
        }
#pragma unroll
        for (int h = 16; h > 0; h >>= 1)
        {
          tv += __shfl_xor_sync(FULL, tv, h);
          qv += __shfl_xor_sync(FULL, qv, h);
          ev += __shfl_xor_sync(FULL, ev, h);
          area += __shfl_xor_sync(FULL, area, h);
        }
        // floats >= 0 order as their bits; the others after this
        auto order = [](float x) {
          const int b = __float_as_int(x);
          return b ^ ((b >> 31) & 0x7fffffff);
        };
        auto value_of = [](int b) { return __int_as_float(b ^ ((b >> 31) & 0x7fffffff)); };
        vm = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(vm)));
        end = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(end)));
        lo = value_of(__reduce_min_sync(FULL, order(lo)));
        hi = value_of(__reduce_max_sync(FULL, order(hi)));
        if (lane == 0)
        {
          times[o + count - 1] = f.kind == 1 ? ((T_END >> 31) << 32) | (T_END & 0x7fffffffull) : T_END;
          lens[i] = (uint32_t)count;
          const Shape s{tv, sqrtf(qv), lo, hi, vm, ev, 0.0f, 0.0f};
          shapes[i] = s;
          // a pair with one like it: |f - g| is about |f|, its square twice that
          // of f, |f g| some five eighths of it
          const Bound bound = f.kind == 1 ? counts_bound(opk, s, s) : general_bound(opk, s, s, end);
          const float total = area * (opk == OPK_L2DIST ? 2.0f : opk == OPK_INNER ? 0.625f : f.kind == 2 ? 0x1p32f : 1.0f);
          risky += bound.within(opk, total) ? 0u : 1u;
          ++seen;
        }
      }
      if (lane == 0 && seen)
      {
        if (risky) atomicAdd(&rec->risky, risky);
        atomicAdd(&rec->packed, seen);
      }
    }

    // ---- arithmetic of the two forms -----------------------------------------------

    // Running sums of one lane's pair.
    //   add      one rectangle: op(F, G) = q, found before its side moved on
    //   good     whether the error bound is small enough against the sum of |terms|
    //   value    the sum as a double, in units of time times op
    //
    // All of them are exact sums, the same however the pair was cut.
    // Kept as 32-bit registers throughout: as 64-bit C++ variables the walk's
    // tied asm operands and the products cost ten more instructions a step
    // (28 against 18 for counts).
    template <int K, bool SG>
    struct Counts
    {
      using V = uint32_t;
      struct Side { uint32_t lo, hi, v; };    // where the element ends (two 31-bit limbs), its value
      struct Q { int32_t q; };
      static constexpr uint32_t BYTES = 12;   // of an element in shared memory
      static constexpr bool DROPS = false;    // whether op drops part of a unit
      int64_t s0 = 0, s1 = 0;                 // sum = s1 2^31 + s0
      int64_t a0 = 0, a1 = 0;                 // signed products: the same of |q|

      static __device__ __forceinline__ uint64_t end() { return ((T_END >> 31) << 32) | (T_END & 0x7fffffffull); }
      static __device__ __forceinline__ uint64_t units(uint64_t t) { return ((t >> 32) << 31) | (t & 0x7fffffffull); }
      static __device__ __forceinline__ Q op(const Side& f, const Side& g)
      {
        // in asm: the compiler would widen the product to 64 bits
        int32_t q;
        if (K == OPK_INNER) asm("mul.lo.s32 %0, %1, %2;" : "=r"(q) : "r"(f.v), "r"(g.v));
        else if (K == OPK_L1) asm("abs.s32 %0, %1;" : "=r"(q) : "r"(f.v - g.v));
        else asm("mul.lo.s32 %0, %1, %1;" : "=r"(q) : "r"(f.v - g.v));
        return Q{q};
      }
      __device__ __forceinline__ void add(uint32_t tl, uint32_t th, uint32_t nl, uint32_t nh, Q q)
      {
        const int32_t lo = (int32_t)(nl - tl), hi = (int32_t)(nh - th);
        s0 += (int64_t)q.q * lo;
        s1 += (int64_t)q.q * hi;
        if (SG)
        {
          const int32_t a = abs(q.q);
          a0 += (int64_t)a * lo;
          a1 += (int64_t)a * hi;
        }
      }
      __device__ __forceinline__ void block()  // s0 stays below 2^63 over a block's 8 steps of 2^28 * 2^31
      {
        s1 += s0 >> 31;
        s0 &= 0x7fffffff;
        if (SG)
        {
          a1 += a0 >> 31;
          a0 &= 0x7fffffff;
        }
      }
      __device__ __forceinline__ void save(uint64_t* c) const
      {
        c[0] = (uint64_t)s0; c[32] = (uint64_t)s1;
        if (SG) { c[64] = (uint64_t)a0; c[96] = (uint64_t)a1; }
      }
      __device__ __forceinline__ void restore(const uint64_t* c)
      {
        s0 = (int64_t)c[0]; s1 = (int64_t)c[32];
        if (SG) { a0 = (int64_t)c[64]; a1 = (int64_t)c[96]; }
      }
      __device__ __forceinline__ bool good(const Shape& f, const Shape& g, uint64_t) const
      {
        const float total = SG ? fmaf((float)a1, 0x1p31f, (float)a0) : fmaf((float)s1, 0x1p31f, (float)s0);
        return counts_bound(K, f, g).within(K, total);
      }
      __device__ __forceinline__ double value() const { return fma((double)s1, 0x1p31, (double)s0); }
      static __device__ __forceinline__ int scale(const Form& f) { return -f.s - (K == OPK_L1 ? f.r : 2 * f.r); }
    };

    template <int K, bool SG>
    struct General
    {
      using V = uint64_t;
      struct Side { uint32_t lo, hi, v, w; };  // where the element ends, its value (low, high word)
      struct Q { uint32_t lo, hi, sign; };     // |op|, all ones where it is negative
      static constexpr uint32_t BYTES = 16;
      static constexpr bool DROPS = K != OPK_L1;
      uint32_t s0 = 0, s1 = 0, s2 = 0, s3 = 0;  // sum of |terms| = s + h 2^64
      uint64_t h = 0;
      uint32_t n0 = 0, n1 = 0, n2 = 0, n3 = 0;  // signed products: that of the negative ones

      static __device__ __forceinline__ uint64_t end() { return T_END; }
      static __device__ __forceinline__ uint64_t units(uint64_t t) { return t; }
      static __device__ __forceinline__ Q op(const Side& f, const Side& g)
      {
        if (K == OPK_INNER)  // magnitudes and signs: the top word of the product
        {
          const uint32_t fw = SG ? f.w & 0x7fffffffu : f.w, gw = SG ? g.w & 0x7fffffffu : g.w;
          uint64_t r = (((uint64_t)f.v * g.v) >> 32) + (uint64_t)f.v * gw;
          r += (uint64_t)fw * g.v;
          const uint64_t q = (r >> 32) + (uint64_t)fw * gw;
          return Q{(uint32_t)q, (uint32_t)(q >> 32), SG ? (uint32_t)((int32_t)(f.w ^ g.w) >> 31) : 0u};
        }
        uint32_t al, ah;
        asm("{\n\t.reg .b32 s;\n\t"
            "sub.cc.u32 %0, %2, %4;\n\t"
            "subc.u32 %1, %3, %5;\n\t"
            "shr.s32 s, %1, 31;\n\t"
            "xor.b32 %0, %0, s;\n\t"
            "xor.b32 %1, %1, s;\n\t"
            "sub.cc.u32 %0, %0, s;\n\t"
            "subc.u32 %1, %1, s;\n\t}"
            : "=&r"(al), "=&r"(ah)
            : "r"(f.v), "r"(f.w), "r"(g.v), "r"(g.w));
        if (K == OPK_L1) return Q{al, ah, 0u};
        const uint64_t r = (((uint64_t)al * al) >> 32) + (uint64_t)al * (ah + ah);  // |d| < 2^63: no carry out
        const uint64_t q = (r >> 32) + (uint64_t)ah * ah;
        return Q{(uint32_t)q, (uint32_t)(q >> 32), 0u};
      }
      __device__ __forceinline__ void add(uint32_t tl, uint32_t th, uint32_t nl, uint32_t nh, Q q)
      {
        uint32_t bl, bh;
        asm("sub.cc.u32 %0, %2, %4;\n\tsubc.u32 %1, %3, %5;"
            : "=&r"(bl), "=r"(bh)
            : "r"(nl), "r"(nh), "r"(tl), "r"(th));
        const uint64_t p = (uint64_t)q.lo * bl;
        uint64_t r = (p >> 32) + (uint64_t)q.lo * bh;
        r += (uint64_t)q.hi * bl;
        if (SG)
        {
          const uint64_t t = (r >> 32) + (uint64_t)q.hi * bh;
          asm("add.cc.u32 %0, %0, %4;\n\taddc.cc.u32 %1, %1, %5;\n\taddc.cc.u32 %2, %2, %6;\n\taddc.u32 %3, %3, %7;"
              : "+r"(s0), "+r"(s1), "+r"(s2), "+r"(s3)
              : "r"((uint32_t)p), "r"((uint32_t)r), "r"((uint32_t)t), "r"((uint32_t)(t >> 32)));
          asm("add.cc.u32 %0, %0, %4;\n\taddc.cc.u32 %1, %1, %5;\n\taddc.cc.u32 %2, %2, %6;\n\taddc.u32 %3, %3, %7;"
              : "+r"(n0), "+r"(n1), "+r"(n2), "+r"(n3)
              : "r"((uint32_t)p & q.sign), "r"((uint32_t)r & q.sign), "r"((uint32_t)t & q.sign),
                "r"((uint32_t)(t >> 32) & q.sign));
        }
        else
        {
          h += (uint64_t)q.hi * bh;
          asm("add.cc.u32 %0, %0, %4;\n\taddc.cc.u32 %1, %1, %5;\n\taddc.cc.u32 %2, %2, %6;\n\taddc.u32 %3, %3, 0;"
              : "+r"(s0), "+r"(s1), "+r"(s2), "+r"(s3)
              : "r"((uint32_t)p), "r"((uint32_t)r), "r"((uint32_t)(r >> 32)));
        }
      }
      __device__ __forceinline__ void block() { }
      __device__ __forceinline__ unsigned __int128 sum() const
      {
        const unsigned __int128 lo = ((uint64_t)s1 << 32) | s0, hi = (((uint64_t)s3 << 32) | s2) + h;
        return (hi << 64) + lo;
      }
      __device__ __forceinline__ unsigned __int128 negative() const
      {
        return ((unsigned __int128)(((uint64_t)n3 << 32) | n2) << 64) + (((uint64_t)n1 << 32) | n0);
      }
      __device__ __forceinline__ void save(uint64_t* c) const
      {
        const unsigned __int128 s = sum();
        c[0] = (uint64_t)s; c[32] = (uint64_t)(s >> 64);
        if (SG) { c[64] = ((uint64_t)n1 << 32) | n0; c[96] = ((uint64_t)n3 << 32) | n2; }
      }
      __device__ __forceinline__ void restore(const uint64_t* c)
      {
        s0 = (uint32_t)c[0]; s1 = (uint32_t)(c[0] >> 32);
        s2 = (uint32_t)c[32]; s3 = (uint32_t)(c[32] >> 32);
        if (SG)
        {
          n0 = (uint32_t)c[64]; n1 = (uint32_t)(c[64] >> 32);
          n2 = (uint32_t)c[96]; n3 = (uint32_t)(c[96] >> 32);
        }
      }
      __device__ __forceinline__ bool good(const Shape& f, const Shape& g, uint64_t T) const
      {
        const unsigned __int128 s = sum();
        const float total = fmaf((float)(uint64_t)(s >> 64), 0x1p64f, (float)(uint64_t)s);
        return general_bound(K, f, g, (float)T).within(K, total);
      }
      __device__ __forceinline__ double value() const
      {
        const __int128 s = (__int128)(SG ? sum() - 2 * negative() : sum());
        const bool neg = SG && s < 0;
        const unsigned __int128 a = (unsigned __int128)(neg ? -s : s);
        const double v = fma((double)(uint64_t)(a >> 64), 0x1p64, (double)(uint64_t)a);
        return neg ? -v : v;
      }
      static __device__ __forceinline__ int scale(const Form& f)
      {
        return K == OPK_L1 ? -f.s - f.r : 64 - f.s - 2 * f.r;
      }
    };

    // ---- the walk -----------------------------------------------------------------

    // A row of a warp in shared memory: times, then values; a lane's column:
    // elements 32 BYTES bytes apart.  (nl, nh): the next breakpoint, the row's
    // on a tie.  One side moves on, with loads for that side alone.
    template <typename A>
    __device__ __forceinline__ void advance(typename A::Side& f, typename A::Side& g, uint32_t& af, uint32_t tof,
                                            uint32_t& ag, uint32_t vof, uint32_t& nl, uint32_t& nh)
    {
      if constexpr (sizeof(typename A::V) == 4)
        // af: address of the row value; its time lies at 2 af + tof
        asm("{\n\t.reg .pred p;\n\t.reg .b32 a, b;\n\t.reg .u64 x, y;\n\t"
            "mov.b64 x, {%0, %1};\n\t"
            "mov.b64 y, {%3, %4};\n\t"
            "setp.le.u64 p, x, y;\n\t"
            "selp.b32 %8, %0, %3, p;\n\t"
            "selp.b32 %9, %1, %4, p;\n\t"
            "@p add.u32 %6, %6, 4;\n\t"
            "@!p add.u32 %7, %7, 384;\n\t"
            "mad.lo.u32 a, %6, 2, %10;\n\t"
            "add.u32 b, %7, %11;\n\t"
            "@p ld.shared.v2.u32 {%0, %1}, [a];\n\t"
            "@p ld.shared.u32 %2, [%6];\n\t"
            "@!p ld.shared.v2.u32 {%3, %4}, [%7];\n\t"
            "@!p ld.shared.u32 %5, [b];\n\t}"
            : "+r"(f.lo), "+r"(f.hi), "+r"(f.v), "+r"(g.lo), "+r"(g.hi), "+r"(g.v), "+r"(af), "+r"(ag), "=&r"(nl),
              "=&r"(nh)
            : "r"(tof), "r"(vof));
      else
        // af: address of the row value; its time lies at af + tof
        asm("{\n\t.reg .pred p;\n\t.reg .b32 a;\n\t.reg .u64 x, y;\n\t"
            "mov.b64 x, {%0, %1};\n\t"
            "mov.b64 y, {%4, %5};\n\t"
            "setp.le.u64 p, x, y;\n\t"
            "selp.b32 %10, %0, %4, p;\n\t"
            "selp.b32 %11, %1, %5, p;\n\t"
            "@p add.u32 %8, %8, 8;\n\t"
            "@!p add.u32 %9, %9, 512;\n\t"
            "add.u32 a, %8, %12;\n\t"
            "@p ld.shared.v2.u32 {%0, %1}, [a];\n\t"
            "@p ld.shared.v2.u32 {%2, %3}, [%8];\n\t"
            "@!p ld.shared.v4.u32 {%4, %5, %6, %7}, [%9];\n\t}"
            : "+r"(f.lo), "+r"(f.hi), "+r"(f.v), "+r"(f.w), "+r"(g.lo), "+r"(g.hi), "+r"(g.v), "+r"(g.w), "+r"(af),
              "+r"(ag), "=&r"(nl), "=&r"(nh)
            : "r"(tof));
    }

    // Steps through one (sub-)window: the row's m elements from t0 / v0, the
    // last ending at the window's end and followed by U copies of itself; the
    // lane's column from address ag.  Nothing passes the row's end, so a
    // column that reaches further is cut there.
    template <typename A>
    __device__ __forceinline__ void walk(A& acc, const uint64_t* t0, const typename A::V* v0, uint32_t ag,
                                         uint32_t vof, uint32_t m, uint32_t steps, uint64_t t)
    {
      using V = typename A::V;
      typename A::Side f, g;
      f.lo = (uint32_t)*t0;
      f.hi = (uint32_t)(*t0 >> 32);
      f.v = (uint32_t)*v0;
      const uint32_t at = (uint32_t)__cvta_generic_to_shared(t0);
      uint32_t af = (uint32_t)__cvta_generic_to_shared(v0);
      const uint32_t tof = sizeof(V) == 4 ? at - 2 * af : at - af;
      const uint32_t af_last = af + (m - 1) * (uint32_t)sizeof(V);
      if constexpr (sizeof(V) == 4)
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%3];\n\tld.shared.u32 %2, [%4];"
                     : "=&r"(g.lo), "=&r"(g.hi), "=r"(g.v)
                     : "r"(ag), "r"(ag + vof)
                     : "memory");
      else
      {
        f.w = (uint32_t)(*v0 >> 32);
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(g.lo), "=r"(g.hi), "=r"(g.v), "=r"(g.w)
                     : "r"(ag)
                     : "memory");
      }
      uint32_t tl = (uint32_t)t, th = (uint32_t)(t >> 32);
      const uint32_t nblk = (steps + U - 1) / U;
      for (uint32_t b = 0; b < nblk; ++b)
      {
        // a lane past its end advances the row on every step: back to the
        // last element, of which U copies follow
        af = min(af, af_last);
#pragma unroll
        for (int u = 0; u < U; ++u)
        {
          const auto q = A::op(f, g);
          uint32_t nl, nh;
          advance<A>(f, g, af, tof, ag, vof, nl, nh);
          acc.add(tl, th, nl, nh, q);
          tl = nl;
          th = nh;
        }
        acc.block();
      }
    }

    template <int K>
    __device__ __forceinline__ double op_f64(double f, double g)
    {
      const double d = f - g;
      return K == OPK_INNER ? f * g : K == OPK_L1 ? fabs(d) : d * d;
    }

    // A pair in double precision, from the CSR points: the merged breakpoints
    // of both in 32 parts of equal number, each walked in naive blocks of 64
    // rectangles under Kahan compensation, as the direct kernels sum, and the
    // parts added neighbour to neighbour.  Nothing in that depends on which PCF
    // comes first.  Few pairs of a row go one after the other, a part to a lane
    // (one lane's chain of dependent loads would hold up the rest of the launch:
    // 23 ms at N = 1200, where one column that ends early fails the test against
    // every row); many go at once, a pair to a lane, part after part, with the
    // same bits (N = 1000 near duplicates, L = 256, L2: 3.60 ms with the pairs
    // at once, 7.95 one after the other, 2.48 in the direct kernel alone).
    //
    // Only what comes before `stop` counts, at or after the time from which
    // every term is 0 (the largest double: no such time): the products of a
    // PCF that ends early are over when it is, the distances of two when both
    // are, and thousands of later elements add nothing (the L2 kernel of 3500 stable ranks with a few
    // such: 2.98 ms with them, 0.98 without).
    __device__ __forceinline__ uint32_t elements_before(const double* f, uint32_t n, double stop)
    {
      uint32_t lo = 1, hi = n;
      while (lo < hi)
      {
        const uint32_t mid = (lo + hi) / 2;
        if (f[2 * mid] < stop) lo = mid + 1; else hi = mid;
      }
      return lo;
    }

    struct DirectPair
    {
      const double *f, *g;
      uint32_t nf, ng, per;  // elements; breakpoints of a part, the end at `stop` one of them
      double stop;           // where both sides' last elements end

      __device__ __forceinline__ DirectPair(const double* f_, uint32_t nf_, const double* g_, uint32_t ng_,
                                            double stop_)
          : f(f_), g(g_), nf(nf_), ng(ng_), stop(stop_)
      {
        if (stop < tmax_of<double>())
        {
          nf = elements_before(f, nf, stop);
          ng = elements_before(g, ng, stop);
        }
        per = (nf + ng - 1 + 31) / 32;
      }
    };

    // The sum over a part.
    struct DirectSum
    {
      double acc = 0.0, comp = 0.0, blk = 0.0;
      uint32_t k = 0;
      __device__ __forceinline__ void flush()
      {
        const double y = blk - comp, s = acc + y;
        comp = isfinite(s) ? (s - acc) - y : 0.0;
        acc = s;
        blk = 0.0;
        k = 0;
      }
      __device__ __forceinline__ void add(double q, double width)
      {
        blk = fma(q, width, blk);
        if (++k == 64) flush();
      }
      __device__ __forceinline__ double end()
      {
        if (k) flush();
        const double x = acc - comp;
        acc = comp = 0.0;
        return x;
      }
    };

    // Where the elements are read: point k's time and value, and the ones
    // after the last, which never come.
    struct DirectSide
    {
      const double* p;
      uint32_t n, next;     // the point that `at` holds
      double v, t, vn;      // the element's value, where it ends, the value after
      double ta, va;        // the point behind that
      double stop;
      __device__ __forceinline__ void read()
      {
        const bool in = next < n;
        ta = in ? p[2 * next] : stop;
        va = in ? p[2 * next + 1] : 0.0;
      }
      __device__ __forceinline__ void start(const double* p_, uint32_t n_, uint32_t k, double stop_)
      {
        p = p_; n = n_; stop = stop_;
        v = p[2 * k + 1];
        next = k + 1;
        read();
        t = ta; vn = va;
        ++next;
        read();
      }
      __device__ __forceinline__ void advance()
      {
        v = vn; t = ta; vn = va;
        ++next;
        read();
      }
    };

    // Parts [part, part + parts) of a pair, each handed to `done` with its sum.
    template <int K, typename F>
    __device__ __forceinline__ void direct_parts(const DirectPair& P, uint32_t part, uint32_t parts, F&& done)
    {
      const uint32_t d = part * P.per;  // breakpoints before the first part
      if (d >= P.nf + P.ng - 1) return;
      // i of them are f's, j are g's
      uint32_t i = d > P.ng - 1 ? d - (P.ng - 1) : 0;
      for (uint32_t hi = min(d, P.nf - 1); i < hi;)
      {
        const uint32_t mid = (i + hi) / 2;
        if (P.f[2 * (mid + 1)] <= P.g[2 * (d - mid)]) i = mid + 1; else hi = mid;
      }
      const uint32_t j = d - i;
      // times >= 0 order as their bits
      uint64_t t = i ? (uint64_t)__double_as_longlong(P.f[2 * i]) : 0;
      if (j) t = max(t, (uint64_t)__double_as_longlong(P.g[2 * j]));
      DirectSide f, g;
      f.start(P.f, P.nf, i, P.stop);
      g.start(P.g, P.ng, j, P.stop);
      const uint64_t stop = (uint64_t)__double_as_longlong(P.stop);
      DirectSum sum;
      for (uint32_t k = 1;; ++k)
      {
        const uint64_t ft = (uint64_t)__double_as_longlong(f.t), gt = (uint64_t)__double_as_longlong(g.t);
        const bool first = ft <= gt;
        const uint64_t tn = first ? ft : gt;
        if (tn != t)
          sum.add(op_f64<K>(f.v, g.v), __longlong_as_double((long long)tn) - __longlong_as_double((long long)t));
        t = tn;
        if (k == P.per || tn == stop)
        {
          done(sum.end());
          if (tn == stop || --parts == 0) break;
          k = 0;
        }
        if (first) f.advance(); else g.advance();
      }
    }

    // The refused pairs of a row, bit l of `redo` for lane l's: this lane's
    // integral, or `res` where it has none of them.  (One call, with all that
    // only refused pairs need inside: two calls in the walk's loop cost it 2 %.)
    template <int K>
    __device__ __noinline__ double walk_again(unsigned redo, const double* f, uint32_t nf, const double* g, uint32_t ng,
                                              uint64_t end, int scale, double res)
    {
      const uint32_t lane = threadIdx.x & 31, steps = 2 * nf;
      // the end's time, rounded up
      const double stop = end == ~0ull ? tmax_of<double>() : ((double)end + 1.0) * pow2(-scale) * (1.0 + 0x1p-50);
      if (__popc(redo) * (12 + steps / 16) > steps)
      {
        if (!(redo >> lane & 1)) return res;
        const DirectPair P(f, nf, g, ng, stop);
        // sums of 2^l neighbours that wait for the next 2^l, as the lanes add
        // them below; parts that are not there are zeros
        double wait[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        uint32_t n = 0;
        auto push = [&](double s) {
          bool carry = true;
#pragma unroll
          for (int l = 0; l < 5; ++l)
            if (carry)
            {
              if (n >> l & 1) s = wait[l] + s;
              else { wait[l] = s; carry = false; }
            }
          if (carry) res = s;
          ++n;
        };
        direct_parts<K>(P, 0, 32, push);
        while (n < 32) push(0.0);
        return res;
      }
      while (redo)
      {
        const int k = __ffs((int)redo) - 1;
        redo &= redo - 1;
        const DirectPair P(f, nf, (const double*)__shfl_sync(FULL, (unsigned long long)g, k), __shfl_sync(FULL, ng, k),
                           __shfl_sync(FULL, stop, k));
        double x = 0.0;
        direct_parts<K>(P, lane, 1, [&](double s) { x = s; });
        __syncwarp();
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) x += __shfl_xor_sync(FULL, x, o);
        if ((int)lane == k) res = x;
      }
      return res;
    }

    // First k in [lo, hi] whose element of this lane's staged column ends
    // after x (STRICT) or at or after x; element hi always does.
    template <bool STRICT>
    __device__ __forceinline__ uint32_t column_find(const unsigned char* col, uint32_t stride, uint32_t lo, uint32_t hi,
                                                    uint64_t x)
    {
      while (lo < hi)
      {
        const uint32_t mid = (lo + hi) >> 1;
        const uint64_t tn = *reinterpret_cast<const uint64_t*>(col + (size_t)mid * stride);
        if (STRICT ? tn > x : tn >= x) hi = mid; else lo = mid + 1;
      }
      return lo;
    }

    // Items, time windows and row pieces as in pairs_window_kernel
    // (pair_kernels.cu): the 32 columns of an item in shared memory, window
    // by window, each warp walking its rows against them.  A PCF that fits
    // the block is one window.  Sums pass from window to window through
    // P.carry, exactly.
    template <int K, typename A>
    __device__ void run_items(const FixedParams& P, const Form& form, unsigned char* smem)
    {
      using V = typename A::V;
      constexpr uint32_t EB = A::BYTES, CS = 32 * EB;  // bytes between a column's elements
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
      __shared__ unsigned long long s_item;
      __shared__ unsigned int s_next_row;
      __shared__ unsigned long long s_bend;
      __shared__ uint32_t s_ck0[32], s_cnt[32], s_cm[32];

      uint32_t* rk0 = reinterpret_cast<uint32_t*>(smem);
      unsigned char* cols = smem + (P.rows_per_item * 4 + 15) / 16 * 16;
      const uint32_t X = fixed_slice_cap(P.smem_bytes - (P.rows_per_item * 4 + 15) / 16 * 16, (uint32_t)nwarps, EB);
      const uint32_t RB = fixed_row_elements(X);
      uint64_t* rt = reinterpret_cast<uint64_t*>(cols + (size_t)X * CS + (size_t)warp * RB * EB);
      V* rv = reinterpret_cast<V*>(rt + RB);
      // this lane's column: element k's time at lcol + k CS, its value vof further
      unsigned char* lcol = cols + (size_t)lane * (sizeof(V) == 4 ? 8 : 16);
      const uint32_t vof = sizeof(V) == 4 ? 256u - 4u * (uint32_t)lane : 8u;
      uint64_t* carry = P.carry + (size_t)blockIdx.x * P.rows_per_item * FIXED_CARRY * 32;

      const uint64_t END = A::end();
      const double unit = pow2(A::scale(form));
      const V* rvals = reinterpret_cast<const V*>(P.r.times + P.r.cap);
      const V* cvals = reinterpret_cast<const V*>(P.c.times + P.c.cap);
      const uint64_t G = ceil_div_u64(P.c.n, 32);

      for (;;)
      {
        if (threadIdx.x == 0) s_item = atomicAdd(P.queue, 1ull);
        __syncthreads();
        if (s_item >= P.n_items) break;
        // from the last item down: in length order a window's longest rows
        // come last, and the longest items are best started first
        const unsigned long long item = P.n_items - 1 - s_item;
        uint64_t c, g;
        if (P.mode == MODE_CROSS) { c = item / G; g = item % G; }
        else tri_decode(item, P.row_begin, P.row_end, P.q, G, &c, &g);
        uint64_t row_lo = P.row_begin + c * 32ull * P.q;
        uint64_t row_hi = row_lo + 32ull * P.q;
        if (row_hi > P.row_end) row_hi = P.row_end;
        const uint64_t col0 = 32ull * g;
        if (P.mode != MODE_CROSS)
        {
          const uint64_t first = col0 + (P.mode == MODE_PDIST ? 1 : 0);
          if (row_lo < first) row_lo = first;
        }
        const uint32_t nrows = row_hi > row_lo ? (uint32_t)(row_hi - row_lo) : 0u;

        // this lane's column; lanes past the last one mirror lane 0's
        const uint64_t cj = col0 + lane;
        const bool cvalid = cj < P.c.n;
        uint64_t corig = P.c.perm ? P.c.perm[cvalid ? cj : col0] : (cvalid ? cj : col0);
        const bool pgood = corig < P.c.n;
        if (!pgood) corig = 0;
        const uint64_t coff = P.c.off[corig];
        const uint32_t cpoints = (uint32_t)(P.c.off[corig + 1] - coff);  // >= 1 (the record)
        const uint32_t clen = P.c.lens[corig];                           // 1 to cpoints, inside the packed arrays
        const uint64_t* ctime = P.c.times + coff;
        const V* cval = cvals + coff;
        const double clast = P.c.pts[2 * (coff + cpoints) - 1];

        if (nrows > 0 && nrows <= P.rows_per_item)
        {
          for (uint32_t r = threadIdx.x; r < nrows; r += blockDim.x) rk0[r] = 0;
          if (threadIdx.x < 32) s_ck0[threadIdx.x] = 0;
          uint64_t Ab = 0;  // the window is [Ab, Be)
          bool first = true;
          for (;;)
          {
            if (threadIdx.x < 32) s_cnt[threadIdx.x] = 0;
            if (threadIdx.x == 0) s_next_row = 0;
            if (warp == 0)
            {
              // the window ends with the earliest X-th element of a column,
              // counted from its first element ending after Ab
              uint32_t k0 = s_ck0[lane];
              while (k0 + 1 < clen && ctime[k0] <= Ab) ++k0;
              s_ck0[lane] = k0;
              uint64_t b = (uint64_t)k0 + X < clen ? ctime[k0 + X - 1] : END;
#pragma unroll
              for (int o = 16; o > 0; o >>= 1)
              {
                const uint64_t y = __shfl_xor_sync(FULL, b, o);
                b = y < b ? y : b;
              }
              if (lane == 0) s_bend = b;
            }
            __syncthreads();
            const uint64_t Be = s_bend;
            const bool last = Be >= END;

            // column slices, cut at the window's end
            {
              const uint32_t k0 = s_ck0[lane];
              const uint32_t avail = min(X, clen - k0);
              uint32_t cnt = 0;
              for (uint32_t k = warp; k < avail; k += nwarps)
              {
                const uint64_t tn = ctime[k0 + k];
                cnt += tn < Be ? 1u : 0u;
                *reinterpret_cast<uint64_t*>(lcol + (size_t)k * CS) = tn < Be ? tn : Be;
                *reinterpret_cast<V*>(lcol + (size_t)k * CS + vof) = cval[k0 + k];
              }
              if (cnt) atomicAdd(&s_cnt[lane], cnt);
            }
            __syncthreads();
            if (warp == 0)
            {
              const uint32_t k0 = s_ck0[lane];
              const uint32_t m = min(s_cnt[lane] + 1u, min(X, clen - k0));
              s_cm[lane] = m;
              s_ck0[lane] = k0 + m - 1;  // reaches the window's end
            }
            __syncthreads();
            const uint32_t cm = s_cm[lane];
            const uint32_t maxmc = __reduce_max_sync(FULL, cm);

            for (;;)
            {
              unsigned r = 0;
              if (lane == 0) r = atomicAdd(&s_next_row, 1u);
              r = __shfl_sync(FULL, r, 0);
              if (r >= nrows) break;
              const uint64_t i = row_lo + r;
              const uint64_t iorig = P.r.perm ? P.r.perm[i] : i;
              if (iorig >= P.r.n) continue;  // a permutation entry out of range: skip the row
              const bool ok =
                  cvalid && pgood && (P.mode == MODE_CROSS || (P.mode == MODE_PDIST ? cj < i : cj <= i));
              if (!__any_sync(FULL, ok)) continue;  // alike in every window
              const uint64_t roff = P.r.off[iorig];
              const uint32_t rpoints = (uint32_t)(P.r.off[iorig + 1] - roff), rlen = P.r.lens[iorig];
              const uint64_t* rtime = P.r.times + roff;
              const V* rval = rvals + roff;

              A acc;
              uint64_t* cslot = carry + (size_t)r * FIXED_CARRY * 32 + lane;
              if (!first) acc.restore(cslot);
              uint32_t k0 = rk0[r], z, m;
              uint64_t Ap = Ab;
              bool first_piece = true;
              for (;;)
              {
                // up to X of the row's elements from k0: z of them end by Ap
                // (skipped), c2 before Be
                uint32_t avail, c2;
                for (;;)
                {
                  avail = min(X, rlen - k0);
                  uint32_t zl = 0, cl = 0;
                  for (uint32_t k = lane; k < avail; k += 32)
                  {
                    const uint64_t e = rtime[k0 + k];
                    rv[k] = rval[k0 + k];
                    rt[k] = e;
                    zl += e <= Ap ? 1u : 0u;
                    cl += e < Be ? 1u : 0u;
                  }
                  z = __reduce_add_sync(FULL, zl);
                  c2 = __reduce_add_sync(FULL, cl);
                  if (z < avail) break;
                  k0 += avail;  // all of them end by Ap; the last element of a row ends at END
                  __syncwarp();
                }
                const bool full = c2 + 1 <= avail;  // the piece reaches Be
                m = full ? (c2 + 1 > z ? c2 + 1 - z : 1u) : avail - z;
                __syncwarp();
                const uint64_t Bp = full ? Be : rt[avail - 1];
                const V vlast = rv[z + m - 1];
                __syncwarp();
                if (lane <= U)  // z + m + U <= X + U < RB
                {
                  rv[z + m - 1 + lane] = vlast;
                  rt[z + m - 1 + lane] = Bp;
                }
                __syncwarp();
                // this lane's column elements meeting [Ap, Bp)
                uint32_t g0 = 0, g1 = cm - 1;
                if (!first_piece) g0 = column_find<true>(lcol, CS, 0, g1, Ap);
                if (!full) g1 = column_find<false>(lcol, CS, g0, g1, Bp);
                const uint32_t ncol = (first_piece && full) ? maxmc : __reduce_max_sync(FULL, g1 - g0 + 1);
                walk(acc, rt + z, rv + z, (uint32_t)__cvta_generic_to_shared(lcol) + g0 * CS, vof, m, m + ncol - 1, Ap);
                __syncwarp();
                if (full) break;
                k0 += z + m;
                Ap = Bp;
                first_piece = false;
              }
              if (lane == 0) rk0[r] = k0 + z + m - 1;  // the element reaching Be starts the next window
              if (!last)
              {
                acc.save(cslot);
                continue;
              }

              const double* rpts = P.r.pts + 2 * roff;
              double res = acc.value() * unit;
              // the last rectangle, to the largest double, where the PCFs'
              // last values leave something of it
              const double rlast = rpts[2 * rpoints - 1];
              if (__any_sync(FULL, ((__double_as_longlong(rlast) | __double_as_longlong(clast)) << 1) != 0))
              {
                const double tail = op_f64<K>(rlast, clast);
                if (tail != 0.0) res = fma(tail, tmax_of<double>(), res);
              }
              // The time from which every term is 0: of products where a side
              // whose last value is 0 changes last, of distances where the
              // later side does, if the last values are alike; else `none`.
              const auto end = [&](bool later_change) -> uint64_t {
                const uint64_t Tr = rlen > 1 ? A::units(rtime[rlen - 2]) : 0, Tc = clen > 1 ? A::units(ctime[clen - 2]) : 0;
                const uint64_t none = later_change ? (Tr > Tc ? Tr : Tc) : ~0ull;
                if (K != OPK_INNER) return rlast == clast ? (Tr > Tc ? Tr : Tc) : none;
                if (rlast == 0.0 && clast == 0.0) return Tr < Tc ? Tr : Tc;
                return rlast == 0.0 ? Tr : clast == 0.0 ? Tc : none;
              };
              const Shape rshape = P.r.shapes[iorig], cshape = P.c.shapes[corig];
              const unsigned redo =
                  __ballot_sync(FULL, ok && !acc.good(rshape, cshape, A::DROPS ? end(true) : 0));
              if (redo)
              {
                res = walk_again<K>(redo, rpts, rpoints, P.c.pts + 2 * coff, cpoints, end(false), form.s, res);
                __syncwarp();
              }
              if (ok)
              {
                if (K == OPK_L2DIST) res = sqrt(res);
                const uint64_t idx = P.mode == MODE_CROSS ? iorig * P.ld + corig : condensed_index(P.mode, iorig, corig);
                const uint64_t rel = idx - P.out_base;  // wraps for idx < out_base
                if (rel < P.out_count) P.out[rel] = res;
              }
            }
            __syncthreads();
            if (last) break;
            Ab = Be;
            first = false;
          }
        }
        __syncthreads();
      }
    }

    template <int K>
    __global__ void __launch_bounds__(FIXED_WARPS * 32, 1) fixed_pairs_kernel(const __grid_constant__ FixedParams P)
    {
      extern __shared__ __align__(16) unsigned char smem_raw[];
      const Form f = form_of(*P.rec, K);
      if (f.kind != 0 && mostly_refused(*P.rec, K))
      {
        // the direct kernel behind this one: its gate, and the elements it
        // reads in the packed arrays' place (launches of other bands may do
        // the same meanwhile, and write the same)
        if (blockIdx.x == 0 && threadIdx.x == 0) *P.gate = 0;
        if (!P.elements) return;
        const uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
        const uint64_t nw = (gridDim.x * (uint64_t)blockDim.x) >> 5;
        for (const FixedSet* s : {&P.r, &P.c})
        {
          if (s == &P.c && P.mode != MODE_CROSS) break;
          for (uint64_t i = w; i < s->n; i += nw)
            write_elements(s->pts, s->off[i], s->off[i + 1] - s->off[i], (Elem<double>*)s->times, threadIdx.x & 31);
        }
        return;
      }
      if (f.kind == 1)
      {
        if (K == OPK_INNER && f.sign) run_items<K, Counts<K, K == OPK_INNER>>(P, f, smem_raw);
        else run_items<K, Counts<K, false>>(P, f, smem_raw);
      }
      else if (f.kind == 2)
      {
        if (K == OPK_INNER && f.sign) run_items<K, General<K, K == OPK_INNER>>(P, f, smem_raw);
        else run_items<K, General<K, false>>(P, f, smem_raw);
      }
    }
  }

  // ---- launchers ----------------------------------------------------------------

  cudaError_t launch_fixed_record(const double* pts, const uint64_t* off, uint64_t n, uint64_t cap, uint32_t longest,
                                  FixedRecord* rec, int sms, cudaStream_t st)
  {
    if (n == 0) return cudaSuccess;
    const unsigned blocks = (unsigned)std::min<uint64_t>((n + 7) / 8, (uint64_t)sms * 8);
    fixed_record_kernel<<<blocks, 256, 0, st>>>(pts, off, n, cap, longest, rec);
    return launched();
  }

  cudaError_t launch_fixed_pack(const double* pts, const uint64_t* off, uint64_t n, uint64_t cap,
                                FixedRecord* rec, int opk, void* packed, Shape* shapes, uint32_t* lens,
                                bool elements, unsigned* gate, int sms, cudaStream_t st)
  {
    if (n == 0) return cudaSuccess;
    const unsigned blocks = (unsigned)std::min<uint64_t>((n + 7) / 8, (uint64_t)sms * 8);
    fixed_pack_kernel<<<blocks, 256, 0, st>>>(pts, off, n, cap, rec, opk, packed, shapes, lens, elements, gate);
    return launched();
  }

  cudaError_t launch_fixed_pairs(const FixedParams& P, int opk, int warps, int grid, cudaStream_t st)
  {
    void (*fn)(const FixedParams) = opk == OPK_L1       ? fixed_pairs_kernel<OPK_L1>
                                    : opk == OPK_L2DIST ? fixed_pairs_kernel<OPK_L2DIST>
                                    : opk == OPK_INNER  ? fixed_pairs_kernel<OPK_INNER>
                                                        : nullptr;
    if (!fn) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P.smem_bytes);
    if (e != cudaSuccess) return e;
    fn<<<grid, warps * 32, P.smem_bytes, st>>>(P);
    return launched();
  }
}
