// Gradients of the float32 L2 kernel and L2 distances as a contraction (sm_103a).
//
// Both gradients see the other PCFs only through one weighted sum,
//   H_i(t) = sum over j of w_ij g_j(t)      (w = dL/dK, or dL/dD / D; S_i = sum of w_ij)
// for PCF i with value v_k on [t_k, t_{k+1}):
//   L2 kernel    dL/dv_k = integral of H_i over the segment
//                dL/dt_k = (v_{k-1} - v_k) H_i(t_k)
//   L2 distance  dL/dv_k = integral of v_k S_i - H_i
//                dL/dt_k = (v_{k-1} - v_k) ((v_{k-1} + v_k) / 2 S_i - H_i(t_k))
// (PCFs with a breakpoint at t_k itself drop out of the time gradient, as in
// the walks of backward.cu, which merge every pair instead.)  Time is cut
// into bins at quantiles of the breakpoints; then
//   * H_i at the bin edges and its integral over whole bins are one matrix
//     product, W (n x n) times the PCFs' edge values and bin integrals
//     (n x 2 bins), in FP32 FMAs;
//   * inside a bin, at a breakpoint t_k of i, H_i adds w_ij times the steps of
//     the other PCFs between the edge and t_k: a list of the bin's breakpoints
//     against the breakpoints of i that lie there.  Its integral is taken over
//     a segment's own part of the bin, not as a difference of two from the
//     edge, which would keep the rounding of the whole bin in a segment of a
//     thousandth of it; and in the last bin from its end, where H is that of
//     zeros, since little is left there of what the edge's value sums.
// Work per PCF pair falls from the merge's 2 L steps, with an atomic each, to
// 2 bins FMAs and L^2 / bins list entries.  Nothing is added atomically, and
// the sums are shorter.  N = 4096, L ~ U{16..512}, L2 kernel, forward and
// backward: 14.4 -> 4.8 ms (the forward is 2.4 of it), error of the gradient
// 8.5e-7 -> 2.5e-7; of each value's gradient against the sum of its own
// |terms|, N = 1000, segments from a millionth of a time unit on: rms 1.2e-8 to
// 1.4e-8 over the first three quarters of the time and 3e-8 to 1.4e-7 behind,
// 2.1e-8 in the walk (with differences from the edge up to 20, rms 5e-2).
//
// For distances each bin's mean value over the PCFs is taken off first: only
// differences count there, and sums of w_ij g_j then stay as small as them.
// Pairs that lie close together beside that are left to the walk (l2_close).
//
// A weight or a value that is not finite, a last value other than 0 (its
// integral has no end), times out of order or a gradient that comes out not
// finite make the walk of backward.cu run instead, decided by a record on
// the device.
#include "sbg_internal.hpp"

#include "backward_l2.cuh"

#include <algorithm>
#include <cmath>

namespace sbg
{
  namespace
  {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr uint32_t SAMPLES = 8192;  // breakpoint times the bin edges come from
    constexpr int ROWS_MAX = 32;        // rows of a near-field CTA (one lane each)
    constexpr int NEAR_THREADS = 1024;
    constexpr int BATCH = 2;            // breakpoints a warp sums for at once
    constexpr int AHEAD = 4;            // list entries a lane has in flight
    constexpr uint32_t BIN_MAX = 8192;  // breakpoints of a bin

    // A time >= 0 as bits that order like it (-0, which passes for 0 in every
    // comparison of times, would order above them all).
    __device__ __forceinline__ uint32_t time_bits(float t) { return t > 0.0f ? __float_as_uint(t) : 0u; }

    // Times from the second breakpoint on (the first is the start whatever it
    // says) must not descend from 0.  The breakpoints behind elements without
    // width are listed, for l2_narrow_kernel: up to n of them, more make the
    // data the walk's.
    __global__ void __launch_bounds__(256) l2_record_kernel(const float* __restrict__ pts,
                                                            const uint64_t* __restrict__ off, uint64_t n,
                                                            uint64_t npts, L2Record* rec,
                                                            uint32_t* __restrict__ narrow)
    {
      const int lane = threadIdx.x & 31;
      const uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
      const uint64_t nw = (gridDim.x * (uint64_t)blockDim.x) >> 5;
      uint32_t tmax = 0, bad = 0;
      for (uint64_t i = w; i < n; i += nw)
      {
        const uint64_t o = off[i], e = off[i + 1];
        if (e <= o || e > npts) { bad = 1; continue; }
        const uint64_t len = e - o;
        for (uint64_t k = lane; k < len; k += 32)
        {
          const float v = pts[2 * (o + k) + 1];
          bad |= !isfinite(v) || (k + 1 == len && v != 0.0f) || (k == 0 && pts[2 * o] != 0.0f) ? 1u : 0u;
          if (k > 0)
          {
            const float t = pts[2 * (o + k)], before = k > 1 ? pts[2 * (o + k - 1)] : 0.0f;
            bad |= !(t >= before) || !(t < FLT_MAX) ? 1u : 0u;
            if (t == before)
            {
              const uint32_t at = atomicAdd(&rec->narrow, 1u);
              if (at < n) narrow[at] = (uint32_t)(o + k);
              else bad = 1;
            }
            tmax = max(tmax, time_bits(t));
          }
        }
      }
      tmax = __reduce_max_sync(FULL, tmax);
      bad = __reduce_or_sync(FULL, bad);
      if (lane == 0)
      {
        if (bad) atomicOr(&rec->bad, 1u);
        atomicMax(&rec->tmax_bits, tmax);
      }
    }

    // Bin edges: quantiles of a sample of the breakpoint times, sorted in
    // shared memory by one CTA; edge 0 is time 0, edge `bins` the last time.
    // Only points that the offsets cover: what stands behind them may be
    // anything, and a NaN would leave the edges out of order.  One point out
    // of each of 8192 equal stretches, at a fraction that runs through [0, 1)
    // in steps of the golden ratio: at a fixed place, PCFs of one length are
    // sampled at the same few of their breakpoints (N = 4096, L = 264: two),
    // whose quantiles leave bins too full to sort.
    __global__ void __launch_bounds__(1024) l2_edges_kernel(const float* __restrict__ pts,
                                                            const uint64_t* __restrict__ off, uint64_t n,
                                                            const L2Record* __restrict__ rec, uint32_t bins,
                                                            float* __restrict__ edges)
    {
      __shared__ float s[SAMPLES];
      if (rec->bad) return;
      const uint64_t o = off[0], covered = off[n] - o;
      for (uint32_t q = threadIdx.x; q < SAMPLES; q += 1024) s[q] = pts[2 * (o + (q * covered + ((uint64_t)(q * 0x9e3779b9u) * covered >> 32)) / SAMPLES)];
      // a stage at distance 32 or less stays within the 64 elements of a warp
      uint32_t before = 64;  // the loads cross warps
      for (uint32_t k = 2; k <= SAMPLES; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1)
        {
          if (j >= 64 || before >= 64) __syncthreads(); else __syncwarp();
#pragma unroll
          for (uint32_t u = 0; u < SAMPLES / 2048; ++u)
          {
            const uint32_t t = threadIdx.x + u * 1024, i = ((t & ~(j - 1)) << 1) | (t & (j - 1));
            const float a = s[i], b = s[i + j];
            if ((a > b) == ((i & k) == 0)) { s[i] = b; s[i + j] = a; }
          }
          before = j;
        }
      __syncthreads();
      const float last = __uint_as_float(rec->tmax_bits);
      for (uint32_t b = threadIdx.x; b <= bins; b += 1024)
        edges[b] = b == 0 ? 0.0f : b == bins ? last : fminf(fmaxf(s[(uint64_t)b * SAMPLES / bins], 0.0f), last);
    }

    // The last bin whose edge is at or before t.
    __device__ __forceinline__ uint32_t bin_of(const float* edges, uint32_t bins, float t)
    {
      uint32_t lo = 0, hi = bins;
      while (hi - lo > 1)
      {
        const uint32_t mid = (lo + hi) >> 1;
        if (edges[mid] <= t) lo = mid; else hi = mid;
      }
      return lo;
    }

    // Counts (FILL = false) or files the breakpoints by bin: a key of the time
    // and the point's index; each point's bin and PCF.
    template <bool FILL>
    __global__ void __launch_bounds__(512) l2_bins_kernel(const float* __restrict__ pts,
                                                          const uint64_t* __restrict__ off, uint64_t n,
                                                          const L2Record* __restrict__ rec, uint32_t bins,
                                                          const float* __restrict__ edges, uint32_t* __restrict__ counts,
                                                          uint64_t* __restrict__ keys, uint16_t* __restrict__ bin,
                                                          uint16_t* __restrict__ owner)
    {
      extern __shared__ float smem[];
      if (rec->bad) return;
      float* se = smem;
      uint32_t* count = reinterpret_cast<uint32_t*>(se + bins);
      uint32_t* place = count + bins;
      for (uint32_t b = threadIdx.x; b < bins; b += blockDim.x)
      {
        se[b] = edges[b];
        count[b] = 0;
      }
      __syncthreads();
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
      const uint64_t i0 = n * blockIdx.x / gridDim.x, i1 = n * (blockIdx.x + 1) / gridDim.x;
      for (uint64_t i = i0 + warp; i < i1; i += nwarps)
      {
        const uint64_t o = off[i], len = off[i + 1] - o;
        for (uint64_t k = 1 + lane; k < len; k += 32)
        {
          uint32_t b;
          if (FILL) b = bin[o + k];
          else
          {
            b = bin_of(se, bins, pts[2 * (o + k)]);
            bin[o + k] = (uint16_t)b;
            owner[o + k] = (uint16_t)i;
          }
          atomicAdd(&count[b], 1u);
        }
      }
      __syncthreads();
      // the counting kernel adds to the totals, the filing one takes its places
      for (uint32_t b = threadIdx.x; b < bins; b += blockDim.x)
        if (count[b])
        {
          const uint32_t base = atomicAdd(&counts[b], count[b]);
          if (FILL) place[b] = base;
        }
      if (!FILL) return;
      __syncthreads();
      for (uint64_t i = i0 + warp; i < i1; i += nwarps)
      {
        const uint64_t o = off[i], len = off[i + 1] - o;
        for (uint64_t k = 1 + lane; k < len; k += 32)
          keys[atomicAdd(&place[bin[o + k]], 1u)] =
              ((uint64_t)time_bits(pts[2 * (o + k)]) << 32) | (uint32_t)(o + k);
      }
    }

    // One bin's breakpoints in order of time (and of the point, at equal
    // times): a bitonic network in shared memory.  A bin of more than
    // BIN_MAX breakpoints (many at one time, which no edge can part) sends
    // the call to the walk.
    __global__ void __launch_bounds__(512) l2_sort_kernel(const float* __restrict__ pts, L2Record* __restrict__ rec,
                                                          const uint32_t* __restrict__ starts,
                                                          const uint64_t* __restrict__ keys,
                                                          const uint16_t* __restrict__ owner, L2Lists lists)
    {
      extern __shared__ uint64_t sk[];
      if (rec->bad) return;
      const uint32_t e0 = starts[blockIdx.x], m = starts[blockIdx.x + 1] - e0;
      if (m > BIN_MAX)
      {
        if (threadIdx.x == 0) atomicOr(&rec->bad_weights, 1u);
        return;
      }
      if (blockIdx.x + 1 == gridDim.x)  // the spare entries that the sums read past the last list
        for (uint32_t x = threadIdx.x; x < 32 * AHEAD; x += blockDim.x)
        {
          lists.event[e0 + m + x] = make_float2(0.0f, 0.0f);
          lists.pcf[e0 + m + x] = 0;
        }
      uint32_t size = 2;
      while (size < m) size <<= 1;
      for (uint32_t x = threadIdx.x; x < size; x += blockDim.x) sk[x] = x < m ? keys[e0 + x] : ~0ull;
      // a stage at distance 32 or less stays within the 64 elements of a warp
      uint32_t before = 64;  // the loads cross warps
      for (uint32_t k = 2; k <= size; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1)
        {
          if (j >= 64 || before >= 64) __syncthreads(); else __syncwarp();
          for (uint32_t t = threadIdx.x; t < size / 2; t += blockDim.x)
          {
            const uint32_t i = ((t & ~(j - 1)) << 1) | (t & (j - 1));
            const uint64_t a = sk[i], b = sk[i + j];
            if ((a > b) == ((i & k) == 0)) { sk[i] = b; sk[i + j] = a; }
          }
          before = j;
        }
      __syncthreads();
      for (uint32_t x = threadIdx.x; x < m; x += blockDim.x)
      {
        const uint64_t key = sk[x];
        const uint32_t pt = (uint32_t)key;
        lists.event[e0 + x] = make_float2(__uint_as_float((uint32_t)(key >> 32)), pts[2 * (uint64_t)pt + 1] - pts[2 * (uint64_t)pt - 1]);
        lists.pcf[e0 + x] = owner[pt];
        lists.point[e0 + x] = pt;
        lists.place[pt] = e0 + x;
      }
    }

    // counts -> starts (bins + 1 of them), and a copy that the filing advances
    __global__ void __launch_bounds__(1024) l2_starts_kernel(const uint32_t* __restrict__ counts, uint32_t bins,
                                                             uint32_t* __restrict__ starts, uint32_t* __restrict__ next)
    {
      __shared__ uint32_t part[1024];
      const uint32_t per = (bins + 1023) / 1024, b0 = threadIdx.x * per, b1 = min(bins, b0 + per);
      uint32_t sum = 0;
      for (uint32_t b = b0; b < b1; ++b) sum += counts[b];
      part[threadIdx.x] = sum;
      __syncthreads();
      for (uint32_t d = 1; d < 1024; d <<= 1)
      {
        const uint32_t x = threadIdx.x >= d ? part[threadIdx.x - d] : 0;
        __syncthreads();
        part[threadIdx.x] += x;
        __syncthreads();
      }
      uint32_t at = part[threadIdx.x] - sum;
      for (uint32_t b = b0; b < b1; ++b)
      {
        starts[b] = at;
        next[b] = at;
        at += counts[b];
      }
      if (threadIdx.x == 1023) starts[bins] = part[1023];
    }

    // First breakpoint k >= 1 of a PCF at or after t (len if none).
    __device__ __forceinline__ uint32_t first_from(const float* p, uint32_t len, float t)
    {
      uint32_t lo = 1, hi = len;
      while (lo < hi)
      {
        const uint32_t mid = (lo + hi) >> 1;
        if (p[2 * (uint64_t)mid] < t) lo = mid + 1; else hi = mid;
      }
      return lo;
    }

    // A bin's mean value just before its edge, over up to 256 PCFs.
    __global__ void __launch_bounds__(256) l2_centres_kernel(const float* __restrict__ pts,
                                                             const uint64_t* __restrict__ off, uint64_t n,
                                                             const L2Record* __restrict__ rec,
                                                             const float* __restrict__ edges, float* __restrict__ centre)
    {
      __shared__ float part[8];
      if (rec->bad) return;
      const uint64_t m = n < 256 ? n : 256;
      float v = 0.0f;
      if (threadIdx.x < m)
      {
        const uint64_t j = threadIdx.x * n / m, o = off[j];
        const uint32_t len = (uint32_t)(off[j + 1] - o);
        v = pts[2 * (o + first_from(pts + 2 * o, len, edges[blockIdx.x]) - 1) + 1] / (float)m;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
      if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
      __syncthreads();
      if (threadIdx.x == 0)
      {
        float c = 0.0f;
        for (int w = 0; w < 8; ++w) c += part[w];
        centre[blockIdx.x] = c;
      }
    }

    // Row j of the table: the PCF just before every edge, then its integral
    // over every bin, each less the bin's centre.  One warp per PCF; rows
    // from n on are zero.
    __global__ void __launch_bounds__(256) l2_table_kernel(const float* __restrict__ pts,
                                                           const uint64_t* __restrict__ off, uint64_t n, uint64_t rows,
                                                           const L2Record* __restrict__ rec, uint32_t bins,
                                                           const float* __restrict__ edges,
                                                           const float* __restrict__ centre, float* __restrict__ table,
                                                           float* __restrict__ norm)
    {
      if (rec->bad) return;
      const uint64_t j = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
      const int lane = threadIdx.x & 31;
      if (j >= rows) return;
      float* out = table + j * 2 * bins;
      const uint64_t o = j < n ? off[j] : 0;
      const uint32_t len = j < n ? (uint32_t)(off[j + 1] - o) : 0;
      const float* p = pts + 2 * o;
      float square = 0.0f;
      for (uint32_t b = lane; b < bins; b += 32)
      {
        float v = 0.0f, area = 0.0f;
        if (j < n)
        {
          const float lo = edges[b], hi = edges[b + 1], c = centre ? centre[b] : 0.0f;
          uint32_t k = first_from(p, len, lo);
          v = p[2 * (uint64_t)(k - 1) + 1] - c;
          float cur = v, at = lo;
          for (; k < len; ++k)
          {
            const float t = p[2 * (uint64_t)k];
            if (!(t < hi)) break;
            area = fmaf(cur, t - at, area);
            square = fmaf(cur * cur, t - at, square);
            cur = p[2 * (uint64_t)k + 1] - c;
            at = t;
          }
          area = fmaf(cur, hi - at, area);
          square = fmaf(cur * cur, hi - at, square);
        }
        out[b] = v;
        out[bins + b] = area;
      }
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) square += __shfl_xor_sync(FULL, square, d);
      if (lane == 0 && j < n) norm[j] = sqrtf(square);
    }

    // Weights of rows [r0, r0 + width) as columns: wt[j][i - r0] = w_ij, 0 on
    // the diagonal and past n.  Tiles of 32 x 32; the condensed entry of (j, i)
    // lies in row max(i, j), so tiles above the diagonal go through shared
    // memory.
    __global__ void __launch_bounds__(256) l2_weights_kernel(const float* __restrict__ g, const float* __restrict__ fwd,
                                                             const float* __restrict__ norm, uint64_t n, bool diag,
                                                             uint64_t r0, uint64_t width, uint64_t rows,
                                                             float* __restrict__ wt, L2Record* rec)
    {
      __shared__ float tile[32][33];
      if (rec->bad) return;  // bad_weights may change while this runs
      const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
      const uint64_t tj = (uint64_t)blockIdx.y * 32, ti = r0 + (uint64_t)blockIdx.x * 32;
      bool bad = false, close = false;
      auto entry = [&](uint64_t a, uint64_t b) {  // a > b
        if (a >= n || b >= n || a <= b) return 0.0f;
        const uint64_t at = diag ? a * (a + 1) / 2 + b : a * (a - 1) / 2 + b;
        float w = g[at];
        if (fwd)
        {
          const float d = fwd[at];
          w = d > 0.0f ? w / d : 0.0f;
          if (w != 0.0f && l2_close(d, norm[a], norm[b]))
          {
            close = true;
            return 0.0f;
          }
        }
        bad |= !isfinite(w);
        return w;
      };
      if (tj > ti)  // rows j below: read along i
      {
        for (int y = ty; y < 32; y += 8)
          if (tj + y < rows) wt[(tj + y) * width + (ti - r0) + tx] = entry(tj + y, ti + tx);
      }
      else
      {
        for (int y = ty; y < 32; y += 8) tile[y][tx] = entry(ti + y, tj + tx);
        __syncthreads();
        for (int y = ty; y < 32; y += 8)
        {
          const uint64_t j = tj + y, i = ti + tx;
          float w = tile[tx][y];  // of (i, j), i > j
          if (tj == ti && j > i) w = tile[y][tx];
          if (j < rows) wt[j * width + (i - r0)] = w;
        }
      }
      if (__any_sync(FULL, bad) && tx == 0) atomicOr(&rec->bad_weights, 1u);
      if (__any_sync(FULL, close) && tx == 0) atomicOr(&rec->close, 1u);
    }

    // ---- C (m x c) = A^T (A: k x m) B (k x c), FP32 ---------------------------------
    //
    // 128 x 128 tiles, 8 x 8 results per thread, operands staged 16 deep with
    // cp.async through four buffers (both are k-major, so tiles copy
    // straight), packed FMAs (two columns per instruction: 32 of them and 12
    // other instructions a k-step instead of 64 and 4).  Bound by the FMA
    // pipe: 28.9 T FMA/s of 39.4 at 4096 x 1792 x 4096.  Sums of 256 terms go
    // to a second set of registers: the rounding of one chain grows with the
    // root of its length.
    constexpr int GT = 128, GK = 16, GS = 4;

    __device__ __forceinline__ void copy16(void* smem, const void* gmem)
    {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem));
    }

    __global__ void __launch_bounds__(256, 1) l2_product_kernel(const float* __restrict__ A, uint64_t m,
                                                                const float* __restrict__ B, uint64_t c, uint64_t k,
                                                                const L2Record* __restrict__ rec, float* __restrict__ C)
    {
      extern __shared__ __align__(16) float smem[];
      if (rec->bad | rec->bad_weights) return;
      float* sa = smem;
      float* sb = smem + GS * GK * GT;
      const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
      const uint64_t m0 = (uint64_t)blockIdx.y * GT, c0 = (uint64_t)blockIdx.x * GT;
      const int steps = (int)(k / GK);
      auto stage = [&](int s) {
        if (s < steps)
        {
          float* da = sa + (s % GS) * GK * GT;
          float* db = sb + (s % GS) * GK * GT;
#pragma unroll
          for (int q = 0; q < 2; ++q)
          {
            const int at = tid + q * 256, row = at >> 5, col = (at & 31) * 4;
            copy16(da + row * GT + col, A + ((uint64_t)s * GK + row) * m + m0 + col);
            copy16(db + row * GT + col, B + ((uint64_t)s * GK + row) * c + c0 + col);
          }
        }
        asm volatile("cp.async.commit_group;");
      };
      uint64_t acc[8][4], total[8][4];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = total[i][j] = 0;
#pragma unroll
      for (int s = 0; s < GS - 1; ++s) stage(s);
      for (int s = 0; s < steps; ++s)
      {
        asm volatile("cp.async.wait_group %0;" ::"n"(GS - 2));
        __syncthreads();
        stage(s + GS - 1);
        const float* pa = sa + (s % GS) * GK * GT + ty * 4;
        const float* pb = sb + (s % GS) * GK * GT + tx * 4;
#pragma unroll
        for (int u = 0; u < GK; ++u)
        {
          float4 a0 = *reinterpret_cast<const float4*>(pa + u * GT), a1 = *reinterpret_cast<const float4*>(pa + u * GT + 64);
          const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(pb + u * GT),
                           b1 = *reinterpret_cast<const ulonglong2*>(pb + u * GT + 64);
          const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
          const uint64_t b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
          for (int i = 0; i < 8; ++i)
          {
            uint64_t aa;
            asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a[i]));
#pragma unroll
            for (int j = 0; j < 4; ++j) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(aa), "l"(b[j]));
          }
        }
        if (s % (256 / GK) == 256 / GK - 1 || s + 1 == steps)
        {
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
            {
              asm("add.rn.f32x2 %0, %0, %1;" : "+l"(total[i][j]) : "l"(acc[i][j]));
              acc[i][j] = 0;
            }
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
      {
        float* out = C + (m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4)) * c + c0 + tx * 4;
        *reinterpret_cast<ulonglong2*>(out) = make_ulonglong2(total[i][0], total[i][1]);
        *reinterpret_cast<ulonglong2*>(out + 64) = make_ulonglong2(total[i][2], total[i][3]);
      }
    }

    // ---- inside the bins, and the gradient ------------------------------------------
    //
    // One CTA per group of up to 32 rows, whose weights lie in shared memory.
    // A warp takes a bin and the rows' breakpoints in it (lane r: row r), two
    // at a time: the bin's list up to a breakpoint's own place, weight times
    // step (H), weight times step times distance, at most the element's part of
    // the bin (its integral there).  Behind a row's last breakpoint of a bin lies
    // what its elements leave of the whole bin's integral, or, of a quarter or
    // less, the rest of the list.  Then each element's gradient from its parts
    // and the whole bins between.
    // Bound by the list reads from L2 (the weights leave L1 no room for the
    // lists) and the gathers from shared memory: 1.4 ms at N = 4096, L ~
    // U{16..512}, 576 bins.  Two breakpoints share a read; four waste as much
    // on the shorter prefixes (5.00 against 5.08 ms forward and backward),
    // one reads 14 GB (1.17 ms at 896 bins, L2 at 12 TB/s).  Unsorted lists
    // with a compare per entry took 1.75 ms at 896 bins.
    template <bool KERNEL>
    __global__ void __launch_bounds__(NEAR_THREADS, 1) l2_gradient_kernel(const __grid_constant__ L2Gradient P)
    {
      extern __shared__ __align__(16) float smem[];
      __shared__ unsigned int s_bin;
      __shared__ float s_sum[ROWS_MAX];
      __shared__ uint32_t s_row[ROWS_MAX];
      // bad_weights may be set by another CTA meanwhile: one answer for all threads
      if (threadIdx.x == 0) s_bin = P.rec->bad | P.rec->bad_weights;
      __syncthreads();
      if (s_bin) return;
      __syncthreads();
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = NEAR_THREADS / 32;
      const uint32_t n = (uint32_t)P.n;
      // Row r of group g is the (g + r groups)-th PCF in length order: the
      // groups' lengths even out (consecutive PCFs left a fifth of the SM
      // time idle at the end).
      const uint32_t span = (uint32_t)(min(P.r0 + P.width, P.n) - P.r0);
      uint32_t rows = 0;
      if (threadIdx.x == 0) s_bin = 0;
      for (uint32_t at = blockIdx.x; at < span && rows < P.rows; at += gridDim.x, ++rows)
        if (threadIdx.x == 0) s_row[rows] = P.order[P.r0 + at];
      __syncthreads();
      // weights: row r of the group at [r n + j].  With all rows in one
      // product the weights are symmetric, and a row is contiguous.
      for (uint32_t r = 0; r < rows; ++r)
      {
        const uint64_t i = s_row[r];
        if (P.n <= P.width)
          for (uint32_t j = threadIdx.x; j < n; j += NEAR_THREADS) smem[(size_t)r * n + j] = P.wt[i * P.width + j];
        else
          for (uint32_t j = threadIdx.x; j < n; j += NEAR_THREADS)
            smem[(size_t)r * n + j] = P.wt[(uint64_t)j * P.width + (i - P.r0)];
      }
      __syncthreads();
      if (!KERNEL)
      {
        for (uint32_t r = warp; r < rows; r += nwarps)
        {
          float s = 0.0f;
          for (uint32_t j = lane; j < n; j += 32) s += smem[(size_t)r * n + j];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
          if (lane == 0) s_sum[r] = s;
        }
        __syncthreads();
      }

      // Some gradient is not finite.  A sum over all PCFs multiplies what
      // overflows (one PCF's integral over a bin, say) by weights of 0 too,
      // which the walk leaves out.
      bool lost = false;

      // One breakpoint, from H at the bin's edge and its bin's sums: H there,
      // its time gradient, and the integral of H over the last `width` before
      // it (area: the part of the bin's list).  Returns that integral.
      auto finish = [&](uint32_t b, uint32_t e0, uint32_t e1, float h0, float width, uint32_t r, uint32_t k, uint32_t at, float t,
                        float h, float area) {
        const uint64_t i = s_row[r], o = P.off[i];
        const float* w = smem + (size_t)r * n;
        const float centre = KERNEL ? 0.0f : P.centre[b];
        float H = h0 + h, sum = KERNEL ? 0.0f : s_sum[r];
        if ((at > e0 && P.lists.event[at - 1].x == t) || (at + 1 < e1 && P.lists.event[at + 1].x == t))
        {
          // other breakpoints at the same time: their PCFs drop out, with
          // the value that H holds of them, after those in front of this
          // one, before those behind it (a PCF's own points stand together,
          // and its own weight is 0)
          float hw = 0.0f, ww = 0.0f;
          for (int side = 0; side < 2; ++side)
            for (uint32_t x = 1 + lane;; x += 32)
            {
              const bool in = side == 0 ? at >= e0 + x : at + x < e1;
              const uint32_t e = in ? (side == 0 ? at - x : at + x) : at;
              const bool tied = in && P.lists.event[e].x == t;
              if (tied)
              {
                const uint32_t j = P.lists.pcf[e], pt = P.lists.point[e];
                const bool counts = side == 0 ? pt + 1 == P.off[j + 1] || P.pts[2 * ((uint64_t)pt + 1)] != t
                                              : pt == P.off[j] + 1 || P.pts[2 * ((uint64_t)pt - 1)] != t;
                if (counts)
                {
                  hw = fmaf(w[j], P.pts[2 * (uint64_t)pt + (side == 0 ? 1 : -1)] - centre, hw);
                  ww += w[j];
                }
              }
              if (!__all_sync(FULL, tied)) break;
            }
#pragma unroll
          for (int d = 16; d > 0; d >>= 1)
          {
            hw += __shfl_xor_sync(FULL, hw, d);
            ww += __shfl_xor_sync(FULL, ww, d);
          }
          H -= hw;
          sum -= ww;
        }
        if (lane == 0)
        {
          const float a = P.pts[2 * (o + k) - 1], c = P.pts[2 * (o + k) + 1];
          float dt = KERNEL ? (a - c) * H : (a - c) * ((0.5f * ((a - centre) + (c - centre))) * sum - H);
          if (KERNEL) dt = fmaf(P.grad_out[i * (i + 1) / 2 + i], (a - c) * (a + c), dt);
          P.grad[2 * (o + k)] = dt;
          P.area[o + k] = fmaf(h0, width, area);
          lost |= !isfinite(dt);
        }
        return fmaf(h0, width, area);
      };
      // A row's last breakpoint of a bin (its h as above): the integral of H
      // from it to the bin's end.  What is left of the whole bin's, or, where
      // that is less than a quarter and would keep the rounding of all of it,
      // the entries from the breakpoint on.
      auto finish_bin = [&](uint32_t b, uint32_t e1, float edge, float hi, uint32_t r, uint32_t k, uint32_t at, float t,
                            float h, float before) {
        const uint64_t i = s_row[r];
        const float* product = P.product + (i - P.r0) * 2 * P.bins;
        float rest = product[P.bins + b] - before;
        if (hi - t < 0.25f * (hi - edge))
        {
          const float* w = smem + (size_t)r * n;
          rest = 0.0f;
          for (uint32_t c0 = at + 1 + lane; c0 < e1 + lane; c0 += 32 * AHEAD)
          {
            float2 ev[AHEAD];
            uint32_t j[AHEAD];
#pragma unroll
            for (int u = 0; u < AHEAD; ++u)
            {
              ev[u] = P.lists.event[c0 + 32 * u];
              j[u] = P.lists.pcf[c0 + 32 * u];
            }
#pragma unroll
            for (int u = 0; u < AHEAD; ++u)
              rest = fmaf(w[j[u]] * (c0 + 32 * u < e1 ? ev[u].y : 0.0f), hi - ev[u].x, rest);
          }
#pragma unroll
          for (int d = 16; d > 0; d >>= 1) rest += __shfl_xor_sync(FULL, rest, d);
          rest = fmaf(product[b] + h, hi - t, rest);
        }
        if (lane == 0) P.rest[P.off[i] + k] = rest;
      };

      // this lane's row
      const uint64_t mine = s_row[lane < (int)rows ? lane : 0];
      const uint64_t moff = P.off[mine];
      const uint32_t mlen = lane < (int)rows ? (uint32_t)(P.off[mine + 1] - moff) : 0;
      const float* mp = P.pts + 2 * moff;
      for (;;)
      {
        unsigned b = 0;
        if (lane == 0) b = atomicAdd(&s_bin, 1u);
        b = __shfl_sync(FULL, b, 0);
        if (b >= P.bins) break;
        b = P.bins - 1 - b;  // the last bin first: it is walked whole for every breakpoint
        const uint32_t e0 = P.starts[b], e1 = P.starts[b + 1];
        if (e0 == e1) continue;
        const float edge = P.edges[b];
        // the row's breakpoints of this bin: [k0, k1); the last bin takes its end too
        const uint32_t k0 = mlen ? first_from(mp, mlen, edge) : 0;
        uint32_t k1 = k0;
        const float hi = P.edges[b + 1];
        if (b + 1 == P.bins) k1 = mlen ? mlen : 0;
        else
          while (k1 < mlen && mp[2 * (uint64_t)k1] < hi) ++k1;
        uint32_t next = k0;
        float before = 0.0f;  // integral of H from the bin's edge to this lane's row's breakpoints so far
        for (;;)
        {
          // up to BATCH breakpoints, a row after another
          float t[BATCH], width[BATCH], h[BATCH], area[BATCH], rest[BATCH];
          uint32_t row[BATCH], el[BATCH], place[BATCH], furthest = 0;
          int count = 0;
#pragma unroll
          for (int q = 0; q < BATCH; ++q)
          {
            const unsigned left = __ballot_sync(FULL, next < k1);
            row[q] = el[q] = place[q] = 0;
            t[q] = width[q] = h[q] = area[q] = rest[q] = 0.0f;
            if (!left) continue;
            row[q] = (uint32_t)__ffs((int)left) - 1;
            el[q] = __shfl_sync(FULL, next, row[q]);
            const uint64_t pt = __shfl_sync(FULL, moff, row[q]) + el[q];
            if (lane == (int)row[q]) ++next;
            t[q] = P.pts[2 * pt];
            width[q] = t[q] - fmaxf(P.pts[2 * pt - 2], edge);  // of the element that ends here, in this bin
            place[q] = P.lists.place[pt];
            furthest = max(furthest, place[q]);
            ++count;
          }
          if (count == 0) break;
          // the weights of a breakpoint's row, by address: no multiplication in the loop
          const float* w[BATCH];
#pragma unroll
          for (int q = 0; q < BATCH; ++q) w[q] = smem + (size_t)row[q] * n;
          // The last bin, where PCF after PCF has ended: back from its end, where
          // H is that of zeros, and nothing is left of what has gone.
          if (b + 1 == P.bins)
          {
            for (uint32_t c0 = e0 + lane; c0 < e1 + lane; c0 += 32 * AHEAD)
            {
              float2 ev[AHEAD];
              uint32_t j[AHEAD];
#pragma unroll
              for (int u = 0; u < AHEAD; ++u)
              {
                ev[u] = P.lists.event[c0 + 32 * u];  // behind the list: zeros
                j[u] = P.lists.pcf[c0 + 32 * u];
              }
#pragma unroll
              for (int u = 0; u < AHEAD; ++u)
#pragma unroll
                for (int q = 0; q < BATCH; ++q)
                {
                  const float x = w[q][j[u]] * ev[u].y;
                  h[q] -= c0 + 32 * u >= place[q] ? x : 0.0f;
                  area[q] = fmaf(-x, fminf(fmaxf(ev[u].x - (t[q] - width[q]), 0.0f), width[q]), area[q]);
                  rest[q] = fmaf(-x, fmaxf(ev[u].x - t[q], 0.0f), rest[q]);
                }
            }
          }
          else for (uint32_t c0 = e0 + lane; c0 < furthest + lane; c0 += 32 * AHEAD)
          {
            float2 ev[AHEAD];
            uint32_t j[AHEAD];
#pragma unroll
            for (int u = 0; u < AHEAD; ++u)
            {
              // past the bin's list: entries of the next one, or zeros, masked below
              ev[u] = P.lists.event[c0 + 32 * u];
              j[u] = P.lists.pcf[c0 + 32 * u];
            }
#pragma unroll
            for (int u = 0; u < AHEAD; ++u)
#pragma unroll
              for (int q = 0; q < BATCH; ++q)
              {
                const float x = w[q][j[u]] * (c0 + 32 * u < place[q] ? ev[u].y : 0.0f);
                h[q] += x;
                area[q] = fmaf(x, fminf(t[q] - ev[u].x, width[q]), area[q]);
              }
          }
#pragma unroll
          for (int q = 0; q < BATCH; ++q)
          {
            if (q >= count) break;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1)
            {
              h[q] += __shfl_xor_sync(FULL, h[q], d);
              area[q] += __shfl_xor_sync(FULL, area[q], d);
            }
            const uint64_t i = s_row[row[q]];
            const bool tail = b + 1 == P.bins;
            const float h0 = !tail ? P.product[(i - P.r0) * 2 * P.bins + b] : KERNEL ? 0.0f : -P.centre[b] * s_sum[row[q]];
            const float part = finish(b, e0, e1, h0, width[q], row[q], el[q], place[q], t[q], h[q], area[q]);
            if (lane == (int)row[q]) before += part;
            if (__shfl_sync(FULL, k1, row[q]) != el[q] + 1) continue;
            if (tail)
            {
#pragma unroll
              for (int d = 16; d > 0; d >>= 1) rest[q] += __shfl_xor_sync(FULL, rest[q], d);
              if (lane == 0) P.rest[P.off[i] + el[q]] = fmaf(h0, hi - t[q], rest[q]);
            }
            else
              finish_bin(b, e1, edge, hi, row[q], el[q], place[q], t[q], h[q], __shfl_sync(FULL, before, row[q]));
          }
        }
      }
      __syncthreads();

      for (uint32_t r = warp; r < rows; r += nwarps)
      {
        const uint64_t i = s_row[r], o = P.off[i];
        const uint32_t len = (uint32_t)(P.off[i + 1] - o);
        const float* hint = P.product + (i - P.r0) * 2 * P.bins + P.bins;
        const float sum = KERNEL ? 0.0f : s_sum[r];
        const float wii = KERNEL ? P.grad_out[i * (i + 1) / 2 + i] : 0.0f;
        for (uint32_t k = lane; k + 1 < len; k += 32)
        {
          const float v = P.pts[2 * (o + k) + 1];
          const float t0 = k ? P.pts[2 * (o + k)] : 0.0f, t1 = P.pts[2 * (o + k + 1)];
          const uint32_t b0 = k ? P.bin[o + k] : 0u, b1 = P.bin[o + k + 1];
          // the part of the first bin, whole bins, the part of the last one
          float H = P.area[o + k + 1], own = 0.0f;
          if (b0 == b1)
          {
            if (!KERNEL) own = (v - P.centre[b0]) * (t1 - t0);
          }
          else
          {
            float whole = k ? P.rest[o + k] : hint[b0];
            if (!KERNEL) own = (v - P.centre[b0]) * (P.edges[b0 + 1] - t0);
            for (uint32_t b = b0 + 1; b < b1; ++b)
            {
              whole += hint[b];
              if (!KERNEL) own = fmaf(v - P.centre[b], P.edges[b + 1] - P.edges[b], own);
            }
            H += whole;
            if (!KERNEL) own = fmaf(v - P.centre[b1], t1 - P.edges[b1], own);
          }
          float dv = KERNEL ? H : fmaf(own, sum, -H);
          if (KERNEL) dv = fmaf(wii, 2.0f * (v * (t1 - t0)), dv);  // the kernel's diagonal
          P.grad[2 * (o + k) + 1] = dv;
          if (k == 0) P.grad[2 * o] = 0.0f;
          lost |= !isfinite(dv);
        }
        // The last element, 0 up to the end of time: of the shorter PCFs most of
        // the bins, by the whole warp.
        {
          const uint32_t k = len - 1, b0 = k ? P.bin[o + k] : 0u;
          float H = 0.0f, own = 0.0f;
          for (uint32_t b = b0 + 1 + lane; b < P.bins; b += 32)
          {
            H += hint[b];
            if (!KERNEL) own = fmaf(-P.centre[b], P.edges[b + 1] - P.edges[b], own);
          }
#pragma unroll
          for (int d = 16; d > 0; d >>= 1)
          {
            H += __shfl_xor_sync(FULL, H, d);
            if (!KERNEL) own += __shfl_xor_sync(FULL, own, d);
          }
          if (lane == 0)
          {
            H += k ? P.rest[o + k] : hint[b0];
            if (!KERNEL) own = fmaf(-P.centre[b0], P.edges[b0 + 1] - (k ? P.pts[2 * (o + k)] : 0.0f), own);
            const float dv = KERNEL ? H : fmaf(own, sum, -H);
            P.grad[2 * (o + k) + 1] = dv;
            if (k == 0) P.grad[2 * o] = 0.0f;
            lost |= !isfinite(dv);
          }
        }
      }
      if (__any_sync(FULL, lost) && lane == 0) atomicOr(&P.rec->bad_weights, 1u);
    }

    // Time gradients behind elements without width, which the walks give the
    // row of a pair alone, the later PCF in length order: a column's step of
    // width 0 passes for a tie.  One CTA per breakpoint, over the earlier PCFs.
    template <bool KERNEL>
    __global__ void __launch_bounds__(256) l2_narrow_kernel(const __grid_constant__ L2Gradient P)
    {
      __shared__ uint32_t s_closed, s_place;
      __shared__ float s_part[8];
      if (threadIdx.x == 0)
      {
        s_closed = P.rec->bad | P.rec->bad_weights;  // bad_weights may be set meanwhile
        s_place = 0;
      }
      __syncthreads();
      if (s_closed) return;
      const uint32_t count = P.rec->narrow;
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      for (uint32_t x = blockIdx.x; x < count; x += gridDim.x)
      {
        const uint64_t pt = P.narrow[x], i = P.owner[pt];
        const float t = P.pts[2 * pt], a = P.pts[2 * pt - 1], c = P.pts[2 * pt + 1];
        // the PCF's place in length order, which stays within its window
        const uint64_t w0 = i / LENGTH_ORDER_WINDOW * LENGTH_ORDER_WINDOW, w1 = min(w0 + LENGTH_ORDER_WINDOW, P.n);
        for (uint64_t p = w0 + threadIdx.x; p < w1; p += 256)
          if (P.order[p] == i) s_place = (uint32_t)p;
        __syncthreads();
        float sum = 0.0f;
        for (uint32_t p = threadIdx.x; p < s_place; p += 256)
        {
          const uint64_t j = P.order[p], hi = max(i, j), lo = min(i, j);
          const uint64_t at = KERNEL ? hi * (hi + 1) / 2 + lo : hi * (hi - 1) / 2 + lo;
          float w = P.grad_out[at];
          if (!KERNEL)
          {
            const float d = P.fwd[at];
            w = d > 0.0f ? w / d : 0.0f;
            if (w != 0.0f && l2_close(d, P.norm[hi], P.norm[lo])) w = 0.0f;
          }
          if (w == 0.0f) continue;
          const uint64_t o = P.off[j];
          const uint32_t len = (uint32_t)(P.off[j + 1] - o), k = first_from(P.pts + 2 * o, len, t);
          if (k < len && P.pts[2 * (o + k)] == t) continue;  // a tie
          const float g = P.pts[2 * (o + k) - 1];
          sum = fmaf(w, KERNEL ? g : 0.5f * (a + c) - g, sum);
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(FULL, sum, d);
        if (lane == 0) s_part[warp] = sum;
        __syncthreads();
        if (threadIdx.x == 0)
        {
          float all = 0.0f;
          for (int q = 0; q < 8; ++q) all += s_part[q];
          float dt = (a - c) * all;
          if (KERNEL) dt = fmaf(P.grad_out[i * (i + 1) / 2 + i], (a - c) * (a + c), dt);
          P.grad[2 * pt] = dt;
          if (!isfinite(dt)) atomicOr(&P.rec->bad_weights, 1u);
        }
        __syncthreads();
      }
    }

    uint64_t up(uint64_t x, uint64_t to) { return (x + to - 1) / to * to; }
  }

  // Bins (a multiple of 64): the product's waves of 128 x 128 tiles, about 75
  // cycles for each k (1.9 waves at N = 4096; the only wave of N = 1021, 104
  // tiles, takes 2.4 times that), against L^2 / bins list entries per pair of PCFs at two
  // cycles for 32 of them (N = 4096, L ~ U{16..512}: 576 bins, product 0.69 ms
  // and lists 1.2; with 896, 1.04 and 0.9 or more), and the table's entries.
  static uint32_t choose_bins(uint64_t n, uint64_t npts, int sms)
  {
    const double mean = (double)npts / (double)n;
    double best = 0;
    uint32_t bins = 64;
    for (uint32_t b = 64; b <= 2048; b += 64)
    {
      const double tiles = std::ceil((double)n / GT) * (2.0 * b / GT);
      const double product = std::ceil(tiles / sms) * (double)n * 75.0;
      const double near = (double)n * (double)n * mean * mean / b / 32.0 * 2.0 / sms;
      const double fill = (double)n * b * 6.0 / sms;
      const double cost = product + near + fill;
      if (b == 64 || cost < best) { best = cost; bins = b; }
    }
    return bins;
  }

  L2BackwardPlan l2_backward_plan(uint64_t n, uint64_t npts, const DeviceInfo& dev)
  {
    L2BackwardPlan p;
    // one row of weights in shared memory (which keeps PCF and bin indices
    // within 16 bits), point indices in 32
    const size_t smem = dev.smem_optin > 2048 ? dev.smem_optin - 1024 : 0;
    if (npts >= 0xffffffffull || n * sizeof(float) > smem) return p;
    // Below about 1e8 pairs times breakpoints the dozen small launches here
    // cost what the walk does (forward and backward: n = 512, L ~ U{4..60} 315
    // us against 266; n = 700, L ~ U{16..512} 575 against 792; n = 1700, L ~
    // U{4..60} 533 against 587); with few PCFs, or several breakpoints of one
    // PCF to a bin, the walk is the more exact one (n = 200, L ~ U{2000..3000}
    // 3.8e-7 of the value gradient against 2.4e-7; from n = 700 on 3.1e-7
    // against 3.9e-7 and more).
    if (n < 300 || npts > 1500 * n || (double)n * (double)npts < 1e8) return p;
    p.bins = choose_bins(n, npts, dev.sms);
    p.k = up(n, 32);
    // weights of at most 1 GB at a time, in whole windows of the length order
    p.width = std::min<uint64_t>(up(n, GT), std::max<uint64_t>(LENGTH_ORDER_WINDOW, (1ull << 28) / p.k / LENGTH_ORDER_WINDOW * LENGTH_ORDER_WINDOW));
    static_assert(LENGTH_ORDER_WINDOW % GT == 0, "panels hold whole tiles");
    const uint64_t rows_max = std::min<uint64_t>(ROWS_MAX, smem / (n * sizeof(float)));
    // as many rows per CTA as fit, fewer where that evens out the last wave
    const uint64_t span = std::min<uint64_t>(p.width, n);
    const uint64_t waves = (span + rows_max * dev.sms - 1) / (rows_max * dev.sms);
    p.rows = (uint32_t)std::min<uint64_t>(rows_max, (span + waves * dev.sms - 1) / (waves * dev.sms));
    p.rows = std::max(p.rows, 1u);
    auto add = [&](size_t bytes) {
      const size_t at = p.bytes;
      p.bytes += up(bytes, 256);
      return at;
    };
    p.record = add(256);
    p.edges = add((p.bins + 1) * 4);
    p.counts = add(p.bins * 4);
    p.starts = add((p.bins + 1) * 4);
    p.next = add(p.bins * 4);
    p.centre = add(p.bins * 4);
    p.norm = add(n * 4);
    p.narrow = add(n * 4);
    p.keys = add(npts * 8);
    p.event = add((npts + 32 * AHEAD) * 8);  // the sums read past a list's end
    p.pcf = add((npts + 32 * AHEAD) * 2);
    p.owner = add(npts * 2);
    p.point = add(npts * 4);
    p.place = add(npts * 4);
    p.area = add(npts * 4);
    p.rest = add(npts * 4);
    p.bin = add(npts * 2);
    p.table = add(p.k * 2 * p.bins * 4);
    p.wt = add(p.k * p.width * 4);
    p.product = add(p.width * 2 * p.bins * 4);
    p.ok = true;
    return p;
  }

  const unsigned* l2_backward(const L2BackwardPlan& p, void* scratch, const float* pts, const uint64_t* off, uint64_t n,
                              uint64_t npts, const float* grad_out, const float* fwd, const uint32_t* order, float* grad,
                              const float** norms, const DeviceInfo& dev, cudaStream_t st)
  {
    char* base = static_cast<char*>(scratch);
    auto f32 = [&](size_t at) { return reinterpret_cast<float*>(base + at); };
    auto u32 = [&](size_t at) { return reinterpret_cast<uint32_t*>(base + at); };
    L2Record* rec = reinterpret_cast<L2Record*>(base + p.record);
    const bool kernel = fwd == nullptr;
    const uint32_t bins = p.bins;
    const unsigned warps8 = (unsigned)std::min<uint64_t>((n + 7) / 8, (uint64_t)dev.sms * 8);
    SBG_CUDA(cudaMemsetAsync(base + p.record, 0, p.starts - p.record, st));  // the record and the counts
    l2_record_kernel<<<warps8, 256, 0, st>>>(pts, off, n, npts, rec, u32(p.narrow));
    SBG_CUDA(launched());
    l2_edges_kernel<<<1, 1024, 0, st>>>(pts, off, n, rec, bins, f32(p.edges));
    SBG_CUDA(launched());
    auto u16 = [&](size_t at) { return reinterpret_cast<uint16_t*>(base + at); };
    uint64_t* keys = reinterpret_cast<uint64_t*>(base + p.keys);
    L2Lists lists{reinterpret_cast<float2*>(base + p.event), u16(p.pcf), u32(p.point), u32(p.place)};
    const unsigned ctas = (unsigned)std::min<uint64_t>((n + 15) / 16, (uint64_t)dev.sms * 2);
    l2_bins_kernel<false><<<ctas, 512, bins * 12, st>>>(pts, off, n, rec, bins, f32(p.edges), u32(p.counts), keys, u16(p.bin),
                                                         u16(p.owner));
    SBG_CUDA(launched());
    l2_starts_kernel<<<1, 1024, 0, st>>>(u32(p.counts), bins, u32(p.starts), u32(p.next));
    SBG_CUDA(launched());
    l2_bins_kernel<true><<<ctas, 512, bins * 12, st>>>(pts, off, n, rec, bins, f32(p.edges), u32(p.next), keys, u16(p.bin),
                                                        u16(p.owner));
    SBG_CUDA(launched());
    const size_t sort_smem = BIN_MAX * sizeof(uint64_t);
    SBG_CUDA(cudaFuncSetAttribute(l2_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sort_smem));
    l2_sort_kernel<<<bins, 512, sort_smem, st>>>(pts, rec, u32(p.starts), keys, u16(p.owner), lists);
    SBG_CUDA(launched());
    if (!kernel)
    {
      l2_centres_kernel<<<bins, 256, 0, st>>>(pts, off, n, rec, f32(p.edges), f32(p.centre));
      SBG_CUDA(launched());
    }
    l2_table_kernel<<<(unsigned)((p.k + 7) / 8), 256, 0, st>>>(pts, off, n, p.k, rec, bins, f32(p.edges),
                                                             kernel ? nullptr : f32(p.centre), f32(p.table),
                                                             f32(p.norm));
    SBG_CUDA(launched());

    const size_t gemm_smem = (size_t)2 * GS * GK * GT * sizeof(float);
    SBG_CUDA(cudaFuncSetAttribute(l2_product_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem));
    const size_t near_smem = (size_t)p.rows * n * sizeof(float);
    void (*near)(const L2Gradient) = kernel ? l2_gradient_kernel<true> : l2_gradient_kernel<false>;
    SBG_CUDA(cudaFuncSetAttribute(near, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)near_smem));
    L2Gradient G{};
    for (uint64_t r0 = 0; r0 < n; r0 += p.width)
    {
      const dim3 tiles((unsigned)(p.width / 32), (unsigned)((p.k + 31) / 32));
      l2_weights_kernel<<<tiles, 256, 0, st>>>(grad_out, fwd, f32(p.norm), n, kernel, r0, p.width, p.k, f32(p.wt), rec);
      SBG_CUDA(launched());
      l2_product_kernel<<<dim3(2 * bins / GT, (unsigned)(p.width / GT)), 256, gemm_smem, st>>>(
          f32(p.wt), p.width, f32(p.table), 2 * bins, p.k, rec, f32(p.product));
      SBG_CUDA(launched());
      G.rec = rec; G.pts = pts; G.off = off; G.order = order; G.n = n; G.r0 = r0; G.width = p.width; G.rows = p.rows; G.bins = bins;
      G.edges = f32(p.edges); G.starts = u32(p.starts); G.centre = f32(p.centre); G.lists = lists;
      G.wt = f32(p.wt); G.product = f32(p.product); G.grad_out = grad_out; G.grad = grad; G.area = f32(p.area); G.rest = f32(p.rest);
      G.bin = u16(p.bin);
      const uint64_t span = std::min<uint64_t>(p.width, n - r0);
      near<<<(unsigned)((span + p.rows - 1) / p.rows), NEAR_THREADS, near_smem, st>>>(G);
      SBG_CUDA(launched());
    }
    G.narrow = u32(p.narrow); G.owner = u16(p.owner); G.fwd = fwd; G.norm = f32(p.norm);
    (kernel ? l2_narrow_kernel<true> : l2_narrow_kernel<false>)<<<(unsigned)std::min<uint64_t>(n, (uint64_t)dev.sms * 8), 256, 0, st>>>(G);
    SBG_CUDA(launched());
    *norms = f32(p.norm);
    return &rec->bad;
  }
}
