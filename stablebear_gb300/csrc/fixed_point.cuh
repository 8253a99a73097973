// Interface of the fixed-point float64 path (fixed_point.cu) to the engine.
#pragma once

#include "pair_kernels.cuh"

namespace sbg
{
  // Warps per CTA unless the caller asks for fewer, one CTA per SM.  Four warps a scheduler cover the walk's
  // latencies, and 128 registers a thread hold it without spills (L1, general
  // values, N = 2500: 1.65 ms with 12 warps, 1.49 with 16, 1.57 with 20, 1.62
  // with 24).
  constexpr int FIXED_WARPS = 16;
  constexpr uint32_t FIXED_CARRY = 4;  // 64-bit words of a pair's running sums

  // What the data of a call is like, gathered on the device (zeroed first).
  struct FixedRecord
  {
    uint64_t tmax_bits, vmax_bits;  // largest time and |value|, as bit patterns
    uint64_t points;
    double vsum;                    // sum of |values|
    uint32_t low;                   // 4096 minus the exponent of the lowest bit set in any value
    uint32_t negative;              // some value is negative
    uint32_t bad;                   // not representable: the direct kernels run
    uint32_t risky;                 // PCFs whose pairs would be walked twice, of
    uint32_t packed;                // these many
    uint32_t pad;
  };

  // What rounding can move of a PCF: the sum of |changes| at times that are no
  // whole number of units, and the root of the sum of their squares; the range of
  // its values where times may round, before 2^52 units; its largest |value|;
  // and for how long, in units, its value is no whole number.  (Values and
  // changes as integer values, general form: over 2^32.)
  struct alignas(16) Shape { float tv, rv, lo, hi, vmax, ev, pad[2]; };

  // One side's PCFs: CSR, processing order, and the packed arrays of `cap`
  // elements (times, then values).
  struct FixedSet
  {
    const double* pts;
    const uint64_t* off;
    const uint32_t* perm;
    uint64_t n;
    const uint64_t* times;
    uint64_t cap;
    const Shape* shapes;
    const uint32_t* lens;  // packed elements of each PCF
  };

  struct FixedParams
  {
    const FixedRecord* rec;
    FixedSet r, c;
    double* out;
    uint64_t out_base, out_count, ld, row_begin, row_end, n_items;
    unsigned long long* queue;  // zeroed before launch
    unsigned* gate;             // of the direct kernel behind: 0 opens it
    uint64_t* carry;            // FIXED_CARRY * 32 words per row of an item and CTA
    uint32_t q, rows_per_item;
    int mode;
    bool elements;              // the direct kernel reads (v, t) elements in the packed arrays' place
    uint32_t smem_bytes;
  };

  // Elements of a column (and row) slice in `bytes` of shared memory, and of
  // a warp's row buffer: the slice and U + 1 more, made even.
  __host__ __device__ inline uint32_t fixed_row_elements(uint32_t X) { return (X + 9 + 1) / 2 * 2; }
  __host__ __device__ inline uint32_t fixed_slice_cap(uint32_t bytes, uint32_t warps, uint32_t elem)
  {
    return (bytes - warps * 12 * elem) / (elem * (32 + warps)) / 4 * 4;
  }

  // longest: the breakpoint count that the call's buffers are sized for.
  cudaError_t launch_fixed_record(const double* pts, const uint64_t* off, uint64_t n, uint64_t cap, uint32_t longest,
                                  FixedRecord* rec, int sms, cudaStream_t st);
  cudaError_t launch_fixed_pack(const double* pts, const uint64_t* off, uint64_t n, uint64_t cap,
                                FixedRecord* rec, int opk, void* packed, Shape* shapes, uint32_t* lens,
                                bool elements, unsigned* gate, int sms, cudaStream_t st);
  cudaError_t launch_fixed_pairs(const FixedParams& P, int opk, int warps, int grid, cudaStream_t st);
}
