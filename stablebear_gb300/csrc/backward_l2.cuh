// Interface of the L2 gradients by contraction (backward_l2.cu) to backward.cu.
#pragma once

#include "sbg_internal.hpp"

namespace sbg
{
  // What the data of a call is like, gathered on the device (zeroed first).
  // bad: the data takes the walk; bad_weights: a weight, an overfull bin or a
  // gradient that is not finite does; close: some pairs of distances do (l2_close).
  // narrow: breakpoints behind elements without width.
  struct L2Record { uint32_t bad, bad_weights, close, tmax_bits, narrow; };

  // A distance far smaller than its two PCFs (less the common part): in
  // v S - H its weight w / D would multiply their size, not their difference,
  // and the rounding with it.  Such pairs keep the walk.  norm: of a PCF less
  // the bins' centres.
  __host__ __device__ inline bool l2_close(float d, float norm_f, float norm_g)
  {
    return d < 0.125f * (norm_f + norm_g);
  }

  // The breakpoints by bin and time: (time, change of the PCF's value), PCF,
  // point; and each point's place there.
  struct L2Lists { float2* event; uint16_t* pcf; uint32_t* point; uint32_t* place; };

  struct L2Gradient
  {
    L2Record* rec;
    const float* pts;
    const uint64_t* off;
    const uint32_t* order;  // the PCFs in length order, panel by panel
    uint64_t n, r0, width;  // PCFs; the rows [r0, r0 + width) of this launch
    uint32_t rows, bins;    // rows per CTA
    const float* edges;     // bins + 1
    const uint32_t* starts; // bins + 1
    const float* centre;    // distances only
    L2Lists lists;
    const float* wt;        // weights, [j][i - r0]
    const float* product;   // [i - r0][2 bins]: H at the edges, its integral over the bins
    const float* grad_out;
    float* grad;            // (npts, 2): [dL/dt, dL/dv]
    float* area;            // integral of H up to the breakpoint, from the one before it or the bin's edge
    float* rest;            // of the last breakpoint in a bin: from it to the bin's end
    const uint16_t* bin;    // the breakpoint's bin
    const uint32_t* narrow; // breakpoints behind elements without width
    const uint16_t* owner;  // the breakpoint's PCF
    const float* fwd;       // distances only, with the PCFs' norms
    const float* norm;
  };

  struct L2BackwardPlan
  {
    bool ok = false;
    uint32_t bins = 0, rows = 0;
    uint64_t k = 0, width = 0;  // rows of the table; rows of the gradient at a time
    size_t bytes = 0;
    size_t record = 0, edges = 0, counts = 0, starts = 0, next = 0, centre = 0, norm = 0, narrow = 0, keys = 0, event = 0, pcf = 0, owner = 0,
           point = 0, place = 0, area = 0, rest = 0, bin = 0, table = 0, wt = 0, product = 0;
  };

  // ok: false where the walk of backward.cu is the better one.
  L2BackwardPlan l2_backward_plan(uint64_t n, uint64_t npts, const DeviceInfo& dev);

  // Launches everything; returns the record: the walk has to run where one of
  // its first three words is set, for the close pairs alone (added to the
  // gradient) where that is the third.  fwd: the distances, or null for the L2
  // kernel; *norms: the PCFs' norms for l2_close.
  const unsigned* l2_backward(const L2BackwardPlan& p, void* scratch, const float* pts, const uint64_t* off, uint64_t n,
                              uint64_t npts, const float* grad_out, const float* fwd, const uint32_t* order, float* grad,
                              const float** norms, const DeviceInfo& dev, cudaStream_t st);
}
