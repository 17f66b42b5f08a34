// wl_reduce.cuh -- per-loop or per-chunk FP64 partial sums -> <W> per group,
// mean and standard error, shared by the single-job and the batched reduction.
#pragma once

#include <math.h>

#include "wl_internal.h"

namespace wl {

// One CTA of kReduceThreads reduces ti instances (a power of two <= 32, the
// fastest thread index, so that a warp reads contiguous partial sums) at one
// flux value; the remaining threads split the groups.  Within a group the
// partial sums are added in chunk order (and within a chunk in loop order
// where the sweep stored its loops one by one, R.inner of them per chunk), and
// the mean and the squared deviations in group order: a result depends
// neither on ti nor on how the sweep was partitioned.  The partial sums hold
// W - 1 per loop; the Richardson weights 8/3, -2, 1/3 (Integrand.c:400) sum to
// one, so <W> = 1 + the same combination of the deviations.
//
// Bound by the latency of its loads when there are few instances (one thread
// per (instance, flux) walked every chunk of the ensemble: 217 us for one
// instance on 1024 loops, 270 us for 96 instances x 3 fluxes on 640 chunks),
// by HBM when there are many.  With the groups split: the whole call for one
// instance on 1024 loops 274 -> 121 us.
template <class Out>
__device__ __forceinline__ void reduce_block(const ReduceShape &R, int i0, int j, int ti,
                                             double *__restrict__ out_group, Out &&out) {
  __shared__ double val[kReduceThreads];  // one round of group values [tg][ti]
  const int tx = threadIdx.x & (ti - 1), gy = threadIdx.x / ti, tg = kReduceThreads / ti;
  const int inst = i0 + tx;
  const bool live = inst < R.ninst;
  const int ng = R.n_chunks / R.cpg;
  const double inv = 1.0 / (double)R.lpg;
  const size_t row = (size_t)R.ninst, step = 3 * (size_t)R.nF * row;
  auto group_value = [&](int g) {
    const double *p = R.partial + ((size_t)g * R.cpg * R.inner * R.nF + j) * 3 * row + inst;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    if (R.inner == 1) {
#pragma unroll 16
      for (int c = 0; c < R.cpg; ++c, p += step) {
        s0 += p[0];
        s1 += p[row];
        s2 += p[2 * row];
      }
    } else {
      for (int c = 0; c < R.cpg; ++c) {
        double t0 = 0.0, t1 = 0.0, t2 = 0.0;
#pragma unroll 8
        for (int l = 0; l < R.inner; ++l, p += step) {
          t0 += p[0];
          t1 += p[row];
          t2 += p[2 * row];
        }
        s0 += t0;
        s1 += t1;
        s2 += t2;
      }
    }
    return 1.0 + (8.0 / 3.0 * (s0 * inv) - 2.0 * (s1 * inv) + 1.0 / 3.0 * (s2 * inv));
  };
  double *og = out_group && live ? out_group + ((size_t)inst * R.nF + j) * ng : nullptr;
  double mean = 0.0, ss = 0.0;
  for (int pass = 0; pass < 2; ++pass) {
    for (int g0 = 0; g0 < ng; g0 += tg) {
      const int g = g0 + gy;
      if (pass == 0 || ng > tg) {  // a single round keeps its values
        if (live && g < ng) {
          double v;
          if (pass && og) {
            v = og[g];
          } else {
            v = group_value(g);
            if (og) og[g] = v;
          }
          val[threadIdx.x] = v;
        }
        __syncthreads();
      }
      if (gy == 0 && live) {
        const int n = min(tg, ng - g0);
        if (pass == 0)
          for (int k = 0; k < n; ++k) mean += val[k * ti + tx];
        else
          for (int k = 0; k < n; ++k) {
            const double d = val[k * ti + tx] - mean;
            ss += d * d;
          }
      }
      if (ng > tg) __syncthreads();  // the round's values are overwritten next
    }
    if (pass == 0) mean /= (double)ng;
  }
  if (gy == 0 && live)
    out((size_t)inst * R.nF + j, mean,
        ng > 1 ? sqrt(ss / ((double)ng * (ng - 1.0))) : 0.0);
}

}  // namespace wl
