// wl_reduce.cuh -- per-loop or per-chunk FP64 partial sums -> <W> per group,
// mean and standard error, shared by the single-job and the batched reduction.
#pragma once

#include <math.h>

#include "wl_internal.h"

namespace wl {

// One CTA of kReduceThreads reduces ti instances (a power of two <= 32, the
// fastest thread index, so that a warp reads contiguous partial sums) at one
// flux value; the remaining threads split the three factors and the groups.
// Within a group the partial sums are added in chunk order (and within a chunk
// in loop order where the sweep stored its loops one by one, R.inner of them per
// chunk), and the mean and the squared deviations in group order: a result
// depends neither on ti nor on how the sweep was partitioned.  The partial sums
// hold W - 1 per loop; the Richardson weights 8/3, -2, 1/3 (Integrand.c:400) sum
// to one, so <W> = 1 + the same combination of the deviations.
//
// Bound by FP64 additions: one takes a warp 62 cycles, however many of its
// lanes add and independent ones too, and an SM 19.  One thread per (instance,
// flux) walking every chunk took 217 us for one instance on 1024 loops and 61
// us for 1024 instances there (cold caches); the groups on threads of their own
// 33 and 58 us (three chains a thread), the factors too, on all SMs, 23 and 32.
// The whole call for one instance: 274 -> 121 -> 74 us (the copies' share too).
template <class Out>
__device__ __forceinline__ void reduce_block(const ReduceShape &R, int i0, int j, int ti,
                                             double *__restrict__ out_group, Out &&out) {
  __shared__ double val[kReduceThreads];  // one round: [tg][3][ti] sums, then [tg][0][ti] values
  const int tx = threadIdx.x & (ti - 1), rest = threadIdx.x / ti;
  const int r = rest % 3, gy = rest / 3, tg = kReduceThreads / ti / 3;
  const int inst = i0 + tx;
  const bool live = inst < R.ninst && gy < tg;
  const int ng = R.n_chunks / R.cpg;
  const double inv = 1.0 / (double)R.lpg;
  const size_t row = (size_t)R.ninst, step = 3 * (size_t)R.nF * row;
  // n values from p on added in order, eight in flight
  auto add_rows = [&](const double *&p, int n, double s) {
    for (; n >= 8; n -= 8) {
      double v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = p[k * step];
      p += 8 * step;
#pragma unroll
      for (int k = 0; k < 8; ++k) s += v[k];
    }
    for (; n > 0; --n, p += step) s += p[0];
    return s;
  };
  auto group_sum = [&](int g) {  // of this thread's factor
    const double *p = R.partial + (((size_t)g * R.cpg * R.inner * R.nF + j) * 3 + r) * row + inst;
    if (R.inner == 1) return add_rows(p, R.cpg, 0.0);
    double s = 0.0;
    for (int c = 0; c < R.cpg; ++c) s += add_rows(p, R.inner, 0.0);
    return s;
  };
  double *og = out_group && live ? out_group + ((size_t)inst * R.nF + j) * ng : nullptr;
  double *const mine = val + (gy * 3 * ti + tx);  // this (group, instance)'s sums
  double mean = 0.0, ss = 0.0;
  for (int pass = 0; pass < 2; ++pass) {
    for (int g0 = 0; g0 < ng; g0 += tg) {
      const int g = g0 + gy;
      if (pass == 0 || ng > tg) {  // a single round keeps its values
        const bool again = pass && og;
        if (live && g < ng && !again) val[threadIdx.x] = group_sum(g);
        __syncthreads();
        if (live && g < ng && r == 0) {
          if (again) {
            mine[0] = og[g];
          } else {
            const double v = 1.0 + (8.0 / 3.0 * (mine[0] * inv) - 2.0 * (mine[ti] * inv) +
                                    1.0 / 3.0 * (mine[2 * ti] * inv));
            mine[0] = v;
            if (og) og[g] = v;
          }
        }
        __syncthreads();
      }
      if (rest == 0 && live) {
        const int n = min(tg, ng - g0);
        if (pass == 0)
          for (int k = 0; k < n; ++k) mean += val[k * 3 * ti + tx];
        else
          for (int k = 0; k < n; ++k) {
            const double d = val[k * 3 * ti + tx] - mean;
            ss += d * d;
          }
      }
      if (ng > tg) __syncthreads();  // the round's values are overwritten next
    }
    if (pass == 0) mean /= (double)ng;
  }
  if (rest == 0 && live)
    out((size_t)inst * R.nF + j, mean,
        ng > 1 ? sqrt(ss / ((double)ng * (ng - 1.0))) : 0.0);
}

}  // namespace wl
