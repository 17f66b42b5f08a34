// wl_internal.h -- launch interfaces between the C-ABI runtime (wl_api.cpp)
// and the kernels (wl_sweep_*.cu, wl_batch.cu, wl_misc.cu, wl_tint.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "wl_types.h"

namespace wl {

// device-side status codes written to the status word of a launch
enum : int { kDevOk = 0, kDevTimeout = 1, kDevBadInstance = 2 };

// Instance-parallel sweep: one lane per instance, one warp per (32 instances,
// unit of loops); every warp streams its loops through shared memory by bulk
// copies and works alone (wl_sweep.cuh).
constexpr int kSweepThreads = 128;
constexpr int kSweepWarps = kSweepThreads / 32;
constexpr int kLandPts = 256;  // points of a warp's landing zone (4 KiB)
// warps resident on the chip: 152 SMs x 4 CTAs (128 registers a thread)
constexpr int kSweepSlots = 152 * 4 * kSweepWarps;

struct SweepArgs {
  const float4 *loops;  // [Nl][ppl]
  int Nl, ppl;
  int ninst;
  const float *cx, *cy;  // [ninst] centre of mass
  const float *rtT;      // [ninst] float(sqrt(T)) as the reference passes it
  const float *tqh, *tql;  // [ninst] 4 T / ppl (spin normalisation 2T/(N/2)), hi + lo
  int nF;
  float F[kMaxF];
  // double-float per-flux constants: cph = F h/3, csp = F h/3 fp_scale
  float cph_hi[kMaxF], cph_lo[kMaxF], csp_hi[kMaxF], csp_lo[kMaxF];
  FieldDev field;
  int chunk_loops;   // loops per partial sum
  int n_chunks;      // Nl / chunk_loops
  int unit_loops;    // loops per warp unit
  int n_units;
  int per_loop;      // the partial sums are stored loop by loop
  int n_tiles;       // warps per unit (set at launch)
  // heavy profiles with few units (sweep_parts): a loop's Kahan blocks go to
  // `parts` warps, part_blocks each, through [Nl][blocks + 2][6][ninst] floats
  int parts, part_blocks;
  float *blocks;
  double *partial;   // [n_chunks][nF][3][ninst], per_loop: [Nl][nF][3][ninst]
  int *status;       // kDevOk / kDevTimeout
  uint32_t wait_tries;
  int kprof, fermion, nint;  // kernel selection inside the persistent batch kernel
  const float4 *bbox;        // lattice: [Nl] unit-loop (xmin, xmax, ymin, ymax)
  // optional [ninst] thread slot -> instance: lattice instances ordered by
  // proper time so that the threads of a warp sum similar numbers of images
  const int *perm;
};

inline __host__ __device__ bool light_profile(int kprof) {
  return kprof == kSmooth || kprof == kStep || kprof == kQuadratic || kprof == kGaussian;
}
// two loops per lane as packed f32x2 pairs (wl_sweep.cuh)
inline __host__ __device__ bool sweep_loop_pairs(int kprof) { return light_profile(kprof); }
// instances per warp (the lattice at 4 intervals: two per lane)
inline __host__ __device__ int warp_instances(int kprof, int nint) {
  return nint == 4 && kprof == kLattice ? 64 : 32;
}
// instances per batch tile (one CTA's warps)
inline __host__ __device__ int sweep_tile_instances(int kprof, int nint) {
  return kSweepWarps * warp_instances(kprof, nint);
}

// Device time of one tile-point relative to the smooth profile at 4
// intervals (tile order, the cut into single loops, processor-sharing split and
// rate estimates): the node count times the profile's cost relative to the smooth
// one at the same interval count, interpolated linearly in nint between 4, 8 and
// 50 (flat outside).  The figures were measured with the CTA tiles (512 instances
// on Nl 1024 x ppl 1024, scalar QED); with the warp units the ratios are, in that
// order, Gaussian 2.1, 2.1, 2.6, lattice at a = 5 lambda 12, 31, 40, periodic 30,
// 30, 34, spline 16, 15, 21, fixflux 73, 70, 91, step and quadratic 1.1 to 1.4.
// They stay because sweep_units' lines are drawn in them and a batch's order by
// the new ones is no better (six uneven jobs 17.9 -> 18.3 ms: Gaussian units ahead
// of smooth ones of the same length).
inline double profile_weight(int kprof, int fermion, int nint) {
  double r[3] = {1.0, 1.0, 1.0};  // at 4, 8, 50 intervals
  switch (kprof) {
    case kGaussian: r[0] = 1.6; r[1] = 1.94; r[2] = 3.95; break;
    case kLattice: r[0] = r[1] = r[2] = 8.0; break;
    case kPeriodic: r[0] = r[1] = 30.4; r[2] = 70.8; break;
    case kSpline: r[0] = r[1] = 12.6; r[2] = 29.2; break;
    case kFixflux:
    case kFixfluxFF: r[0] = r[1] = 180.0; r[2] = 400.0; break;
    default: break;
  }
  double w;
  if (nint <= 4) w = r[0];
  else if (nint <= 8) w = r[0] + (r[1] - r[0]) * (nint - 4) / 4.0;
  else if (nint <= 50) w = r[1] + (r[2] - r[1]) * (nint - 8) / 42.0;
  else w = r[2];
  return (fermion ? w * 1.15 : w) * (nint + 1) / 5.0;
}

// CTAs of a sweep of so many warp units (0: too many; a warp finds its unit as
// blockIdx.x * kSweepWarps + warp in 32 bits)
inline unsigned sweep_ctas(long long items) {
  const long long ctas = (items + kSweepWarps - 1) / kSweepWarps;
  return ctas > (1ll << 32) / kSweepWarps ? 0u : (unsigned)ctas;
}

// warp units of a sweep by whole chunks
inline double sweep_chunk_items(const SweepArgs &a, int kprof, int nint) {
  const int per = warp_instances(kprof, nint);
  return (double)((a.ninst + per - 1) / per) * a.n_chunks;
}
// How the loops of a sweep are cut into warp units.  By whole chunks of
// chunk_loops (one partial sum per chunk), or, where that gives the launch too
// few units to fill the chip evenly, into the smallest units (a loop, or the
// two of a packed pair) whose loops are stored one by one; the reduction adds
// them in the same order, so a result does not depend on the choice.
//   items: the launch's units by whole chunks, w = items / kSweepSlots waves of
// them.  Chunks leave part of the last wave idle: a launch alone on the chip gains
// 10 % from single loops at 0.84 waves or just above one, 4 % at 1.7, and most of
// the chip below a quarter; one beside other launches, which fill the idle part,
// nothing.  Single loops cost 48 nF bytes of traffic per (loop, instance) and 3 nF
// of the reduction's FP64 additions, which in a chunk's walk overlap its FP32 work:
// with x = nF / (ppl weight), among others 28 % of the time at x = 1/16, 9-14 % at
// 1/64, 3-4 % at 1/128, 1 % at 1/256.  alone: the call waits for its results, so
// its launches share the chip with other contexts' only; the lines lie where the
// two sides meet alone (0.012) and where a launch among others loses at most 3 %
// (0.005; the Gaussian profile's longer walks wait for instructions by chunks,
// spinor, 1024 instances x 64 points 194 us by single loops, 208 by chunks: 0.015
// for it).  Smooth scalar on 1024 loops, three wl_eval_device calls in flight, by
// single loops -> chunks: 1024 instances x 64 points 92 -> 80 us, 512 x 4 F x 256
// points 176 -> 156; 96 instances x 3 F on 5120 x 2048 stay single loops (1.20 ms,
// 3.14 in 128-thread tiles of 256 instances).  Above 16 waves the sums would also
// outgrow the gain (0.24 GB per flux value at wl_eval's 8 loops per chunk; a
// batch's larger chunks: batch_plan).
inline void sweep_units(SweepArgs &a, int kprof, int fermion, int nint, double items,
                        bool alone = true) {
  const int loops = a.n_chunks * a.chunk_loops, unit = sweep_loop_pairs(kprof) ? 2 : 1;
  const double w = items / kSweepSlots, x = a.nF / (a.ppl * profile_weight(kprof, fermion, nint));
  const double line = kprof == kGaussian ? 0.015 : alone ? 0.012 : 0.005;
  const bool split = w <= 16.0 && x * w * (w < 1.0 ? w : 1.0) < line;
  a.per_loop = a.chunk_loops == 1 || split;
  a.unit_loops = a.per_loop ? unit : a.chunk_loops;
  a.n_units = (loops + a.unit_loops - 1) / a.unit_loops;
}
constexpr double kNoSplit = 1e300;  // items of a launch that keeps whole chunks

// Kahan blocks of a loop's walk: 8 groups, counted from the loop's first walked
// group (1) up to group 64 and from multiples of 64 groups (256 points) after it
inline __host__ __device__ int loop_blocks(int nq) {
  return nq <= 64 ? (nq + 6) / 8 : 8 + (nq - 64 + 7) / 8;
}
inline __host__ __device__ int block_begin(int b) { return b < 8 ? 1 + 8 * b : 8 * b; }

// A heavy profile's launch of fewer than two waves of single-loop units (8 CTAs
// per SM, sweep_min_ctas): its loops are cut further, at their Kahan blocks, into
// about four waves of warps (at most 8 blocks, a landing zone, each); a second
// kernel adds the blocks in the walk's order.  Sets a.parts (0: not cut) and
// returns the floats needed.
//   Bound by latency there: fixflux, 64 instances on 512 x 512 points (1024
// units), issued in a fifth of the cycles: 48.2 -> 26.9 ms, and 21 with 8 CTAs
// per SM; periodic, 128 instances on 1024 x 512 (4096 units): 32.7 -> 23.9 ms.
// Two waves instead of four 5 % slower, eight the same.
inline size_t sweep_parts(SweepArgs &a, bool heavy) {
  constexpr size_t kMost = (size_t)64 << 20;  // floats (256 MB)
  const long long units = (long long)((a.ninst + 31) / 32) * a.n_chunks * a.chunk_loops;
  a.parts = 0;
  if (!heavy || !a.per_loop || units >= 4 * kSweepSlots) return 0;
  const int nb = loop_blocks(a.ppl / 4);
  int parts = (int)((8 * kSweepSlots + units - 1) / units);
  if (parts < (nb + 7) / 8) parts = (nb + 7) / 8;
  if (parts > nb) parts = nb;
  const size_t need = (size_t)a.n_chunks * a.chunk_loops * (nb + 2) * 6 * a.ninst;
  if (parts < 2 || need > kMost) return 0;
  a.part_blocks = (nb + parts - 1) / parts;
  a.parts = (nb + a.part_blocks - 1) / a.part_blocks;
  return need;
}
inline bool heavy_profile(int kprof) {
  return kprof == kPeriodic || kprof == kSpline || kprof == kFixflux || kprof == kFixfluxFF;
}

// Persistent multi-job sweep: a queue of tiles (job, instance tile, loop
// chunk) drained by one CTA per slot; jobs differ in ensemble, profile,
// instances, flux values and loops per tile.
struct BatchTile {
  int job, tile_x, chunk, cost;
};
// Partial sums [n_chunks * inner][nF][3][ninst] of one job: cpg chunks per group
// of lpg loops, each chunk one sum (inner = 1) or its inner loops one by one.
struct ReduceShape {
  const double *partial;
  int n_chunks, cpg, inner, lpg, ninst, nF;
};
constexpr int kReduceThreads = 256;
// Instances per CTA of a reduction: 32 (a warp reads 256 contiguous bytes)
// when that fills the chip, else fewer, down to the 4 of a 32-byte sector: the
// FP64 additions (2 lanes per SM per clock) then run on all SMs, and more groups
// at once.
inline int reduce_instances(int ninst, int nF) {
  int ti = 32;
  while (ti > 1 && ti / 2 >= ninst) ti /= 2;
  while (ti > 4 && (long long)((ninst + ti - 1) / ti) * nF < 304) ti /= 2;
  return ti;
}
struct ReduceJob {  // per job: where its partial sums and outputs live
  ReduceShape shape;
  double *out_group, *out_mean, *out_sem;
  int ti, first;  // instances per CTA, first CTA of the job
};
// CTAs of one job's reduction
inline int reduce_blocks(const ReduceJob &r) {
  return (r.shape.ninst + r.ti - 1) / r.ti * r.shape.nF;
}
struct BatchArgs {
  const SweepArgs *jobs;
  const BatchTile *tiles;
  int ntiles;
  int *counter;  // next tile to take
};
cudaError_t launch_batch(const BatchArgs &a, int grid, cudaStream_t s);
cudaError_t launch_batch_reduce(const ReduceJob *jobs, int njobs, int blocks, cudaStream_t s);
// largest number of batch-kernel CTAs resident per SM
int batch_max_ctas_per_sm();
// every profile batches; the heavy ones (periodic, spline, fixflux) are not
// instantiated in the persistent kernel (their tiles would triple its
// compilation time) and run as chunk-range launches of their own sweep
// kernel beside it, with the same partial-sum layout
bool batch_supports(int kprof, int nint);
bool batch_in_kernel(int kprof);
bool plain_supports(int kprof);

// Loop-parallel sweep: one warp per (loop, instance), lanes over groups of
// four points; per-loop results.  Used for few instances and for EV().
constexpr int kLoopWarps = 4;  // warps per CTA

struct LoopArgs {
  const float4 *loops;
  int Nl, ppl;
  int ninst;
  const float *cx, *cy, *rtT, *tqh, *tql;
  int nF;
  float F[kMaxF];
  float cph_hi[kMaxF], cph_lo[kMaxF], csp_hi[kMaxF], csp_lo[kMaxF];
  FieldDev field;
  double *partial;  // [Nl][nF][3][ninst]  (chunk = one loop)
  float4 *scal;     // optional [ninst][Nl] Wsscal of F[0]
  float4 *ferm;     // optional [ninst][Nl] Wsferm of F[0]
  const float4 *bbox;  // lattice: [Nl] unit-loop bounding boxes
  // optional (one instance): the ensemble's fingerprint (point_hash, zeroed by
  // the caller), from the very points the sweep reads
  unsigned long long *fingerprint;
  int split;  // two warps per (loop, instance)
};

// plain per-instance kernel (the batching baseline), light profiles only
cudaError_t launch_plain(int kprof, bool fermion, int nint, const LoopArgs &a, int inst,
                         cudaStream_t st);

// returns cudaErrorInvalidValue for an unsupported (profile, nint)
cudaError_t launch_sweep(int profile, bool fermion, int nint, const SweepArgs &a,
                         cudaStream_t s);
cudaError_t launch_loopwarp(int profile, bool fermion, int nint, const LoopArgs &a,
                            cudaStream_t s);

// partial sums -> per-group <W>, mean and SEM over groups
// (status_out, may be NULL: receives the status word as a double)
cudaError_t launch_group_reduce(const ReduceShape &r, double *out_group, double *out_mean,
                                double *out_sem, const int *status, double *status_out,
                                cudaStream_t s);

// EV(): mean over an index list of per-loop W factors (partial with
// ninst = 1, nF = 1) and the Richardson combination; writes one double.
cudaError_t launch_list_mean(const double *partial, const int *list, int n, double *out,
                             cudaStream_t s);
// the same for the ngroups lists of n consecutive loops (g n .. g n + n - 1),
// one double per group, each summed exactly as launch_list_mean sums it
cudaError_t launch_group_list_means(const double *partial, int n, int ngroups, double *out,
                                    cudaStream_t s);

// device-resident instances (cx, cy, T) -> the sweep's float arrays
// [cx | cy | rtT | tq_hi | tq_lo]; flags T <= 0 or non-finite values in *status
cudaError_t launch_instance_setup(const double *cx, const double *cy, const double *T,
                                  int ninst, int ppl, float *out, int *status,
                                  cudaStream_t s);

// pipe throughput probes: kind 0 FP32 FMA chains, 1 MUFU rcp chains;
// each thread performs iters * 8 operations
// one CTA waiting (bounded) on an mbarrier that gets its arrival or not
cudaError_t launch_wait_selftest(int *status, uint32_t max_tries, int arrive, cudaStream_t s);
cudaError_t launch_peak_probe(int kind, int blocks, int threads, int iters, float *sink,
                              cudaStream_t s);

// FP64 proper-time integral + jackknife (wl_tint.cu)
struct TintArgs {
  const double *groups;  // [nrho * nT][nF][ng]   instance i = r * nT + k
  const double *rho;     // [nrho] centre of mass x (y = 0, as rhogrand, EffAct.c:23-25)
  const double *T;       // [nT]
  const double *w;       // [nT] quadrature weights in T (dT, Simpson on ln T)
  const double *F;       // [nF]
  int nrho, nT, nF, ng, nbins;
  int profile, fermion;
  double l2, a, lmin, m2, e;
  double rimg2;   // lattice: (rimage / a)^2
  double xcm_x;   // scratch: the centre of mass of the current evaluation
  double *igrand;  // optional [nrho][nF][nT][ng]
  double *Ig;      // [nrho][nF][ng]
  double *leff, *err;  // [nrho][nF]
  // optional: the launch's status word, copied as a double behind the results
  const int *status;
  double *status_out;
};
cudaError_t launch_tint(const TintArgs &a, cudaStream_t s);

// perm[0..n) = instances in decreasing rtT, then by the centre's position in
// its lattice cell (one CTA, bucketed; the order inside a bucket is arbitrary
// and changes no result)
cudaError_t launch_order_instances(const float *cx, const float *cy, const float *rtT, int n,
                                   float inv_a, int *perm, cudaStream_t s);

// 64-bit fingerprint of the (x, y) coordinates of npts float4 points (zeroes
// *out first; EV()'s check that a cached ensemble was not rewritten)
cudaError_t launch_fingerprint(const float4 *loops, size_t npts, unsigned long long *out,
                               cudaStream_t s);

// per-loop bounding boxes of an ensemble (lattice image selection)
cudaError_t launch_loop_bbox(const float4 *loops, int Nl, int ppl, float4 *out, cudaStream_t s);

// seeded unit loops
cudaError_t launch_vloops(uint64_t seed, int first, int Nl, int ppl, float4 *out,
                          cudaStream_t s);

constexpr int kInstArrays = 5;  // cx, cy, rtT, tq_hi, tq_lo

}  // namespace wl
