// wl_batch.cu -- persistent multi-job sweep and its batched reduction.
//
// Many evaluations of uneven size (different ensembles, profiles, flux
// values, instance counts, loops per tile) run as one launch: every warp takes
// units from a global queue (atomicAdd on a counter) until it is empty and
// runs the same code as the single-job sweep (warp_unit), so a job's partial
// sums -- and its results -- do not depend on the batch.  The host orders tiles
// by decreasing cost so the queue drains evenly.
#include "wl_device.cuh"
#include "wl_internal.h"
#include "wl_reduce.cuh"
#include "wl_sweep.cuh"

namespace wl {

namespace {

// The persistent kernel's CTAs are single warps (a slot of the launch's grid is
// four of them): a warp that finds the queue empty leaves at once, where in a
// CTA of four each waited for the slowest (an uneven batch of six jobs 18.7 ->
// 18.4 ms).
// Dynamic shared memory: the warp's stage, its barrier, its job's parameters.
constexpr int kBatchBar = kLatStageBytes;
constexpr int kBatchJob = kBatchBar + 16;
constexpr int kBatchSmem = kBatchJob + 16 * (((int)sizeof(SweepArgs) + 15) / 16);
extern __shared__ __align__(128) unsigned char batch_smem[];

__device__ __forceinline__ SweepArgs &warp_job() {
  return *reinterpret_cast<SweepArgs *>(batch_smem + kBatchJob);
}
__device__ __forceinline__ WarpStage batch_stage() {
  float4 *const land = reinterpret_cast<float4 *>(batch_smem);
  return WarpStage{land, land + kLandPts, reinterpret_cast<uint64_t *>(batch_smem + kBatchBar), 0u};
}

// A called function per kind: each is allocated registers on its own (inlined,
// the 28 of them spilled 420 bytes and the kernel ran an uneven batch of six
// jobs in 43.9 ms; called, and with the lattice units first, 20.0 ms; CTA tiles
// of 256 instances, 33 ms).  It finds its stage and job in shared memory itself:
// through pointer arguments the walk's loads were generic ones, and the field's
// constants were loaded at every segment (4000 smooth instances on 4096 x 1024
// points, scalar, 20.0 -> 18.5 ms).
// Takes and returns the stage's count of copies; ~0u: a copy timed out.
template <int P, bool FERM, int NINT, bool PAIR>
__device__ __noinline__ uint32_t unit_called(int tile, int l0, int l1, size_t row,
                                             uint32_t copies) {
  const SweepArgs &A = warp_job();
  WarpStage W = batch_stage();
  W.copies = copies;
  bool ok;
  if constexpr (P == kLattice && PAIR)
    ok = warp_unit_lattice<FERM, false, const FieldDev>(A, tile, l0, l1, row, W);
  else
    ok = warp_unit<P, FERM, NINT, PAIR, const FieldDev>(A, tile, l0, l1, row, W);
  return ok ? W.copies : ~0u;
}

// One warp's unit of a job: loop pairs for the light profiles, two instances
// per lane for the lattice at 4 intervals -- as the single-job sweep, so such a
// job's loops match it bit for bit -- one loop at a time otherwise.
template <bool FERM, int NINT>
__device__ __forceinline__ uint32_t run_unit(int kprof, int tile, int l0, int l1, size_t row,
                                             uint32_t copies) {
  switch (kprof) {
    case kSmooth: return unit_called<kSmooth, FERM, NINT, true>(tile, l0, l1, row, copies);
    case kSmoothWide:
      if constexpr (NINT == 4)
        return unit_called<kSmoothWide, FERM, 4, true>(tile, l0, l1, row, copies);
      return copies;
    case kGaussian: return unit_called<kGaussian, FERM, NINT, true>(tile, l0, l1, row, copies);
    case kStep: return unit_called<kStep, FERM, NINT, true>(tile, l0, l1, row, copies);
    case kQuadratic: return unit_called<kQuadratic, FERM, NINT, true>(tile, l0, l1, row, copies);
    case kLattice:
      if constexpr (NINT == 4)
        return unit_called<kLattice, FERM, 4, true>(tile, l0, l1, row, copies);
      if constexpr (NINT == 0)
        return unit_called<kLattice, FERM, 0, false>(tile, l0, l1, row, copies);
      return copies;
    default: return copies;
  }
}

constexpr int kBatchMinSlots = 4;  // per SM

// Every warp takes units from the queue (a tile holds kSweepWarps of them) and
// works alone.
__global__ void __launch_bounds__(32, kBatchMinSlots * kSweepWarps)
    batch_kernel(const __grid_constant__ BatchArgs B) {
  const int lane = threadIdx.x;
  SweepArgs &job = warp_job();
  warp_stage_init(batch_stage().bar);
  uint32_t copies = 0;
  int have = -1;  // the job whose parameters this warp holds
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(B.counter, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t / kSweepWarps >= B.ntiles) break;
    const BatchTile d = B.tiles[t / kSweepWarps];
    if (d.job != have) {  // copied word by word
      const int *src = reinterpret_cast<const int *>(B.jobs + d.job);
      int *dst = reinterpret_cast<int *>(&job);
      for (int i = lane; i < (int)(sizeof(SweepArgs) / 4); i += 32) dst[i] = src[i];
      __syncwarp();
      have = d.job;
    }
    const int tile = d.tile_x * kSweepWarps + t % kSweepWarps;
    if (tile >= job.n_tiles) continue;
    int l0, l1;
    const size_t row = unit_loops(job, d.chunk, l0, l1);
    // 4 and 50 intervals (the reference's) unrolled, any other count at run time
    const int k = job.kprof == kSmooth && job.nint == 4 && smooth_clamp_idle(job.field)
                      ? kSmoothWide
                      : job.kprof;
    const bool n50 = job.nint == 50 && light_profile(k);
    if (job.fermion) {
      if (job.nint == 4) copies = run_unit<true, 4>(k, tile, l0, l1, row, copies);
      else if (n50) copies = run_unit<true, 50>(k, tile, l0, l1, row, copies);
      else copies = run_unit<true, 0>(k, tile, l0, l1, row, copies);
    } else {
      if (job.nint == 4) copies = run_unit<false, 4>(k, tile, l0, l1, row, copies);
      else if (n50) copies = run_unit<false, 50>(k, tile, l0, l1, row, copies);
      else copies = run_unit<false, 0>(k, tile, l0, l1, row, copies);
    }
    if (copies == ~0u) break;  // a copy timed out: the status is set, stop taking units
    __syncwarp();              // the job's parameters may be rewritten next
  }
}

// the jobs' reductions as one launch: a CTA's job by binary search
__global__ void __launch_bounds__(kReduceThreads)
    batch_reduce_kernel(const ReduceJob *__restrict__ jobs, int njobs) {
  const int b = blockIdx.x;
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (jobs[mid].first <= b) lo = mid;
    else hi = mid - 1;
  }
  const ReduceJob J = jobs[lo];
  const int nx = (J.shape.ninst + J.ti - 1) / J.ti;
  reduce_block(J.shape, (b - J.first) % nx * J.ti, (b - J.first) / nx, J.ti, J.out_group,
               [&](size_t at, double mean, double sem) {
                 J.out_mean[at] = mean;
                 J.out_sem[at] = sem;
               });
}

// The plain per-instance kernel: one thread per loop walking its points from
// global memory (AoS float4, strided by ppl between threads), the structure of
// the reference's ExpectValue (intEV.cu:573-582) with this library's segment
// arithmetic; one launch per instance.
template <int P, bool FERM, int NINT>
__global__ void __launch_bounds__(128) plain_kernel(const __grid_constant__ LoopArgs A, int inst) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= A.Nl) return;
  const float cx = A.cx[inst], cy = A.cy[inst], s = A.rtT[inst];
  const df tq = {A.tqh[inst], A.tql[inst]};
  const FieldDev &F = A.field;
  const float4 *w = A.loops + (size_t)l * A.ppl;
  ImgRange img = {0, -1, 0, -1, 1};  // lattice: this loop's images
  if constexpr (P == kLattice) img = image_range(A.bbox[l], s, cx, cy, F);
  auto pt = [&](int p, float &x, float &y) {
    const float4 v = w[p];
    x = fmaf(s, v.x, cx);
    y = fmaf(s, v.y, cy);
  };
  float ph[3] = {0.f, 0.f, 0.f}, sp[3] = {0.f, 0.f, 0.f};
  float z0x, z0y, z1x, z1y, z2x, z2y, z3x, z3y;
  pt(0, z0x, z0y);
  pt(1, z1x, z1y);
  pt(2, z2x, z2y);
  pt(3, z3x, z3y);
  seg<P, FERM, NINT>(z1x, z1y, z3x, z3y, F, img, ph[0], sp[0]);
  float zAx = z0x, zAy = z0y, zBx = z2x, zBy = z2y, zOx = z3x, zOy = z3y;
  for (int q = 1; q < A.ppl / 4; ++q) {
    float P0x, P0y, P1x, P1y, P2x, P2y, P3x, P3y;
    pt(4 * q, P0x, P0y);
    pt(4 * q + 1, P1x, P1y);
    pt(4 * q + 2, P2x, P2y);
    pt(4 * q + 3, P3x, P3y);
    seg<P, FERM, NINT>(zAx, zAy, P0x, P0y, F, img, ph[2], sp[2]);
    seg<P, FERM, NINT>(zOx, zOy, P1x, P1y, F, img, ph[0], sp[0]);
    seg<P, FERM, NINT>(zBx, zBy, P2x, P2y, F, img, ph[1], sp[1]);
    seg<P, FERM, NINT>(P1x, P1y, P3x, P3y, F, img, ph[0], sp[0]);
    zAx = P0x; zAy = P0y;
    zBx = P2x; zBy = P2y;
    zOx = P3x; zOy = P3y;
  }
  seg<P, FERM, NINT>(zOx, zOy, z1x, z1y, F, img, ph[0], sp[0]);
  seg<P, FERM, NINT>(zBx, zBy, z2x, z2y, F, img, ph[1], sp[1]);
  seg<P, FERM, NINT>(zAx, zAy, z0x, z0y, F, img, ph[2], sp[2]);
  const df G[3] = {df{ph[0], 0.f}, df{ph[1], 0.f}, df{ph[2], 0.f}};
  const df H[3] = {df{sp[0], 0.f}, df{sp[1], 0.f}, df{sp[2], 0.f}};
  loop_epilogue<FERM>(G, H, A.cph_hi, A.cph_lo, A.csp_hi, A.csp_lo, tq, A.nF,
                      [&](int j, double d0, double d1, double d2) {
                        double *o = A.partial + ((size_t)(l * A.nF + j) * 3) * A.ninst + inst;
                        o[0] = d0;
                        o[A.ninst] = d1;
                        o[2 * (size_t)A.ninst] = d2;
                      });
}

template <bool FERM, int NINT>
cudaError_t plain_dispatch(int kprof, const LoopArgs &a, int inst, cudaStream_t st) {
  const dim3 grid((a.Nl + 127) / 128);
  switch (kprof) {
    case kSmooth: plain_kernel<kSmooth, FERM, NINT><<<grid, 128, 0, st>>>(a, inst); break;
    case kGaussian: plain_kernel<kGaussian, FERM, NINT><<<grid, 128, 0, st>>>(a, inst); break;
    case kStep: plain_kernel<kStep, FERM, NINT><<<grid, 128, 0, st>>>(a, inst); break;
    case kQuadratic: plain_kernel<kQuadratic, FERM, NINT><<<grid, 128, 0, st>>>(a, inst); break;
    case kLattice: plain_kernel<kLattice, FERM, NINT><<<grid, 128, 0, st>>>(a, inst); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_plain(int kprof, bool fermion, int nint, const LoopArgs &a, int inst,
                         cudaStream_t st) {
  if (fermion)
    return nint == 4 ? plain_dispatch<true, 4>(kprof, a, inst, st)
                     : plain_dispatch<true, 0>(kprof, a, inst, st);
  return nint == 4 ? plain_dispatch<false, 4>(kprof, a, inst, st)
                   : plain_dispatch<false, 0>(kprof, a, inst, st);
}

bool batch_supports(int kprof, int nint) {
  (void)nint;
  return kprof >= kStep && kprof <= kLattice;
}

bool batch_in_kernel(int kprof) { return light_profile(kprof) || kprof == kLattice; }

bool plain_supports(int kprof) { return light_profile(kprof) || kprof == kLattice; }

int batch_max_ctas_per_sm() {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_kernel, 32, kBatchSmem) !=
      cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return n >= kSweepWarps ? n / kSweepWarps : 1;
}

// The queue's counter counts kSweepWarps units per tile in 32 bits, so a launch
// takes at most kBatchLaunchTiles tiles and a larger batch several launches (a
// 64-bit counter: served requests 3 % slower).
constexpr int kBatchLaunchTiles = 1 << 28;

cudaError_t launch_batch(const BatchArgs &a, int grid, cudaStream_t s) {
  BatchArgs b = a;
  for (int first = 0; first < a.ntiles; first += b.ntiles) {
    b.tiles = a.tiles + first;
    b.ntiles = a.ntiles - first < kBatchLaunchTiles ? a.ntiles - first : kBatchLaunchTiles;
    if (first > 0) {
      const cudaError_t e = cudaMemsetAsync(b.counter, 0, sizeof(int), s);
      if (e != cudaSuccess) return e;
    }
    batch_kernel<<<grid * kSweepWarps, 32, kBatchSmem, s>>>(b);
  }
  return cudaGetLastError();
}

cudaError_t launch_batch_reduce(const ReduceJob *jobs, int njobs, int blocks, cudaStream_t s) {
  batch_reduce_kernel<<<blocks, kReduceThreads, 0, s>>>(jobs, njobs);
  return cudaGetLastError();
}

}  // namespace wl
