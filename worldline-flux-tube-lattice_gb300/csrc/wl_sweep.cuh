// wl_sweep.cuh -- the two Wilson-loop sweep kernels.
//
// Both compute, per (loop, instance), the reference kernel's per-loop phases
// (ExpectValue -> WilsonLoop, intEV.cu:508-582) and the EVMean factors
// (Integrand.c:352-390), and write FP64 partial sums of the W factors.
//
// sweep kernels (instance-parallel): lane = instance (centre of mass, proper
//   time), warp = 32 instances x a unit of loops.  Every warp works alone: it
//   streams its own loops through shared memory with bulk copies
//   (cp.async.bulk + mbarrier, the next piece in flight while one is walked),
//   and every lane walks every staged point, so each shared-memory load is a
//   warp-wide broadcast and the ensemble comes from HBM about once per launch
//   (the warps of other instances read it from L2).  Within a loop the points
//   are visited in order; the three sub-loops (N/2: odd points, N/4a: i = 0
//   mod 4, N/4b: i = 2 mod 4; intEV.cu:461-506) advance together, one group of
//   four points (four segments) at a time, and each segment adds to its
//   sub-loop in the reference's order.  Phases accumulate in FP32 with Kahan
//   compensation per block of 8 groups; W factors accumulate in FP64.
//
// loopwarp_kernel (loop-parallel): warp = (loop, instance), lanes over the
//   groups of four points; per-loop results (EV() and few-instance calls).
#pragma once

#include <type_traits>

#include "wl_device.cuh"
#include "wl_internal.h"

namespace wl {

// the fixflux segment's per-warp queues assume CTAs of kFfWarps warps
static_assert(kSweepThreads == 32 * kFfWarps && kLoopWarps == kFfWarps,
              "fixflux queues: 4 warps per CTA");

// ------------------------------------------------------ staging per warp --
// A warp's staging area: the landing zone of its bulk copies, the compact copy of
// a piece's coordinates that the lanes walk, and for sweep_kernel's loop pairs the
// first points of the loops and the chunk's running sums.  `copies` counts the pieces this
// warp has waited for (its barrier's phase continues across units).
struct WarpStage {
  float4 *land;   // [kLandPts] float4 points as the ensemble holds them
  float4 *comp;   // the piece's coordinates, laid out for its walk
  uint64_t *bar;  // the warp's mbarrier
  uint32_t copies;
  // pairs: points 0..2 of the walked loops, as in comp
  __device__ float4 *first() const { return land + kLandPts * 3 / 2; }
  // pairs: [kMaxF][3][32 lanes]
  __device__ double *sums() const { return reinterpret_cast<double *>(first() + 4); }
};

__device__ __forceinline__ void warp_stage_init(uint64_t *bar) {
  if ((threadIdx.x & 31) == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  __syncwarp();
}

// Waits (bounded) for the piece in flight; on a time-out waits once more, so
// that the copy does not land after the warp has left, and reports.
__device__ __forceinline__ bool warp_stage_wait(const SweepArgs &A, WarpStage &W) {
  const uint32_t par = W.copies & 1u;
  const bool ok = mbar_wait_bounded(W.bar, par, A.wait_tries);
  if (!__all_sync(0xffffffffu, ok)) {
    mbar_wait_bounded(W.bar, par, A.wait_tries);
    if ((threadIdx.x & 31) == 0) atomicExch(A.status, kDevTimeout);
    return false;
  }
  ++W.copies;
  return true;
}

// W - 1 of one loop at one instance into the partial sums: stored on its own
// (per_loop) or added to its chunk's sum, which the same lane keeps in loop
// order (acc: not the chunk's first loop).
__device__ __forceinline__ void put_loop(const SweepArgs &A, size_t row, int j, int ic, bool acc,
                                         double d0, double d1, double d2) {
  double *o = A.partial + (row * A.nF + j) * 3 * A.ninst + ic;
  const size_t n = (size_t)A.ninst;
  if (acc) {
    d0 += o[0];
    d1 += o[n];
    d2 += o[2 * n];
  }
  o[0] = d0;
  o[n] = d1;
  o[2 * n] = d2;
}

// The same for sweep_kernel's loop pairs, a chunk's sums kept in the warp's shared memory
// until its last loop (`last`).  Added to in global memory they took a round trip
// per loop and flux, one after another (the stores may alias the next loads): 1024
// Gaussian instances at four fluxes on 1024 loops of 64 points 321 -> 306 us.
__device__ __forceinline__ void put_pair_loop(const SweepArgs &A, const WarpStage &W, size_t row,
                                              int j, int ic, bool live, bool acc, bool last,
                                              double d0, double d1, double d2) {
  double *const s = W.sums() + j * 96 + (threadIdx.x & 31);
  if (acc) {
    d0 += s[0];
    d1 += s[32];
    d2 += s[64];
  }
  if (!last) {
    s[0] = d0;
    s[32] = d1;
    s[64] = d2;
  } else if (live) {
    double *o = A.partial + (row * A.nF + j) * 3 * A.ninst + ic;
    o[0] = d0;
    o[A.ninst] = d1;
    o[2 * (size_t)A.ninst] = d2;
  }
}

// scalar and pair arithmetic of the walk under one name
__device__ __forceinline__ float vset(float, float a) { return a; }
__device__ __forceinline__ float2 vset(float2, float a) { return f2(a); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return fma2(a, b, c); }
__device__ __forceinline__ void vkahan(float &s, float &c, float x) { kahan_add(s, c, x); }
__device__ __forceinline__ void vkahan(float2 &s, float2 &c, float2 x) { kahan_add2(s, c, x); }
__device__ __forceinline__ float vlane(float v, int) { return v; }
__device__ __forceinline__ float vlane(float2 v, int h) { return h ? v.y : v.x; }
template <bool PAIR>
struct Vec {
  using T = float;
};
template <>
struct Vec<true> {
  using T = float2;
};

// one segment; EDGE: a loop's opening or a closing segment
template <int P, bool FERM, int NINT, bool EDGE = false>
__device__ __forceinline__ void vseg(float zix, float ziy, float zjx, float zjy,
                                     const FieldDev &F, const ImgRange &img, float &ph,
                                     float &sp) {
  seg<P, FERM, NINT, kSqRound>(zix, ziy, zjx, zjy, F, img, ph, sp);
}
template <int P, bool FERM, int NINT, bool EDGE = false>
__device__ __forceinline__ void vseg(float2 zix, float2 ziy, float2 zjx, float2 zjy,
                                     const FieldDev &F, const ImgRange &, float2 &ph,
                                     float2 &sp) {
  seg2<P, FERM, NINT, EDGE>(zix, ziy, zjx, zjy, F, ph, sp);
}

// end of the Kahan block that holds group q (loop_blocks)
__device__ __forceinline__ int block_end(int q) {
  return q < 64 ? min(((q - 1) & ~7) + 9, 64) : (q & ~7) + 8;
}

// Groups of a walk in straight-line code: 4 where they fit the registers (smooth,
// the scalar step profile: 5 % over 2 at 512 points per loop), 2 elsewhere (scalar
// quadratic 1-4 % over 4, 9-12 % at four fluxes), 1 around a run-time node loop.  The
// persistent kernel (MIXED) runs several kinds of unit on an SM at once, whose
// code then competes for the instruction cache: 1 for the kinds that get 4 here
// (served smooth and Gaussian requests 4.9e11 segments/s at 4, 5.4e11 at 2,
// 5.57e11 at 1; the other kinds at 1 too 5.52e11).
template <int P, bool FERM, int NINT, bool MIXED>
constexpr int walk_unroll() {
  if (NINT == 0) return 1;
  if (NINT == 4 && (smooth_profile(P) || (P == kStep && !FERM))) return MIXED ? 1 : 4;
  return 2;
}
static_assert(walk_unroll<kStep, false, 4, false>() == 4 &&
                  walk_unroll<kStep, false, 4, true>() == 1 &&
                  walk_unroll<kStep, true, 4, false>() == 2 &&
                  walk_unroll<kQuadratic, false, 4, false>() == 2 &&
                  walk_unroll<kSmoothWide, true, 4, false>() == 4,
              "profiles as the comment names them");

// One unit of a warp: instances [32 tile, +32), one per lane, over loops
// [l0, l1).  PAIR: the lane walks loops l and l + 1 together as a packed pair:
// every FP32 operation of a segment is one f32x2 operation on the two loops
// (each half rounds as the scalar walk does), and the staged piece interleaves
// the two loops' coordinates (x, x', y, y'), so that one 16-byte broadcast load
// gives both operands already packed.
//   Bound by the SM's dispatch: a packed operation takes two of its cycles, so
// a pair-segment of the smooth spinor profile spends 68 on FP32 arithmetic, 10
// on reciprocals (80 on the MUFU) and ~13 on clamps, loads and loop control.
// Tiles of 256 instances on one loop (two per thread, a CTA barrier per piece)
// left lanes dead below 256 instances and slots empty below ~600 CTAs.
// Measured, 256-instance tiles -> warp units: 96 instances x 3 fluxes on 5120 x
// 2048 points 3.14 -> 1.15 ms; 8192 instances there 101.3 -> 98.6 ms (8.8e11
// segments/s); smooth scalar at 50 intervals, 3160 instances on 5120 x 1024,
// 152.3 -> 143.5 ms.  Run-time interval counts, one instance per thread -> loop
// pairs: Gaussian spinor at 16 intervals, 333 instances on 1500 x 516, 4.83 ->
// 2.65 ms.  One lane per instance, one CTA per chunk -> one warp per loop, 50
// intervals: periodic, 128 instances on 1024 x 512, 103 -> 32.7 ms; fixflux, 64
// instances on 512 x 512, 375 -> 92 ms (48 with its segment's smaller code).
//   row: the partial-sum row of loop l0 (per_loop) or of the unit's chunk.
// Returns false if a copy timed out.
template <int P, bool FERM, int NINT, bool PAIR, class Field = const FieldDev &>
__device__ __forceinline__ bool warp_unit(const SweepArgs &A, int tile, int l0, int l1,
                                          size_t row, WarpStage &W) {
  using V = typename Vec<PAIR>::T;
  constexpr int kLoops = PAIR ? 2 : 1;         // loops walked together
  constexpr int kPiece = kLandPts / kLoops;    // points per staged piece
  // the persistent kernel (Field by value) keeps the longer forms below: called
  // units of long loops lose 3 % by the shorter ones (served smooth requests 8.04e11
  // -> 7.82e11 segments/s, an uneven batch of six jobs 18.0 -> 18.6 ms)
  constexpr bool kMixed = !std::is_reference<Field>::value;
  constexpr int kUnroll = walk_unroll<P, FERM, NINT, kMixed>();
  constexpr bool kSums = PAIR && !kMixed;  // put_pair_loop
  // the loops' first points kept in shared memory for their closing segments; read
  // again from the ensemble a pair waits for them (50 intervals: Gaussian scalar 3 %,
  // smooth spinor 1 %), but the smooth scalar kernel at 50 compiles to a faster walk
  // that way (3160 instances on 2048 x 1024 points 56.8 ms, 57.7 with them kept)
  constexpr bool kFirst = kSums && !(smooth_profile(P) && !FERM && NINT == 50);
  const int lane = threadIdx.x & 31;
  const int slot = tile * 32 + lane;
  const bool live = slot < A.ninst;
  const int sl = live ? slot : A.ninst - 1;
  // every per-instance read and the partial-sum write go through ic: a lane's
  // result does not depend on which slot it runs in
  const int ic = A.perm ? A.perm[sl] : sl;
  Field F = A.field;  // by value where A is not in the constant bank
  const V cx = vset(V(), A.cx[ic]), cy = vset(V(), A.cy[ic]), s = vset(V(), A.rtT[ic]);

  auto issue = [&](int l, int p0) {  // points p0.. of the kLoops loops from l
    const uint32_t bytes = (uint32_t)(min(kPiece, A.ppl - p0) * (int)sizeof(float4));
    const bool two = PAIR && l + 1 < l1;
    mbar_arrive_expect_tx(W.bar, two ? 2 * bytes : bytes);
    const float4 *src = A.loops + (size_t)l * A.ppl + p0;
    bulk_g2s(W.land, src, bytes, W.bar);
    if (two) bulk_g2s(W.land + kPiece, src + A.ppl, bytes, W.bar);
  };
  if (lane == 0) issue(l0, 0);

  // running sums of the current loops: phase and spin, each with compensation
  V ph[3], pc[3], sp[3], sc[3], bp[3], bs[3];
  const V zero = vset(V(), 0.f);
  // previous point of each sub-loop
  V zAx = zero, zAy = zero, zBx = zero, zBy = zero, zOx = zero, zOy = zero;
#pragma unroll
  for (int r = 0; r < 3; ++r) ph[r] = pc[r] = sp[r] = sc[r] = bp[r] = bs[r] = zero;
  ImgRange img = {0, -1, 0, -1, 1};  // lattice images of the current loop
  const int nq = A.ppl >> 2;

  int l = l0, p0 = 0;  // the piece's loops and first point
#pragma unroll 1
  while (l < l1) {
    const int np = min(kPiece, A.ppl - p0);
    const bool last = p0 + kPiece >= A.ppl;
    if (!warp_stage_wait(A, W)) return false;
    // compact copy of the piece, then the landing zone is free for the next
    if constexpr (PAIR) {
      const int o = l + 1 < l1 ? kPiece : 0;
      for (int i = lane; i < np; i += 32) {
        const float2 a = *reinterpret_cast<const float2 *>(W.land + i);
        const float2 b = *reinterpret_cast<const float2 *>(W.land + o + i);
        const float4 v = make_float4(a.x, b.x, a.y, b.y);
        W.comp[i] = v;
        if (kFirst && p0 == 0 && i < 3) W.first()[i] = v;
      }
    } else {
      for (int i = lane; i < np; i += 32)
        reinterpret_cast<float2 *>(W.comp)[i] = *reinterpret_cast<const float2 *>(W.land + i);
    }
    __syncwarp();
    const int ln = last ? l + kLoops : l, pn = last ? 0 : p0 + kPiece;
    if (lane == 0 && ln < l1) issue(ln, pn);

    auto pt = [&](int p, V &x, V &y) {
      if constexpr (PAIR) {
        const float4 v = W.comp[p - p0];
        x = fma2(s, make_float2(v.x, v.y), cx);
        y = fma2(s, make_float2(v.z, v.w), cy);
      } else {
        const float2 v = reinterpret_cast<const float2 *>(W.comp)[p - p0];
        x = fmaf(s, v.x, cx);
        y = fmaf(s, v.y, cy);
      }
    };

    int q = p0 >> 2;
    const int qend = (p0 + np) >> 2;
    if (p0 == 0) {  // first piece of a loop: points 0..3 open the sub-loops
#pragma unroll
      for (int r = 0; r < 3; ++r) ph[r] = pc[r] = sp[r] = sc[r] = zero;
      if constexpr (P == kLattice && !PAIR)
        img = image_range(A.bbox[l], A.rtT[ic], A.cx[ic], A.cy[ic], F);
      V z1x, z1y;
      pt(0, zAx, zAy);
      pt(1, z1x, z1y);
      pt(2, zBx, zBy);
      pt(3, zOx, zOy);
      vseg<P, FERM, NINT, true>(z1x, z1y, zOx, zOy, F, img, ph[0], sp[0]);  // N/2: 1 -> 3
      q = 1;
    }
    while (q < qend) {
      const int be = min(block_end(q), nq), qe = min(be, qend);
      auto group = [&](int qq) {
        V P0x, P0y, P1x, P1y, P2x, P2y, P3x, P3y;
        pt(4 * qq, P0x, P0y);
        pt(4 * qq + 1, P1x, P1y);
        pt(4 * qq + 2, P2x, P2y);
        pt(4 * qq + 3, P3x, P3y);
        vseg<P, FERM, NINT>(zAx, zAy, P0x, P0y, F, img, bp[2], bs[2]);  // N/4a: 4q-4 -> 4q
        vseg<P, FERM, NINT>(zOx, zOy, P1x, P1y, F, img, bp[0], bs[0]);  // N/2 : 4q-1 -> 4q+1
        vseg<P, FERM, NINT>(zBx, zBy, P2x, P2y, F, img, bp[1], bs[1]);  // N/4b: 4q-2 -> 4q+2
        vseg<P, FERM, NINT>(P1x, P1y, P3x, P3y, F, img, bp[0], bs[0]);  // N/2 : 4q+1 -> 4q+3
        zAx = P0x; zAy = P0y;
        zBx = P2x; zBy = P2y;
        zOx = P3x; zOy = P3y;
      };
      if constexpr (Profile<P>::kHeavy || P == kLattice) {
#pragma unroll 1
        for (; q < qe; ++q) group(q);
      } else {
#pragma unroll kUnroll
        for (; q < qe; ++q) group(q);
      }
      if (q == be) {  // the block is complete (it may span two pieces)
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          vkahan(ph[r], pc[r], bp[r]);
          if (FERM) vkahan(sp[r], sc[r], bs[r]);
          bp[r] = bs[r] = zero;
        }
      }
    }

    if (last) {  // last piece: closing segments back to points 1, 0, 2
      // (kept since the first piece in registers they would take six, twelve on a
      // pair, through the whole walk)
      V tp[3] = {zero, zero, zero}, ts[3] = {zero, zero, zero};
      const float2 *g = reinterpret_cast<const float2 *>(A.loops + (size_t)l * A.ppl);
      auto gpt = [&](int p, V &x, V &y) {
        if constexpr (kFirst) {
          const float4 v = W.first()[p];
          x = fma2(s, make_float2(v.x, v.y), cx);
          y = fma2(s, make_float2(v.z, v.w), cy);
        } else if constexpr (PAIR) {
          const float2 a = __ldg(&g[2 * p]);
          const float2 b = l + 1 < l1 ? __ldg(&g[2 * ((size_t)A.ppl + p)]) : a;
          x = fma2(s, make_float2(a.x, b.x), cx);
          y = fma2(s, make_float2(a.y, b.y), cy);
        } else {
          const float2 a = __ldg(&g[2 * p]);
          x = fmaf(s, a.x, cx);
          y = fmaf(s, a.y, cy);
        }
      };
      V zx, zy;
      gpt(1, zx, zy);
      vseg<P, FERM, NINT, true>(zOx, zOy, zx, zy, F, img, tp[0], ts[0]);  // N/2 : N-1 -> 1
      gpt(2, zx, zy);
      vseg<P, FERM, NINT, true>(zBx, zBy, zx, zy, F, img, tp[1], ts[1]);  // N/4b: N-2 -> 2
      gpt(0, zx, zy);
      vseg<P, FERM, NINT, true>(zAx, zAy, zx, zy, F, img, tp[2], ts[2]);  // N/4a: N-4 -> 0
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        vkahan(ph[r], pc[r], tp[r]);
        vkahan(sp[r], sc[r], ts[r]);
      }
      const df tq = {A.tqh[ic], A.tql[ic]};
#pragma unroll 1
      for (int h = 0; h < kLoops; ++h) {  // per-loop epilogue of each half
        if (l + h >= l1) break;
        const df G[3] = {fast_two_sum(vlane(ph[0], h), -vlane(pc[0], h)),
                         fast_two_sum(vlane(ph[1], h), -vlane(pc[1], h)),
                         fast_two_sum(vlane(ph[2], h), -vlane(pc[2], h))};
        const df H[3] = {fast_two_sum(vlane(sp[0], h), -vlane(sc[0], h)),
                         fast_two_sum(vlane(sp[1], h), -vlane(sc[1], h)),
                         fast_two_sum(vlane(sp[2], h), -vlane(sc[2], h))};
        const size_t at = A.per_loop ? row + (l - l0) + h : row;
        const bool acc = !A.per_loop && l + h > l0;
        loop_epilogue<FERM, kSums && NINT != 50>(G, H, A.cph_hi, A.cph_lo, A.csp_hi, A.csp_lo, tq, A.nF,
                            [&](int j, double w0, double w1, double w2) {
                              if constexpr (kSums)
                                put_pair_loop(A, W, at, j, ic, live, acc,
                                              A.per_loop || l + h == l1 - 1, w0, w1, w2);
                              else if (live)
                                put_loop(A, at, j, ic, acc, w0, w1, w2);
                            });
      }
    }
    __syncwarp();  // every lane is done with the compact piece
    l = ln;
    p0 = pn;
  }
  return true;
}

// ------------------------------------------------ lattice, images outer --
// One segment u_i -> u_j for two images at once (packed pair; u = the loop
// point minus the image centre R, scaled): the Gaussian tube's Simpson
// integral in units of x = rho^2 / lambda^2 (exact mode), each half as
// segment_lattice evaluates one image.  Adds cross * S to ph and the spin
// integral to sp (its 1/l2 scale is applied per loop).
//
// Far nodes: at x > 18, e^-x < 1.6e-8 is below half an ulp of 1, so the
// FP32 integrand (1 - e^-x)/x is exactly 1/x; the spin integrand e^-x is
// taken as 0 there (a change below 1.6e-8 of a node's largest value,
// whichever path runs).  With VOTE, when every node of the segment, in both
// halves and on every active lane of the warp, is far, the segment takes the
// reciprocals alone -- one MUFU operation per node instead of two, and none
// of the small-x polynomial -- with results bit-identical to the full path,
// so an instance's sums still do not depend on its warp-mates.  The walks
// over blocks of staged points decide once per block instead (kLatSub).
// With MID the caller knows every node is at x >= 0.5: the integrand's
// large-x form alone (gauss_q2_big), the same bits as gauss_q2 there.
constexpr float kLatFar = 18.0f;

template <bool FERM, bool VOTE = true, bool MID = false>
__device__ __forceinline__ void lat_seg2(float2 uix, float2 uiy, float2 ujx, float2 ujy,
                                         float2 il2, float2 &ph, float2 &sp) {
  const float2 dx = add2(ujx, neg2(uix)), dy = add2(ujy, neg2(uiy));
  const float2 as = mul2(fma2(uix, uix, mul2(uiy, uiy)), il2);
  // b/l2 alone: 2b/l2, the linear coefficient, is its exact double, which
  // the node polynomial takes through exact halvings and doublings of t
  const float2 bs = mul2(fma2(uix, dx, mul2(uiy, dy)), il2);
  const float2 cs = mul2(fma2(dx, dx, mul2(dy, dy)), il2);
  const float2 cross = mul2(fma2(uix, dy, neg2(mul2(uiy, dx))), il2);
  float2 x[5];
  x[0] = as;
  x[4] = add2(fma2(bs, f2(2.0f), as), cs);  // (as + 2bs) + cs
#pragma unroll
  for (int j = 1; j < 4; j++) {
    const float t = (float)j * 0.25f;
    x[j] = fma2(fma2(cs, f2(0.5f * t), bs), f2(2.0f * t), as);  // as + t (2bs + cs t)
  }
  float xmin = fminf(x[0].x, x[0].y);
#pragma unroll
  for (int j = 1; j < 5; j++) xmin = fminf(xmin, fminf(x[j].x, x[j].y));
  if (VOTE && __all_sync(__activemask(), xmin > kLatFar)) {
    // 1/x at every node; the Simpson sum in the full path's order
    float2 r[5];
#pragma unroll
    for (int j = 0; j < 5; j++) r[j] = rcp2(x[j]);
    const float2 so = add2(r[1], r[3]);
    const float2 se = r[2];
    ph = fma2(cross, fma2(f2(4.0f), so, fma2(f2(2.0f), se, add2(r[0], r[4]))), ph);
    if (FERM) sp = add2(sp, f2(0.0f));
    return;
  }
  float2 q[5], e[5];
#pragma unroll
  for (int j = 0; j < 5; j++) {
    if (MID)  // every node at x >= 0.5 (the caller's block test); il2 > 0
      gauss_q2_big(x[j], q[j], e[j], il2.x < 0.0f ? 1.0f : -1.0f);
    else
      gauss_q2(x[j], q[j], e[j]);
    if (FERM)
      e[j] = make_float2(x[j].x > kLatFar ? 0.0f : e[j].x, x[j].y > kLatFar ? 0.0f : e[j].y);
  }
  ph = fma2(cross, fma2(f2(4.0f), add2(q[1], q[3]), fma2(f2(2.0f), q[2], add2(q[0], q[4]))), ph);
  if (FERM)
    sp = add2(sp, fma2(f2(4.0f), add2(e[1], e[3]), fma2(f2(2.0f), e[2], add2(e[0], e[4]))));
}

// The far path of lat_seg2 alone (no vote): for a walk whose every node is
// known to be far -- the same operations as lat_seg2 takes when its warp
// agrees, so the sums are bit-identical to either path of lat_seg2.  The
// spin integrand is 0 at every far node and its sum is left as it is (the
// full path would add +0 to a sum that is never -0).
__device__ __forceinline__ void lat_seg2_far(float2 uix, float2 uiy, float2 ujx, float2 ujy,
                                             float2 il2, float2 &ph) {
  const float2 dx = add2(ujx, neg2(uix)), dy = add2(ujy, neg2(uiy));
  const float2 as = mul2(fma2(uix, uix, mul2(uiy, uiy)), il2);
  const float2 bs = mul2(fma2(uix, dx, mul2(uiy, dy)), il2);
  const float2 cs = mul2(fma2(dx, dx, mul2(dy, dy)), il2);
  const float2 cross = mul2(fma2(uix, dy, neg2(mul2(uiy, dx))), il2);
  float2 r[5];
  r[0] = rcp2(as);
  r[4] = rcp2(add2(fma2(bs, f2(2.0f), as), cs));
#pragma unroll
  for (int j = 1; j < 4; j++) {
    const float t = (float)j * 0.25f;
    r[j] = rcp2(fma2(fma2(cs, f2(0.5f * t), bs), f2(2.0f * t), as));
  }
  ph = fma2(cross, fma2(f2(4.0f), add2(r[1], r[3]), fma2(f2(2.0f), r[2], add2(r[0], r[4]))), ph);
}

// A walk of an image over a block of kLatSub staged points is far when the
// block's points (and the earlier points its segments start from) lie in a
// box whose nearest point to the image centre is at x = rho^2/lambda^2 > 19:
// every Simpson node lies on a segment inside the box, and its x computed in
// FP32 stays above 18 (the rounding of rho^2 at these sizes is far below the
// 5 % margin).  Such a walk takes lat_seg2_far; any other takes the full
// path of lat_seg2 without its vote (a far node gives the same sums either
// way).  Measured on the a = 2, 5, 10 lambda lattice workloads against one
// walk per segment with a vote: boxes of 32 points with vote-free near walks
// 11-13 % faster; boxes of 64, 128, 256 points 0.5-3 % slower than 32; the
// near walk with the vote kept 4-9 % slower.  The warps of an SM are in
// different walks at any time, so the walks' instructions have to stay in the
// instruction cache together: with the far and near walks unrolled by two
// groups "no instruction" was the top stall (3.2 cycles per issue); one group
// each (the middle walk keeps two) took 512 instances on 1024 x 1024 points,
// a = 5 lambda, spinor, from 15.5 to 10.6 ms.
constexpr float kLatFarChunk = 19.0f;
// A block whose box stays at x > 0.55 from the image centres has every node
// at x >= 0.5 (the same margin argument), where the integrand takes its
// large-x form: the walk skips the small-x polynomial and its selects.
constexpr float kLatMidChunk = 0.55f;
constexpr int kLatSub = 32;  // staged points per far-test box
constexpr int kLatNSub = kLandPts / kLatSub;
static_assert(kLandPts % kLatSub == 0 && kLatSub % 4 == 0, "whole groups per box");

// the rarely taken opening / closing segments as one called copy
template <bool FERM>
__device__ __noinline__ float4 lat_seg2_called(float2 uix, float2 uiy, float2 ujx, float2 ujy,
                                               float2 il2, float4 acc) {
  float2 ph = make_float2(acc.x, acc.y), sp = make_float2(acc.z, acc.w);
  lat_seg2<FERM>(uix, uiy, ujx, ujy, il2, ph, sp);
  return make_float4(ph.x, ph.y, sp.x, sp.y);
}

// Lattice unit of a warp at 4 intervals with the images outer: two instances
// A, B per lane (slots t and t + 32 of the unit's 64 in the instance order),
// one loop at a time.  For every staged piece of a loop, the images of the two
// (loop, instance) pairs walk all of the piece's segments two at a time as
// packed f32x2 pairs: A's image p beside B's image p while both have one, then
// the longer list's remaining images two at a time -- ceil((K_A + K_B) / 2)
// walks, and at step p the lanes of a warp hold images in the same position
// relative to similar instances.  A loop point minus an image centre is
// image-independent up to the shift, so the walk starts from the raw unit-loop
// points, staged with each coordinate twice (x, x, y, y) so that one 16-byte
// broadcast load gives both packed operands; per image pair the walk is uniform
// across the warp (no per-segment image loop, no row logic).  An instance's
// images are its range of image_range() flattened row by row (k -> m0 + k / w,
// n0 + k % w), its rows trimmed to the |R| disk where the range crosses it; an
// unused half is computed and not added.  Each image's walk over the piece is
// summed in FP32 and added once, in image order, to its instance's
// Kahan-compensated loop totals: an instance's sums do not depend on its
// partner or on the unit's other instances.  Warps do not wait for one another:
// the image counts of a CTA's four warps differ, and a barrier per piece (128
// threads, 256 instances per tile) held them to the largest; 512 instances on
// 1024 x 1024 points, a = 5 lambda, spinor: 29.0 -> 18.0 ms alone.

// shared-memory rows of the loop totals: [instance A/B][phase, its
// compensation, spin, its compensation][sub-loop] x 32 lanes (kept out of
// registers: they are touched once per image walk)
constexpr int kLatTotRows = 2 * 4 * 3;
// compact points of a lattice piece: the 4 before it, the piece, the loop's first 4
constexpr int kLatPts = kLandPts + 8, kLatFirst = kLandPts + 4;

// MIDWALK: walk the blocks between near and far with the large-x form alone
// (the single-job kernel; inside the persistent batch kernel the extra walk
// measured 3 % slower on the uneven batch, so its units keep two walks --
// the sums are the same bits either way)
template <bool FERM, bool MIDWALK, class Field = const FieldDev &>
__device__ __forceinline__ bool warp_unit_lat(const SweepArgs &A, int tile, int l0, int l1,
                                              size_t row, WarpStage &W, float (*tot)[32],
                                              float4 *box) {
  const int lane = threadIdx.x & 31;
  // slots t and t + 32: a unit holding 32 or fewer instances gives each lane
  // at most one (the lanes of a warp still hold consecutive slots)
  const int sA = tile * 64 + lane, sB = sA + 32;
  const bool liveA = sA < A.ninst, liveB = sB < A.ninst;
  const int slA = liveA ? sA : A.ninst - 1, slB = liveB ? sB : A.ninst - 1;
  const int iA = A.perm ? A.perm[slA] : slA, iB = A.perm ? A.perm[slB] : slB;
  const int npc = (A.ppl + kLandPts - 1) / kLandPts;
  const int K = (l1 - l0) * npc;
  Field F = A.field;

  auto issue = [&](int k) {
    const int l = l0 + k / npc, p0 = k % npc * kLandPts;
    const uint32_t bytes = (uint32_t)(min(kLandPts, A.ppl - p0) * (int)sizeof(float4));
    mbar_arrive_expect_tx(W.bar, bytes);
    bulk_g2s(W.land, A.loops + (size_t)l * A.ppl + p0, bytes, W.bar);
  };
  if (lane == 0) issue(0);

  const float2 il2 = f2(F.inv_l2);
  // loop totals per instance (h = 0: A, 1: B), Kahan-compensated, in tot[]
  auto T = [&](int h, int v, int r) -> float & { return tot[(h * 4 + v) * 3 + r][lane]; };
  auto tot_add = [&](int h, int r, float vp, float vs) {
    float a = T(h, 0, r), ac = T(h, 1, r);
    kahan_add(a, ac, vp);
    T(h, 0, r) = a;
    T(h, 1, r) = ac;
    if (FERM) {
      float b = T(h, 2, r), bc = T(h, 3, r);
      kahan_add(b, bc, vs);
      T(h, 2, r) = b;
      T(h, 3, r) = bc;
    }
  };

#pragma unroll 1
  for (int k = 0; k < K; ++k) {
    const int c = k % npc;
    const int l = l0 + k / npc;
    const int p0 = c * kLandPts;
    const int np = min(kLandPts, A.ppl - p0), p1 = p0 + np;
    if (!warp_stage_wait(A, W)) return false;
    // compact points: the last 4 of the piece before stay in front of this one
    // (a piece that another follows is full), the first 4 of the loop behind
    if (c > 0) {
      float4 v;
      if (lane < 4) v = W.comp[kLandPts + lane];
      __syncwarp();
      if (lane < 4) W.comp[lane] = v;
    }
    for (int i = lane; i < np; i += 32) {
      const float2 a = *reinterpret_cast<const float2 *>(W.land + i);
      const float4 v = make_float4(a.x, a.x, a.y, a.y);
      W.comp[4 + i] = v;
      if (c == 0 && i < 4) W.comp[kLatFirst + i] = v;
    }
    __syncwarp();
    if (lane == 0 && k + 1 < K) issue(k + 1);
    if (c == 0) {
#pragma unroll
      for (int w = 0; w < kLatTotRows; ++w) tot[w][lane] = 0.f;
    }
    const bool last = c == npc - 1;
    // bounding boxes (unit loop) of the points each block of kLatSub staged
    // points' segments touch: the block's points and the four before it (the
    // previous piece's for the first block)
#pragma unroll 1
    for (int b = 0; b < kLatNSub; ++b) {
      const int lo = max(b * kLatSub - 4, c == 0 ? 0 : -4);
      const int hi = min((b + 1) * kLatSub, np);
      float x0 = INFINITY, x1 = -INFINITY, y0 = INFINITY, y1 = -INFINITY;
      for (int i = lo + lane; i < hi; i += 32) {
        const float4 v = W.comp[4 + i];
        x0 = fminf(x0, v.x);
        x1 = fmaxf(x1, v.x);
        y0 = fminf(y0, v.z);
        y1 = fmaxf(y1, v.z);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
        x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
        y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
        y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
      }
      if (lane == 0) box[b] = make_float4(x0, x1, y0, y1);
    }
    __syncwarp();
    // the nearest point of block b's box, scaled and shifted as U() maps the
    // points (fma(s, w, c - R) is monotone in w), is far from the image centre
    auto block_x = [&](int b, float sc, float crx, float cry) {
      const float4 bb = box[b];
      const float lx = fmaf(sc, bb.x, crx), hx = fmaf(sc, bb.y, crx);
      const float ly = fmaf(sc, bb.z, cry), hy = fmaf(sc, bb.w, cry);
      const float ex = fmaxf(fmaxf(lx, -hx), 0.0f), ey = fmaxf(fmaxf(ly, -hy), 0.0f);
      return fmaf(ex, ex, ey * ey) * F.inv_l2;
    };
    // this loop's images of each instance
    const float4 bb = A.bbox[l];
    const ImgRange gA = image_range(bb, A.rtT[iA], A.cx[iA], A.cy[iA], F);
    const ImgRange gB = image_range(bb, A.rtT[iB], A.cx[iB], A.cy[iB], F);
    const int widA = max(gA.n1 - gA.n0 + 1, 1), widB = max(gB.n1 - gB.n0 + 1, 1);
    // row m of a range trimmed to the disk m^2 + n^2 <= (rimage/a)^2 (the
    // criterion image_range uses for `inside`)
    auto row_of = [&](const ImgRange &g, int m, int &lo, int &hi) {
      const float mm = (float)(m * m);
      int nx = (int)floorf(sqrtf(fmaxf(F.rimg2 - mm, 0.0f)));
      while (nx >= 0 && mm + (float)(nx * nx) > F.rimg2) --nx;
      while (mm + (float)((nx + 1) * (nx + 1)) <= F.rimg2) ++nx;
      lo = max(g.n0, -nx);
      hi = min(g.n1, nx);
    };
    auto count = [&](const ImgRange &g, int wid) {
      if (g.m1 < g.m0 || g.n1 < g.n0) return 0;
      if (g.inside) return (g.m1 - g.m0 + 1) * wid;
      int n = 0;
      for (int m = g.m0; m <= g.m1; ++m) {
        int lo, hi;
        row_of(g, m, lo, hi);
        n += max(hi - lo + 1, 0);
      }
      return n;
    };
    // a slot past the tile's instances walks nothing
    const int nA = liveA ? count(gA, widA) : 0, nB = liveB ? count(gB, widB) : 0;
    const int mn = min(nA, nB), mx = max(nA, nB);
    const int steps = mn + (mx - mn + 1) / 2;
    const int qa = c == 0 ? 1 : (p0 >> 2), qend = p1 >> 2;
    const float4 *const pts = W.comp + 4 - p0;  // loop point p of the piece
    for (int p = 0; p < steps; ++p) {
      // the step's two images: (A p, B p), then the longer list two at a time
      int jx, jy;
      bool bx, by;
      if (p < mn) {
        jx = jy = p;
        bx = false;
        by = true;
      } else {
        jx = mn + 2 * (p - mn);
        jy = jx + 1;
        bx = by = nB > nA;
      }
      auto image = [&](int j, bool isB, bool &ok, float &s, float &crx, float &cry) {
        const ImgRange &g = isB ? gB : gA;
        const int wd = isB ? widB : widA, n = isB ? nB : nA;
        int jj = min(j, n - 1), m, nn;
        if (g.inside) {
          m = g.m0 + jj / wd;
          nn = g.n0 + jj % wd;
        } else {  // the rows trimmed to the disk, in order
          m = g.m0;
          nn = g.n0;
          for (int mr = g.m0; mr <= g.m1; ++mr) {
            int lo, hi;
            row_of(g, mr, lo, hi);
            const int cnt = max(hi - lo + 1, 0);
            if (jj < cnt) {
              m = mr;
              nn = lo + jj;
              break;
            }
            jj -= cnt;
          }
        }
        ok = j < n;
        const int ic = isB ? iB : iA;
        s = A.rtT[ic];
        crx = fmaf(-(float)m, F.a, A.cx[ic]);
        cry = fmaf(-(float)nn, F.a, A.cy[ic]);
      };
      bool okx, oky;
      float sx, sy, cxx, cxy, cyx, cyy;
      image(jx, bx, okx, sx, cxx, cyx);
      image(jy, by, oky, sy, cxy, cyy);
      const float2 s2 = make_float2(sx, sy);
      const float2 crx = make_float2(cxx, cxy), cry = make_float2(cyx, cyy);
      // point minus image centre, scaled: u = s w + (c - R)
      auto U = [&](const float4 &w, float2 &ux, float2 &uy) {
        ux = fma2(s2, make_float2(w.x, w.y), crx);
        uy = fma2(s2, make_float2(w.z, w.w), cry);
      };
      float2 bp[3] = {f2(0.f), f2(0.f), f2(0.f)}, bs[3] = {f2(0.f), f2(0.f), f2(0.f)};
      float2 uAx, uAy, uBx, uBy, uOx, uOy;
      if (c == 0) {  // the N/2 sub-loop's first segment 1 -> 3; sub-loops open at 0, 2, 3
        float2 u1x, u1y, u3x, u3y;
        U(pts[1], u1x, u1y);
        U(pts[3], u3x, u3y);
        const float4 r = lat_seg2_called<FERM>(u1x, u1y, u3x, u3y, il2,
                                               make_float4(0.f, 0.f, 0.f, 0.f));
        bp[0] = make_float2(r.x, r.y);
        bs[0] = make_float2(r.z, r.w);
        U(pts[0], uAx, uAy);
        U(pts[2], uBx, uBy);
        uOx = u3x;
        uOy = u3y;
      } else {  // the previous piece's last points of each sub-loop
        U(pts[p0 - 4], uAx, uAy);
        U(pts[p0 - 2], uBx, uBy);
        U(pts[p0 - 1], uOx, uOy);
      }
      auto group4 = [&](int q, auto &&segf) {
        float2 P0x, P0y, P1x, P1y, P2x, P2y, P3x, P3y;
        U(pts[4 * q], P0x, P0y);
        U(pts[4 * q + 1], P1x, P1y);
        U(pts[4 * q + 2], P2x, P2y);
        U(pts[4 * q + 3], P3x, P3y);
        segf(uAx, uAy, P0x, P0y, 2);  // N/4a: 4q-4 -> 4q
        segf(uOx, uOy, P1x, P1y, 0);  // N/2 : 4q-1 -> 4q+1
        segf(uBx, uBy, P2x, P2y, 1);  // N/4b: 4q-2 -> 4q+2
        segf(P1x, P1y, P3x, P3y, 0);  // N/2 : 4q+1 -> 4q+3
        uAx = P0x; uAy = P0y;
        uBx = P2x; uBy = P2y;
        uOx = P3x; uOy = P3y;
      };
      auto far_seg = [&](float2 ix, float2 iy, float2 jx, float2 jy, int r) {
        lat_seg2_far(ix, iy, jx, jy, il2, bp[r]);
      };
      auto mid_seg = [&](float2 ix, float2 iy, float2 jx, float2 jy, int r) {
        lat_seg2<FERM, false, true>(ix, iy, jx, jy, il2, bp[r], bs[r]);
      };
      auto near_seg = [&](float2 ix, float2 iy, float2 jx, float2 jy, int r) {
        lat_seg2<FERM, false>(ix, iy, jx, jy, il2, bp[r], bs[r]);
      };
#pragma unroll 1
      for (int b = 0; b < kLatNSub; ++b) {
        const int q0 = max(qa, (p0 + b * kLatSub) >> 2);
        const int q1 = min(qend, (p0 + (b + 1) * kLatSub) >> 2);
        // an unused half is not added: it never holds the warp back
        const float xb = fminf(okx ? block_x(b, sx, cxx, cyx) : INFINITY,
                               oky ? block_x(b, sy, cxy, cyy) : INFINITY);
        const unsigned am = __activemask();
        if (__all_sync(am, xb > kLatFarChunk)) {
          // every node of the block's walk is far: reciprocals only, no
          // per-segment vote, four segments of straight-line work per group
#pragma unroll 1
          for (int q = q0; q < q1; ++q) group4(q, far_seg);
        } else if (MIDWALK && __all_sync(am, xb > kLatMidChunk)) {
          // no node near an image centre: the integrand's large-x form alone
#pragma unroll 2
          for (int q = q0; q < q1; ++q) group4(q, mid_seg);
        } else {
#pragma unroll 1
          for (int q = q0; q < q1; ++q) group4(q, near_seg);
        }
      }
      if (last) {  // closing segments back to points 1, 2, 0
        float2 ux, uy;
        float4 r;
        U(W.comp[kLatFirst + 1], ux, uy);
        r = lat_seg2_called<FERM>(uOx, uOy, ux, uy, il2,
                                  make_float4(bp[0].x, bp[0].y, bs[0].x, bs[0].y));
        bp[0] = make_float2(r.x, r.y);
        bs[0] = make_float2(r.z, r.w);
        U(W.comp[kLatFirst + 2], ux, uy);
        r = lat_seg2_called<FERM>(uBx, uBy, ux, uy, il2,
                                  make_float4(bp[1].x, bp[1].y, bs[1].x, bs[1].y));
        bp[1] = make_float2(r.x, r.y);
        bs[1] = make_float2(r.z, r.w);
        U(W.comp[kLatFirst], ux, uy);
        r = lat_seg2_called<FERM>(uAx, uAy, ux, uy, il2,
                                  make_float4(bp[2].x, bp[2].y, bs[2].x, bs[2].y));
        bp[2] = make_float2(r.x, r.y);
        bs[2] = make_float2(r.z, r.w);
      }
      // each image's piece sums into its instance's totals, in image order
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        if (okx) tot_add(bx ? 1 : 0, r, bp[r].x, bs[r].x);
        if (oky) tot_add(by ? 1 : 0, r, bp[r].y, bs[r].y);
      }
    }
    __syncwarp();
    if (last) {
      const size_t at = A.per_loop ? row + (l - l0) : row;
      const bool acc = !A.per_loop && l > l0;
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {  // per-loop epilogue of each instance
        const int ih = h ? iB : iA;
        const bool live = h ? liveB : liveA;
        const df G[3] = {fast_two_sum(T(h, 0, 0), -T(h, 1, 0)),
                         fast_two_sum(T(h, 0, 1), -T(h, 1, 1)),
                         fast_two_sum(T(h, 0, 2), -T(h, 1, 2))};
        const df H[3] = {fast_two_sum(T(h, 2, 0), -T(h, 3, 0)),
                         fast_two_sum(T(h, 2, 1), -T(h, 3, 1)),
                         fast_two_sum(T(h, 2, 2), -T(h, 3, 2))};
        const df tq = {A.tqh[ih], A.tql[ih]};
        loop_epilogue<FERM>(G, H, A.cph_hi, A.cph_lo, A.csp_hi, A.csp_lo, tq, A.nF,
                            [&](int j, double d0, double d1, double d2) {
                              if (live) put_loop(A, at, j, ih, acc, d0, d1, d2);
                            });
      }
    }
    __syncwarp();  // every lane is done with the compact piece
  }
  return true;
}

// ------------------------------------------------------------- kernels --
// bytes of dynamic shared memory per warp
constexpr int kStageBytes = kLandPts * 16 + kLandPts * 8;
constexpr int kPairStageBytes = kStageBytes + 4 * 16 + kMaxF * 3 * 32 * 8;
constexpr int kLatStageBytes =
    kLandPts * 16 + kLatPts * 16 + kLatTotRows * 32 * 4 + kLatNSub * 16;
template <int P, bool PAIR>
constexpr int stage_bytes() {
  return !PAIR ? kStageBytes : P == kLattice ? kLatStageBytes : kPairStageBytes;
}

__device__ __forceinline__ WarpStage warp_stage(unsigned char *smem, uint64_t *bars, int bytes) {
  const int w = threadIdx.x >> 5;
  float4 *const land = reinterpret_cast<float4 *>(smem + w * bytes);
  return WarpStage{land, land + kLandPts, bars + w, 0u};
}

// the lattice's totals and block boxes behind its compact points
template <bool FERM, bool MIDWALK, class Field = const FieldDev &>
__device__ __forceinline__ bool warp_unit_lattice(const SweepArgs &A, int tile, int l0, int l1,
                                                  size_t row, WarpStage &W) {
  float4 *const box = W.comp + kLatPts;
  return warp_unit_lat<FERM, MIDWALK, Field>(A, tile, l0, l1, row, W,
                                      reinterpret_cast<float(*)[32]>(box + kLatNSub), box);
}

// loops [l0, l1) of unit u and the partial-sum row of its first
__device__ __forceinline__ size_t unit_loops(const SweepArgs &A, int u, int &l0, int &l1) {
  l0 = u * A.unit_loops;
  l1 = min(l0 + A.unit_loops, A.n_chunks * A.chunk_loops);
  return A.per_loop ? (size_t)l0 : (size_t)u;
}

// CTAs per SM a sweep is compiled for.  The heavy profiles wait on chains of
// divisions and exponentials, not on a pipe, and gain from more warps than from
// registers (spills included): over 4 CTAs fixflux 8 per SM 19-21 % faster,
// periodic 8 1-12 %, spline 6 9-22 % (512 instances on 512 loops, 8 and 50
// intervals); the light profiles lose 2-6 % at 5 or 6.
template <int P>
constexpr int sweep_min_ctas() {
  return !Profile<P>::kHeavy ? 4 : P == kSpline ? 6 : 8;
}

// warp -> (unit, instance tile): the tiles of a unit on consecutive warps, so
// that they share its loops in L2; the lattice's units of a tile instead, its
// first tiles holding the instances with the most images: the light ones then
// fill the end (512 instances on 1024 x 1024 points, a = 5: 13.4 -> 10.4 ms)
template <int P, bool FERM, int NINT, bool PAIR>
__global__ void __launch_bounds__(kSweepThreads, sweep_min_ctas<P>())
    sweep_kernel(const __grid_constant__ SweepArgs A) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[kSweepWarps];
  const unsigned item = blockIdx.x * kSweepWarps + (threadIdx.x >> 5);
  constexpr bool kLat4 = P == kLattice && PAIR;
  const unsigned u = kLat4 ? item % (unsigned)A.n_units : item / (unsigned)A.n_tiles;
  const int tile = kLat4 ? item / (unsigned)A.n_units : item % (unsigned)A.n_tiles;
  if (u >= (unsigned)A.n_units || tile >= A.n_tiles) return;  // whole warp
  WarpStage W = warp_stage(smem, bars, stage_bytes<P, PAIR>());
  warp_stage_init(W.bar);
  int l0, l1;
  const size_t row = unit_loops(A, u, l0, l1);
  if constexpr (kLat4)
    warp_unit_lattice<FERM, true>(A, tile, l0, l1, row, W);
  else
    warp_unit<P, FERM, NINT, PAIR>(A, tile, l0, l1, row, W);
}

// One part of a heavy profile's loop (SweepArgs::parts): the FP32 sums of its
// Kahan blocks, of the opening segment (part 0) and of the closing ones (last),
// exactly as warp_unit forms them, stored for loop_finish_kernel.
template <int P, bool FERM>
__global__ void __launch_bounds__(kSweepThreads, sweep_min_ctas<P>())
    sweep_part_kernel(const __grid_constant__ SweepArgs A) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[kSweepWarps];
  const int lane = threadIdx.x & 31;
  const unsigned item = blockIdx.x * kSweepWarps + (threadIdx.x >> 5);
  const unsigned u = item / (unsigned)A.n_tiles;
  const int l = u / (unsigned)A.parts, part = u % (unsigned)A.parts;
  if (l >= A.n_chunks * A.chunk_loops) return;  // whole warp
  WarpStage W = warp_stage(smem, bars, kStageBytes);
  warp_stage_init(W.bar);
  const int slot = (item % (unsigned)A.n_tiles) * 32 + lane;
  const bool live = slot < A.ninst;
  const int ic = live ? slot : A.ninst - 1;
  const FieldDev &F = A.field;
  const float cx = A.cx[ic], cy = A.cy[ic], s = A.rtT[ic];
  const int nq = A.ppl >> 2, nb = loop_blocks(nq);
  const int b0 = part * A.part_blocks, b1 = min(b0 + A.part_blocks, nb);
  const int q0 = block_begin(b0), q1 = min(block_begin(b1), nq);
  const float4 *const loop = A.loops + (size_t)l * A.ppl;
  if (lane == 0) {
    const uint32_t bytes = (uint32_t)((q1 - q0) * 4 * (int)sizeof(float4));
    mbar_arrive_expect_tx(W.bar, bytes);
    bulk_g2s(W.land, loop + 4 * q0, bytes, W.bar);
  }
  auto scale = [&](float2 v, float &x, float &y) {
    x = fmaf(s, v.x, cx);
    y = fmaf(s, v.y, cy);
  };
  auto gpt = [&](int p, float &x, float &y) {
    scale(__ldg(reinterpret_cast<const float2 *>(loop + p)), x, y);
  };
  auto pt = [&](int p, float &x, float &y) {
    scale(*reinterpret_cast<const float2 *>(W.land + (p - 4 * q0)), x, y);
  };
  float *const out = A.blocks + (size_t)l * (nb + 2) * 6 * A.ninst + ic;
  auto put = [&](int b, const float *ph, const float *sp) {
    if (!live) return;
    float *o = out + (size_t)b * 6 * A.ninst;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      o[(size_t)r * A.ninst] = ph[r];
      if (FERM) o[(size_t)(3 + r) * A.ninst] = sp[r];
    }
  };
  const ImgRange img = {0, -1, 0, -1, 1};
  float zAx, zAy, zBx, zBy, zOx, zOy;  // previous point of each sub-loop
  gpt(4 * q0 - 4, zAx, zAy);
  gpt(4 * q0 - 2, zBx, zBy);
  gpt(4 * q0 - 1, zOx, zOy);
  if (part == 0) {
    float ph[3] = {0.f, 0.f, 0.f}, sp[3] = {0.f, 0.f, 0.f}, x, y;
    gpt(1, x, y);
    seg<P, FERM, 0, kSqRound>(x, y, zOx, zOy, F, img, ph[0], sp[0]);  // N/2: 1 -> 3
    put(0, ph, sp);
  }
  if (!warp_stage_wait(A, W)) return;
#pragma unroll 1
  for (int b = b0; b < b1; ++b) {
    float bp[3] = {0.f, 0.f, 0.f}, bs[3] = {0.f, 0.f, 0.f};
    const int qe = min(block_begin(b + 1), nq);
#pragma unroll 1
    for (int q = block_begin(b); q < qe; ++q) {
      float P0x, P0y, P1x, P1y, P2x, P2y, P3x, P3y;
      pt(4 * q, P0x, P0y);
      pt(4 * q + 1, P1x, P1y);
      pt(4 * q + 2, P2x, P2y);
      pt(4 * q + 3, P3x, P3y);
      seg<P, FERM, 0, kSqRound>(zAx, zAy, P0x, P0y, F, img, bp[2], bs[2]);  // N/4a: 4q-4 -> 4q
      seg<P, FERM, 0, kSqRound>(zOx, zOy, P1x, P1y, F, img, bp[0], bs[0]);  // N/2 : 4q-1 -> 4q+1
      seg<P, FERM, 0, kSqRound>(zBx, zBy, P2x, P2y, F, img, bp[1], bs[1]);  // N/4b: 4q-2 -> 4q+2
      seg<P, FERM, 0, kSqRound>(P1x, P1y, P3x, P3y, F, img, bp[0], bs[0]);  // N/2 : 4q+1 -> 4q+3
      zAx = P0x; zAy = P0y;
      zBx = P2x; zBy = P2y;
      zOx = P3x; zOy = P3y;
    }
    put(1 + b, bp, bs);
  }
  if (part == A.parts - 1) {
    float tp[3] = {0.f, 0.f, 0.f}, ts[3] = {0.f, 0.f, 0.f}, x, y;
    gpt(1, x, y);
    seg<P, FERM, 0, kSqRound>(zOx, zOy, x, y, F, img, tp[0], ts[0]);  // N/2 : N-1 -> 1
    gpt(2, x, y);
    seg<P, FERM, 0, kSqRound>(zBx, zBy, x, y, F, img, tp[1], ts[1]);  // N/4b: N-2 -> 2
    gpt(0, x, y);
    seg<P, FERM, 0, kSqRound>(zAx, zAy, x, y, F, img, tp[2], ts[2]);  // N/4a: N-4 -> 0
    put(1 + nb, tp, ts);
  }
}

// the parts' sums of one (loop, instance) in the walk's order, and its epilogue
// (one instantiation per profile: the units are compiled with different options)
template <int P, bool FERM>
__global__ void __launch_bounds__(128) loop_finish_kernel(const __grid_constant__ SweepArgs A) {
  const long long at = (long long)blockIdx.x * 128 + threadIdx.x;
  const int l = (int)(at / A.ninst), i = (int)(at % A.ninst);
  if (l >= A.n_chunks * A.chunk_loops) return;
  const int nb = loop_blocks(A.ppl >> 2);
  const float *b = A.blocks + (size_t)l * (nb + 2) * 6 * A.ninst + i;
  const size_t n = (size_t)A.ninst;
  float ph[3] = {b[0], 0.f, 0.f}, pc[3] = {0.f, 0.f, 0.f};
  float sp[3] = {FERM ? b[3 * n] : 0.f, 0.f, 0.f}, sc[3] = {0.f, 0.f, 0.f};
#pragma unroll 2
  for (int k = 0; k <= nb; ++k) {  // the blocks, then the closing segments
    b += 6 * n;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      kahan_add(ph[r], pc[r], b[r * n]);
      if (FERM) kahan_add(sp[r], sc[r], b[(3 + r) * n]);
    }
  }
  const df G[3] = {fast_two_sum(ph[0], -pc[0]), fast_two_sum(ph[1], -pc[1]),
                   fast_two_sum(ph[2], -pc[2])};
  const df H[3] = {fast_two_sum(sp[0], -sc[0]), fast_two_sum(sp[1], -sc[1]),
                   fast_two_sum(sp[2], -sc[2])};
  const df tq = {A.tqh[i], A.tql[i]};
  loop_epilogue<FERM>(G, H, A.cph_hi, A.cph_lo, A.csp_hi, A.csp_lo, tq, A.nF,
                      [&](int j, double w0, double w1, double w2) {
                        put_loop(A, l, j, i, false, w0, w1, w2);
                      });
}

// One warp per (loop, instance), or (A.split) two: the N/2 sub-loop's segments
// on one, both N/4 sub-loops' on the other -- the same work each, and the same
// sums, since the sub-loops' accumulators are separate.  Bound by latency when
// few (loop, instance) pairs leave the SMs with a few warps each: one instance
// on 512 loops of 512 points, fixflux at 50 intervals, 1.06 -> 0.59 ms with two.
//   LEAN: one warp per pair and no fingerprint, the form of launches that fill the
// chip.  The role tests and hashes of the other took the light profiles from 32-40
// to 40-48 registers and the lattice from 72 to 92, and with them the SM's warps:
// 25 instances on 512 x 1820 points, lattice spinor, 224 -> 233 us.
//   With A.fingerprint the warps also hash the points they read: EV() checks a
// cached ensemble against that, and a pass of its own over the ensemble took
// 20 us beside the 60 us of the sweep (5120 loops of 1024 points, 50
// intervals); 79 such EV() sweeps of integrateT 10.8 -> 9.9 ms.
//   (kSqRound / kSqFuse: the roundings the four calls were compiled to, written
// out so that results keep their bits.)
template <int P, bool FERM, int NINT, bool LEAN>
__global__ void __launch_bounds__(kLoopWarps * 32)
    loopwarp_kernel(const __grid_constant__ LoopArgs A) {
  __shared__ float quarter[kLoopWarps][4];  // split: sums of the N/4 sub-loops
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool split = !LEAN && A.split;
  unsigned long long *const fingerprint = LEAN ? nullptr : A.fingerprint;
  const int l = split ? blockIdx.x * (kLoopWarps / 2) + (w >> 1) : blockIdx.x * kLoopWarps + w;
  const bool half = !split || !(w & 1), quarters = !split || (w & 1);
  const int inst = blockIdx.y;
  const bool on = l < A.Nl;  // whole warp
  if (!split && !on) return;
  const float cx = A.cx[inst], cy = A.cy[inst], s = A.rtT[inst];
  const FieldDev &F = A.field;
  const float2 *pts = reinterpret_cast<const float2 *>(A.loops + (size_t)(on ? l : 0) * A.ppl);
  auto pt = [&](int p, float &x, float &y) {
    const float2 v = __ldg(&pts[2 * p]);
    x = fmaf(s, v.x, cx);
    y = fmaf(s, v.y, cy);
    return v;
  };
  // group q covers points 4q..4q+3 and the four segments ending there; the
  // previous points of group 0 wrap to the end of the loop (closing segments)
  const int nq = on ? A.ppl >> 2 : 0;
  ImgRange img = {0, -1, 0, -1, 1};
  if constexpr (P == kLattice)
    if (on) img = image_range(A.bbox[l], s, cx, cy, F);
  float ph[3] = {0.f, 0.f, 0.f}, sp[3] = {0.f, 0.f, 0.f};
  unsigned long long hash = 0;
  // a point that this group is the first to read: hashed before its segments, so
  // that no coordinate lives through them
  auto own = [&](int p, float &x, float &y) {
    const float2 v = pt(p, x, y);
    if (fingerprint) hash += point_hash(v, (size_t)l * A.ppl + p);
  };
  for (int q = lane; q < nq; q += 32) {
    const int pa = (q == 0 ? A.ppl : 4 * q) - 4;
    if constexpr (LEAN) {
      float zAx, zAy, zBx, zBy, zOx, zOy, P0x, P0y, P1x, P1y, P2x, P2y, P3x, P3y;
      pt(pa, zAx, zAy);
      pt(pa + 2, zBx, zBy);
      pt(pa + 3, zOx, zOy);
      pt(4 * q, P0x, P0y);
      pt(4 * q + 1, P1x, P1y);
      pt(4 * q + 2, P2x, P2y);
      pt(4 * q + 3, P3x, P3y);
      seg<P, FERM, NINT, kSqFuse>(zAx, zAy, P0x, P0y, F, img, ph[2], sp[2]);
      seg<P, FERM, NINT, kSqRound>(zOx, zOy, P1x, P1y, F, img, ph[0], sp[0]);
      seg<P, FERM, NINT, kSqRound>(zBx, zBy, P2x, P2y, F, img, ph[1], sp[1]);
      seg<P, FERM, NINT, kSqRound>(P1x, P1y, P3x, P3y, F, img, ph[0], sp[0]);
    } else {
      if (half) {
        float zOx, zOy, P1x, P1y, P3x, P3y;
        pt(pa + 3, zOx, zOy);
        own(4 * q + 1, P1x, P1y);
        own(4 * q + 3, P3x, P3y);
        seg<P, FERM, NINT, kSqRound>(zOx, zOy, P1x, P1y, F, img, ph[0], sp[0]);
        seg<P, FERM, NINT, kSqRound>(P1x, P1y, P3x, P3y, F, img, ph[0], sp[0]);
      }
      if (quarters) {
        float zAx, zAy, zBx, zBy, P0x, P0y, P2x, P2y;
        pt(pa, zAx, zAy);
        pt(pa + 2, zBx, zBy);
        own(4 * q, P0x, P0y);
        own(4 * q + 2, P2x, P2y);
        seg<P, FERM, NINT, kSqFuse>(zAx, zAy, P0x, P0y, F, img, ph[2], sp[2]);
        seg<P, FERM, NINT, kSqRound>(zBx, zBy, P2x, P2y, F, img, ph[1], sp[1]);
      }
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      ph[r] += __shfl_xor_sync(0xffffffffu, ph[r], off);
      if (FERM) sp[r] += __shfl_xor_sync(0xffffffffu, sp[r], off);
    }
  }
  if (fingerprint) {
    for (int off = 16; off > 0; off >>= 1) hash += __shfl_xor_sync(0xffffffffu, hash, off);
    if (lane == 0 && on) atomicAdd(fingerprint, hash);
  }
  if (split) {
    if (lane == 0 && quarters) {
      quarter[w][0] = ph[1];
      quarter[w][1] = ph[2];
      quarter[w][2] = sp[1];
      quarter[w][3] = sp[2];
    }
    __syncthreads();
    if (lane == 0 && half) {
      ph[1] = quarter[w + 1][0];
      ph[2] = quarter[w + 1][1];
      sp[1] = quarter[w + 1][2];
      sp[2] = quarter[w + 1][3];
    }
  }
  if (lane == 0 && half && on) {
    const df tq = {A.tqh[inst], A.tql[inst]};
    const df G[3] = {df{ph[0], 0.f}, df{ph[1], 0.f}, df{ph[2], 0.f}};
    const df H[3] = {df{sp[0], 0.f}, df{sp[1], 0.f}, df{sp[2], 0.f}};
    loop_epilogue<FERM>(G, H, A.cph_hi, A.cph_lo, A.csp_hi, A.csp_lo, tq, A.nF,
                        [&](int j, double w0, double w1, double w2) {
                          double *o = A.partial + ((size_t)(l * A.nF + j) * 3) * A.ninst + inst;
                          o[0] = w0;
                          o[A.ninst] = w1;
                          o[2 * (size_t)A.ninst] = w2;
                        });
    // Wsscal / Wsferm of the first flux value (intEV.cu:553-561)
    const size_t o = (size_t)inst * A.Nl + l;
    auto val = [](df x) { return x.hi + x.lo; };
    const df cph0 = {A.cph_hi[0], A.cph_lo[0]};
    if (A.scal)
      A.scal[o] = make_float4(val(df_mul(cph0, G[0])), val(df_mul(cph0, G[1])),
                              val(df_mul(cph0, G[2])), 0.0f);
    if (FERM && A.ferm) {
      const df csp0 = df_mul(df{A.csp_hi[0], A.csp_lo[0]}, tq);
      A.ferm[o] = make_float4(val(df_mul(csp0, H[0])), 2.0f * val(df_mul(csp0, H[1])),
                              2.0f * val(df_mul(csp0, H[2])), 0.0f);
    }
  }
}

// instantiation + dispatch over (fermion, nint) for one profile
template <int P, bool FERM, int NINT, bool PAIR>
cudaError_t sweep_launch(SweepArgs a, cudaStream_t s) {
  constexpr bool kLat4 = P == kLattice && PAIR;
  const int per = kLat4 ? 64 : 32;
  a.n_tiles = (a.ninst + per - 1) / per;
  const long long items = (long long)a.n_tiles * a.n_units;
  const unsigned ctas = sweep_ctas(items);
  if (!ctas) return cudaErrorInvalidConfiguration;
  constexpr size_t smem = (size_t)kSweepWarps * stage_bytes<P, PAIR>();
  auto k = sweep_kernel<P, FERM, NINT, PAIR>;
  if (smem > 48 * 1024) {  // a per-device attribute
    const cudaError_t e =
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  k<<<ctas, kSweepThreads, smem, s>>>(a);
  return cudaGetLastError();
}

template <int P, bool FERM>
cudaError_t sweep_parts_launch(SweepArgs a, cudaStream_t s) {
  a.n_tiles = (a.ninst + 31) / 32;
  const long long loops = (long long)a.n_chunks * a.chunk_loops;
  const long long items = loops * a.parts * a.n_tiles;
  const unsigned ctas = sweep_ctas(items);
  if (!ctas) return cudaErrorInvalidConfiguration;
  sweep_part_kernel<P, FERM><<<ctas, kSweepThreads, kSweepWarps * kStageBytes, s>>>(a);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  loop_finish_kernel<P, FERM><<<(unsigned)((loops * a.ninst + 127) / 128), 128, 0, s>>>(a);
  return cudaGetLastError();
}

template <int P>
cudaError_t sweep_dispatch(bool fermion, int nint, const SweepArgs &a, cudaStream_t s) {
  constexpr bool kLight = P == kSmooth || P == kStep || P == kQuadratic || P == kGaussian;
  if constexpr (P == kSmooth) {
    if (nint == 4 && smooth_clamp_idle(a.field))
      return fermion ? sweep_launch<kSmoothWide, true, 4, true>(a, s)
                     : sweep_launch<kSmoothWide, false, 4, true>(a, s);
  }
#define WL_SWEEP_CASE(NI, PAIR)                                     \
  if (NI == 0 || nint == NI)                                        \
    return fermion ? sweep_launch<P, true, NI, PAIR>(a, s)          \
                   : sweep_launch<P, false, NI, PAIR>(a, s);
  if constexpr (kLight || P == kLattice) {
    WL_SWEEP_CASE(4, true)  // light: packed pairs; lattice: images outer
  }
  if constexpr (kLight) {
    // the reference's interval count: packed pairs too (smooth: a share of the
    // reciprocals on the FP32 pipe); measured over one instance per thread:
    // smooth +20 % / +13 % (scalar / spinor), Gaussian +56 % / +54 %, step
    // +4 % / +31 %, quadratic +35 % / +24 %
    WL_SWEEP_CASE(50, true)
  }
  if constexpr (Profile<P>::kHeavy) {
    if (a.parts)
      return fermion ? sweep_parts_launch<P, true>(a, s) : sweep_parts_launch<P, false>(a, s);
  }
  // other interval counts, the heavy profiles one loop at a time
  WL_SWEEP_CASE(0, kLight)
#undef WL_SWEEP_CASE
  return cudaErrorInvalidValue;
}

template <int P>
cudaError_t loopwarp_dispatch(bool fermion, int nint, const LoopArgs &a, cudaStream_t s) {
  const int per = a.split ? kLoopWarps / 2 : kLoopWarps;  // loops per CTA
  const dim3 grid((a.Nl + per - 1) / per, a.ninst);
  // a heavy profile's segments hold more registers than either form
  const bool lean = !Profile<P>::kHeavy && !a.split && !a.fingerprint;
#define WL_LOOP_CASE(FE, NI)                                                       \
  if (fermion == FE && (NI == 0 || nint == NI)) {                                  \
    if (lean)                                                                      \
      loopwarp_kernel<P, FE, NI, !Profile<P>::kHeavy><<<grid, kLoopWarps * 32, 0, s>>>(a); \
    else                                                                           \
      loopwarp_kernel<P, FE, NI, false><<<grid, kLoopWarps * 32, 0, s>>>(a);       \
    return cudaGetLastError();                                                     \
  }
  if constexpr (!Profile<P>::kHeavy) {
    WL_LOOP_CASE(true, 4)
    WL_LOOP_CASE(false, 4)
  }
  if constexpr (!Profile<P>::kHeavy && P != kLattice) {
    WL_LOOP_CASE(true, 50)
    WL_LOOP_CASE(false, 50)
  }
  WL_LOOP_CASE(true, 0)
  WL_LOOP_CASE(false, 0)
#undef WL_LOOP_CASE
  return cudaErrorInvalidValue;
}

}  // namespace wl
