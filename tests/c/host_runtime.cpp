/* The C-ABI runtime (csrc/wl_api.cpp) on the host alone: the CUDA runtime and
 * the kernel launchers are replaced by stand-ins that record what the library
 * asks for.  Asynchronous copies are carried out only when their stream is
 * waited for -- the latest moment the CUDA runtime may read or write their host
 * side -- and a host buffer that is rewritten or released before is reported.
 * Usage: host_runtime <scenario>; prints "name value" lines. */
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>

#include <new>
#include <string>

#include "wl_internal.h"
#include "wl_legacy.h"
#include "wlgpu.h"

namespace {

struct Block {
  char *p;
  size_t n;
};
struct Copy {
  char *dst;
  const char *src;
  size_t n;
  bool to_host;
  unsigned char *seen;  // the source's contents when the copy was enqueued
};
constexpr int kMany = 4096;
Block g_dev[kMany];
int g_ndev = 0;
Copy g_copy[kMany];
int g_ncopy = 0;
long g_released = 0, g_rewritten = 0, g_syncs = 0, g_kernels = 0;
size_t g_bytes = 0, g_largest = 0;  // device memory held, the largest allocation
bool g_report = true;
wl::SweepArgs g_jobs[64];
int g_sweeps_cut = 0;

void run_copies() {
  for (int i = 0; i < g_ncopy; ++i) {
    Copy &c = g_copy[i];
    if (!c.to_host && memcmp(c.seen, c.src, c.n)) ++g_rewritten;
    memcpy(c.dst, c.src, c.n);
    free(c.seen);
  }
  g_ncopy = 0;
}
void host_released(const void *p, size_t n) {
  for (int i = 0; i < g_ncopy; ++i) {
    const char *h = g_copy[i].to_host ? g_copy[i].dst : g_copy[i].src;
    if (h >= (const char *)p && h < (const char *)p + n) ++g_released;
  }
}
bool on_device(const void *p) {
  for (int i = 0; i < g_ndev; ++i)
    if ((const char *)p >= g_dev[i].p && (const char *)p < g_dev[i].p + g_dev[i].n) return true;
  return false;
}

}  // namespace

// every host buffer of the library comes from here: 16 bytes in front hold its size
void *operator new(size_t n) {
  char *p = (char *)malloc(n + 16);
  if (!p) abort();
  memcpy(p, &n, sizeof(n));
  return p + 16;
}
void operator delete(void *q) noexcept {
  if (!q) return;
  char *p = (char *)q - 16;
  size_t n;
  memcpy(&n, p, sizeof(n));
  host_released(q, n);
  free(p);
}
void operator delete(void *q, size_t) noexcept { operator delete(q); }

extern "C" {
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **, unsigned int,
                                             unsigned long long,
                                             cudaDriverEntryPointQueryResult *) {
  return cudaErrorNotSupported;
}
cudaError_t cudaMalloc(void **out, size_t n) {
  *out = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (*out == MAP_FAILED || g_ndev == kMany) return cudaErrorMemoryAllocation;
  g_dev[g_ndev++] = {(char *)*out, n};
  g_bytes += n;
  if (n > g_largest) g_largest = n;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  run_copies();  // cudaFree waits for the device
  for (int i = 0; i < g_ndev; ++i)
    if (g_dev[i].p == p) {
      g_bytes -= g_dev[i].n;
      munmap(p, g_dev[i].n);
      g_dev[i] = g_dev[--g_ndev];
      break;
    }
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  memset(a, 0, sizeof(*a));
  a->type = on_device(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  run_copies();
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  if (g_ncopy == kMany) return cudaErrorUnknown;
  Copy c = {(char *)d, (const char *)s, n, k == cudaMemcpyDeviceToHost, nullptr};
  c.seen = (unsigned char *)malloc(n + 1);
  memcpy(c.seen, s, n);
  g_copy[g_ncopy++] = c;
  return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
  return memset(d, v, n), cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  return *s = (cudaStream_t)0x10, cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return run_copies(), ++g_syncs, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
  return *e = nullptr, cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = (cudaEvent_t)0x20, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return run_copies(), cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
}

namespace wl {
static cudaError_t kernels(int n) { return g_kernels += n, cudaSuccess; }
cudaError_t launch_tint(const TintArgs &, cudaStream_t) { return kernels(1); }
cudaError_t launch_batch(const BatchArgs &b, int, cudaStream_t) {
  int n = 0;
  for (int t = 0; t < b.ntiles; ++t)
    if (b.tiles[t].job >= n) n = b.tiles[t].job + 1;
  for (int j = 0; j < n && j < 64; ++j) g_jobs[j] = b.jobs[j];
  return kernels(1);
}
cudaError_t launch_plain(int, bool, int, const LoopArgs &, int, cudaStream_t) { return kernels(1); }
cudaError_t launch_sweep(int, bool, int, const SweepArgs &a, cudaStream_t) {
  g_sweeps_cut += a.parts > 0;
  return kernels(a.parts > 0 ? 2 : 1);  // a cut sweep adds its blocks in a second kernel
}
cudaError_t launch_vloops(uint64_t, int, int, int, float4 *, cudaStream_t) { return kernels(1); }
bool batch_supports(int, int) { return true; }
bool plain_supports(int k) { return light_profile(k) || k == kLattice; }
bool batch_in_kernel(int k) { return light_profile(k) || k == kLattice; }
int batch_max_ctas_per_sm() { return 4; }
cudaError_t launch_loopwarp(int, bool, int, const LoopArgs &, cudaStream_t) { return kernels(1); }
cudaError_t launch_list_mean(const double *, const int *, int, double *, cudaStream_t) { return kernels(1); }
cudaError_t launch_loop_bbox(const float4 *, int, int, float4 *, cudaStream_t) { return kernels(1); }
cudaError_t launch_peak_probe(int, int, int, int, float *, cudaStream_t) { return kernels(1); }
cudaError_t launch_fingerprint(const float4 *, size_t, unsigned long long *, cudaStream_t) { return kernels(1); }
cudaError_t launch_batch_reduce(const ReduceJob *, int, int, cudaStream_t) { return kernels(1); }
cudaError_t launch_group_reduce(const ReduceShape &, double *, double *, double *, const int *,
                                double *, cudaStream_t) {
  return kernels(1);
}
cudaError_t launch_wait_selftest(int *, unsigned, int, cudaStream_t) { return kernels(1); }
cudaError_t launch_instance_setup(const double *, const double *, const double *, int, int, float *,
                                  int *, cudaStream_t) {
  return kernels(1);
}
cudaError_t launch_order_instances(const float *, const float *, const float *, int, float, int *,
                                   cudaStream_t) {
  return kernels(1);
}
cudaError_t launch_group_list_means(const double *, int, int, double *, cudaStream_t) { return kernels(1); }
}  // namespace wl

// ------------------------------------------------------------ scenarios --
static void say(const char *name, double v) { printf("%s %.17g\n", name, v); }
static void need(int status, const char *what) {
  if (status == WL_OK) return;
  fprintf(stderr, "%s: status %d\n", what, status);
  exit(2);
}
static wl_field field_of(int profile, int fermion, int nint) {
  wl_field f;
  memset(&f, 0, sizeof(f));
  f.profile = profile;
  f.fermion = fermion;
  f.nint = nint;
  f.mode = profile == WL_PROFILE_LATTICE ? WL_MODE_EXACT : WL_MODE_REFCOMPAT;
  f.lambda2 = 0.5;
  f.tubedist = 2.0;
  f.lmin = 0.2;
  f.rimage = 24.0;
  return f;
}
static int ensemble(wl_ctx *c, int Nl, int ppl) {
  int h = 0;
  need(wl_ensemble_generate(c, 1, 0, Nl, ppl, &h), "generate");
  return h;
}

// host buffers of the proper-time integral's copies
static void tint_staging(wl_ctx *c) {
  const int h = ensemble(c, 256, 64);
  const wl_field f = field_of(WL_PROFILE_SMOOTH, 0, 4);
  double rho[5], T[9], F[2] = {0.5, 1.0}, leff[10], err[10];
  for (int i = 0; i < 5; ++i) rho[i] = 0.5 * i;
  for (int k = 0; k < 9; ++k) T[k] = exp(0.3 * k);
  for (int rep = 0; rep < 2; ++rep)
    need(wl_tint(c, h, &f, 5, rho, 9, T, 2, F, 64, 2, leff, err, nullptr), "tint");
  need(wl_effective_action(c, h, &f, 1.0, WL_TRULE_SUBST, 5, nullptr, 64, 3, leff, err, nullptr,
                           nullptr),
       "effective action");
  say("released", (double)g_released);
  say("rewritten", (double)g_rewritten);
}

// waits of the stream per EV() sweep and per wl_loops() call
static void loop_waits(wl_ctx *c) {
  const int Nl = 256, ppl = 64, h = ensemble(c, Nl, ppl);
  const wl_field f = field_of(WL_PROFILE_SMOOTH, 0, 50);
  const float *loops = nullptr;
  need(wl_ensemble_info(c, h, &loops, nullptr, nullptr), "info");
  struct Wparams p;
  memset(&p, 0, sizeof(p));
  p.Nl = Nl;
  p.Nppl = ppl;
  p.F = 1.0;
  p.l2 = 0.5;
  p.ng = Nl / 128;
  p.worldlines = (float4 *)loops;
  cudaMalloc((void **)&p.Wsscal_d, sizeof(float4) * Nl);
  int list[128];
  for (int j = 0; j < 128; ++j) list[j] = j;
  EV(0.5, &p, list);  // the first call makes the context
  long before = g_syncs;
  for (int k = 0; k < 10; ++k) EV(1.0 + k, &p, list);
  say("ev", (double)(g_syncs - before) / 10);
  before = g_syncs;
  for (int k = 0; k < 10; ++k) need(wl_loops(c, h, &f, 0.1, 0, 1.0 + k, 1.0, nullptr, nullptr), "loops");
  say("loops", (double)(g_syncs - before) / 10);
  say("rewritten", (double)g_rewritten);
}

// wl_last_launches() against the kernels that were enqueued
static void launches(wl_ctx *c) {
  static double cx[64], cy[64], T[64], out[4096];
  for (int i = 0; i < 64; ++i) cx[i] = 0.05 * i, T[i] = 0.1 + 0.1 * i;
  const double F[1] = {1.0}, rho[2] = {0.1, 0.5};
  double *dev = nullptr;
  cudaMalloc((void **)&dev, sizeof(double) * 64);
  for (int i = 0; i < 64; ++i) dev[i] = T[i];
  const int h = ensemble(c, 256, 512);
  int worst = 0;
  long before;
  auto count = [&](int status, const char *what) {
    need(status, what);
    int n = -1;
    wl_last_launches(c, &n, nullptr);
    const int off = abs(n - (int)(g_kernels - before));
    if (off > worst) worst = off;
    before = g_kernels;
  };
  const int profiles[] = {WL_PROFILE_SMOOTH, WL_PROFILE_LATTICE, WL_PROFILE_FIXFLUX,
                          WL_PROFILE_PERIODIC, WL_PROFILE_SPLINE};
  for (int p : profiles) {
    const wl_field f = field_of(p, 0, 4);
    // first use: the lattice's boxes and the spline's table
    need(wl_eval(c, h, &f, 1, cx, cy, T, 1, F, 128, nullptr, out, nullptr), "eval");
    before = g_kernels;
    for (int n : {1, 40})
      count(wl_eval(c, h, &f, n, cx, cy, T, 1, F, 128, nullptr, out, nullptr), "eval");
    count(wl_eval_device(c, h, &f, 40, dev, dev, dev, 1, F, 128, nullptr, nullptr, nullptr),
          "eval_device");
    count(wl_tint(c, h, &f, 2, rho, 2 * 16 + 1, [] {
            static double t[33];
            for (int k = 0; k < 33; ++k) t[k] = exp(0.1 * k);
            return t;
          }(), 1, F, 128, 2, out, out + 2, nullptr), "tint");
    wl_job J[2];
    memset(J, 0, sizeof(J));
    for (wl_job &j : J) {
      j.handle = h;
      j.ninst = 40;
      j.cx = cx;
      j.cy = cy;
      j.T = T;
      j.nF = 1;
      j.F[0] = 1.0;
      j.group = 128;
      j.field = f;
    }
    J[1].field = field_of(WL_PROFILE_SMOOTH, 1, 4);
    count(wl_batch_eval(c, 2, J, 0), "batch");
  }
  say("cut", (double)g_sweeps_cut);  // the heavy profiles did take the cut path
  say("off", (double)worst);
}

static wl_job job_of(int h, const wl_field &f, int n, int nF, const double *v, const double *T) {
  wl_job j;
  memset(&j, 0, sizeof(j));
  j.handle = h;
  j.field = f;
  j.ninst = n;
  j.cx = j.cy = v;
  j.T = T;
  j.nF = nF;
  for (int k = 0; k < nF; ++k) j.F[k] = 0.5;
  j.group = 128;
  return j;
}

// device memory of a batch whose chunks are whole groups (ppl 64, groups of
// 128), just under the number of units at which jobs stop being cut
static void batch_scratch(wl_ctx *c) {
  const int n = 31100, Nl = 5120, h = ensemble(c, Nl, 64);
  double *v = new double[n], *T = new double[n];
  for (int i = 0; i < n; ++i) v[i] = 0.1, T[i] = 1.0;
  g_largest = 0;
  wl_job j = job_of(h, field_of(WL_PROFILE_GAUSSIAN, 1, 50), n, 4, v, T);
  need(wl_batch_eval(c, 1, &j, 0), "batch");
  say("largest", (double)g_largest);
  say("chunk_sums", 8.0 * Nl / 128 * 4 * 3 * n);
  // small jobs are still cut into single loops
  wl_job k = job_of(h, field_of(WL_PROFILE_SMOOTH, 1, 50), 40, 1, v, T);
  need(wl_batch_eval(c, 1, &k, 0), "batch");
  say("small_per_loop", g_jobs[0].per_loop);
}

// a light job's cut, alone and beside a heavy job that runs in a launch of its own
static void batch_side(wl_ctx *c) {
  const int n = 4000, Nl = 5120, h = ensemble(c, Nl, 4096), h2 = ensemble(c, 1024, 1024);
  double *v = new double[n], *T = new double[n];
  for (int i = 0; i < n; ++i) v[i] = 0.1, T[i] = 1.0;
  wl_job j[2] = {job_of(h2, field_of(WL_PROFILE_SMOOTH, 0, 4), 300, 1, v, T),
                 job_of(h, field_of(WL_PROFILE_FIXFLUX, 0, 50), n, 1, v, T)};
  for (int k = 1; k <= 2; ++k) {
    need(wl_batch_eval(c, k, j, 0), "batch");
    say(k == 1 ? "alone" : "beside", g_jobs[0].per_loop);
  }
}

// EV() configured for the lattice: launches nothing, returns NaN
static void ev_lattice(wl_ctx *c) {
  const int Nl = 128, ppl = 64, h = ensemble(c, Nl, ppl);
  const float *loops = nullptr;
  need(wl_ensemble_info(c, h, &loops, nullptr, nullptr), "info");
  need(wl_legacy_configure(WL_PROFILE_LATTICE, 2.0, 0.1, 4, WL_MODE_EXACT), "configure");
  struct Wparams p;
  memset(&p, 0, sizeof(p));
  p.Nl = Nl;
  p.Nppl = ppl;
  p.F = 1.0;
  p.l2 = 0.5;
  p.ng = 1;
  p.worldlines = (float4 *)loops;
  cudaMalloc((void **)&p.Wsscal_d, sizeof(float4) * Nl);
  int list[128];
  for (int j = 0; j < 128; ++j) list[j] = j;
  const long before = g_kernels;
  say("nan", isnan(EV(0.5, &p, list)));
  say("kernels", (double)(g_kernels - before));
}

// every launch the host lets through has its last warp's unit index in 32 bits
static void sweep_grid() {
  bool ok = wl::sweep_ctas(1) == 1 && wl::sweep_ctas(4) == 1 && wl::sweep_ctas(5) == 2;
  for (int b = 3; b < 62; ++b)
    for (int d = -1; d <= 1; ++d) {
      const long long items = (1ll << b) + d;
      const unsigned ctas = wl::sweep_ctas(items);
      if (items <= 1ll << 32) ok &= (long long)ctas * wl::kSweepWarps >= items;
      ok &= (unsigned long long)ctas * wl::kSweepWarps <= 1ull << 32;
    }
  say("ok", ok);
}

// smooth_clamp_idle(): where it says so, lambda^2 + max(a, clamp) and lambda^2 + a
// are the same float for every a below the clamp; elsewhere they differ somewhere
static void clamp_idle() {
  int wrong = 0, idle = 0;
  const float widths[] = {1e-7f, 0.01f, 0.2f, 0.24999999f, 0.25f, 0.3f, 0.49999997f, 0.5f, 1.0f, 300.0f};
  for (float l2 : widths)
    for (float clamp : {1e-8f, 1e-30f, -INFINITY}) {
      wl::FieldDev f;
      memset(&f, 0, sizeof(f));
      f.l2 = l2;
      f.clampA = clamp;
      bool same = true;
      for (float a = 0.0f; clamp > 0.0f && a <= clamp; a = a * 1.01f + 1e-44f) {
        volatile float x = l2 + fmaxf(a, clamp), y = l2 + a;
        same &= x == y;
      }
      wrong += same != wl::smooth_clamp_idle(f);
      idle += same;
    }
  say("wrong", wrong);
  say("idle", idle);
}

// which launches are cut into single loops: 10 alone on the chip, 1 among others
static void cut_rule() {
  struct Case {
    const char *name;
    int profile, fermion, nint, ninst, nF, Nl, ppl, chunk;
  };
  const Case cases[] = {
      {"short_loops_full_chip", WL_PROFILE_SMOOTH, 0, 4, 1024, 1, 1024, 64, 8},
      {"four_fluxes", WL_PROFILE_SMOOTH, 0, 4, 512, 4, 1024, 256, 8},
      {"scan", WL_PROFILE_SMOOTH, 1, 4, 96, 3, 5120, 2048, 8},
      {"long_loops_full_chip", WL_PROFILE_SMOOTH, 0, 4, 1024, 1, 1024, 1024, 8},
      {"heavier_nodes", WL_PROFILE_GAUSSIAN, 1, 16, 333, 2, 1500, 516, 5},
      {"just_above_a_wave", WL_PROFILE_SMOOTH, 0, 4, 513, 2, 1152, 232, 8},
      {"few_units", WL_PROFILE_SMOOTH, 0, 4, 40, 4, 1024, 64, 8},
      {"many_waves", WL_PROFILE_SMOOTH, 1, 4, 8192, 3, 5120, 2048, 8}};
  for (const Case &k : cases) {
    wl::SweepArgs a;
    memset(&a, 0, sizeof(a));
    a.ninst = k.ninst;
    a.nF = k.nF;
    a.ppl = k.ppl;
    a.chunk_loops = k.chunk;
    a.n_chunks = k.Nl / k.chunk;
    const double items = wl::sweep_chunk_items(a, k.profile, k.nint);
    wl::sweep_units(a, k.profile, k.fermion, k.nint, items, true);
    const int alone = a.per_loop;
    wl::sweep_units(a, k.profile, k.fermion, k.nint, items, false);
    say(k.name, 10 * alone + a.per_loop);
    if (a.n_units != (k.Nl + a.unit_loops - 1) / a.unit_loops) exit(4);
  }
}

int main(int argc, char **argv) {
  const std::string s = argc > 1 ? argv[1] : "";
  wl_ctx *c = nullptr;
  need(wl_ctx_create(0, &c), "context");
  if (s == "tint_staging") tint_staging(c);
  else if (s == "loop_waits") loop_waits(c);
  else if (s == "launches") launches(c);
  else if (s == "batch_scratch") batch_scratch(c);
  else if (s == "batch_side") batch_side(c);
  else if (s == "ev_lattice") ev_lattice(c);
  else if (s == "sweep_grid") sweep_grid();
  else if (s == "clamp_idle") clamp_idle();
  else if (s == "cut_rule") cut_rule();
  else return 3;
  wl_ctx_destroy(c);
  return 0;
}
