// The per-step sweep kernels: one Douglas ADI timestep in scaled delta form (see hs2g_compile.cu for the
// algebra and hs2g_internal.cuh for the coefficient layout).  Replaces, per timestep, the reference's
// source-field assembly and three permute / CSR mat-vec / tridiagonal-solve stages
// (alternatingdirection_c_pyx.pyx:294-416, tridiag.pyx:46-69).
//
// FP64 is the binding resource on GB300 (about 0.6e12 DFMA/s against ~6.5 TB/s of HBM and 32-bit integer units 64
// times as wide), so the step is arranged for the fewest FP64 operations: the stencil in integers and 2 recurrence
// FMAs per voxel in the x sweep, 2 FMAs per voxel in the y sweep, 2 FMAs and 1 add per voxel in the z sweep.
//   x sweep: hs2g_x.cuh
//   y, z sweeps: one warp per 16 neighbouring lines, both ends of each line at once, rows copied ahead into shared
//            memory and coefficients from tables per line class (hs2g_pair.cuh, hs2g_classes.cu).
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "hs2g_internal.cuh"
#include "hs2g_pair.cuh"
#include "hs2g_x.cuh"

namespace hs2g {
namespace {

// Where a launch's class source values come from: nowhere, the kernel's parameter table, or row ds->step of the
// handle's device schedule (an inactive row or one past the schedule's end gives zeros).
enum XSource { kNoSource, kTable, kRow };
template <int SRC>
using XTable = typename std::conditional<SRC == kTable, QTable, int>::type;

// the class source values of the launch into shared memory (SRC), before the kernel waits for the previous one
template <int SRC>
__device__ __forceinline__ void x_sources(XProblem<double>& P, const XTable<SRC>& qt, const DevSchedule* ds, double* sq) {
  if constexpr (SRC == kTable)
    for (int e = threadIdx.x; e < HS2G_MAX_CLASSES; e += blockDim.x) sq[e] = qt.q[e];
  if constexpr (SRC == kRow) {
    const int64_t st = ds->step;
    const bool on = st >= 0 && st < ds->n && ds->active[st];
    for (int e = threadIdx.x; e < HS2G_MAX_CLASSES; e += blockDim.x) sq[e] = on ? ds->q[st * HS2G_MAX_CLASSES + e] : 0.0;
    P.qshape = ds->shape;
  }
}
// The stencil of the x-lines [begin, end): a CTA per kXStencilLines lines and per gridDim.y-th chunk of columns.
template <int SRC, bool SHARED, typename IX>
__global__ void __launch_bounds__(32 * kXStencilWarps, kXStencilCtas) x_stencil_kernel(XProblem<double> P, XTable<SRC> qt,
                                                                           const DevSchedule* ds, int64_t begin,
                                                                           int64_t end) {
  __shared__ XLine<IX> lines[kXStencilLines];
  __shared__ double sq[SRC == kNoSource ? 1 : HS2G_MAX_CLASSES];
  x_sources<SRC>(P, qt, ds, sq);
  wait_prior_grid();  // T comes from the previous step's z sweep, which used W0 as its scratch
  x_stencil_lines<double, SRC != kNoSource, SHARED, IX>(P, begin + blockIdx.x * (int64_t)kXStencilLines, end, blockIdx.y,
                                                gridDim.y, lines, sq);
}
// The whole x sweep of [begin, end), 16 lines per CTA.
template <int SRC, bool SHARED, typename IX>
__global__ void __launch_bounds__(kXFusedThreads, 3) x_fused_kernel(XProblem<double> P, XTable<SRC> qt,
                                                                    const DevSchedule* ds, int64_t begin, int64_t end) {
  extern __shared__ __align__(16) unsigned char x_sm[];
  x_sources<SRC>(P, qt, ds, reinterpret_cast<double*>(x_sm));
  wait_prior_grid();
  x_fused_lines<SRC != kNoSource, SHARED, IX>(P, begin + blockIdx.x * (int64_t)16, end, x_sm);
}
// The x line solves of [begin, end) in W0, 16 lines per warp.
template <bool TABLE, bool KEEP>
__global__ void __launch_bounds__(32 * kPairMaxWarps) x_solve_kernel(XProblem<double> P, int64_t begin, int64_t end,
                                                                     int64_t smem_per_warp) {
  extern __shared__ __align__(16) unsigned char x_sm[];
  const int64_t L0 = begin + (blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5)) * x_lines<true>();
  if (L0 >= end) return;
  wait_prior_grid();
  x_solve_lines<double, true, TABLE, KEEP>(P, L0, (int)min((int64_t)x_lines<true>(), end - L0),
                                           reinterpret_cast<double*>(x_sm + (threadIdx.x >> 5) * smem_per_warp));
}

// 32-bit index arithmetic when every voxel index, with the pad column of an odd nx, is below 2^31
bool x_index32(const Dims& d, const Coeffs& c) { return d.nz * d.ny * c.px < ((int64_t)1 << 31); }

using XSolveKernel = void (*)(XProblem<double>, int64_t, int64_t, int64_t);
XSolveKernel x_solve_for(bool table, bool keep) {
  return table ? (keep ? x_solve_kernel<true, true> : x_solve_kernel<true, false>)
               : (keep ? x_solve_kernel<false, true> : x_solve_kernel<false, false>);
}
template <int SRC, bool SHARED>
cudaError_t launch_x(const StepArgs& a, const Coeffs& c, const XTable<SRC>& q, const DevSchedule* ds, int64_t begin,
                     int64_t end, cudaStream_t s) {
  if (end <= begin) return cudaSuccess;
  const XProblem<double> P{a.d.nz, a.d.ny, a.d.nx, a.T_in, c.xb, c.bidx, c.nchunks, c.a0, c.b0, c.cls0,
                           a.vclass, a.qdense, a.qshape, a.W0, c.px};
  if (c.cls0 && (x_index32(a.d, c) ? x_fused<int32_t>(a.d.nx, end - begin) : x_fused<int64_t>(a.d.nx, end - begin))) {
    const dim3 grid((unsigned)((end - begin + 15) / 16)), block(kXFusedThreads);
    if (x_index32(a.d, c))
      return launch_kernel(x_fused_kernel<SRC, SHARED, int32_t>, grid, block, x_fused_smem<int32_t>(a.d.nx), s, a.pdl_x, P, q, ds,
                           begin, end);
    return launch_kernel(x_fused_kernel<SRC, SHARED, int64_t>, grid, block, x_fused_smem<int64_t>(a.d.nx), s, a.pdl_x, P, q, ds,
                         begin, end);
  }
  // a CTA walks its lines' chunks, or takes every second, fourth ... of them until there are CTAs enough for the GPU
  const int64_t ctas = (end - begin + kXStencilLines - 1) / kXStencilLines;
  unsigned split = 1;
  while (split < c.nchunks && split < 32768 && ctas * split < kSMs * 8) split *= 2;
  const dim3 grid((unsigned)ctas, split), block(32 * kXStencilWarps);
  cudaError_t e = x_index32(a.d, c)
                      ? launch_kernel(x_stencil_kernel<SRC, SHARED, int32_t>, grid, block, 0, s, a.pdl_x, P, q, ds, begin, end)
                      : launch_kernel(x_stencil_kernel<SRC, SHARED, int64_t>, grid, block, 0, s, a.pdl_x, P, q, ds, begin, end);
  if (e != cudaSuccess) return e;
  const int64_t groups = (end - begin + x_lines<true>() - 1) / x_lines<true>();
  const PairShape sh = c.cls0 ? x_solve_shape<double, true, true>(a.d.nx, groups)
                              : x_solve_shape<double, true, false>(a.d.nx, groups);
  return launch_kernel(x_solve_for(c.cls0 != nullptr, sh.keep), dim3((unsigned)((groups + sh.warps - 1) / sh.warps)),
                       dim3(32 * sh.warps), sh.smem, s, a.pdl, P, begin, end, (int64_t)(sh.smem / sh.warps));
}
cudaError_t launch_x_any(const StepArgs& a, const Coeffs& c, const QTable& q, int64_t begin, int64_t end,
                         cudaStream_t s) {
  if (a.has_qtab || a.qdense)
    return c.bidx ? launch_x<kTable, true>(a, c, q, nullptr, begin, end, s)
                  : launch_x<kTable, false>(a, c, q, nullptr, begin, end, s);
  return c.bidx ? launch_x<kNoSource, true>(a, c, 0, nullptr, begin, end, s)
                : launch_x<kNoSource, false>(a, c, 0, nullptr, begin, end, s);
}

// The y sweep (ADD_T false: W1 = s2 * dT1 from W0 = sigma * dT0; rows of lines k) and the z sweep (ADD_T: T_out =
// T_in + dT2 from W1 = s2 * dT1; rows of lines j; W0 the scratch of the forward values, T_in may be T_out) over the
// rows of lines [begin, end).  One warp per group of 16 neighbouring lines.
struct PairArgs {
  Dims d;
  int64_t px;
  const double* W;
  const double* a;
  const double* b;
  const int32_t* cls;
  const double* T;
  double* out;
  double* Z;
  int64_t begin, end;
};
// the 16 lines of group grp; their number, 0 past the last group
template <bool ADD_T, bool TABLE>
__device__ __forceinline__ int pair_group(const PairArgs& g, int64_t grp, PairLines<double>& p) {
  const int64_t nx = g.d.nx, gpr = (nx + 15) / 16;  // groups per row of lines
  const int64_t row = g.begin + grp / gpr, i0 = (grp % gpr) * 16;
  if (row >= g.end) return 0;
  const int64_t w = ADD_T ? row * g.px + i0 : row * g.d.ny * g.px + i0;  // first line's first row in the padded arrays
  const int64_t wst = ADD_T ? g.d.ny * g.px : g.px;
  p.W = g.W + w;
  p.wst = p.cst = p.zst = wst;
  p.a = TABLE ? g.a : g.a + w;
  p.b = TABLE ? g.b : g.b + w;
  p.cls = TABLE ? g.cls + row * nx + i0 : nullptr;
  p.T = ADD_T ? g.T + row * nx + i0 : nullptr;
  p.out = g.out + (ADD_T ? row * nx + i0 : w);
  p.st = ADD_T ? g.d.nxy() : wst;
  p.Z = g.Z + w;
  return (int)min((int64_t)16, nx - i0);
}
template <bool ADD_T, bool KEEP, bool TABLE, int TVEC>
__global__ void __launch_bounds__(32 * kPairMaxWarps) pair_sweep_kernel(PairArgs g, int64_t smem_per_warp) {
  extern __shared__ __align__(16) unsigned char pair_sm[];
  PairLines<double> p{};
  const int width = pair_group<ADD_T, TABLE>(g, blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5), p);
  if (!width) return;
  wait_prior_grid();
  pair_solve<double, true, ADD_T, KEEP, TABLE, 2, TVEC>(
      p, (int)(ADD_T ? g.d.nz : g.d.ny), width, reinterpret_cast<double*>(pair_sm + (threadIdx.x >> 5) * smem_per_warp));
}
__global__ void copy_layer_kernel(Dims d, const double* __restrict__ T, int layer, double* __restrict__ dst) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t < d.nxy()) dst[t] = T[(int64_t)layer * d.nxy() + t];
}

// Temperature of the z = 0 surface estimated from layers 0 and 1 as the reference's
// insulating_z_min_surface_temperature(T, dz) does (surface_temperature.py:4-36): the mean of a quadratic with
// zero slope at the surface through the two layer centres, c = T0 - (0.25 a) dz^2 with a = (T1 - T0)/(2 dz^2),
// and the linear extrapolation T0 - (T1 - T0)/2.  Same operations in the same order, each rounding explicit.
__device__ __forceinline__ double surface_value(double t0, double t1, double dz2) {
  const double a = __ddiv_rn(__dsub_rn(t1, t0), __dmul_rn(2.0, dz2));
  const double c = __dsub_rn(t0, __dmul_rn(__dmul_rn(0.25, a), dz2));
  const double lin = __dsub_rn(t0, __ddiv_rn(__dsub_rn(t1, t0), 2.0));
  return __ddiv_rn(__dadd_rn(lin, c), 2.0);
}
__global__ void surface_estimate_kernel(int64_t nxy, const double* __restrict__ T, double dz2,
                                        double* __restrict__ dst) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t < nxy) dst[t] = surface_value(T[t], T[nxy + t], dz2);
}

inline unsigned blocks(int64_t n, int per) { return (unsigned)((n + per - 1) / per); }
// History of a step into row ds->row of hist: layer `layer` of T, or (dz2 > 0) the surface estimate; the last
// CTA to finish advances the row (every CTA read it at its start).
__global__ void history_row_kernel(int64_t nxy, const double* __restrict__ T, int layer, double dz2,
                                   double* __restrict__ hist, DevSchedule* ds) {
  __shared__ int64_t s_row;
  wait_prior_grid();
  if (threadIdx.x == 0) s_row = *(volatile int64_t*)&ds->row;
  __syncthreads();
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t < nxy)
    hist[s_row * nxy + t] = dz2 > 0.0 ? surface_value(T[t], T[nxy + t], dz2) : T[(int64_t)layer * nxy + t];
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&ds->hist_done, 1u) == gridDim.x - 1) {
      ds->row = s_row + 1;
      ds->hist_done = 0;
      __threadfence();
    }
  }
}

__global__ void schedule_flags_kernel(const double* __restrict__ q, int64_t nrows, uint8_t* __restrict__ active) {
  const int64_t r = blockIdx.x * (int64_t)(blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= nrows) return;
  bool any = false;
  for (int c = lane; c < HS2G_MAX_CLASSES; c += 32) any |= q[r * HS2G_MAX_CLASSES + c] != 0.0;
  any = __any_sync(0xffffffffu, any);
  if (lane == 0) active[r] = any ? 1 : 0;
}


// FP64 issue-rate probe: 8 independent FMA chains per thread, registers only, one store per thread.
__global__ void fp64_probe_kernel(double* out, int iters, double a, double b) {
  double acc[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = (double)(threadIdx.x + k);
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = fma(acc[k], a, b);
  }
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += acc[k];
  out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

}  // namespace

cudaError_t fp64_fma_rate(double* fma_per_s) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const int blocksN = sms * 4, threads = 256, iters = 4096;
  double* out = nullptr;
  e = cudaMalloc(&out, sizeof(double) * blocksN * threads);
  if (e != cudaSuccess) return e;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  float best = 1e30f;
  for (int rep = 0; rep < 5; ++rep) {
    cudaEventRecord(e0, 0);
    fp64_probe_kernel<<<blocksN, threads>>>(out, iters, 0.999999, 1e-7);
    cudaEventRecord(e1, 0);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (rep > 0 && ms < best) best = ms;
  }
  e = cudaGetLastError();
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  *fma_per_s = (double)blocksN * threads * iters * 8 / (best * 1e-3);
  return e;
}

namespace {
using PairKernel = void (*)(PairArgs, int64_t);
template <bool ADD_T>
PairKernel pair_kernel(bool keep, bool table, bool t16) {
  // T moves 16 bytes at a time when its rows start on 16-byte boundaries (an even nx)
  if (table)
    return keep ? (ADD_T && !t16 ? pair_sweep_kernel<ADD_T, true, true, 1> : pair_sweep_kernel<ADD_T, true, true, 2>)
                : (ADD_T && !t16 ? pair_sweep_kernel<ADD_T, false, true, 1> : pair_sweep_kernel<ADD_T, false, true, 2>);
  return keep ? (ADD_T && !t16 ? pair_sweep_kernel<ADD_T, true, false, 1> : pair_sweep_kernel<ADD_T, true, false, 2>)
              : (ADD_T && !t16 ? pair_sweep_kernel<ADD_T, false, false, 1> : pair_sweep_kernel<ADD_T, false, false, 2>);
}
template <bool ADD_T>
cudaError_t launch_pair(const PairArgs& g, cudaStream_t s, bool pdl) {
  if (g.end <= g.begin) return cudaSuccess;
  const int64_t n = ADD_T ? g.d.nz : g.d.ny, groups = (g.end - g.begin) * ((g.d.nx + 15) / 16);
  const bool table = g.cls != nullptr;
  const bool t16 = g.d.nx % 2 == 0 && ((reinterpret_cast<uintptr_t>(g.T) & 15) == 0);
  const PairShape sh = table ? pair_shape<double, true, ADD_T, true>(n, groups) : pair_shape<double, true, ADD_T, false>(n, groups);
  return launch_kernel(pair_kernel<ADD_T>(sh.keep, table, t16), dim3((unsigned)((groups + sh.warps - 1) / sh.warps)),
                       dim3(32 * sh.warps), sh.smem, s, pdl, g, (int64_t)(sh.smem / sh.warps));
}
// the y and z sweeps of a step, with events before each and after the last when ev is given
cudaError_t launch_yz(const StepArgs& a, const Coeffs& c, cudaStream_t s, cudaEvent_t* ev) {
  cudaError_t e = launch_y(a, c, s);
  if (e != cudaSuccess) return e;
  if (ev) cudaEventRecord(ev[2], s);
  e = launch_z_rows(a, c, 0, a.d.ny, s);
  if (e != cudaSuccess) return e;
  if (ev) cudaEventRecord(ev[3], s);
  return cudaGetLastError();
}
}  // namespace

cudaError_t sweeps_prepare(const Dims& d, const Coeffs& c) {
  constexpr size_t kDefault = 48 * 1024, kMost = 226 * 1024;
  cudaError_t e = cudaSuccess;
  // A CTA has up to kPairMaxWarps warps' shares, at most kMost.  The limit belongs to the kernel, not to the problem:
  // always the same value, so that a small problem never takes from what an earlier one needs.
  auto allow = [&](const void* kernel, size_t smem) {
    if (smem > kDefault && e == cudaSuccess)
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost);
  };
  const bool tx = c.cls0 != nullptr, ty = c.cls1 != nullptr, tz = c.cls2 != nullptr;
  auto most = [](size_t keep, size_t ring) { return kPairMaxWarps * std::max(keep, ring); };
  for (int keep = 0; keep < 2; ++keep) {
    allow((const void*)x_solve_for(tx, keep), most(tx ? x_solve_smem<double, true, true, true>(d.nx) : x_solve_smem<double, true, false, true>(d.nx),
                                                   x_solve_smem<double, true, false, false>(d.nx)));
    allow((const void*)pair_kernel<false>(keep, ty, true),
          most(ty ? pair_smem<double, true, false, true, true>(d.ny) : pair_smem<double, true, false, true, false>(d.ny),
               pair_smem<double, true, false, false, false>(d.ny)));
    for (int t16 = 0; t16 < 2; ++t16)
      allow((const void*)pair_kernel<true>(keep, tz, t16),
            most(tz ? pair_smem<double, true, true, true, true>(d.nz) : pair_smem<double, true, true, true, false>(d.nz),
                 pair_smem<double, true, true, false, false>(d.nz)));
  }
  auto allow_fused = [&](auto shared) {
    constexpr bool S = decltype(shared)::value;
    for (const void* k : {(const void*)x_fused_kernel<kNoSource, S, int32_t>, (const void*)x_fused_kernel<kTable, S, int32_t>,
                          (const void*)x_fused_kernel<kRow, S, int32_t>, (const void*)x_fused_kernel<kNoSource, S, int64_t>,
                          (const void*)x_fused_kernel<kTable, S, int64_t>, (const void*)x_fused_kernel<kRow, S, int64_t>})
      allow(k, x_fused_smem<int64_t>(d.nx));
  };
  if (c.bidx)
    allow_fused(std::true_type());
  else
    allow_fused(std::false_type());
  return e;
}

cudaError_t launch_step_events(const StepArgs& a, const Coeffs& c, const QTable& q, cudaStream_t s,
                               cudaEvent_t ev[4]) {
  if (ev) cudaEventRecord(ev[0], s);
  const cudaError_t e = launch_x_any(a, c, q, 0, a.d.nz * a.d.ny, s);
  if (e != cudaSuccess) return e;
  if (ev) cudaEventRecord(ev[1], s);
  return launch_yz(a, c, s, ev);
}

cudaError_t launch_step(const StepArgs& a, const Coeffs& c, const QTable& q, cudaStream_t s) {
  return launch_step_events(a, c, q, s, nullptr);
}

cudaError_t launch_step_row(const StepArgs& a, const Coeffs& c, const DevSchedule* ds, cudaStream_t s) {
  const cudaError_t e = c.bidx ? launch_x<kRow, true>(a, c, 0, ds, 0, a.d.nz * a.d.ny, s)
                               : launch_x<kRow, false>(a, c, 0, ds, 0, a.d.nz * a.d.ny, s);
  if (e != cudaSuccess) return e;
  return launch_yz(a, c, s, nullptr);
}

cudaError_t launch_history_row(const Dims& d, const double* T, int layer, double dz2, double* hist, DevSchedule* ds,
                               cudaStream_t s, bool pdl) {
  return launch_kernel(history_row_kernel, dim3(blocks(d.nxy(), 256)), dim3(256), 0, s, pdl, d.nxy(), T, layer, dz2,
                       hist, ds);
}

cudaError_t launch_schedule_flags(const double* q, int64_t nrows, uint8_t* active, cudaStream_t s) {
  if (nrows <= 0) return cudaSuccess;
  schedule_flags_kernel<<<blocks(nrows, 8), 256, 0, s>>>(q, nrows, active);
  return cudaGetLastError();
}

double surface_dz2(double dz) {
  // dz^2 as the reference's dz**2.0 computes it: the C library's pow, which can differ from dz*dz by an ulp (the
  // volatile exponent keeps the compiler from replacing the call by a multiplication)
  volatile double two = 2.0;
  return std::pow(dz, (double)two);
}

cudaError_t launch_x_range(const StepArgs& a, const Coeffs& c, const QTable& q, int64_t line_begin,
                           int64_t line_end, cudaStream_t s) {
  return launch_x_any(a, c, q, line_begin, line_end, s);
}

cudaError_t launch_y(const StepArgs& a, const Coeffs& c, cudaStream_t s) {
  return launch_pair<false>(PairArgs{a.d, c.px, a.W0, c.a1, c.b1, c.cls1, nullptr, a.W1, a.W1, 0, a.d.nz}, s, a.pdl);
}

cudaError_t launch_z_rows(const StepArgs& a, const Coeffs& c, int64_t j_begin, int64_t j_end, cudaStream_t s) {
  return launch_pair<true>(PairArgs{a.d, c.px, a.W1, c.a2, c.b2, c.cls2, a.T_in, a.T_out, a.W0, j_begin, j_end}, s,
                           a.pdl);
}

cudaError_t launch_copy_layer(const Dims& d, const double* T, int layer, double* dst, cudaStream_t s) {
  copy_layer_kernel<<<blocks(d.nxy(), 256), 256, 0, s>>>(d, T, layer, dst);
  return cudaGetLastError();
}

cudaError_t launch_surface_estimate(int64_t nxy, const double* T, double dz, double* dst, cudaStream_t s) {
  const double dz2 = surface_dz2(dz);
  surface_estimate_kernel<<<blocks(nxy, 256), 256, 0, s>>>(nxy, T, dz2, dst);
  return cudaGetLastError();
}

}  // namespace hs2g
