// Batched timestep: many independent problems of uneven size advanced together.
//
// All instances live in one concatenated device state (instance b's fields start at voxel offset off[b], each
// (nz_b, ny_b, nx_b) C-ordered).  A step is four sweep kernels over flattened work lists, a CTA per work item -- the x
// stencil and the x solve: 64 x-lines of an instance (the stencil a CTA per 16 of them and, split, per part of their
// columns); y and z: kPairMaxWarps groups of neighbouring lines, a group per warp -- with the instances of the longest
// lines first, and a step-counter increment.  They are captured once in a CUDA graph and replayed; the per-step source
// tables are uploaded once and selected on the device by the step counter, so the graph never changes.
//
// The arithmetic per line is that of the single-problem kernels (hs2g_sweep.cu, scaled delta-form Douglas
// ADI), templated on the storage type: double (results equal to the single-problem path bit for bit) or float
// (coefficients compiled in double, rounded once; its error against double is measured by the caller).
// hs2g_batch_autotune chooses, timed on the batch, how many CTAs share an item's columns in the stencil and whether
// each axis's forward values stay in shared memory.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "hs2g_internal.cuh"
#include "hs2g_pair.cuh"
#include "hs2g_x.cuh"

namespace hs2g {
namespace {

struct Inst {
  Dims d;
  int64_t off;      // voxel offset in the concatenated fields
  int64_t nchunks;  // 32-column chunks per x-line
  int64_t woff;     // offset of the instance in W0 and W1, whose rows have pitch px (nx rounded up to 16 bytes)
  int64_t px;
  const void* pool;      // stencil blocks, and their index per (line, chunk) or null
  const int32_t* bidx;
  // x, y and z line coefficients: in voxel order (row pitch px), or with cls tables per line class
  const void* a[3];
  const void* b[3];
  const int32_t* cls[3];
};

struct XWork {
  int32_t inst;
  int32_t pad;
  int64_t L0;  // first x-line of the block
};
struct LWork {
  int32_t inst;
  int32_t pad;
  int64_t g0;  // first group of neighbouring lines (y: rows of lines k, z: rows of lines j)
};

template <typename R>
struct BatchView {
  const Inst* inst;
  R* T;
  R* W0;
  R* W1;
  const uint8_t* vclass;
  const R* qtabs;          // [nsched][ninst][nclass]
  const uint8_t* active;   // [nsched][ninst] any source active
  const int* step;         // device step counter
  int nsched, ninst, nclass;
  const XWork* xw;
  const LWork* yw;
  const LWork* zw;
};


template <typename R>
__device__ __forceinline__ XProblem<R> x_problem(const BatchView<R>& v, const Inst& I) {
  return {I.d.nz, I.d.ny, I.d.nx, v.T + I.off, (const R*)I.pool, I.bidx, I.nchunks, (const R*)I.a[0], (const R*)I.b[0],
          I.cls[0], v.vclass + I.off, nullptr, nullptr, v.W0 + I.woff, I.px};
}
// x sweep: a work item is kXItemLines consecutive x-lines of one instance.  The stencil takes a CTA per item and
// gridDim.y-th chunk of columns (IX = int32_t when every instance has fewer than 2^31 voxels); the line solves a warp
// per 16 (FP64) or 32 (FP32) lines of an item.  DENSE: some instance keeps its blocks, or line coefficients, in voxel order.
constexpr int kXItemLines = 64;
template <typename R, bool DENSE, typename IX>
__global__ void __launch_bounds__(32 * kXStencilWarps, kXStencilCtas) batch_stencil_kernel(BatchView<R> v) {
  __shared__ XLine<IX> lines[kXStencilLines];
  __shared__ R sq[HS2G_MAX_CLASSES];
  constexpr int SUB = kXItemLines / kXStencilLines;
  const XWork item = v.xw[blockIdx.x / SUB];
  const Inst& I = v.inst[item.inst];
  const int64_t L0 = item.L0 + (int)(blockIdx.x % SUB) * kXStencilLines, end = I.d.nz * I.d.ny;
  if (L0 >= end || blockIdx.y >= I.nchunks) return;
  const XProblem<R> P = x_problem(v, I);
  const int step = *v.step;
  if (step < v.nsched && v.active[(int64_t)step * v.ninst + item.inst]) {
    const R* q = v.qtabs + ((int64_t)step * v.ninst + item.inst) * v.nclass;
    for (int c = threadIdx.x; c < HS2G_MAX_CLASSES; c += 32 * kXStencilWarps) sq[c] = c < v.nclass ? q[c] : R(0);
    if (!DENSE || P.bidx)
      x_stencil_lines<R, true, true, IX>(P, L0, end, blockIdx.y, gridDim.y, lines, sq);
    else
      x_stencil_lines<R, true, false, IX>(P, L0, end, blockIdx.y, gridDim.y, lines, sq);
  } else {
    if (!DENSE || P.bidx)
      x_stencil_lines<R, false, true, IX>(P, L0, end, blockIdx.y, gridDim.y, lines, sq);
    else
      x_stencil_lines<R, false, false, IX>(P, L0, end, blockIdx.y, gridDim.y, lines, sq);
  }
}
template <typename R, bool KEEP, bool DENSE>
__global__ void __launch_bounds__(32 * kPairMaxWarps) batch_x_solve_kernel(BatchView<R> v, int64_t smem_per_warp) {
  extern __shared__ __align__(16) unsigned char batch_x_sm[];
  constexpr bool TWO = sizeof(R) == 8;
  const XWork item = v.xw[blockIdx.x];
  const Inst& I = v.inst[item.inst];
  const int64_t L0 = item.L0 + (threadIdx.x >> 5) * x_lines<TWO>(), end = I.d.nz * I.d.ny;
  if (L0 >= end) return;
  const int count = (int)min((int64_t)x_lines<TWO>(), end - L0);
  R* sm = reinterpret_cast<R*>(batch_x_sm + (threadIdx.x >> 5) * smem_per_warp);
  if (!DENSE || I.cls[0])
    x_solve_lines<R, TWO, true, KEEP>(x_problem(v, I), L0, count, sm);
  else
    x_solve_lines<R, TWO, false, KEEP>(x_problem(v, I), L0, count, sm);
}

// y lines (W1 = s2*dT1 from W0 = sigma*dT0) and z lines (ADD_T: T += dT2 from W1 = s2*dT1, W0 as scratch): a CTA takes
// one work item, kPairMaxWarps groups of 16 (FP64, both ends) or 32 (FP32) neighbouring lines of one instance, a
// group per warp.  DENSE: some instance keeps its coefficients in voxel order.
template <typename R, bool ADD_T, bool KEEP, bool DENSE>
__global__ void __launch_bounds__(32 * kPairMaxWarps) batch_pair_kernel(BatchView<R> v, int64_t smem_per_warp) {
  extern __shared__ __align__(16) unsigned char batch_sm[];
  constexpr bool TWO = sizeof(R) == 8;
  constexpr int G = pair_lines<TWO>(), VEC = 16 / sizeof(R);
  const LWork item = (ADD_T ? v.zw : v.yw)[blockIdx.x];
  const Inst& I = v.inst[item.inst];
  const int64_t nx = I.d.nx, ny = I.d.ny, gpr = (nx + G - 1) / G;
  const int64_t grp = item.g0 + (threadIdx.x >> 5);
  const int64_t row = grp / gpr, i0 = (grp % gpr) * G;
  if (row >= (ADD_T ? ny : I.d.nz)) return;
  const int64_t w = ADD_T ? row * I.px + i0 : row * ny * I.px + i0, wst = ADD_T ? ny * I.px : I.px;
  constexpr int AX = ADD_T ? 2 : 1;
  const int32_t* cls = I.cls[AX];
  PairLines<R> p{};
  p.W = (ADD_T ? v.W1 : v.W0) + I.woff + w;
  p.wst = p.cst = p.zst = wst;
  p.a = (const R*)I.a[AX] + (cls ? 0 : w);
  p.b = (const R*)I.b[AX] + (cls ? 0 : w);
  p.cls = cls ? cls + row * nx + i0 : nullptr;
  p.T = ADD_T ? v.T + I.off + row * nx + i0 : nullptr;
  p.out = ADD_T ? v.T + I.off + row * nx + i0 : v.W1 + I.woff + w;
  p.st = ADD_T ? nx * ny : wst;
  p.Z = (ADD_T ? v.W0 : v.W1) + I.woff + w;
  const int n = (int)(ADD_T ? I.d.nz : ny), width = (int)min((int64_t)G, nx - i0);
  R* sm = reinterpret_cast<R*>(batch_sm + (threadIdx.x >> 5) * smem_per_warp);
  const bool t16 = !ADD_T || (nx % VEC == 0 && I.off % VEC == 0);
  if (!DENSE || cls) {
    if (t16)
      pair_solve<R, TWO, ADD_T, KEEP, true, VEC, VEC>(p, n, width, sm);
    else
      pair_solve<R, TWO, ADD_T, KEEP, true, VEC, 1>(p, n, width, sm);
  } else {
    if (t16)
      pair_solve<R, TWO, ADD_T, KEEP, false, VEC, VEC>(p, n, width, sm);
    else
      pair_solve<R, TWO, ADD_T, KEEP, false, VEC, 1>(p, n, width, sm);
  }
}

__global__ void batch_advance_kernel(int* step) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *step += 1;
}

template <typename R>
__global__ void convert_kernel(const double* __restrict__ src, R* __restrict__ dst, int64_t n) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    dst[e] = (R)src[e];
}
template <typename R>
__global__ void widen_kernel(const R* __restrict__ src, double* __restrict__ dst, int64_t n) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    dst[e] = (double)src[e];
}

struct Tuning {
  int x_split;                  // the stencil's CTAs per item: each takes every x_split-th chunk of columns
  bool x_keep, y_keep, z_keep;  // the forward values of the x / y / z lines stay in shared memory
};

}  // namespace

// ---------------------------------------------------------------------------------------------------------
// Batch object
// ---------------------------------------------------------------------------------------------------------
struct Batch {
  int device = 0;
  int precision = 64;
  int ninst = 0;
  cudaStream_t stream = nullptr;
  std::vector<Inst> inst;
  std::vector<int64_t> offsets;  // [ninst+1] voxel offsets
  int64_t nvox = 0;
  Inst* inst_dev = nullptr;
  void* T = nullptr;  // R*
  void* W0 = nullptr;
  void* W1 = nullptr;
  std::vector<void*> coef_mem;  // the instances' coefficients
  int64_t nw = 0;               // elements of W0 and W1
  uint8_t* vclass = nullptr;
  void* qtabs = nullptr;
  uint8_t* active = nullptr;
  int nsched = 0, nclass = 1;
  int* step = nullptr;
  XWork* xw = nullptr;
  LWork* yw = nullptr;
  LWork* zw = nullptr;
  int64_t nxw = 0, nyw = 0, nzw = 0;
  Tuning tune{1, true, true, true};
  int64_t max_nx = 0, max_ny = 0, max_nz = 0;  // longest x, y and z line
  bool dense[3] = {false, false, false};  // some instance keeps its x / y / z coefficients in voxel order
  bool dense_blocks = false;              // and its stencil blocks
  bool ix32 = false;  // every instance's voxels and stencil blocks below 2^31 elements: 32-bit x-sweep indices
  cudaGraphExec_t graph = nullptr;
  int64_t bytes = 0;
  size_t elem() const { return precision == 64 ? 8 : 4; }
};

namespace {

template <typename R>
BatchView<R> view(const Batch& b) {
  BatchView<R> v{};
  v.inst = b.inst_dev;
  v.T = (R*)b.T;
  v.W0 = (R*)b.W0;
  v.W1 = (R*)b.W1;
  v.vclass = b.vclass;
  v.qtabs = (const R*)b.qtabs;
  v.active = b.active;
  v.step = b.step;
  v.nsched = b.nsched;
  v.ninst = b.ninst;
  v.nclass = b.nclass;
  v.xw = b.xw;
  v.yw = b.yw;
  v.zw = b.zw;
  return v;
}

template <typename R>
using BatchPairKernel = void (*)(BatchView<R>, int64_t);
template <typename R, bool ADD_T>
BatchPairKernel<R> batch_pair_for(bool keep, bool dense) {
  return keep ? (dense ? batch_pair_kernel<R, ADD_T, true, true> : batch_pair_kernel<R, ADD_T, true, false>)
              : (dense ? batch_pair_kernel<R, ADD_T, false, true> : batch_pair_kernel<R, ADD_T, false, false>);
}
// launch shape of an axis (force_keep: -1 by rule); CTAs have kPairMaxWarps warps
template <typename R, bool ADD_T>
PairShape batch_shape(const Batch& b, int force_keep) {
  constexpr bool TWO = sizeof(R) == 8;
  const int64_t len = ADD_T ? b.max_nz : b.max_ny, groups = (ADD_T ? b.nzw : b.nyw) * kPairMaxWarps;
  PairShape sh = b.dense[ADD_T ? 2 : 1] ? pair_shape<R, TWO, ADD_T, false>(len, groups, force_keep)
                                : pair_shape<R, TWO, ADD_T, true>(len, groups, force_keep);
  size_t each = b.dense[ADD_T ? 2 : 1] ? pair_smem<R, TWO, ADD_T, true, false>(len) : pair_smem<R, TWO, ADD_T, true, true>(len);
  if (each * kPairMaxWarps > 226 * 1024) sh.keep = false;
  if (!sh.keep) each = b.dense[ADD_T ? 2 : 1] ? pair_smem<R, TWO, ADD_T, false, false>(len) : pair_smem<R, TWO, ADD_T, false, true>(len);
  sh.warps = kPairMaxWarps;
  sh.smem = each * kPairMaxWarps;
  return sh;
}
template <typename R, bool ADD_T>
cudaError_t launch_batch_pair(const Batch& b, const BatchView<R>& v, bool keep, cudaStream_t s) {
  const PairShape sh = batch_shape<R, ADD_T>(b, keep ? 1 : 0);
  const int64_t work = ADD_T ? b.nzw : b.nyw;
  batch_pair_for<R, ADD_T>(sh.keep, b.dense[ADD_T ? 2 : 1])<<<(unsigned)work, 32 * kPairMaxWarps, sh.smem, s>>>(
      v, (int64_t)(sh.smem / kPairMaxWarps));
  return cudaGetLastError();
}
template <typename R>
BatchPairKernel<R> batch_x_solve_for(bool keep, bool dense) {
  return keep ? (dense ? batch_x_solve_kernel<R, true, true> : batch_x_solve_kernel<R, true, false>)
              : (dense ? batch_x_solve_kernel<R, false, true> : batch_x_solve_kernel<R, false, false>);
}
// the same for the x line solves, whose CTAs have a warp per x_lines of an item
template <typename R>
PairShape batch_x_shape(const Batch& b, int force_keep) {
  constexpr bool TWO = sizeof(R) == 8;
  const int warps = kXItemLines / x_lines<TWO>();
  const int64_t groups = b.nxw * warps;
  PairShape sh = b.dense[0] ? x_solve_shape<R, TWO, false>(b.max_nx, groups, force_keep)
                            : x_solve_shape<R, TWO, true>(b.max_nx, groups, force_keep);
  size_t each = b.dense[0] ? x_solve_smem<R, TWO, false, true>(b.max_nx) : x_solve_smem<R, TWO, true, true>(b.max_nx);
  if (each * warps > 226 * 1024) sh.keep = false;
  if (!sh.keep) each = b.dense[0] ? x_solve_smem<R, TWO, false, false>(b.max_nx) : x_solve_smem<R, TWO, true, false>(b.max_nx);
  sh.warps = warps;
  sh.smem = each * warps;
  return sh;
}
template <typename R>
cudaError_t batch_prepare() {
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < 4 && e == cudaSuccess; ++k)
    e = cudaFuncSetAttribute((const void*)batch_x_solve_for<R>(k & 1, k & 2), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             226 * 1024);
  for (int k = 0; k < 8 && e == cudaSuccess; ++k) {
    const void* f = k & 4 ? (const void*)batch_pair_for<R, true>(k & 1, k & 2) : (const void*)batch_pair_for<R, false>(k & 1, k & 2);
    e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
  }
  return e;
}

template <typename R>
cudaError_t launch_axis(const Batch& b, int axis, const Tuning& t, cudaStream_t s) {
  BatchView<R> v = view<R>(b);
  if (axis == 0) {
    const dim3 grid((unsigned)(b.nxw * (kXItemLines / kXStencilLines)), (unsigned)t.x_split);
    const auto stencil = b.dense_blocks ? (b.ix32 ? batch_stencil_kernel<R, true, int32_t> : batch_stencil_kernel<R, true, int64_t>)
                                        : (b.ix32 ? batch_stencil_kernel<R, false, int32_t> : batch_stencil_kernel<R, false, int64_t>);
    stencil<<<grid, 32 * kXStencilWarps, 0, s>>>(v);
    const PairShape sh = batch_x_shape<R>(b, t.x_keep ? 1 : 0);
    batch_x_solve_for<R>(sh.keep, b.dense[0])<<<(unsigned)b.nxw, 32 * sh.warps, sh.smem, s>>>(
        v, (int64_t)(sh.smem / sh.warps));
  } else if (axis == 1) {
    return launch_batch_pair<R, false>(b, v, t.y_keep, s);
  } else if (axis == 2) {
    return launch_batch_pair<R, true>(b, v, t.z_keep, s);
  } else {
    batch_advance_kernel<<<1, 32, 0, s>>>(b.step);
  }
  return cudaGetLastError();
}

cudaError_t launch_axis_any(const Batch& b, int axis, const Tuning& t, cudaStream_t s) {
  return b.precision == 64 ? launch_axis<double>(b, axis, t, s) : launch_axis<float>(b, axis, t, s);
}

cudaError_t launch_step_batch(const Batch& b, cudaStream_t s) {
  cudaError_t e = cudaSuccess;
  for (int axis = 0; axis < 4 && e == cudaSuccess; ++axis) e = launch_axis_any(b, axis, b.tune, s);
  return e;
}

}  // namespace

// Work lists: blocks of consecutive x-lines, and of groups of y and z lines, per instance, longest lines first.
void batch_build_work(Batch& b, std::vector<XWork>& xw, std::vector<LWork>& yw, std::vector<LWork>& zw) {
  xw.clear();
  yw.clear();
  zw.clear();
  const int per = b.precision == 64 ? pair_lines<true>() : pair_lines<false>();
  auto groups = [&](const Dims& d) { return (d.nx + per - 1) / per; };  // of neighbouring lines in a row of lines
  std::vector<int> order(b.ninst);
  for (int i = 0; i < b.ninst; ++i) order[i] = i;
  auto by = [&](auto len) {
    std::vector<int> o = order;
    std::stable_sort(o.begin(), o.end(), [&](int p, int q) { return len(b.inst[p].d) > len(b.inst[q].d); });
    return o;
  };
  for (int ib : by([](const Dims& d) { return d.nx; })) {
    const Dims& d = b.inst[ib].d;
    for (int64_t L0 = 0; L0 < d.nz * d.ny; L0 += kXItemLines) xw.push_back(XWork{ib, 0, L0});
  }
  for (int ib : by([](const Dims& d) { return d.ny; })) {
    const Dims& d = b.inst[ib].d;
    for (int64_t g0 = 0; g0 < d.nz * groups(d); g0 += kPairMaxWarps) yw.push_back(LWork{ib, 0, g0});
  }
  for (int ib : by([](const Dims& d) { return d.nz; })) {
    const Dims& d = b.inst[ib].d;
    for (int64_t g0 = 0; g0 < d.ny * groups(d); g0 += kPairMaxWarps) zw.push_back(LWork{ib, 0, g0});
  }
}

cudaError_t batch_upload_work(Batch& b) {
  std::vector<XWork> xw;
  std::vector<LWork> yw, zw;
  batch_build_work(b, xw, yw, zw);
  if (b.xw) cudaFree(b.xw);
  if (b.yw) cudaFree(b.yw);
  if (b.zw) cudaFree(b.zw);
  b.xw = nullptr;
  b.yw = b.zw = nullptr;
  cudaError_t e = cudaMalloc(&b.xw, sizeof(XWork) * std::max<size_t>(1, xw.size()));
  if (e == cudaSuccess) e = cudaMalloc(&b.yw, sizeof(LWork) * std::max<size_t>(1, yw.size()));
  if (e == cudaSuccess) e = cudaMalloc(&b.zw, sizeof(LWork) * std::max<size_t>(1, zw.size()));
  if (e == cudaSuccess) e = cudaMemcpy(b.xw, xw.data(), sizeof(XWork) * xw.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b.yw, yw.data(), sizeof(LWork) * yw.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b.zw, zw.data(), sizeof(LWork) * zw.size(), cudaMemcpyHostToDevice);
  b.nxw = (int64_t)xw.size();
  b.nyw = (int64_t)yw.size();
  b.nzw = (int64_t)zw.size();
  return e;
}

cudaError_t batch_convert(const double* src, void* dst, int64_t n, int precision, cudaStream_t s) {
  if (precision == 64) return cudaMemcpyAsync(dst, src, sizeof(double) * n, cudaMemcpyDeviceToDevice, s);
  convert_kernel<float><<<1024, 256, 0, s>>>(src, (float*)dst, n);
  return cudaGetLastError();
}

cudaError_t batch_widen(const void* src, double* dst, int64_t n, int precision, cudaStream_t s) {
  if (precision == 64) return cudaMemcpyAsync(dst, src, sizeof(double) * n, cudaMemcpyDeviceToDevice, s);
  widen_kernel<float><<<1024, 256, 0, s>>>((const float*)src, dst, n);
  return cudaGetLastError();
}

cudaError_t batch_step(Batch& b, cudaStream_t s) { return launch_step_batch(b, s); }

cudaError_t batch_time_axis(Batch& b, int axis, const Tuning& t, int reps, float* ms) {
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaError_t e = launch_axis_any(b, axis, t, b.stream);  // warm-up
  cudaEventRecord(e0, b.stream);
  for (int r = 0; r < reps && e == cudaSuccess; ++r) e = launch_axis_any(b, axis, t, b.stream);
  cudaEventRecord(e1, b.stream);
  if (e == cudaSuccess) e = cudaEventSynchronize(e1);
  float v = 0.f;
  cudaEventElapsedTime(&v, e0, e1);
  *ms = v / reps;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return e;
}

// Candidate launch shapes per axis, timed on the batch itself.  Returns the report in `report`.
cudaError_t batch_autotune(Batch& b, std::string& report) {
  Tuning best = b.tune;
  char line[256];
  cudaError_t e = cudaSuccess;
  // x: the stencil's CTAs per item, and the line solves' forward values in shared or global memory
  {
    float bt = 1e30f;
    for (int keep = 1; keep >= 0; --keep)
      for (int split : {1, 2, 4}) {
        Tuning t = best;
        t.x_split = split;
        t.x_keep = keep != 0;
        float ms;
        if ((e = batch_time_axis(b, 0, t, 2, &ms)) != cudaSuccess) return e;
        snprintf(line, sizeof line, "x split %d, forward values in %s memory: %.3f ms\n", split,
                 keep ? "shared" : "global", ms);
        report += line;
        if (ms < bt) bt = ms, best.x_split = split, best.x_keep = keep != 0;
      }
  }
  // y and z: forward values in shared memory or through global memory
  for (int axis = 1; axis <= 2; ++axis) {
    float bt = 1e30f;
    for (int keep = 1; keep >= 0; --keep) {
      Tuning t = best;
      (axis == 1 ? t.y_keep : t.z_keep) = keep != 0;
      float ms;
      if ((e = batch_time_axis(b, axis, t, 2, &ms)) != cudaSuccess) return e;
      snprintf(line, sizeof line, "%s forward values in %s memory: %.3f ms\n", axis == 1 ? "y" : "z",
               keep ? "shared" : "global", ms);
      report += line;
      if (ms < bt) bt = ms, (axis == 1 ? best.y_keep : best.z_keep) = keep != 0;
    }
  }
  b.tune = best;
  snprintf(line, sizeof line, "chosen: x split %d, x values in %s memory, y in %s, z in %s\n", best.x_split,
           best.x_keep ? "shared" : "global", best.y_keep ? "shared" : "global", best.z_keep ? "shared" : "global");
  report += line;
  return e;
}

}  // namespace hs2g

// ---------------------------------------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------------------------------------
struct hs2g_batch {
  hs2g::Batch b;
};

namespace {

using hs2g::Batch;

struct BatchDeviceGuard {
  int prev = -1;
  bool ok = false;
  explicit BatchDeviceGuard(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    ok = (prev == dev) || (cudaSetDevice(dev) == cudaSuccess);
  }
  ~BatchDeviceGuard() {
    int cur = -1;
    if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
  }
};

int bfail(int code, const char* msg) { return hs2g::set_last_error(code, msg); }
int bcuda(cudaError_t e, const char* what) {
  cudaGetLastError();  // a failed allocation leaves its error as the last error: clear it for later checks
  char buf[256];
  snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
  return hs2g::set_last_error(e == cudaErrorMemoryAllocation ? HS2G_ERR_NOMEM : HS2G_ERR_CUDA, buf);
}

template <typename T>
cudaError_t balloc(Batch& b, T** p, int64_t count) {
  const size_t bytes = sizeof(T) * (size_t)std::max<int64_t>(1, count);
  cudaError_t e = cudaMalloc((void**)p, bytes);
  if (e == cudaSuccess) b.bytes += (int64_t)bytes;
  else *p = nullptr;
  return e;
}

void batch_free(Batch& b) {
  if (b.graph) cudaGraphExecDestroy(b.graph);
  b.graph = nullptr;
  for (void* p : {(void*)b.inst_dev, b.T, b.W0, b.W1, (void*)b.vclass, b.qtabs, (void*)b.active,
                  (void*)b.step, (void*)b.xw, (void*)b.yw, (void*)b.zw})
    if (p) cudaFree(p);
  for (void* p : b.coef_mem) cudaFree(p);
  if (b.stream) cudaStreamDestroy(b.stream);
}

// Compile instance `ib` of problem p into the batch (FP64 workspace ws, then into the batch's storage type).
int compile_instance(Batch& b, int ib, const hs2g_class_problem& p, double* ws, bool search, unsigned long long* err) {
  hs2g::Inst& I = b.inst[ib];
  const hs2g::Dims& d = I.d;
  const int64_t n = d.nvox(), np = d.nz * d.ny * I.px;
  const int64_t nfz = (d.nz + 1) * d.nxy(), nfy = d.nz * (d.ny + 1) * d.nx, nfx = d.nz * d.ny * (d.nx + 1);
  cudaStream_t s = b.stream;
  // workspace layout (doubles): faces z, y, x | M s2 sigma | a0 b0 | a1 b1 a2 b2 | bytes:
  // compute mask, material, boundary classes | material table | boundary forms
  double* fz = ws;
  double* fy = fz + nfz;
  double* fx = fy + nfy;
  double* M = fx + nfx;
  double* s2 = M + n;
  double* sg = s2 + n;
  double* c2 = sg + n;
  double* c4 = c2 + 2 * np;
  uint8_t* u8 = reinterpret_cast<uint8_t*>(c4 + 4 * np);
  uint8_t* comp = u8;
  uint8_t* mat = comp + n;
  uint8_t* bz = mat + n;
  uint8_t* by = bz + nfz;
  uint8_t* bx = by + nfy;
  hs2g_material* mats = reinterpret_cast<hs2g_material*>((reinterpret_cast<uintptr_t>(bx + nfx) + 255) & ~uintptr_t(255));
  hs2g_face_form* forms = reinterpret_cast<hs2g_face_form*>(
      (reinterpret_cast<uintptr_t>(mats + HS2G_MAX_CLASSES) + 255) & ~uintptr_t(255));
  // then the faces' values per class and material pair, and the scratch of the search for equal lines and blocks
  unsigned char* table = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(forms + 3 * HS2G_MAX_CLASSES) + 255) & ~uintptr_t(255));
  unsigned char* scratch = search ? table + ((hs2g::face_table_bytes(p.nmat, p.nbnd) + 255) & ~size_t(255)) : nullptr;
  cudaError_t e = cudaSuccess;
  auto up = [&](void* dst, const void* src, size_t bytes) {
    if (e == cudaSuccess) e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
  };
  up(mat, p.material, (size_t)n);
  up(bz, p.boundary_z, (size_t)nfz);
  up(by, p.boundary_y, (size_t)nfy);
  up(bx, p.boundary_x, (size_t)nfx);
  up(mats, p.materials, sizeof(hs2g_material) * p.nmat);
  up(forms, p.forms, sizeof(hs2g_face_form) * p.nbnd * 3);
  if (p.volumetric) up(b.vclass + I.off, p.volumetric, (size_t)n);
  else if (e == cudaSuccess) e = cudaMemsetAsync(b.vclass + I.off, 0, (size_t)n, s);
  const uint8_t* bclass[3] = {bz, by, bx};
  double* G[3] = {fz, fy, fx};
  if (e == cudaSuccess) e = hs2g::launch_faces(d, mat, bclass, mats, p.nmat, forms, p.nbnd, G, err, table, s);
  if (e == cudaSuccess) e = hs2g::launch_capacity_from_classes(d, mat, mats, p.nmat, M, comp, err, s);
  if (e != cudaSuccess) return bcuda(e, "batch compile");
  unsigned long long v = 0;
  if ((e = cudaMemcpyAsync(&v, err, sizeof v, cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
      (e = cudaStreamSynchronize(s)) != cudaSuccess)
    return bcuda(e, "batch compile");
  if (v) {
    char buf[160];
    const int code = -(int)(v >> 56);
    snprintf(buf, sizeof buf, "instance %d: invalid problem (error %d at axis %d index %llu)", ib, code,
             (int)((v >> 54) & 3), (unsigned long long)(v & ((1ull << 54) - 1)));
    return bfail(code, buf);
  }
  hs2g::Coeffs c{};
  c.nchunks = I.nchunks;
  c.px = I.px;
  const bool f64 = b.precision == 64;
  c.a0 = c2;
  c.b0 = c2 + np;
  c.a1 = c4;
  c.b1 = c4 + np;
  c.a2 = c4 + 2 * np;
  c.b2 = c4 + 3 * np;
  const hs2g::Faces faces{fz, fy, fx, {}};
  if ((e = hs2g::launch_factor(d, faces, M, comp, s2, sg, c, s, f64)) != cudaSuccess) return bcuda(e, "batch factor");
  hs2g::Compressed kept;
  if ((e = hs2g::compress_coeffs(d, faces, comp, s2, c, b.precision, scratch, &kept, s)) != cudaSuccess)
    return bcuda(e, "batch factor");
  for (void* m : {kept.mem, kept.own})
    if (m) b.coef_mem.push_back(m);
  I.pool = kept.blocks.pool;
  I.bidx = kept.blocks.bidx;
  if (!I.bidx) b.dense_blocks = true;
  b.bytes += (int64_t)kept.blocks.bytes;
  const double* coeffs[3][2] = {{c.a0, c.b0}, {c.a1, c.b1}, {c.a2, c.b2}};
  // in one allocation: float tables beside the classes, and the arrays where the lines have too many classes (whole
  // 256 bytes each)
  int64_t count[3] = {}, total = 0;
  for (int ax = 0; ax < 3; ++ax) {
    const hs2g::LineTables& t = kept.lines[ax];
    I.cls[ax] = t.cls;
    if (t.cls) b.bytes += (int64_t)t.bytes;
    else b.dense[ax] = true;
    if (t.cls && f64) {  // the tables as they are
      I.a[ax] = t.a;
      I.b[ax] = t.b;
    } else {
      count[ax] = t.cls ? t.nclass * (ax == 0 ? d.nx : ax == 1 ? d.ny : d.nz) : np;
      total += 2 * ((count[ax] + 63) & ~int64_t(63));
    }
  }
  if (total) {
    unsigned char* m = nullptr;
    if ((e = cudaMalloc(&m, b.elem() * total)) != cudaSuccess) return bcuda(e, "batch factor");
    b.coef_mem.push_back(m);
    b.bytes += (int64_t)b.elem() * total;
    for (int ax = 0; ax < 3; ++ax) {
      const hs2g::LineTables& t = kept.lines[ax];
      const void** dst[2] = {&I.a[ax], &I.b[ax]};
      for (int q = 0; q < 2 && count[ax] && e == cudaSuccess; ++q) {
        *dst[q] = m;
        e = hs2g::batch_convert(t.cls ? (q ? t.b : t.a) : coeffs[ax][q], m, count[ax], b.precision, s);
        m += b.elem() * ((count[ax] + 63) & ~int64_t(63));
      }
    }
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  return e == cudaSuccess ? HS2G_OK : bcuda(e, "batch factor");
}

int capture(Batch& b) {
  if (b.graph) {
    cudaGraphExecDestroy(b.graph);
    b.graph = nullptr;
  }
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamBeginCapture(b.stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return bcuda(e, "graph capture");
  cudaError_t le = hs2g::batch_step(b, b.stream);
  e = cudaStreamEndCapture(b.stream, &g);
  if (le != cudaSuccess) return bcuda(le, "graph capture: launch");
  if (e != cudaSuccess) return bcuda(e, "graph capture");
  e = cudaGraphInstantiate(&b.graph, g, 0);
  cudaGraphDestroy(g);
  return e == cudaSuccess ? HS2G_OK : bcuda(e, "graph instantiate");
}

}  // namespace

extern "C" {

int hs2g_batch_create(int n, const hs2g_class_problem* problems, int precision, int device, hs2g_batch** out) {
  if (!out || !problems || n < 1 || n > (1 << 20) || (precision != 64 && precision != 32))
    return bfail(HS2G_ERR_ARG, "hs2g_batch_create: bad argument");
  *out = nullptr;
  for (int i = 0; i < n; ++i) {
    const hs2g_class_problem& p = problems[i];
    if (p.nz < 1 || p.ny < 1 || p.nx < 1 || !p.materials || !p.forms || !p.material || !p.boundary_z ||
        !p.boundary_y || !p.boundary_x || p.nmat < 1 || p.nmat > HS2G_MAX_CLASSES || p.nbnd < 1 ||
        p.nbnd > HS2G_MAX_CLASSES)
      return bfail(HS2G_ERR_ARG, "hs2g_batch_create: bad problem");
  }
  BatchDeviceGuard g(device);
  if (!g.ok) return bfail(HS2G_ERR_CUDA, "hs2g_batch_create: cannot select device");
  hs2g_batch* hb = new hs2g_batch();
  Batch& b = hb->b;
  b.device = device;
  b.precision = precision;
  b.ninst = n;
  auto bail = [&](int rc) {
    std::string msg = hs2g_last_error();
    batch_free(b);
    delete hb;
    hs2g::set_last_error(rc, msg.c_str());
    return rc;
  };
  cudaError_t e = cudaStreamCreateWithFlags(&b.stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    delete hb;
    return bcuda(e, "cudaStreamCreate");
  }
  int64_t off = 0, ws = 0, ws_least = 0;  // workspace with and without the scratch of the search
  b.offsets.push_back(0);
  for (int i = 0; i < n; ++i) {
    hs2g::Inst I{};
    I.d = hs2g::Dims{problems[i].nz, problems[i].ny, problems[i].nx};
    I.off = off;
    I.nchunks = (I.d.nx + 31) / 32;
    I.woff = b.nw;
    const int64_t quad = 16 / (int64_t)b.elem();
    I.px = (I.d.nx + quad - 1) / quad * quad;
    b.nw += I.d.nz * I.d.ny * I.px;
    b.inst.push_back(I);
    const hs2g::Dims& d = I.d;
    const int64_t nn = d.nvox();
    off += nn + (nn & 1);  // keep every instance 16-byte aligned
    b.offsets.push_back(off);
    const int64_t faces = (d.nz + 1) * d.nxy() + d.nz * (d.ny + 1) * d.nx + d.nz * d.ny * (d.nx + 1);
    const int64_t need = faces + 3 * nn + 6 * d.nz * d.ny * I.px + (faces + 3 * nn) / 8 + 2048 +
                         (int64_t)(sizeof(hs2g_material) * HS2G_MAX_CLASSES + sizeof(hs2g_face_form) * 3 *
                                   HS2G_MAX_CLASSES) / 8 + 512 +
                         (int64_t)hs2g::face_table_bytes(problems[i].nmat, problems[i].nbnd) / 8;
    ws_least = std::max(ws_least, need);
    ws = std::max(ws, need + (int64_t)hs2g::compress_scratch(d) / 8);
  }
  b.nvox = off;
  b.ix32 = true;
  for (const hs2g::Inst& I : b.inst)
    b.ix32 = b.ix32 && I.d.nz * I.d.ny * I.px < ((int64_t)1 << 31);
  const size_t el = b.elem();
  double* wsp = nullptr;
  unsigned long long* err = nullptr;
  bool search = true;
  auto workspace = [&]() {
    cudaError_t w = cudaMalloc(&wsp, sizeof(double) * ws);
    if (w == cudaErrorMemoryAllocation) {  // no room for the search: everything in voxel order
      cudaGetLastError();
      search = false;
      w = cudaMalloc(&wsp, sizeof(double) * ws_least);
    }
    return w;
  };
  if ((e = balloc(b, &b.inst_dev, n)) != cudaSuccess || (e = balloc(b, (char**)&b.T, b.nvox * el)) != cudaSuccess ||
      (e = balloc(b, (char**)&b.W0, b.nw * el)) != cudaSuccess ||
      (e = balloc(b, (char**)&b.W1, b.nw * el)) != cudaSuccess ||
      (e = balloc(b, &b.vclass, b.nvox)) != cudaSuccess || (e = balloc(b, &b.step, 1)) != cudaSuccess ||
      (e = workspace()) != cudaSuccess ||
      (e = cudaMalloc(&err, sizeof(unsigned long long))) != cudaSuccess) {
    if (wsp) cudaFree(wsp);
    if (err) cudaFree(err);
    hs2g::set_last_error(HS2G_ERR_NOMEM, "hs2g_batch_create: device allocation failed");
    return bail(HS2G_ERR_NOMEM);
  }
  cudaMemsetAsync(b.T, 0, b.nvox * el, b.stream);
  cudaMemsetAsync(b.W0, 0, b.nw * el, b.stream);
  cudaMemsetAsync(b.W1, 0, b.nw * el, b.stream);
  cudaMemsetAsync(b.vclass, 0, b.nvox, b.stream);
  cudaMemsetAsync(b.step, 0, sizeof(int), b.stream);
  const int64_t bytes = b.bytes;
  auto compile_all = [&]() {
    int rc = HS2G_OK;
    for (int i = 0; i < n && rc == HS2G_OK; ++i) {
      cudaMemsetAsync(err, 0, sizeof(unsigned long long), b.stream);
      rc = compile_instance(b, i, problems[i], wsp, search, err);
    }
    return rc;
  };
  int rc = compile_all();
  if (rc == HS2G_ERR_NOMEM && search) {  // the coefficients did not fit beside the scratch
    cudaStreamSynchronize(b.stream);
    for (void* m : b.coef_mem) cudaFree(m);
    b.coef_mem.clear();
    b.bytes = bytes;
    b.dense[0] = b.dense[1] = b.dense[2] = b.dense_blocks = false;
    cudaFree(wsp);
    wsp = nullptr;
    search = false;
    if (cudaMalloc(&wsp, sizeof(double) * ws_least) == cudaSuccess)
      rc = compile_all();
    else
      cudaGetLastError();
  }
  cudaFree(wsp);
  cudaFree(err);
  if (rc != HS2G_OK) return bail(rc);
  e = cudaMemcpyAsync(b.inst_dev, b.inst.data(), sizeof(hs2g::Inst) * n, cudaMemcpyHostToDevice, b.stream);
  if (e != cudaSuccess) return bail(bcuda(e, "instances"));
  if ((e = hs2g::batch_upload_work(b)) != cudaSuccess) return bail(bcuda(e, "work lists"));
  for (const hs2g::Inst& I : b.inst) {
    b.max_nx = std::max(b.max_nx, I.d.nx);
    b.max_ny = std::max(b.max_ny, I.d.ny);
    b.max_nz = std::max(b.max_nz, I.d.nz);
  }
  if (precision == 64) {
    e = hs2g::batch_prepare<double>();
    b.tune.x_keep = hs2g::batch_x_shape<double>(b, -1).keep;
    b.tune.y_keep = hs2g::batch_shape<double, false>(b, -1).keep;
    b.tune.z_keep = hs2g::batch_shape<double, true>(b, -1).keep;
  } else {
    e = hs2g::batch_prepare<float>();
    b.tune.x_keep = hs2g::batch_x_shape<float>(b, -1).keep;
    b.tune.y_keep = hs2g::batch_shape<float, false>(b, -1).keep;
    b.tune.z_keep = hs2g::batch_shape<float, true>(b, -1).keep;
  }
  if (e != cudaSuccess) return bail(bcuda(e, "configure sweep kernels"));
  if ((e = cudaStreamSynchronize(b.stream)) != cudaSuccess) return bail(bcuda(e, "batch create"));
  *out = hb;
  return HS2G_OK;
}

void hs2g_batch_destroy(hs2g_batch* hb) {
  if (!hb) return;
  BatchDeviceGuard g(hb->b.device);
  cudaStreamSynchronize(hb->b.stream);
  batch_free(hb->b);
  delete hb;
}

int hs2g_batch_layout(const hs2g_batch* hb, int64_t* offsets, int64_t* dims) {
  if (!hb) return bfail(HS2G_ERR_ARG, "null batch");
  const Batch& b = hb->b;
  for (int i = 0; i <= b.ninst && offsets; ++i) offsets[i] = b.offsets[i];
  for (int i = 0; i < b.ninst && dims; ++i) {
    dims[3 * i] = b.inst[i].d.nz;
    dims[3 * i + 1] = b.inst[i].d.ny;
    dims[3 * i + 2] = b.inst[i].d.nx;
  }
  return HS2G_OK;
}

int64_t hs2g_batch_device_bytes(const hs2g_batch* hb) { return hb ? hb->b.bytes : 0; }

int hs2g_batch_set_temperature(hs2g_batch* hb, const double* T, int flags) {
  if (!hb || !T) return bfail(HS2G_ERR_ARG, "null argument");
  Batch& b = hb->b;
  BatchDeviceGuard g(b.device);
  const bool dev = flags & HS2G_DEVICE;
  cudaError_t e = cudaSuccess;
  if (b.precision == 64) {
    e = cudaMemcpyAsync(b.T, T, sizeof(double) * b.nvox, dev ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                        b.stream);
  } else {
    const double* src = T;
    double* tmp = nullptr;
    if (!dev) {
      if ((e = cudaMallocAsync(&tmp, sizeof(double) * b.nvox, b.stream)) == cudaSuccess)
        e = cudaMemcpyAsync(tmp, T, sizeof(double) * b.nvox, cudaMemcpyHostToDevice, b.stream);
      src = tmp;
    }
    if (e == cudaSuccess) e = hs2g::batch_convert(src, b.T, b.nvox, 32, b.stream);
    if (tmp) cudaFreeAsync(tmp, b.stream);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(b.stream);
  return e == cudaSuccess ? HS2G_OK : bcuda(e, "set temperature");
}

int hs2g_batch_get_temperature(hs2g_batch* hb, double* T, int flags) {
  if (!hb || !T) return bfail(HS2G_ERR_ARG, "null argument");
  Batch& b = hb->b;
  BatchDeviceGuard g(b.device);
  const bool dev = flags & HS2G_DEVICE;
  cudaError_t e = cudaSuccess;
  if (b.precision == 64) {
    e = cudaMemcpyAsync(T, b.T, sizeof(double) * b.nvox, dev ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                        b.stream);
  } else {
    double* dst = T;
    double* tmp = nullptr;
    if (!dev) {
      e = cudaMallocAsync(&tmp, sizeof(double) * b.nvox, b.stream);
      dst = tmp;
    }
    if (e == cudaSuccess) e = hs2g::batch_widen(b.T, dst, b.nvox, 32, b.stream);
    if (e == cudaSuccess && tmp) e = cudaMemcpyAsync(T, tmp, sizeof(double) * b.nvox, cudaMemcpyDeviceToHost, b.stream);
    if (tmp) cudaFreeAsync(tmp, b.stream);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(b.stream);
  return e == cudaSuccess ? HS2G_OK : bcuda(e, "get temperature");
}

int hs2g_batch_set_sources(hs2g_batch* hb, int nsteps, int nclass, const double* qtabs) {
  if (!hb || nsteps < 0 || nclass < 1 || nclass > HS2G_MAX_CLASSES || (nsteps > 0 && !qtabs))
    return bfail(HS2G_ERR_ARG, "hs2g_batch_set_sources: bad argument");
  Batch& b = hb->b;
  BatchDeviceGuard g(b.device);
  cudaStreamSynchronize(b.stream);
  if (b.qtabs) cudaFree(b.qtabs);
  if (b.active) cudaFree(b.active);
  b.qtabs = nullptr;
  b.active = nullptr;
  const int64_t nq = (int64_t)nsteps * b.ninst * nclass;
  std::vector<uint8_t> act((size_t)std::max<int64_t>(1, (int64_t)nsteps * b.ninst), 0);
  for (int64_t s = 0; s < (int64_t)nsteps * b.ninst; ++s)
    for (int c = 0; c < nclass; ++c)
      if (qtabs[s * nclass + c] != 0.0) act[(size_t)s] = 1;
  cudaError_t e = cudaMalloc(&b.qtabs, b.elem() * (size_t)std::max<int64_t>(1, nq));
  if (e == cudaSuccess) e = cudaMalloc(&b.active, act.size());
  if (e == cudaSuccess) e = cudaMemcpy(b.active, act.data(), act.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess && nq > 0) {
    if (b.precision == 64) {
      e = cudaMemcpy(b.qtabs, qtabs, sizeof(double) * nq, cudaMemcpyHostToDevice);
    } else {
      std::vector<float> f((size_t)nq);
      for (int64_t i = 0; i < nq; ++i) f[(size_t)i] = (float)qtabs[i];
      e = cudaMemcpy(b.qtabs, f.data(), sizeof(float) * nq, cudaMemcpyHostToDevice);
    }
  }
  if (e == cudaSuccess) e = cudaMemset(b.step, 0, sizeof(int));
  b.nsched = nsteps;
  b.nclass = nclass;
  if (b.graph) {
    cudaGraphExecDestroy(b.graph);
    b.graph = nullptr;
  }
  return e == cudaSuccess ? HS2G_OK : bcuda(e, "set sources");
}

int hs2g_batch_set_clock(hs2g_batch* hb, int step) {
  if (!hb || step < 0) return bfail(HS2G_ERR_ARG, "bad argument");
  BatchDeviceGuard g(hb->b.device);
  cudaError_t e = cudaMemcpyAsync(hb->b.step, &step, sizeof(int), cudaMemcpyHostToDevice, hb->b.stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(hb->b.stream);
  return e == cudaSuccess ? HS2G_OK : bcuda(e, "set clock");
}

int hs2g_batch_run(hs2g_batch* hb, int nsteps, int flags, double* elapsed_ms) {
  if (!hb || nsteps < 0) return bfail(HS2G_ERR_ARG, "bad argument");
  Batch& b = hb->b;
  BatchDeviceGuard g(b.device);
  if (!b.qtabs) {
    int rc = hs2g_batch_set_sources(hb, 0, 1, nullptr);
    if (rc) return rc;
  }
  if (!b.graph) {
    int rc = capture(b);
    if (rc) return rc;
  }
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (elapsed_ms) {
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, b.stream);
  }
  cudaError_t e = cudaSuccess;
  for (int s = 0; s < nsteps && e == cudaSuccess; ++s) e = cudaGraphLaunch(b.graph, b.stream);
  if (elapsed_ms) cudaEventRecord(e1, b.stream);
  if (e == cudaSuccess && (elapsed_ms || (flags & HS2G_SYNC))) e = cudaStreamSynchronize(b.stream);
  if (elapsed_ms) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    *elapsed_ms = ms;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
  }
  return e == cudaSuccess ? HS2G_OK : bcuda(e, "batch run");
}

int hs2g_batch_autotune(hs2g_batch* hb, char* report, int report_len) {
  if (!hb) return bfail(HS2G_ERR_ARG, "null batch");
  Batch& b = hb->b;
  BatchDeviceGuard g(b.device);
  if (!b.qtabs) {
    int rc = hs2g_batch_set_sources(hb, 0, 1, nullptr);
    if (rc) return rc;
  }
  // the z sweep updates T in place: tune on a saved copy and restore it afterwards
  void* save = nullptr;
  const size_t bytes = b.elem() * (size_t)b.nvox;
  cudaError_t e = cudaMalloc(&save, bytes);
  if (e != cudaSuccess) return bcuda(e, "autotune");
  e = cudaMemcpyAsync(save, b.T, bytes, cudaMemcpyDeviceToDevice, b.stream);
  std::string rep;
  if (e == cudaSuccess) e = hs2g::batch_autotune(b, rep);
  cudaError_t e2 = cudaMemcpyAsync(b.T, save, bytes, cudaMemcpyDeviceToDevice, b.stream);
  cudaStreamSynchronize(b.stream);
  cudaFree(save);
  if (b.graph) {
    cudaGraphExecDestroy(b.graph);
    b.graph = nullptr;
  }
  if (report && report_len > 0) {
    strncpy(report, rep.c_str(), (size_t)report_len - 1);
    report[report_len - 1] = 0;
  }
  if (e != cudaSuccess) return bcuda(e, "autotune");
  return e2 == cudaSuccess ? HS2G_OK : bcuda(e2, "autotune restore");
}

}  // extern "C"
