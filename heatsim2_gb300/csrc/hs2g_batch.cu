// Batched timestep: many independent problems of uneven size advanced together.
//
// All instances live in one concatenated device state (instance b's fields start at voxel offset off[b], each
// (nz_b, ny_b, nx_b) C-ordered).  The three sweeps are persistent kernels that walk flattened work lists --
// x: (instance, 32 x-lines), y: (instance, 128 y-lines), z: (instance, 128 z-lines) -- ordered longest lines
// first so the static round-robin over the persistent grid balances uneven instances.  One timestep (three
// sweeps + a step-counter increment) is captured once in a CUDA graph and replayed; the per-step source
// tables are uploaded once and selected on the device by the step counter, so the graph never changes.
//
// The arithmetic per line is that of the single-problem kernels (hs2g_sweep.cu, scaled delta-form Douglas
// ADI), templated on the storage type: double (results equal to the single-problem path bit for bit) or float
// (coefficients compiled in double, rounded once; its error against double is measured by the caller).
// Block sizes and persistent grid sizes per axis are chosen by hs2g_batch_autotune (timed on the batch).
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "hs2g_internal.cuh"
#include "hs2g_pair.cuh"

namespace hs2g {
namespace {

struct Inst {
  Dims d;
  int64_t off;      // voxel offset in the concatenated fields
  int64_t xb_off;   // element offset of the instance's stencil blocks
  int64_t nchunks;  // 32-column chunks per x-line
  int64_t woff;     // offset of the instance in W0 and W1, whose rows have pitch px (nx rounded up to 16 bytes)
  int64_t px;
  // y and z coefficients (axis 0: y, 1: z): rows of pitch px like W0, or with cls tables per line class
  const void* a[2];
  const void* b[2];
  const int32_t* cls[2];
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
  const R* xb;
  const R* a0;
  const R* b0;
  const uint8_t* vclass;
  const R* qtabs;          // [nsched][ninst][nclass]
  const uint8_t* active;   // [nsched][ninst] any source active
  const int* step;         // device step counter
  int nsched, ninst, nclass;
  const XWork* xw;
  int64_t nx_work;
  const LWork* yw;
  int64_t ny_work;
  const LWork* zw;
  int64_t nz_work;
};

constexpr int kMaxBatchClasses = HS2G_MAX_CLASSES;

// IX: index type of the voxel, line and stencil-block arithmetic within an instance (int32_t when every
// instance and its stencil blocks have fewer than 2^31 elements)
template <typename R, bool HAS_Q, typename IX = int64_t>
__device__ __forceinline__ R batch_stencil(const Inst& I, const R* __restrict__ T, const R* __restrict__ xb,
                                           const uint8_t* __restrict__ vclass, const R* sq, IX L, int ch,
                                           int lane) {
  const Dims& d = I.d;
  const IX nx = (IX)d.nx, ny = (IX)d.ny, nz = (IX)d.nz;
  const IX i = (IX)ch * 32 + lane;
  const IX k = L / ny, j = L - k * ny;
  const IX p = L * nx + i;
  const IX nxy = nx * ny;
  const R* __restrict__ w = xb + I.xb_off + ((L * (IX)I.nchunks + ch) * kXBlockCoeffs) * 32 + lane;
  const R* Ti = T + I.off;
  const R t = Ti[p];
  const R txl = i > 0 ? Ti[p - 1] : t;
  const R txh = i + 1 < nx ? Ti[p + 1] : t;
  const R tyl = j > 0 ? Ti[p - nx] : t;
  const R tyh = j + 1 < ny ? Ti[p + nx] : t;
  const R tzl = k > 0 ? Ti[p - nxy] : t;
  const R tzh = k + 1 < nz ? Ti[p + nxy] : t;
  R r = w[kWc * 32] * t;
  r = fma(w[kWxl * 32], txl, r);
  r = fma(w[kWxh * 32], txh, r);
  r = fma(w[kWyl * 32], tyl, r);
  r = fma(w[kWyh * 32], tyh, r);
  r = fma(w[kWzl * 32], tzl, r);
  r = fma(w[kWzh * 32], tzh, r);
  if (HAS_Q) r = fma(w[kWq * 32], sq[vclass[I.off + p]], r);
  return r;
}

// One block of 32 x-lines of one instance (CTA of 128 threads), same structure as sweep_x_kernel.
template <typename R, bool HAS_Q, typename IX = int64_t>
__device__ void batch_x_block(const BatchView<R>& v, const Inst& I, int64_t L0_, const R* sq, R (*sr)[33],
                              R (*sa)[33]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Dims& d = I.d;
  const IX nx = (IX)d.nx, L0 = (IX)L0_;
  const IX nlines = (IX)(d.nz * d.ny);
  const int nchunks = (int)I.nchunks;
  R* W0 = v.W0 + I.woff;
  const IX px = (IX)I.px;
  const R* a0 = v.a0 + I.off;
  const R* b0 = v.b0 + I.off;
  R carry = 0;
  for (int ch = 0; ch < nchunks; ++ch) {
    const IX i = (IX)ch * 32 + lane;
#pragma unroll
    for (int ll = 0; ll < 8; ++ll) {
      const int l = warp * 8 + ll;
      const IX L = L0 + l;
      R r = 0, a = 0;
      if (L < nlines && i < nx) {
        r = batch_stencil<R, HAS_Q, IX>(I, v.T, v.xb, v.vclass, sq, L, ch, lane);
        a = a0[L * nx + i];
      }
      sr[l][lane] = r;
      sa[l][lane] = a;
    }
    __syncthreads();
    if (warp == 0) {
      const int cw = (int)min((int64_t)32, d.nx - (int64_t)ch * 32);
      R z = carry;
      if (cw == 32) {  // full chunks unrolled: the shared loads of later rows issue ahead of the chain
#pragma unroll 4
        for (int cc = 0; cc < 32; ++cc) {
          z = fma(-sa[lane][cc], z, sr[lane][cc]);
          sr[lane][cc] = z;
        }
      } else {
        for (int cc = 0; cc < cw; ++cc) {
          z = fma(-sa[lane][cc], z, sr[lane][cc]);
          sr[lane][cc] = z;
        }
      }
      carry = z;
    }
    __syncthreads();
#pragma unroll
    for (int ll = 0; ll < 8; ++ll) {
      const int l = warp * 8 + ll;
      const IX L = L0 + l;
      if (L < nlines && i < nx) W0[L * px + i] = sr[l][lane];
    }
    __syncthreads();
  }
  carry = 0;
  for (int ch = nchunks - 1; ch >= 0; --ch) {
    const IX i = (IX)ch * 32 + lane;
#pragma unroll
    for (int ll = 0; ll < 8; ++ll) {
      const int l = warp * 8 + ll;
      const IX L = L0 + l;
      R z = 0, b = 0;
      if (L < nlines && i < nx) {
        z = W0[L * px + i];
        b = b0[L * nx + i];
      }
      sr[l][lane] = z;
      sa[l][lane] = b;
    }
    __syncthreads();
    if (warp == 0) {
      const int cw = (int)min((int64_t)32, d.nx - (int64_t)ch * 32);
      R x = carry;
      if (cw == 32) {
#pragma unroll 4
        for (int cc = 31; cc >= 0; --cc) {
          x = fma(-sa[lane][cc], x, sr[lane][cc]);
          sr[lane][cc] = x;
        }
      } else {
        for (int cc = cw - 1; cc >= 0; --cc) {
          x = fma(-sa[lane][cc], x, sr[lane][cc]);
          sr[lane][cc] = x;
        }
      }
      carry = x;
    }
    __syncthreads();
#pragma unroll
    for (int ll = 0; ll < 8; ++ll) {
      const int l = warp * 8 + ll;
      const IX L = L0 + l;
      if (L < nlines && i < nx) W0[L * px + i] = sr[l][lane];
    }
    __syncthreads();
  }
}

// 72 registers (7 CTAs of 128 threads per SM): more loads in flight per thread than at 64 registers, which
// left the kernel load-latency bound (2.25e10 against 2.47e10 voxel-steps/s on the 256-instance batch).
// IX = int32_t (every batch whose instances have fewer than 2^31 voxels and stencil-block elements): 32-bit
// line, voxel and block arithmetic within an instance, 9.55 against 10.65 ms per FP64 step of that batch (the
// same for the y and z sweeps changed nothing there).
template <typename R, typename IX = int64_t>
__global__ void __launch_bounds__(128, 7) batch_x_kernel(BatchView<R> v) {
  __shared__ R sr[32][33];
  __shared__ R sa[32][33];
  __shared__ R sq[kMaxBatchClasses];
  const int step = *v.step;
  const bool sched = step < v.nsched;
  for (int64_t w = blockIdx.x; w < v.nx_work; w += gridDim.x) {
    const XWork item = v.xw[w];
    const Inst I = v.inst[item.inst];
    const bool has_q = sched && v.active[(int64_t)step * v.ninst + item.inst];
    if (has_q) {
      const R* q = v.qtabs + ((int64_t)step * v.ninst + item.inst) * v.nclass;
      for (int c = threadIdx.x; c < kMaxBatchClasses; c += blockDim.x) sq[c] = c < v.nclass ? q[c] : R(0);
      __syncthreads();
      batch_x_block<R, true, IX>(v, I, item.L0, sq, sr, sa);
    } else {
      batch_x_block<R, false, IX>(v, I, item.L0, sq, sr, sa);
    }
  }
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
  const int32_t* cls = I.cls[ADD_T];
  PairLines<R> p;
  p.W = (ADD_T ? v.W1 : v.W0) + I.woff + w;
  p.wst = p.cst = p.zst = wst;
  p.a = (const R*)I.a[ADD_T] + (cls ? 0 : w);
  p.b = (const R*)I.b[ADD_T] + (cls ? 0 : w);
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
  int x_grid;
  bool y_keep, z_keep;  // the forward values of the y / z lines stay in shared memory
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
  int64_t nvox = 0, xb_len = 0;
  Inst* inst_dev = nullptr;
  void* T = nullptr;  // R*
  void* W0 = nullptr;
  void* W1 = nullptr;
  void* coef = nullptr;  // a0 and b0, nvox R each
  std::vector<void*> line_mem;  // the instances' y and z coefficients
  int64_t nw = 0;               // elements of W0 and W1
  void* xb = nullptr;
  uint8_t* vclass = nullptr;
  void* qtabs = nullptr;
  uint8_t* active = nullptr;
  int nsched = 0, nclass = 1;
  int* step = nullptr;
  XWork* xw = nullptr;
  LWork* yw = nullptr;
  LWork* zw = nullptr;
  int64_t nxw = 0, nyw = 0, nzw = 0;
  Tuning tune{0, true, true};
  int64_t max_ny = 0, max_nz = 0;  // longest y and z line
  bool dense[2] = {false, false};  // some instance keeps its y / z coefficients in voxel order
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
  R* c = (R*)b.coef;
  v.a0 = c;
  v.b0 = c + b.nvox;
  v.xb = (const R*)b.xb;
  v.vclass = b.vclass;
  v.qtabs = (const R*)b.qtabs;
  v.active = b.active;
  v.step = b.step;
  v.nsched = b.nsched;
  v.ninst = b.ninst;
  v.nclass = b.nclass;
  v.xw = b.xw;
  v.nx_work = b.nxw;
  v.yw = b.yw;
  v.ny_work = b.nyw;
  v.zw = b.zw;
  v.nz_work = b.nzw;
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
  PairShape sh = b.dense[ADD_T] ? pair_shape<R, TWO, ADD_T, false>(len, groups, force_keep)
                                : pair_shape<R, TWO, ADD_T, true>(len, groups, force_keep);
  size_t each = b.dense[ADD_T] ? pair_smem<R, TWO, ADD_T, true, false>(len) : pair_smem<R, TWO, ADD_T, true, true>(len);
  if (each * kPairMaxWarps > 226 * 1024) sh.keep = false;
  if (!sh.keep) each = b.dense[ADD_T] ? pair_smem<R, TWO, ADD_T, false, false>(len) : pair_smem<R, TWO, ADD_T, false, true>(len);
  sh.warps = kPairMaxWarps;
  sh.smem = each * kPairMaxWarps;
  return sh;
}
template <typename R, bool ADD_T>
cudaError_t launch_batch_pair(const Batch& b, const BatchView<R>& v, bool keep, cudaStream_t s) {
  const PairShape sh = batch_shape<R, ADD_T>(b, keep ? 1 : 0);
  const int64_t work = ADD_T ? b.nzw : b.nyw;
  batch_pair_for<R, ADD_T>(sh.keep, b.dense[ADD_T])<<<(unsigned)work, 32 * kPairMaxWarps, sh.smem, s>>>(
      v, (int64_t)(sh.smem / kPairMaxWarps));
  return cudaGetLastError();
}
template <typename R>
cudaError_t batch_prepare() {
  cudaError_t e = cudaSuccess;
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
    if (b.ix32)
      batch_x_kernel<R, int32_t><<<(unsigned)std::max(1, t.x_grid), 128, 0, s>>>(v);
    else
      batch_x_kernel<R><<<(unsigned)std::max(1, t.x_grid), 128, 0, s>>>(v);
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

// Work lists: blocks of 32 x-lines, and of the line solves' y and z lines, per instance, longest lines first.
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
    for (int64_t L0 = 0; L0 < d.nz * d.ny; L0 += 32) xw.push_back(XWork{ib, 0, L0});
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
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b.device);
  Tuning best = b.tune;
  char line[256];
  cudaError_t e = cudaSuccess;
  // x: persistent grid size (CTAs of 128 threads)
  {
    float bt = 1e30f;
    // per = 0: one CTA per work item, the hardware's block scheduler doing the balancing
    for (int per : {4, 5, 6, 7, 8, 10, 0}) {
      Tuning t = best;
      t.x_grid = (int)std::min<int64_t>(std::min<int64_t>(b.nxw, 1 << 30), per ? (int64_t)sms * per : b.nxw);
      float ms;
      if ((e = batch_time_axis(b, 0, t, 2, &ms)) != cudaSuccess) return e;
      snprintf(line, sizeof line, "x grid %d: %.3f ms\n", t.x_grid, ms);
      report += line;
      if (ms < bt) bt = ms, best.x_grid = t.x_grid;
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
  snprintf(line, sizeof line, "chosen: x grid %d, y values in %s memory, z values in %s memory\n", best.x_grid,
           best.y_keep ? "shared" : "global", best.z_keep ? "shared" : "global");
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
  for (void* p : {(void*)b.inst_dev, b.T, b.W0, b.W1, b.coef, b.xb, (void*)b.vclass, b.qtabs, (void*)b.active,
                  (void*)b.step, (void*)b.xw, (void*)b.yw, (void*)b.zw})
    if (p) cudaFree(p);
  for (void* p : b.line_mem) cudaFree(p);
  if (b.stream) cudaStreamDestroy(b.stream);
}

int64_t xb_elems(const hs2g::Dims& d) { return d.nz * d.ny * ((d.nx + 31) / 32) * hs2g::kXBlockCoeffs * 32; }

// Compile instance `ib` of problem p into the batch (FP64 workspace ws, then into the batch's storage type).
int compile_instance(Batch& b, int ib, const hs2g_class_problem& p, double* ws, unsigned long long* err) {
  hs2g::Inst& I = b.inst[ib];
  const hs2g::Dims& d = I.d;
  const int64_t n = d.nvox(), np = d.nz * d.ny * I.px;
  const int64_t nfz = (d.nz + 1) * d.nxy(), nfy = d.nz * (d.ny + 1) * d.nx, nfx = d.nz * d.ny * (d.nx + 1);
  cudaStream_t s = b.stream;
  // workspace layout (doubles): faces z, y, x | M s2 sigma | a0 b0 | a1 b1 a2 b2 | x blocks | bytes:
  // compute mask, material, boundary classes | material table | boundary forms
  double* fz = ws;
  double* fy = fz + nfz;
  double* fx = fy + nfy;
  double* M = fx + nfx;
  double* s2 = M + n;
  double* sg = s2 + n;
  double* c2 = sg + n;
  double* c4 = c2 + 2 * n;
  double* xbw = c4 + 4 * np;
  uint8_t* u8 = reinterpret_cast<uint8_t*>(xbw + xb_elems(d));
  uint8_t* comp = u8;
  uint8_t* mat = comp + n;
  uint8_t* bz = mat + n;
  uint8_t* by = bz + nfz;
  uint8_t* bx = by + nfy;
  hs2g_material* mats = reinterpret_cast<hs2g_material*>((reinterpret_cast<uintptr_t>(bx + nfx) + 255) & ~uintptr_t(255));
  hs2g_face_form* forms = reinterpret_cast<hs2g_face_form*>(
      (reinterpret_cast<uintptr_t>(mats + HS2G_MAX_CLASSES) + 255) & ~uintptr_t(255));
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
  if (e == cudaSuccess) e = hs2g::launch_faces(d, 0, mat, bz, mats, p.nmat, forms, p.nbnd, fz, err, s);
  if (e == cudaSuccess) e = hs2g::launch_faces(d, 1, mat, by, mats, p.nmat, forms, p.nbnd, fy, err, s);
  if (e == cudaSuccess) e = hs2g::launch_faces(d, 2, mat, bx, mats, p.nmat, forms, p.nbnd, fx, err, s);
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
  c.a0 = f64 ? (double*)b.coef + I.off : c2;
  c.b0 = f64 ? (double*)b.coef + b.nvox + I.off : c2 + n;
  c.a1 = c4;
  c.b1 = c4 + np;
  c.a2 = c4 + 2 * np;
  c.b2 = c4 + 3 * np;
  c.xb = f64 ? (double*)b.xb + I.xb_off : xbw;
  if (!f64 && (e = cudaMemsetAsync(xbw, 0, sizeof(double) * xb_elems(d), s)) != cudaSuccess)
    return bcuda(e, "batch compile");
  if ((e = hs2g::launch_factor(d, fz, fy, fx, M, comp, s2, sg, c, s, f64)) != cudaSuccess)
    return bcuda(e, "batch factor");
  if (!f64) {
    for (int a = 0; a < 2 && e == cudaSuccess; ++a)
      e = hs2g::batch_convert(c2 + a * n, (float*)b.coef + a * b.nvox + I.off, n, 32, s);
    if (e == cudaSuccess) e = hs2g::batch_convert(xbw, (float*)b.xb + I.xb_off, xb_elems(d), 32, s);
  }
  // the y and z coefficients: tables per line class, or the arrays where the lines have too many classes
  for (int ax = 0; ax < 2 && e == cudaSuccess; ++ax) {
    const double *a = ax ? c.a2 : c.a1, *bb = ax ? c.b2 : c.b1;
    hs2g::LineTables t;
    e = ax ? hs2g::classify_lines(a, bb, d.ny, d.nx, I.px, d.nz, d.ny * I.px, &t, s)
           : hs2g::classify_lines(a, bb, d.nz, d.nx, d.ny * I.px, d.ny, I.px, &t, s);
    if (e != cudaSuccess) break;
    const int64_t count = t.cls ? t.nclass * (ax ? d.nz : d.ny) : np;
    if (t.cls) {
      b.line_mem.push_back(t.cls);
      b.bytes += (int64_t)sizeof(int32_t) * (ax ? d.ny : d.nz) * d.nx;
      a = t.a;
      bb = t.b;
    } else {
      b.dense[ax] = true;
    }
    I.cls[ax] = t.cls;
    const void** dst[2] = {&I.a[ax], &I.b[ax]};
    const double* src[2] = {a, bb};
    for (int q = 0; q < 2; ++q) {
      if (t.cls && f64) {  // the tables as they are
        b.line_mem.push_back((void*)src[q]);
        *dst[q] = src[q];
      } else {
        void* m = nullptr;
        if (e == cudaSuccess) e = cudaMalloc(&m, b.elem() * count);
        if (e == cudaSuccess) {
          b.line_mem.push_back(m);
          *dst[q] = m;
          e = hs2g::batch_convert(src[q], m, count, b.precision, s);
        }
      }
      b.bytes += (int64_t)b.elem() * count;
    }
    if (t.cls && !f64) {
      cudaStreamSynchronize(s);
      cudaFree(t.a);
      cudaFree(t.b);
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
  int64_t off = 0, xoff = 0, ws = 0;
  b.offsets.push_back(0);
  for (int i = 0; i < n; ++i) {
    hs2g::Inst I{};
    I.d = hs2g::Dims{problems[i].nz, problems[i].ny, problems[i].nx};
    I.off = off;
    I.xb_off = xoff;
    I.nchunks = (I.d.nx + 31) / 32;
    I.woff = b.nw;
    const int64_t quad = 16 / (int64_t)b.elem();
    I.px = (I.d.nx + quad - 1) / quad * quad;
    b.nw += I.d.nz * I.d.ny * I.px;
    b.inst.push_back(I);
    const hs2g::Dims& d = I.d;
    const int64_t nn = d.nvox();
    off += nn + (nn & 1);  // keep every instance 16-byte aligned
    xoff += xb_elems(d);
    b.offsets.push_back(off);
    const int64_t faces = (d.nz + 1) * d.nxy() + d.nz * (d.ny + 1) * d.nx + d.nz * d.ny * (d.nx + 1);
    const int64_t need = faces + 5 * nn + 4 * d.nz * d.ny * I.px + xb_elems(d) + (faces + 3 * nn) / 8 + 2048 +
                         (int64_t)(sizeof(hs2g_material) * HS2G_MAX_CLASSES + sizeof(hs2g_face_form) * 3 *
                                   HS2G_MAX_CLASSES) / 8 + 256;
    ws = std::max(ws, need);
  }
  b.nvox = off;
  b.xb_len = xoff;
  b.ix32 = true;
  for (const hs2g::Inst& I : b.inst)
    b.ix32 = b.ix32 && I.d.nz * I.d.ny * I.px < ((int64_t)1 << 31) && xb_elems(I.d) < ((int64_t)1 << 31);
  const size_t el = b.elem();
  double* wsp = nullptr;
  unsigned long long* err = nullptr;
  if ((e = balloc(b, &b.inst_dev, n)) != cudaSuccess || (e = balloc(b, (char**)&b.T, b.nvox * el)) != cudaSuccess ||
      (e = balloc(b, (char**)&b.W0, b.nw * el)) != cudaSuccess ||
      (e = balloc(b, (char**)&b.W1, b.nw * el)) != cudaSuccess ||
      (e = balloc(b, (char**)&b.coef, 2 * b.nvox * el)) != cudaSuccess ||
      (e = balloc(b, (char**)&b.xb, b.xb_len * el)) != cudaSuccess ||
      (e = balloc(b, &b.vclass, b.nvox)) != cudaSuccess || (e = balloc(b, &b.step, 1)) != cudaSuccess ||
      (e = cudaMalloc(&wsp, sizeof(double) * ws)) != cudaSuccess ||
      (e = cudaMalloc(&err, sizeof(unsigned long long))) != cudaSuccess) {
    if (wsp) cudaFree(wsp);
    if (err) cudaFree(err);
    hs2g::set_last_error(HS2G_ERR_NOMEM, "hs2g_batch_create: device allocation failed");
    return bail(HS2G_ERR_NOMEM);
  }
  cudaMemsetAsync(b.xb, 0, b.xb_len * el, b.stream);
  cudaMemsetAsync(b.T, 0, b.nvox * el, b.stream);
  cudaMemsetAsync(b.W0, 0, b.nw * el, b.stream);
  cudaMemsetAsync(b.W1, 0, b.nw * el, b.stream);
  cudaMemsetAsync(b.coef, 0, 2 * b.nvox * el, b.stream);
  cudaMemsetAsync(b.vclass, 0, b.nvox, b.stream);
  cudaMemsetAsync(b.step, 0, sizeof(int), b.stream);
  int rc = HS2G_OK;
  for (int i = 0; i < n && rc == HS2G_OK; ++i) {
    cudaMemsetAsync(err, 0, sizeof(unsigned long long), b.stream);
    rc = compile_instance(b, i, problems[i], wsp, err);
  }
  cudaFree(wsp);
  cudaFree(err);
  if (rc != HS2G_OK) return bail(rc);
  e = cudaMemcpyAsync(b.inst_dev, b.inst.data(), sizeof(hs2g::Inst) * n, cudaMemcpyHostToDevice, b.stream);
  if (e != cudaSuccess) return bail(bcuda(e, "instances"));
  if ((e = hs2g::batch_upload_work(b)) != cudaSuccess) return bail(bcuda(e, "work lists"));
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  b.tune.x_grid = (int)std::min<int64_t>(b.nxw, (int64_t)sms * 7);  // the x kernel's 7 resident CTAs per SM
  for (const hs2g::Inst& I : b.inst) {
    b.max_ny = std::max(b.max_ny, I.d.ny);
    b.max_nz = std::max(b.max_nz, I.d.nz);
  }
  if (precision == 64) {
    e = hs2g::batch_prepare<double>();
    b.tune.y_keep = hs2g::batch_shape<double, false>(b, -1).keep;
    b.tune.z_keep = hs2g::batch_shape<double, true>(b, -1).keep;
  } else {
    e = hs2g::batch_prepare<float>();
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
