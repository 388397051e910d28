// Adjoint of the ADI timestep: gradients of a top-surface misfit with respect to per-voxel conductivity k,
// volumetric heat capacity C = rho*c and source amplitude q, for one problem or a batch of independent
// problems of uneven size advanced together (no counterpart in the reference, which has no derivatives).
//
// Model per instance (every voxel computed, exterior faces insulating, interior faces conducting with the
// arithmetic face mean of boundary_conducting, G_f = (k_lo + k_hi) / (2 d^2)), M = C/dt, source s_n * q at
// step n.  The step is the Douglas delta form of the forward path (hs2g_sweep.cu):
//     r0 = L T + s_n q,  A_x y0 = r0,  A_y y1 = M y0,  A_z y2 = M y1,  T' = T + y2,   A_a = M - L_a / 2.
// Loss per instance J = sum_n sum_{top layer k=0} (T_{n+1} - d_n)^2.
// Discrete adjoint of one step, lambda the adjoint of T' (including the misfit gradient at T'):
//     mu2 = A_z^-T lambda,  mu1 = A_y^-T (M mu2),  mu0 = A_x^-T (M mu1),  lambda_T = lambda + L mu0
//     dJ/dG_f (face q|p on axis a, q the lower voxel) += -(mu0_p - mu0_q)(T_p - T_q)
//                                                       - (mu_a,p - mu_a,q)(y_a,p - y_a,q) / 2
//     dJ/dM_p += mu2 y1 + mu1 y0 - mu0 y0 - mu1 y1 - mu2 y2,     dJ/dq_p += s_n mu0_p
// with (mu_a, y_a) = (mu0, y0), (mu1, y1), (mu2, y2) for a = x, y, z (L is symmetric).  A_a = M - L_a/2 is
// symmetric too, so A_a^-T = A_a^-1: the adjoint's line solves are the forward ones, with the same factors.
//
// Memory: T is checkpointed every `ckpt` steps in the forward pass (ceil(nsteps/ckpt) states); the backward
// pass recomputes a segment from its checkpoint, keeping T_n, y0, y1, y2 of each of its steps (4*ckpt states,
// allocated by the first backward pass), then sweeps the segment backwards.
// Concatenated layout: instance i occupies voxels [off_i, off_i + nz*ny*px) of every field, x rows of an odd nx padded
// by one column, so that every copy of the line solves moves 16 bytes, and instances starting on 32-byte sectors (the
// caller's arrays have no pad; they are packed and unpacked on the way).  Pad voxels hold zero temperatures, conductances and increments.  Each
// kernel covers all instances in one launch (lines or voxels of the whole batch, the instance found by binary search).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "hs2g_internal.cuh"
#include "hs2g_few.cuh"
#include "hs2g_pair.cuh"
#include "hs2g_x.cuh"

namespace hs2g {
namespace {

constexpr int kTh = 128;

struct AInst {
  int64_t off;              // first voxel
  int64_t nz, ny, nx;
  int64_t px;               // pitch of the x rows
  int64_t ext;              // first voxel in the caller's arrays
  double idx2, idy2, idz2;  // 1/d^2 per axis
  int64_t obs_off;          // first observation of the instance (nsteps * ny * nx each)
};

struct AView {
  const AInst* inst;
  const int64_t* vox_off;   // ninst + 1 voxel prefix
  const int64_t* line_off;  // 3 * (ninst + 1) line prefixes, axis-major (x, y, z)
  const int64_t* grp_off;   // the same of groups of 16 lines, one warp's in the line solves
  int ninst;
  int64_t nvox;
};

inline unsigned nblk(int64_t n) { return (unsigned)std::max<int64_t>(1, (n + kTh - 1) / kTh); }

// index of the last prefix entry <= v (prefix[0] = 0; instances are non-empty so the prefix increases)
__device__ __forceinline__ int find_inst(const int64_t* prefix, int n, int64_t v) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(prefix + mid) <= v) lo = mid; else hi = mid - 1;
  }
  return lo;
}

struct Line {
  int64_t base, stride, len;
};

// global line t of axis (0 = x, 1 = y, 2 = z) -> first voxel, stride, length
__device__ __forceinline__ Line line_at(const AView& v, int axis, int64_t t) {
  const int64_t* pre = v.line_off + axis * (v.ninst + 1);
  const int i = find_inst(pre, v.ninst, t);
  const AInst& in = v.inst[i];
  const int64_t l = t - pre[i], nxy = in.ny * in.px;
  if (axis == 0) return Line{in.off + l * in.px, 1, in.nx};
  if (axis == 1) return Line{in.off + (l / in.px) * nxy + l % in.px, in.px, in.ny};
  return Line{in.off + l, nxy, in.nz};
}

struct Vox {
  int i, j, k, nx, ny, nz, px, nxy;  // nxy: voxels from one layer to the next
  int inst;
  bool in;  // false: a pad of its row, or between two instances
};
// voxel p -> instance and (k, j, i); 32-bit divisions (hs2g_adjoint_create refuses batches of 2^31 voxels)
__device__ __forceinline__ Vox vox_at(const AView& v, int64_t p) {
  const int n = find_inst(v.vox_off, v.ninst, p);
  const AInst& in = v.inst[n];
  const uint32_t l = (uint32_t)(p - in.off), px = (uint32_t)in.px, ny = (uint32_t)in.ny;
  const uint32_t row = l / px, k = row / ny;
  Vox r;
  r.inst = n;
  r.nx = (int)in.nx; r.ny = (int)in.ny; r.nz = (int)in.nz; r.px = (int)in.px; r.nxy = (int)(in.px * in.ny);
  r.i = l - row * px; r.j = row - k * ny; r.k = k;
  r.in = r.i < r.nx && r.k < r.nz;
  return r;
}

// a field between the caller's arrays and the padded ones (the pads zero)
template <typename E>
__global__ void adj_pack_kernel(AView v, const E* __restrict__ src, E* __restrict__ dst) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= v.nvox) return;
  const Vox x = vox_at(v, p);
  dst[p] = x.in ? src[v.inst[x.inst].ext + (x.k * x.ny + x.j) * x.nx + x.i] : E(0);
}
__global__ void adj_unpack_kernel(AView v, const double* __restrict__ src, double* __restrict__ dst) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= v.nvox) return;
  const Vox x = vox_at(v, p);
  if (x.in) dst[v.inst[x.inst].ext + (x.k * x.ny + x.j) * x.nx + x.i] = src[p];
}

// per-voxel low-face conductances of each axis from k (zero on the exterior), M = C / dt
__global__ void adj_setup_kernel(AView v, const double* __restrict__ k, const double* __restrict__ C, double inv_dt,
                                 double* __restrict__ gx, double* __restrict__ gy, double* __restrict__ gz,
                                 double* __restrict__ M) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= v.nvox) return;
  const Vox x = vox_at(v, p);
  if (!x.in) {
    gx[p] = gy[p] = gz[p] = 0.0;
    M[p] = 1.0;
    return;
  }
  const AInst& in = v.inst[x.inst];
  const double kp = k[p];
  gx[p] = x.i > 0 ? 0.5 * (k[p - 1] + kp) * in.idx2 : 0.0;
  gy[p] = x.j > 0 ? 0.5 * (k[p - x.px] + kp) * in.idy2 : 0.0;
  gz[p] = x.k > 0 ? 0.5 * (k[p - x.nxy] + kp) * in.idz2 : 0.0;
  M[p] = C[p] * inv_dt;
}

// A fixed-temperature voxel gets this capacity: its row of every stage matrix is then M times the identity to
// within 1e-290, its increments vanish against T, and the stage matrices stay symmetric (the reference's
// identity rows with couplings from computed neighbours are not), so the adjoint's transposed solves remain
// the forward solves.
constexpr double kFixedCapacity = 1e300;

// Whether s v is more than a zero: without the FP64 unit, whose instructions are what the voxel kernels wait for.  (A
// product with zero is NaN when v is infinite or NaN.)
__device__ __forceinline__ bool adds_something(double s, double v) {
  return ((uint64_t)__double_as_longlong(s) << 1) != 0 ||
         ((uint64_t)__double_as_longlong(v) << 1) >= (uint64_t(0x7ff) << 53);
}
// false, unknown to the compiler: `while (again) { ...; again = never(); }` is a branch that stays one, where the FP64
// instructions of an `if` would be issued with a predicate, whether or not it holds
__device__ __forceinline__ bool never() {
  unsigned zero;
  asm volatile("mov.u32 %0, 0;" : "=r"(zero));
  return zero != 0;
}

// The same with face classes and fixed voxels: the conductance of a face of class c on axis a is the class's
// affine form f0 + flo k_lo + fhi k_hi, the k of a fixed side replaced by its computed neighbour's
// (crank_nicolson.pyx:298-338); a face between two fixed voxels conducts nothing.  A class index past the
// table records an error.
__global__ void adj_setup_faces_kernel(AView v, const double* __restrict__ k, const double* __restrict__ C,
                                       double inv_dt, const uint8_t* __restrict__ fcls, int nclass,
                                       const double* __restrict__ forms, const uint8_t* __restrict__ fixed,
                                       double* __restrict__ gx, double* __restrict__ gy, double* __restrict__ gz,
                                       double* __restrict__ M, int* __restrict__ err) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= v.nvox) return;
  const Vox x = vox_at(v, p);
  if (!x.in) {
    gx[p] = gy[p] = gz[p] = 0.0;
    M[p] = 1.0;
    return;
  }
  const bool fp = fixed && fixed[p];
  M[p] = fp ? kFixedCapacity : C[p] * inv_dt;
  double* out[3] = {gz, gy, gx};
  const bool has_low[3] = {x.k > 0, x.j > 0, x.i > 0};
  const int64_t step[3] = {x.nxy, x.px, 1};
  for (int a = 0; a < 3; ++a) {
    double G = 0.0;
    if (has_low[a]) {
      const int64_t q = p - step[a];
      const bool fq = fixed && fixed[q];
      const int c = fcls[a * v.nvox + p];
      if (c >= nclass) {
        atomicExch(err, 1);
      } else if (!(fp && fq)) {
        const double* f = forms + ((int64_t)(x.inst * nclass + c) * 3 + a) * 3;
        const double klo = fq ? k[p] : k[q], khi = fp ? k[q] : k[p];
        G = fma(f[2], khi, fma(f[1], klo, f[0]));
      }
    }
    out[a][p] = G;
  }
}

// D = the sum of a voxel's six face conductances (the diagonal of -L)
__global__ void adj_diag_kernel(AView v, const double* __restrict__ gx, const double* __restrict__ gy,
                                const double* __restrict__ gz, double* __restrict__ D) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= v.nvox) return;
  const Vox x = vox_at(v, p);
  if (!x.in) {
    D[p] = 0.0;
    return;
  }
  double d = gx[p] + gy[p] + gz[p];
  if (x.i + 1 < x.nx) d += gx[p + 1];
  if (x.j + 1 < x.ny) d += gy[p + x.px];
  if (x.k + 1 < x.nz) d += gz[p + x.nxy];
  D[p] = d;
}

// Factors of A_a = M - L_a/2 per line, eliminated from both ends towards the middle row m (len/2 on y and z lines,
// (len-1)/2 on x lines, where the upper end starts on a 16-byte boundary): with p_r the pivots and h_r the
// conductance towards the middle,
//     z_r = W_r - a_r z_{r -+ 1},   x_r = z_r - b_r x_{r +- 1}   (lower, upper end),
//     x_m = W_m - a_m z_{m-1} - b_m z_{m+1},   W = rhs scale.
// Kept: -a = G / (2 p) of the face away from the middle, -b = G / (2 p) of the face towards it, ip = 1 / p (x: half of
// it, see adj_update_kernel) and mip = M / p, the scale of b = rhs and of b = M rhs.  A pair of lanes takes a line, one
// end each.  FP64 arithmetic bounds the kernel on many lines: one reciprocal per row and b from it by one correction step,
// 5.86 million voxels 688 us on the three axes against 865 with two divisions.  The step is Markstein's (Computation of
// elementary functions on the IBM RISC System/6000 processor, 1990): y the rounded reciprocal, q = y in to within two
// units of its last place, q + (in - q p) y with two fused multiply-adds is in / p to within half a unit and 2^-103 of
// it.  It wants y and q normal numbers and the remainder in - q p exact: p is at most 1e300 (a fixed voxel's row), whose
// y is one, and q is for every conductance above 1e-7 there (below, it is off by units of 5e-324, which nothing sees).
__global__ void adj_factor_kernel(AView v, int axis, int64_t nlines, const double* __restrict__ M,
                                  const double* __restrict__ g, double* __restrict__ a, double* __restrict__ b,
                                  double* __restrict__ ip, double* __restrict__ mip) {
  const int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 1;
  const bool upper = threadIdx.x & 1, live = t < nlines;
  const Line ln = live ? line_at(v, axis, t) : Line{0, 0, 0};
  const int64_t m = axis == 0 ? (ln.len - 1) / 2 : ln.len / 2;
  const int64_t rows = upper ? ln.len - 1 - m : m;
  const int64_t d = upper ? -ln.stride : ln.stride;
  int64_t p = ln.base + (upper ? (ln.len - 1) * ln.stride : 0);
  const double one = axis == 0 ? 0.5 : 1.0;
  double away = 0.0, drop = 0.0;  // half the conductance away from the middle, and what it takes from the pivot
  for (int64_t r = 0; r < rows; ++r, p += d) {
    const double in = 0.5 * g[upper ? p : p + ln.stride];
    const double m0 = M[p], piv = m0 + (away + in) - drop, inv = 1.0 / piv;
    double bb = __dmul_rn(in, inv);
    bb = __fma_rn(__fma_rn(-bb, piv, in), inv, bb);  // in / piv
    a[p] = away * inv;
    b[p] = bb;
    ip[p] = one * inv;
    mip[p] = __dmul_rn(m0, inv);
    drop = in * bb;
    away = in;
  }
  const double away_up = __shfl_xor_sync(0xffffffffu, away, 1), drop_up = __shfl_xor_sync(0xffffffffu, drop, 1);
  if (live && !upper) {  // p is the middle row
    const double m0 = M[p], piv = m0 + (away + away_up) - drop - drop_up, inv = 1.0 / piv;
    a[p] = away * inv;
    b[p] = away_up * inv;
    ip[p] = one * inv;
    mip[p] = __dmul_rn(m0, inv);
  }
}

// r0 = s q - D T_p + sum over faces of G T_nbr at voxel p = (k, j, i) of an (nz, ny, nx) instance (D = the sum
// of the six G): 8 FP64 operations against 13 for the face-by-face differences (skipping the source where s = 0, as
// adj_update_kernel does, made it slower: 110 us against 97 for 5.86 million voxels); temperatures are offsets
// from their initial mean, so the cancellation in -D T_p + sum G T_nbr stays at the rounding of the increments
__device__ __forceinline__ double residual_at(const double* __restrict__ T, const double* __restrict__ gx,
                                              const double* __restrict__ gy, const double* __restrict__ gz,
                                              const double* __restrict__ D, const double* __restrict__ q, double s,
                                              int64_t p, const Vox& x) {
  double r = __fma_rn(-D[p], T[p], __dmul_rn(s, q[p]));
  if (x.i > 0) r = __fma_rn(gx[p], T[p - 1], r);
  if (x.i + 1 < x.nx) r = __fma_rn(gx[p + 1], T[p + 1], r);
  if (x.j > 0) r = __fma_rn(gy[p], T[p - x.px], r);
  if (x.j + 1 < x.ny) r = __fma_rn(gy[p + x.px], T[p + x.px], r);
  if (x.k > 0) r = __fma_rn(gz[p], T[p - x.nxy], r);
  if (x.k + 1 < x.nz) r = __fma_rn(gz[p + x.nxy], T[p + x.nxy], r);
  return r;
}

// the right-hand sides of the forward x stage, W = r0 ip (half of them, as ip is halved).  FP64 arithmetic bounds it:
// 5.86 million voxels 97 us.
__global__ void adj_resid_kernel(AView v, const double* __restrict__ T, const double* __restrict__ gx,
                                 const double* __restrict__ gy, const double* __restrict__ gz,
                                 const double* __restrict__ D, const double* __restrict__ q, double s,
                                 const double* __restrict__ ip, double* __restrict__ W) {
  wait_prior_grid();  // the previous kernel on the stream (programmatic dependent launch)
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= v.nvox) return;
  const Vox x = vox_at(v, p);
  W[p] = x.in ? __dmul_rn(residual_at(T, gx, gy, gz, D, q, s, p, x), ip[p]) : 0.0;
}

// The line solves take the sweeps' code (hs2g_x.cuh, hs2g_pair.cuh) with coefficients per voxel: one warp per 16
// neighbouring lines, both ends at once, operands copied ahead in 16-byte pieces.  A voxel's right-hand side is
// multiplied by its scale on the way from shared memory, b = M rhs with mip, b = rhs with ip.  The same kernel serves
// a small problem and a batch, whether the forward values stay in shared memory or go through the output, so an
// instance's results do not depend on what it is solved with.
// A few lines are bound by the latency of a half line's chain, many by memory (32 to 56 bytes per voxel).  Against one
// thread per line, or one warp per 32 lines with a second one copying: y lines of six instances of 0.4 to 1.8 million
// voxels 138 -> 55 us, of 32x128x128 26 -> 16 us; x with its residual 177 -> 152 us and 33 -> 27 us; z of 32 rows alike.
// x lines, y = A_x^-1 (M rhs); SCALE false: in place from y = W
template <bool SCALE, bool KEEP>
__global__ void __launch_bounds__(32 * kPairMaxWarps) adj_x_kernel(AView v, int64_t ngroups, const double* rhs,
                                                                   const double* __restrict__ a,
                                                                   const double* __restrict__ b,
                                                                   const double* __restrict__ scale, double* y,
                                                                   int64_t smem_per_warp) {
  extern __shared__ __align__(16) unsigned char adj_sm[];
  const int warp = threadIdx.x >> 5;
  const int64_t grp = blockIdx.x * (int64_t)(blockDim.x >> 5) + warp;
  if (grp >= ngroups) return;
  const int i = find_inst(v.grp_off, v.ninst, grp);
  const AInst& in = v.inst[i];
  XProblem<double> P{};
  P.nz = in.nz;
  P.ny = in.ny;
  P.nx = in.nx;
  P.px = in.px;
  P.a0 = a + in.off;
  P.b0 = b + in.off;
  P.W0 = y + in.off;
  P.in = rhs + in.off;
  P.sc = scale + in.off;
  const int64_t L0 = (grp - v.grp_off[i]) * 16;
  wait_prior_grid();  // the previous kernel on the stream (programmatic dependent launch)
  x_solve_lines<double, true, false, KEEP, SCALE>(P, L0, (int)min((int64_t)16, in.nz * in.ny - L0),
                                                  reinterpret_cast<double*>(adj_sm + warp * smem_per_warp));
}
template <bool SCALE>
__global__ void __launch_bounds__(kFewThreads, 4) adj_few_x_kernel(AView v, const double* rhs,
                                                                   const double* __restrict__ a,
                                                                   const double* __restrict__ b,
                                                                   const double* __restrict__ scale, double* y) {
  extern __shared__ __align__(16) unsigned char adj_sm[];
  const int i = find_inst(v.grp_off, v.ninst, blockIdx.x);
  const AInst& in = v.inst[i];
  const int64_t L0 = (blockIdx.x - v.grp_off[i]) * 16, at = in.off + L0 * in.px;
  few_x_solve<SCALE>(rhs + at, scale + at, a + at, b + at, y + at, in.px, (int)in.nx,
                     (int)min((int64_t)16, in.nz * in.ny - L0), reinterpret_cast<double*>(adj_sm),
                     [] { wait_prior_grid(); });
}

// y (axis 1) or z (axis 2) lines, y = A_a^-1 (scale rhs); with T_out, T_out = T_in + 2 y (which may be the same; y is
// half the increment), y itself only when given, Z the scratch of the forward values, and with obs the top layer's
// T_out - obs of step obs_step in obs's place
struct APair {
  int axis;
  const double *rhs, *a, *b, *scale;
  double *y, *Z;
  const double* T_in;
  double *T_out, *obs;
  int64_t obs_step;
};
// the 16 lines of group grp: their rows and number, and this lane's observation (null: none)
template <bool ADD_T>
__device__ __forceinline__ void apair_lines(const AView& v, const APair& g, int64_t grp, PairLines<double>& p, int& n,
                                            int& width, double*& ob) {
  const int lane = threadIdx.x & 31;
  const int64_t* pre = v.grp_off + g.axis * (v.ninst + 1);
  const int i = find_inst(pre, v.ninst, grp);
  const AInst& in = v.inst[i];
  const int64_t l = grp - pre[i], px = in.px, nxy = in.ny * px;
  // y: 16 of a layer's px lines, z: 16 of all ny px (the pads' among them)
  const int64_t gpr = (px + 15) / 16;
  const int64_t first = g.axis == 1 ? (l % gpr) * 16 : l * 16;
  width = (int)min((int64_t)16, (g.axis == 1 ? px : nxy) - first);
  n = (int)(g.axis == 1 ? in.ny : in.nz);
  const int64_t base = in.off + (g.axis == 1 ? (l / gpr) * nxy : 0) + first;
  p.W = g.rhs + base;
  p.a = g.a + base;
  p.b = g.b + base;
  p.sc = g.scale + base;
  p.wst = p.cst = p.st = p.zst = g.axis == 1 ? px : nxy;
  p.out = (ADD_T ? g.T_out : g.y) + base;
  if (ADD_T) {
    p.T = g.T_in + base;
    p.X = g.y ? g.y + base : nullptr;
  }
  p.Z = (ADD_T ? g.Z : g.y) + base;
  ob = nullptr;
  if (ADD_T && g.obs && lane < width) {
    const uint32_t at = (uint32_t)first + lane, j = at / (uint32_t)px, c = at - j * (uint32_t)px;
    if (c < in.nx) ob = g.obs + in.obs_off + g.obs_step * in.ny * in.nx + j * in.nx + c;
  }
}
template <bool ADD_T, bool KEEP>
__global__ void __launch_bounds__(32 * kPairMaxWarps) adj_pair_kernel(AView v, APair g, int64_t ngroups,
                                                                      int64_t smem_per_warp) {
  extern __shared__ __align__(16) unsigned char adj_sm[];
  const int warp = threadIdx.x >> 5;
  const int64_t grp = blockIdx.x * (int64_t)(blockDim.x >> 5) + warp;
  if (grp >= ngroups) return;
  PairLines<double> p{};
  int n, width;
  double* ob;
  apair_lines<ADD_T>(v, g, grp, p, n, width, ob);
  wait_prior_grid();  // the previous kernel on the stream (programmatic dependent launch)
  const double seen = ob ? *ob : 0.0;
  pair_solve<double, true, ADD_T, KEEP, false, 2, 2, true>(p, n, width,
                                                            reinterpret_cast<double*>(adj_sm + warp * smem_per_warp));
  if (ob) *ob = p.out[threadIdx.x & 31] - seen;  // row 0 is stored by the lower end's lane
}
template <bool ADD_T>
__global__ void __launch_bounds__(kFewThreads, 4) adj_few_pair_kernel(AView v, APair g) {
  extern __shared__ __align__(16) unsigned char adj_sm[];
  PairLines<double> p{};
  int n, width;
  double* ob;
  apair_lines<ADD_T>(v, g, blockIdx.x, p, n, width, ob);
  if (threadIdx.x >= 32) ob = nullptr;
  double seen = 0.0;
  few_solve<ADD_T>(p, n, width, reinterpret_cast<double*>(adj_sm), [&] {
    wait_prior_grid();  // the previous kernel on the stream (programmatic dependent launch)
    if (ob) seen = *ob;
  });
  if (ADD_T && g.obs) {
    __syncthreads();  // row 0 is another warp's store
    if (ob) *ob = p.out[threadIdx.x] - seen;
  }
}

// lambda = misfit gradient of the last observation, 2 (T_N - d_{N-1}) on the top layer, 0 below; diff: the forward
// pass's differences T - d
__global__ void adj_seed_kernel(AView v, const double* __restrict__ diff, int64_t obs_step, double* __restrict__ lam) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= v.nvox) return;
  const Vox x = vox_at(v, p);
  const AInst& in = v.inst[x.inst];
  lam[p] = x.in && x.k == 0 ? 2.0 * diff[in.obs_off + (obs_step * x.ny + x.j) * x.nx + x.i] : 0.0;
}

// lambda += L mu0 (+ the misfit gradient of observation obs_step, from diff, when obs_step >= 0), and the
// gradient accumulation of one step; one thread per voxel, each voxel owning its three low faces.
// FP64 arithmetic bounds it, so what can be had without is: the increments h = y / 2 are halved (the x stage's scale
// is, exactly, and with it what follows), which takes the factors 1/2 out of the face gradients; a voxel's
// difference of mu0 to the left is formed once and shared through shared memory with the neighbour that needs it, as
// are T and h0; the source gradient is skipped where s = 0.  gM accumulates half its value.  (T + h0 is not formed per
// voxel, which would save one more operation: where T is large against the differences of h0 it loses their digits.)
// 30 operations (31 with a source) against 34, five CTAs to an SM (48 registers): 5.86 million voxels 342 us
// against 375 (22 fields of 8 bytes take 154).
constexpr int kUpdateThreads = 256;
__global__ void __launch_bounds__(kUpdateThreads, 5) adj_update_kernel(
    AView v, const double* __restrict__ gx, const double* __restrict__ gy, const double* __restrict__ gz,
    const double* __restrict__ T, const double* __restrict__ h0, const double* __restrict__ h1,
    const double* __restrict__ h2, const double* __restrict__ mu0, const double* __restrict__ mu1,
    const double* __restrict__ mu2, double s, const double* __restrict__ diff, int64_t obs_step,
    double* __restrict__ lam, double* __restrict__ ggx, double* __restrict__ ggy, double* __restrict__ ggz,
    double* __restrict__ gM, double* __restrict__ gq) {
  __shared__ double sT[kUpdateThreads + 1], sh[kUpdateThreads + 1], sd[kUpdateThreads + 1];
  const int t = threadIdx.x;
  const int64_t p0 = blockIdx.x * (int64_t)kUpdateThreads, p = p0 + t;
  Vox x{};
  if (p < v.nvox) x = vox_at(v, p);
  wait_prior_grid();  // the previous kernel on the stream (programmatic dependent launch)
  double m0 = 0.0, Tp = 0.0, a0 = 0.0, d0x = 0.0;
  if (x.in) {
    m0 = mu0[p];
    Tp = T[p];
    a0 = h0[p];
    if (x.i > 0) d0x = m0 - mu0[p - 1];
  }
  sT[t + 1] = Tp;
  sh[t + 1] = a0;
  sd[t] = d0x;
  // the neighbours beyond the block (read by voxels of their row alone): T and h0 on the left, mu0's difference on the right
  if (t == 0 && p0 > 0) {
    sT[0] = T[p0 - 1];
    sh[0] = h0[p0 - 1];
  }
  if (t == 32 && p0 + kUpdateThreads < v.nvox) sd[kUpdateThreads] = mu0[p0 + kUpdateThreads] - mu0[p0 + kUpdateThreads - 1];
  __syncthreads();
  if (!x.in) return;
  const double m1 = mu1[p], m2 = mu2[p], a1 = h1[p], a2 = h2[p];
  double l = lam[p];
  if (x.i > 0) {
    l = fma(-gx[p], d0x, l);
    ggx[p] = fma(-d0x, (a0 - sh[t]) + (Tp - sT[t]), ggx[p]);
  }
  if (x.j > 0) {
    const int64_t q = p - x.px;
    const double d0 = m0 - mu0[q];
    l = fma(-gy[p], d0, l);
    ggy[p] = fma(-(m1 - mu1[q]), a1 - h1[q], fma(-d0, Tp - T[q], ggy[p]));
  }
  if (x.k > 0) {
    const int64_t q = p - x.nxy;
    const double d0 = m0 - mu0[q];
    l = fma(-gz[p], d0, l);
    ggz[p] = fma(-(m2 - mu2[q]), a2 - h2[q], fma(-d0, Tp - T[q], ggz[p]));
  }
  if (x.i + 1 < x.nx) l = fma(gx[p + 1], sd[t + 1], l);
  if (x.j + 1 < x.ny) l = fma(gy[p + x.px], mu0[p + x.px] - m0, l);
  if (x.k + 1 < x.nz) l = fma(gz[p + x.nxy], mu0[p + x.nxy] - m0, l);
  bool again = obs_step >= 0 && x.k == 0;
  while (again) {
    l += 2.0 * diff[v.inst[x.inst].obs_off + (obs_step * x.ny + x.j) * x.nx + x.i];
    again = never();
  }
  lam[p] = l;
  // half of mu2 y1 + mu1 y0 - mu0 y0 - mu1 y1 - mu2 y2 = mu2 (y1 - y2) + mu1 (y0 - y1) - mu0 y0
  gM[p] = fma(m2, a1 - a2, fma(m1, a0 - a1, fma(-m0, a0, gM[p])));
  again = adds_something(s, m0);
  while (again) {
    gq[p] = fma(s, m0, gq[p]);
    again = never();
  }
}

// s + v as an unevaluated pair: returns the rounded sum, err receives its exact rounding error (Knuth's TwoSum)
__device__ __forceinline__ double two_sum(double s, double v, double& err) {
  const double t = s + v;
  const double bp = t - s;
  err = (s - (t - bp)) + (v - bp);
  return t;
}

// misfits of the steps from step0, as compensated pairs: block (c, i, s) sums the squares of the differences T - obs
// of step step0 + s (left in obs's place by the forward z solves) over its slice of instance i's top layer with per-thread Neumaier sums and a TwoSum tree (256 threads, fixed order) and writes
// part[2*((step*ninst + i)*kMisfitBlocks + c)] and the next entry (rounded sum, error); summing the pairs
// exactly on the host leaves the loss with no summation error that would swamp the small loss differences
// finite-difference checks take
constexpr int kMisfitBlocks = 32;
__global__ void adj_misfit_kernel(AView v, const double* __restrict__ diff, int64_t step0, double* __restrict__ part) {
  __shared__ double sh_hi[256], sh_lo[256];
  const AInst& in = v.inst[blockIdx.y];
  const int64_t m = in.ny * in.nx, step = step0 + blockIdx.z;
  const double* o = diff + in.obs_off + step * m;
  double hi = 0.0, lo = 0.0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
    const double r = o[e];
    const double sq = r * r;
    double err;
    hi = two_sum(hi, sq, err);
    lo += err + fma(r, r, -sq);  // the square's own rounding error, exactly
  }
  sh_hi[threadIdx.x] = hi;
  sh_lo[threadIdx.x] = lo;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      double err;
      const double s2 = two_sum(sh_hi[threadIdx.x], sh_hi[threadIdx.x + w], err);
      sh_lo[threadIdx.x] += sh_lo[threadIdx.x + w] + err;
      sh_hi[threadIdx.x] = s2;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const int64_t at = 2 * ((step * v.ninst + blockIdx.y) * kMisfitBlocks + blockIdx.x);
    part[at] = sh_hi[0];
    part[at + 1] = sh_lo[0];
  }
}

// chain to the parameters: gk from the face gradients (G = (k_lo + k_hi) / (2 d^2)), gC = 2 gM / dt (gM is half)
__global__ void adj_chain_kernel(AView v, const double* __restrict__ ggx, const double* __restrict__ ggy,
                                 const double* __restrict__ ggz, const double* __restrict__ gM, double two_inv_dt,
                                 double* __restrict__ gk, double* __restrict__ gC) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= v.nvox) return;
  const Vox x = vox_at(v, p);
  if (!x.in) return;
  const AInst& in = v.inst[x.inst];
  double fx = 0.0, fy = 0.0, fz = 0.0;
  if (x.i > 0) fx += ggx[p];
  if (x.i + 1 < x.nx) fx += ggx[p + 1];
  if (x.j > 0) fy += ggy[p];
  if (x.j + 1 < x.ny) fy += ggy[p + x.px];
  if (x.k > 0) fz += ggz[p];
  if (x.k + 1 < x.nz) fz += ggz[p + x.nxy];
  gk[p] = 0.5 * (in.idx2 * fx + in.idy2 * fy + in.idz2 * fz);
  gC[p] = gM[p] * two_inv_dt;
}

// The chain with face classes: d G_f / d k of each side from the face's affine form (both coefficients to the
// computed side of a face with a fixed neighbour); no gradient for fixed voxels' k, C and q.
__global__ void adj_chain_faces_kernel(AView v, const double* __restrict__ ggx, const double* __restrict__ ggy,
                                       const double* __restrict__ ggz, const double* __restrict__ gM, double two_inv_dt,
                                       const uint8_t* __restrict__ fcls, int nclass, const double* __restrict__ forms,
                                       const uint8_t* __restrict__ fixed, double* __restrict__ gk,
                                       double* __restrict__ gC, double* __restrict__ gq) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= v.nvox) return;
  const Vox x = vox_at(v, p);
  if (!x.in) return;
  const bool fp = fixed && fixed[p];
  if (fp) {
    gk[p] = 0.0;
    gC[p] = 0.0;
    gq[p] = 0.0;
    return;
  }
  const double* gg[3] = {ggz, ggy, ggx};
  const int64_t coord[3] = {x.k, x.j, x.i}, len[3] = {x.nz, x.ny, x.nx}, step[3] = {x.nxy, x.px, 1};
  double acc = 0.0;
  for (int a = 0; a < 3; ++a) {
    if (coord[a] > 0) {  // low face: p is its hi side
      const int64_t q = p - step[a];
      const int c = min((int)fcls[a * v.nvox + p], nclass - 1);
      const double* f = forms + ((int64_t)(x.inst * nclass + c) * 3 + a) * 3;
      const bool fq = fixed && fixed[q];
      acc = fma(gg[a][p], fq ? f[1] + f[2] : f[2], acc);
    }
    if (coord[a] + 1 < len[a]) {  // high face (the low face of r): p is its lo side
      const int64_t r = p + step[a];
      const int c = min((int)fcls[a * v.nvox + r], nclass - 1);
      const double* f = forms + ((int64_t)(x.inst * nclass + c) * 3 + a) * 3;
      const bool fr = fixed && fixed[r];
      acc = fma(gg[a][r], fr ? f[1] + f[2] : f[1], acc);
    }
  }
  gk[p] = acc;
  gC[p] = gM[p] * two_inv_dt;
}

}  // namespace
}  // namespace hs2g

struct hs2g_adjoint {
  int device = 0;
  double dt = 0.0;
  cudaStream_t stream = nullptr;
  bool own_stream = true;
  int ninst = 0;
  int64_t n = 0, next = 0;       // voxels with the pads of the rows, and without (the caller's arrays)
  int64_t nobs_step = 0;         // top-layer voxels of all instances (observations per step)
  int64_t nlines[3] = {0, 0, 0}, ngroups[3] = {0, 0, 0};
  int64_t max_len[3] = {0, 0, 0};  // longest line of each axis over the instances
  std::vector<hs2g::AInst> host_inst;
  std::vector<int64_t> host_ext_off;  // the caller's layout
  hs2g::AInst* inst = nullptr;
  int64_t* vox_off = nullptr;
  int64_t* line_off = nullptr;
  int64_t* grp_off = nullptr;
  // parameters and derived fields
  double *k = nullptr, *C = nullptr, *q = nullptr, *M = nullptr, *D = nullptr;
  double* g[3] = {nullptr, nullptr, nullptr};
  // face classes and fixed voxels (hs2g_adjoint_set_faces): without them every interior face conducts with the
  // arithmetic mean of k and every voxel is computed
  uint8_t* fcls = nullptr;   // 3 * n: class of each voxel's low face on z, y, x
  uint8_t* fixed = nullptr;  // n, or null
  double* forms = nullptr;   // [ninst][nclass][3][3]
  int nclass = 0;
  int* err = nullptr;
  // line factors of A_x, A_y, A_z (adj_factor_kernel)
  double *ca[3] = {nullptr, nullptr, nullptr}, *cb[3] = {nullptr, nullptr, nullptr},
         *ip[3] = {nullptr, nullptr, nullptr}, *mip[3] = {nullptr, nullptr, nullptr};
  // run state
  bool have_params = false;
  int nsteps = 0, ckpt = 1;
  std::vector<double> sched;
  double* obs = nullptr;    // nsteps * nobs_step, replaced by T - obs as the forward pass goes
  double* ckpts = nullptr;  // ceil(nsteps / ckpt) * n
  double* seg = nullptr;    // ckpt * 4 * n: T, y0, y1, y2 of each step of a segment
  double* seg2 = nullptr;   // a second segment store: the next segment is recomputed while this one is swept
  int stored_from = -1;     // the last forward pass left the states of the segments from here on in the stores (-1: none)
  cudaStream_t rec_stream = nullptr;  // the recompute stream
  cudaEvent_t ev_rec[2] = {nullptr, nullptr}, ev_done[2] = {nullptr, nullptr}, ev_start = nullptr;
  double* T = nullptr;      // forward state
  double *lam = nullptr, *mu[3] = {nullptr, nullptr, nullptr};
  double *gg[3] = {nullptr, nullptr, nullptr}, *gM = nullptr, *gq = nullptr;
  double* parts = nullptr;  // 2 * kMisfitBlocks * nsteps * ninst misfit parts (compensated pairs)
  int64_t obs_cap = 0, ckpt_cap = 0, seg_cap = 0, seg2_cap = 0, parts_cap = 0;
  int64_t fixed_bytes = 0;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

namespace {

using hs2g::kTh;
using hs2g::nblk;
using hs2g::launch_kernel;

// The kernels of a step are launched with programmatic dependent launch (each waits for the previous kernel at its
// start; no kernel triggers early): the launch latency at each kernel boundary is hidden.  HS2G_PDL=0 turns it
// off.
bool adj_pdl() {
  static const bool on = [] {
    const char* e = getenv("HS2G_PDL");
    return !(e && strcmp(e, "0") == 0);
  }();
  return on;
}

int afail(int code, const char* m) { return hs2g::set_last_error(code, m); }
int acuda(cudaError_t e, const char* what) {
  cudaGetLastError();  // a failed allocation leaves its error as the last error: clear it for later checks
  char buf[256];
  snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
  return hs2g::set_last_error(e == cudaErrorMemoryAllocation ? HS2G_ERR_NOMEM : HS2G_ERR_CUDA, buf);
}

struct AGuard {
  int prev = -1;
  bool ok = false;
  explicit AGuard(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    ok = (prev == dev) || (cudaSetDevice(dev) == cudaSuccess);
  }
  ~AGuard() {
    int cur = -1;
    if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
  }
};

hs2g::AView view(const hs2g_adjoint* a) {
  return hs2g::AView{a->inst, a->vox_off, a->line_off, a->grp_off, a->ninst, a->n};
}

cudaError_t grow(double** p, int64_t* cap, int64_t need) {
  if (*p && *cap >= need) return cudaSuccess;
  if (*p) cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  cudaError_t e = cudaMalloc(p, sizeof(double) * std::max<int64_t>(1, need));
  if (e == cudaSuccess) *cap = need;
  return e;
}

// a field from the caller's array, or to it (through stage, in the caller's layout, when the rows have pads)
template <typename E>
cudaError_t copy_in(const hs2g_adjoint* a, E* dst, const E* src, cudaMemcpyKind kind, double* stage, cudaStream_t st) {
  if (a->n == a->next) return cudaMemcpyAsync(dst, src, sizeof(E) * a->n, kind, st);
  E* tmp = reinterpret_cast<E*>(stage);
  const cudaError_t e = cudaMemcpyAsync(tmp, src, sizeof(E) * a->next, kind, st);
  if (e != cudaSuccess) return e;
  hs2g::adj_pack_kernel<E><<<nblk(a->n), kTh, 0, st>>>(view(a), tmp, dst);
  return cudaGetLastError();
}
cudaError_t copy_out(const hs2g_adjoint* a, double* dst, const double* src, cudaMemcpyKind kind, double* stage,
                     cudaStream_t st) {
  if (a->n == a->next) return cudaMemcpyAsync(dst, src, sizeof(double) * a->n, kind, st);
  hs2g::adj_unpack_kernel<<<nblk(a->n), kTh, 0, st>>>(view(a), src, stage);
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? e : cudaMemcpyAsync(dst, stage, sizeof(double) * a->next, kind, st);
}

// y = A_x^-1 (M rhs); without rhs in place, y = A_x^-1 of right-hand sides already scaled
template <bool SCALE>
cudaError_t xsolve(const hs2g_adjoint* a, cudaStream_t st, const double* rhs, double* y) {
  const int64_t groups = a->ngroups[0];
  const size_t few = hs2g::few_x_smem<SCALE>(a->max_len[0]);
  if (hs2g::few_lines(groups, few))
    return launch_kernel(hs2g::adj_few_x_kernel<SCALE>, dim3((unsigned)groups), dim3(hs2g::kFewThreads), few, st,
                         adj_pdl(), view(a), SCALE ? rhs : y, a->ca[0], a->cb[0], a->mip[0], y);
  const hs2g::PairShape sh = hs2g::x_solve_shape<double, true, false, SCALE>(a->max_len[0], groups);
  return launch_kernel(sh.keep ? hs2g::adj_x_kernel<SCALE, true> : hs2g::adj_x_kernel<SCALE, false>,
                       dim3((unsigned)((groups + sh.warps - 1) / sh.warps)), dim3(32 * sh.warps), sh.smem, st,
                       adj_pdl(), view(a), groups, SCALE ? rhs : y, a->ca[0], a->cb[0], a->mip[0], y,
                       (int64_t)(sh.smem / sh.warps));
}
template <bool ADD_T>
cudaError_t pair_launch(const hs2g_adjoint* a, cudaStream_t st, const hs2g::APair& g) {
  const int64_t groups = a->ngroups[g.axis];
  const size_t few = hs2g::few_smem(a->max_len[g.axis]);
  if (hs2g::few_lines(groups, few))
    return launch_kernel(hs2g::adj_few_pair_kernel<ADD_T>, dim3((unsigned)groups), dim3(hs2g::kFewThreads), few, st,
                         adj_pdl(), view(a), g);
  const hs2g::PairShape sh = hs2g::pair_shape<double, true, ADD_T, false, true>(a->max_len[g.axis], groups);
  return launch_kernel(sh.keep ? hs2g::adj_pair_kernel<ADD_T, true> : hs2g::adj_pair_kernel<ADD_T, false>,
                       dim3((unsigned)((groups + sh.warps - 1) / sh.warps)), dim3(32 * sh.warps), sh.smem, st,
                       adj_pdl(), view(a), g, groups, (int64_t)(sh.smem / sh.warps));
}
// y = A_a^-1 (M rhs) on the y or z lines (weighted false: A_a^-1 rhs)
cudaError_t ysolve(const hs2g_adjoint* a, cudaStream_t st, int axis, bool weighted, const double* rhs, double* y) {
  hs2g::APair g{};
  g.axis = axis;
  g.rhs = rhs;
  g.a = a->ca[axis];
  g.b = a->cb[axis];
  g.scale = weighted ? a->mip[axis] : a->ip[axis];
  g.y = y;
  return pair_launch<false>(a, st, g);
}
// the forward z stage: y2 = A_z^-1 (M y1) (stored when keep_y), T_out = T_in + 2 y2, and T_out - obs of step obs_step
// >= 0 in obs's place
cudaError_t zstep(const hs2g_adjoint* a, cudaStream_t st, const double* y1, double* y2, bool keep_y, const double* T_in,
                  double* T_out, int64_t obs_step) {
  return pair_launch<true>(a, st, hs2g::APair{2, y1, a->ca[2], a->cb[2], a->mip[2], keep_y ? y2 : nullptr, y2, T_in,
                                              T_out, obs_step >= 0 ? a->obs : nullptr, obs_step});
}

// one forward step T_in -> T_out on stream st (T_out may alias T_in; NULL skips it), y0, y1 and with keep_y y2 left in
// place; obs_step >= 0: as zstep
cudaError_t fwd_step(hs2g_adjoint* a, cudaStream_t st, const double* T_in, double* T_out, double* y0, double* y1,
                     double* y2, bool keep_y, double s, int64_t obs_step) {
  cudaError_t e = launch_kernel(hs2g::adj_resid_kernel, dim3(nblk(a->n)), dim3(kTh), 0, st, adj_pdl(), view(a), T_in,
                                a->g[0], a->g[1], a->g[2], a->D, a->q, s, a->ip[0], y0);
  if (e == cudaSuccess) e = xsolve<false>(a, st, nullptr, y0);
  if (e == cudaSuccess) e = ysolve(a, st, 1, true, y0, y1);
  if (e == cudaSuccess)
    e = T_out ? zstep(a, st, y1, y2, keep_y, T_in, T_out, obs_step) : ysolve(a, st, 2, true, y1, y2);
  return e;
}

// adjoint of one step: lambda (the adjoint of T_{n+1}) -> the adjoint of T_n, gradients accumulated.
// A_a is symmetric, so the transposed solves A_a^-T are the forward line solves.
cudaError_t bwd_step(hs2g_adjoint* a, const double* Tn, const double* y0, const double* y1, const double* y2,
                     double s, int64_t obs_step) {
  cudaStream_t st = a->stream;
  cudaError_t e = ysolve(a, st, 2, false, a->lam, a->mu[2]);
  if (e == cudaSuccess) e = ysolve(a, st, 1, true, a->mu[2], a->mu[1]);
  if (e == cudaSuccess) e = xsolve<true>(a, st, a->mu[1], a->mu[0]);
  if (e == cudaSuccess)
    e = launch_kernel(hs2g::adj_update_kernel,
                      dim3((unsigned)((a->n + hs2g::kUpdateThreads - 1) / hs2g::kUpdateThreads)),
                      dim3(hs2g::kUpdateThreads), 0, st, adj_pdl(), view(a), a->g[0], a->g[1],
                      a->g[2], Tn, y0, y1, y2, a->mu[0], a->mu[1], a->mu[2], s, a->obs, obs_step, a->lam, a->gg[0],
                      a->gg[1], a->gg[2], a->gM, a->gq);
  return e;
}

void adj_free(hs2g_adjoint* a) {
  void* ptrs[] = {a->inst, a->vox_off, a->line_off, a->grp_off, a->k, a->C, a->q, a->M, a->D, a->g[0], a->g[1],
                  a->g[2], a->ca[0], a->ca[1], a->ca[2], a->cb[0], a->cb[1], a->cb[2], a->ip[0], a->ip[1], a->ip[2],
                  a->mip[0], a->mip[1], a->mip[2],
                  a->obs, a->ckpts, a->seg, a->seg2, a->T, a->lam, a->mu[0], a->mu[1], a->mu[2], a->gg[0], a->gg[1],
                  a->gg[2], a->gM, a->gq, a->parts, a->fcls, a->fixed, a->forms, a->err};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  if (a->ev0) cudaEventDestroy(a->ev0);
  if (a->ev1) cudaEventDestroy(a->ev1);
  cudaEvent_t evs[] = {a->ev_rec[0], a->ev_rec[1], a->ev_done[0], a->ev_done[1], a->ev_start};
  for (cudaEvent_t ev : evs)
    if (ev) cudaEventDestroy(ev);
  if (a->rec_stream) cudaStreamDestroy(a->rec_stream);
  if (a->stream && a->own_stream) cudaStreamDestroy(a->stream);
}

cudaMemcpyKind in_kind(int flags) { return (flags & HS2G_DEVICE) ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice; }
cudaMemcpyKind out_kind(int flags) { return (flags & HS2G_DEVICE) ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost; }

void read_elapsed(hs2g_adjoint* a, double* elapsed_ms) {
  if (!elapsed_ms) return;
  float ms = 0.f;
  *elapsed_ms = cudaEventElapsedTime(&ms, a->ev0, a->ev1) == cudaSuccess ? ms : -1.0;
}

}  // namespace

extern "C" {

int hs2g_adjoint_create(int n, const hs2g_adjoint_grid* grids, double dt, int device, hs2g_adjoint** out) {
  if (!out) return afail(HS2G_ERR_ARG, "hs2g_adjoint_create: null output");
  *out = nullptr;
  if (n < 1 || !grids || !(dt > 0) || !std::isfinite(dt))
    return afail(HS2G_ERR_ARG, "hs2g_adjoint_create: bad argument");
  std::vector<hs2g::AInst> inst((size_t)n);
  std::vector<int64_t> vox_off((size_t)n + 1, 0), line_off(3 * ((size_t)n + 1), 0), grp_off(line_off), ext_off(vox_off);
  int64_t nobs = 0;
  const int64_t limit = int64_t(1) << 40;
  for (int i = 0; i < n; ++i) {
    const hs2g_adjoint_grid& g = grids[i];
    if (g.nz < 1 || g.ny < 1 || g.nx < 1 || !(g.dz > 0) || !(g.dy > 0) || !(g.dx > 0) || !std::isfinite(g.dz) ||
        !std::isfinite(g.dy) || !std::isfinite(g.dx))
      return afail(HS2G_ERR_ARG, "hs2g_adjoint_create: bad grid");
    if (g.ny > limit / g.nx || g.nz > limit / (g.ny * g.nx)) return afail(HS2G_ERR_ARG, "hs2g_adjoint_create: grid too large");
    hs2g::AInst& a = inst[i];
    a.off = vox_off[i];
    a.ext = ext_off[i];
    a.nz = g.nz;
    a.ny = g.ny;
    a.nx = g.nx;
    // (whole 32-byte sectors would be two columns more of memory and nothing faster: four instances of 40x130x33, 20 steps
    // and their gradients 3.42 ms against 3.33, of 48x192x189 21.4 against 21.6)
    a.px = (g.nx + 1) / 2 * 2;
    a.idx2 = 1.0 / (g.dx * g.dx);
    a.idy2 = 1.0 / (g.dy * g.dy);
    a.idz2 = 1.0 / (g.dz * g.dz);
    a.obs_off = nobs;  // in units of nsteps, scaled when the step count is known
    nobs += g.ny * g.nx;
    ext_off[i + 1] = ext_off[i] + g.nz * g.ny * g.nx;
    // (six instances of 3.4 million voxels, 37 steps: 24.7 ms where the later ones start off the sectors, 24.0 so)
    vox_off[i + 1] = vox_off[i] + g.nz * g.ny * a.px;
    if (i + 1 < n) vox_off[i + 1] = (vox_off[i + 1] + 3) / 4 * 4;
    if (ext_off[i + 1] > limit) return afail(HS2G_ERR_ARG, "hs2g_adjoint_create: batch too large");
    const int64_t lines[3] = {g.nz * g.ny, g.nz * a.px, g.ny * a.px};
    const int64_t groups[3] = {(lines[0] + 15) / 16, g.nz * ((a.px + 15) / 16), (lines[2] + 15) / 16};
    for (int ax = 0; ax < 3; ++ax) {
      line_off[ax * (n + 1) + i + 1] = line_off[ax * (n + 1) + i] + lines[ax];
      grp_off[ax * (n + 1) + i + 1] = grp_off[ax * (n + 1) + i] + groups[ax];
    }
  }
  // the kernels index voxels with 32 bits; 2^31 voxels would need 515 GB for the 30 per-voxel fields
  if (ext_off[n] > 0x7fffffff || vox_off[n] > 0x7fffffff)
    return afail(HS2G_ERR_ARG, "hs2g_adjoint_create: batch too large (2^31 voxels)");
  AGuard guard(device);
  if (!guard.ok) return afail(HS2G_ERR_CUDA, "hs2g_adjoint_create: cannot select device");
  hs2g_adjoint* a = new hs2g_adjoint();
  a->device = device;
  a->dt = dt;
  a->ninst = n;
  a->n = vox_off[n];
  a->next = ext_off[n];
  a->nobs_step = nobs;
  for (int ax = 0; ax < 3; ++ax) {
    a->nlines[ax] = line_off[ax * (n + 1) + n];
    a->ngroups[ax] = grp_off[ax * (n + 1) + n];
  }
  for (const auto& in : inst) {
    a->max_len[0] = std::max(a->max_len[0], in.nx);
    a->max_len[1] = std::max(a->max_len[1], in.ny);
    a->max_len[2] = std::max(a->max_len[2], in.nz);
  }
  a->host_inst = inst;
  a->host_ext_off = ext_off;
  cudaError_t e = cudaStreamCreateWithFlags(&a->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreate(&a->ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&a->ev1);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&a->rec_stream, cudaStreamNonBlocking);
  for (int b = 0; b < 2 && e == cudaSuccess; ++b) {
    e = cudaEventCreateWithFlags(&a->ev_rec[b], cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&a->ev_done[b], cudaEventDisableTiming);
  }
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&a->ev_start, cudaEventDisableTiming);
  // (a CTA has at most 227 KB, less what it takes beside its own)
  const void* solves[] = {(const void*)hs2g::adj_pair_kernel<false, false>, (const void*)hs2g::adj_pair_kernel<false, true>,
                          (const void*)hs2g::adj_pair_kernel<true, false>,  (const void*)hs2g::adj_pair_kernel<true, true>,
                          (const void*)hs2g::adj_x_kernel<false, false>,    (const void*)hs2g::adj_x_kernel<false, true>,
                          (const void*)hs2g::adj_x_kernel<true, false>,     (const void*)hs2g::adj_x_kernel<true, true>,
                          (const void*)hs2g::adj_few_pair_kernel<false>,    (const void*)hs2g::adj_few_pair_kernel<true>,
                          (const void*)hs2g::adj_few_x_kernel<false>,       (const void*)hs2g::adj_few_x_kernel<true>};
  for (const void* f : solves)
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
  if (e == cudaSuccess) e = cudaMalloc(&a->inst, sizeof(hs2g::AInst) * n);
  if (e == cudaSuccess) e = cudaMalloc(&a->vox_off, sizeof(int64_t) * (n + 1));
  if (e == cudaSuccess) e = cudaMalloc(&a->line_off, sizeof(int64_t) * 3 * (n + 1));
  if (e == cudaSuccess) e = cudaMalloc(&a->grp_off, sizeof(int64_t) * 3 * (n + 1));
  double** per_voxel[] = {&a->k, &a->C, &a->q, &a->M, &a->D, &a->g[0], &a->g[1], &a->g[2], &a->ca[0],
                          &a->ca[1], &a->ca[2], &a->cb[0], &a->cb[1], &a->cb[2], &a->ip[0], &a->ip[1], &a->ip[2], &a->mip[0],
                          &a->mip[1], &a->mip[2], &a->T,
                          &a->lam, &a->mu[0], &a->mu[1], &a->mu[2], &a->gg[0], &a->gg[1], &a->gg[2], &a->gM,
                          &a->gq};
  const int nfields = (int)(sizeof(per_voxel) / sizeof(per_voxel[0]));
  for (double** p : per_voxel)
    if (e == cudaSuccess) e = cudaMalloc(p, sizeof(double) * a->n);
  // the pads of the rows, which no solve of x lines writes
  for (double** p : per_voxel)
    if (e == cudaSuccess && a->n != a->next) e = cudaMemsetAsync(*p, 0, sizeof(double) * a->n, a->stream);
  if (e == cudaSuccess) e = cudaMemcpy(a->inst, inst.data(), sizeof(hs2g::AInst) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(a->vox_off, vox_off.data(), sizeof(int64_t) * (n + 1), cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(a->line_off, line_off.data(), sizeof(int64_t) * 3 * (n + 1), cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(a->grp_off, grp_off.data(), sizeof(int64_t) * 3 * (n + 1), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaStreamSynchronize(a->stream);
  if (e != cudaSuccess) {
    const int rc = acuda(e, "hs2g_adjoint_create");
    adj_free(a);
    delete a;
    return rc;
  }
  a->fixed_bytes = (int64_t)nfields * a->n * (int64_t)sizeof(double);
  *out = a;
  return HS2G_OK;
}

void hs2g_adjoint_destroy(hs2g_adjoint* a) {
  if (!a) return;
  AGuard guard(a->device);
  cudaStreamSynchronize(a->stream);
  adj_free(a);
  delete a;
}

int hs2g_adjoint_set_stream(hs2g_adjoint* a, void* stream) {
  if (!a) return afail(HS2G_ERR_ARG, "null handle");
  if (!a->own_stream && a->stream == (cudaStream_t)stream) return HS2G_OK;
  AGuard guard(a->device);
  cudaStreamSynchronize(a->stream);
  if (a->own_stream) cudaStreamDestroy(a->stream);
  a->stream = (cudaStream_t)stream;  // NULL = the legacy default stream
  a->own_stream = false;
  return HS2G_OK;
}

int hs2g_adjoint_layout(const hs2g_adjoint* a, int64_t* offsets) {
  if (!a || !offsets) return afail(HS2G_ERR_ARG, "null argument");
  for (int i = 0; i <= a->ninst; ++i) offsets[i] = a->host_ext_off[i];
  return HS2G_OK;
}

int64_t hs2g_adjoint_device_bytes(const hs2g_adjoint* a) {
  if (!a) return 0;
  return a->fixed_bytes +
         (int64_t)sizeof(double) * (a->obs_cap + a->ckpt_cap + a->seg_cap + a->seg2_cap + a->parts_cap);
}

int hs2g_adjoint_set_parameters(hs2g_adjoint* a, const double* k, const double* C, const double* q, int flags) {
  if (!a || !k || !C || !q) return afail(HS2G_ERR_ARG, "hs2g_adjoint_set_parameters: null argument");
  AGuard guard(a->device);
  cudaStream_t st = a->stream;
  const int64_t n = a->n;
  const cudaMemcpyKind kind = in_kind(flags);
  a->have_params = false;
  a->nsteps = 0;
  a->stored_from = -1;
  cudaError_t e = copy_in(a, a->k, k, kind, a->mu[0], st);
  if (e == cudaSuccess) e = copy_in(a, a->C, C, kind, a->mu[1], st);
  if (e == cudaSuccess) e = copy_in(a, a->q, q, kind, a->mu[2], st);
  if (e != cudaSuccess) return acuda(e, "hs2g_adjoint_set_parameters");
  const hs2g::AView v = view(a);
  if (a->forms) {
    e = cudaMemsetAsync(a->err, 0, sizeof(int), st);
    if (e != cudaSuccess) return acuda(e, "hs2g_adjoint_set_parameters");
    hs2g::adj_setup_faces_kernel<<<nblk(n), kTh, 0, st>>>(v, a->k, a->C, 1.0 / a->dt, a->fcls, a->nclass, a->forms,
                                                          a->fixed, a->g[0], a->g[1], a->g[2], a->M, a->err);
  } else {
    hs2g::adj_setup_kernel<<<nblk(n), kTh, 0, st>>>(v, a->k, a->C, 1.0 / a->dt, a->g[0], a->g[1], a->g[2], a->M);
  }
  hs2g::adj_diag_kernel<<<nblk(n), kTh, 0, st>>>(v, a->g[0], a->g[1], a->g[2], a->D);
  for (int ax = 0; ax < 3; ++ax)
    hs2g::adj_factor_kernel<<<nblk(2 * a->nlines[ax]), kTh, 0, st>>>(v, ax, a->nlines[ax], a->M, a->g[ax], a->ca[ax],
                                                                    a->cb[ax], a->ip[ax], a->mip[ax]);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return acuda(e, "hs2g_adjoint_set_parameters");
  if (a->forms) {
    int bad = 0;
    e = cudaMemcpy(&bad, a->err, sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return acuda(e, "hs2g_adjoint_set_parameters");
    if (bad) return afail(HS2G_ERR_ARG, "hs2g_adjoint_set_parameters: a face class index is past the forms table");
  }
  a->have_params = true;
  return HS2G_OK;
}

int hs2g_adjoint_set_faces(hs2g_adjoint* a, int nclass, const double* forms, const uint8_t* face_z,
                           const uint8_t* face_y, const uint8_t* face_x, const uint8_t* fixed, int flags) {
  if (a && nclass == 0) {  // back to the default: every interior face conducting, every voxel computed
    AGuard guard(a->device);
    cudaStreamSynchronize(a->stream);
    void* ptrs[] = {a->forms, a->fcls, a->fixed};
    for (void* p : ptrs)
      if (p) cudaFree(p);
    a->forms = nullptr;
    a->fcls = a->fixed = nullptr;
    a->nclass = 0;
    a->have_params = false;
    a->nsteps = 0;
    a->stored_from = -1;
    return HS2G_OK;
  }
  if (!a || nclass < 1 || nclass > HS2G_MAX_CLASSES || !forms || !face_z || !face_y || !face_x)
    return afail(HS2G_ERR_ARG, "hs2g_adjoint_set_faces: bad argument");
  const int64_t nf = (int64_t)a->ninst * nclass * 9;
  for (int64_t t = 0; t < nf; ++t)
    if (!std::isfinite(forms[t])) return afail(HS2G_ERR_ARG, "hs2g_adjoint_set_faces: non-finite face form");
  AGuard guard(a->device);
  cudaStream_t st = a->stream;
  const int64_t n = a->n;
  const cudaMemcpyKind kind = in_kind(flags);
  cudaError_t e = cudaSuccess;
  if (a->forms && a->nclass != nclass) {
    cudaFree(a->forms);
    a->forms = nullptr;
  }
  if (!a->forms) e = cudaMalloc(&a->forms, sizeof(double) * nf);
  if (e == cudaSuccess && !a->fcls) e = cudaMalloc(&a->fcls, 3 * (size_t)n);
  if (e == cudaSuccess && !a->err) e = cudaMalloc(&a->err, sizeof(int));
  if (e == cudaSuccess && fixed && !a->fixed) e = cudaMalloc(&a->fixed, (size_t)n);
  if (e != cudaSuccess) {
    cudaFree(a->forms);
    a->forms = nullptr;
    return acuda(e, "hs2g_adjoint_set_faces: device allocation");
  }
  a->nclass = nclass;
  e = cudaMemcpyAsync(a->forms, forms, sizeof(double) * nf, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = copy_in(a, a->fcls, face_z, kind, a->mu[0], st);
  if (e == cudaSuccess) e = copy_in(a, a->fcls + n, face_y, kind, a->mu[1], st);
  if (e == cudaSuccess) e = copy_in(a, a->fcls + 2 * n, face_x, kind, a->mu[2], st);
  if (e == cudaSuccess && fixed) e = copy_in(a, a->fixed, fixed, kind, a->lam, st);
  if (e == cudaSuccess && !fixed && a->fixed) {
    cudaFree(a->fixed);
    a->fixed = nullptr;
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return acuda(e, "hs2g_adjoint_set_faces");
  a->have_params = false;  // the faces apply from the next hs2g_adjoint_set_parameters
  a->nsteps = 0;
  a->stored_from = -1;
  return HS2G_OK;
}

int hs2g_adjoint_forward(hs2g_adjoint* a, int nsteps, const double* schedule, const double* T0, const double* obs,
                         int ckpt, double* loss, double* T_out, int flags, double* elapsed_ms) {
  if (!a || nsteps < 1 || !schedule || !T0 || !obs || ckpt < 1 || !loss)
    return afail(HS2G_ERR_ARG, "hs2g_adjoint_forward: bad argument");
  if (!a->have_params) return afail(HS2G_ERR_STATE, "hs2g_adjoint_forward: parameters not set");
  for (int s = 0; s < nsteps; ++s)
    if (!std::isfinite(schedule[s])) return afail(HS2G_ERR_ARG, "hs2g_adjoint_forward: non-finite schedule");
  AGuard guard(a->device);
  cudaStream_t st = a->stream;
  const int64_t n = a->n;
  ckpt = std::min(ckpt, nsteps);
  const int64_t nck = (nsteps + ckpt - 1) / ckpt;
  a->nsteps = 0;
  cudaError_t e = cudaStreamSynchronize(st);  // buffers may be reallocated below
  if (e == cudaSuccess) e = grow(&a->obs, &a->obs_cap, (int64_t)nsteps * a->nobs_step);
  if (e == cudaSuccess) e = grow(&a->ckpts, &a->ckpt_cap, nck * n);
  if (e == cudaSuccess) e = grow(&a->parts, &a->parts_cap, (int64_t)2 * hs2g::kMisfitBlocks * nsteps * a->ninst);
  if (e != cudaSuccess) return acuda(e, "hs2g_adjoint_forward: device allocation");
  std::vector<hs2g::AInst> inst = a->host_inst;
  for (auto& in : inst) in.obs_off *= nsteps;
  e = cudaMemcpyAsync(a->inst, inst.data(), sizeof(hs2g::AInst) * a->ninst, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(a->obs, obs, sizeof(double) * nsteps * a->nobs_step, in_kind(flags), st);
  if (e == cudaSuccess) e = copy_in(a, a->T, T0, in_kind(flags), a->mu[0], st);
  if (e == cudaSuccess) e = cudaEventRecord(a->ev0, st);
  a->sched.assign(schedule, schedule + nsteps);
  a->stored_from = -1;
  // The states of the last two segments (T, y0, y1, y2 of each step, the layout the recompute writes) go straight into
  // the two stores, which the backward pass sweeps first, when the stores already exist from an earlier backward pass:
  // that pass then recomputes neither.  The same kernels compute the same states, so the gradients do not change.
  // (With the last segment alone, six instances of 5.86 million voxels, 40 steps in segments of 10: 41.3 ms; with both
  // 39.2.)
  const int64_t seg_need = (int64_t)ckpt * 4 * n;
  double* stores[2] = {a->seg, a->seg2};
  int64_t from = nck;
  if (a->seg && a->seg_cap >= seg_need && (nck == 1 || (a->seg2 && a->seg2_cap >= seg_need)))
    from = std::max<int64_t>(0, nck - 2);
  const hs2g::AView v = view(a);
  for (int s = 0; s < nsteps && e == cudaSuccess; ++s) {
    const int sg = s / ckpt, j = s - sg * ckpt;
    const bool kept = sg >= from;
    double* slot = kept ? stores[sg & 1] + (int64_t)j * 4 * n : nullptr;
    if (j == 0) {
      e = cudaMemcpyAsync(a->ckpts + (int64_t)sg * n, a->T, sizeof(double) * n, cudaMemcpyDeviceToDevice, st);
      if (kept && e == cudaSuccess) e = cudaMemcpyAsync(slot, a->T, sizeof(double) * n, cudaMemcpyDeviceToDevice, st);
    }
    if (e != cudaSuccess) break;
    if (kept)  // a segment's last state goes back to T
      e = fwd_step(a, st, slot, j + 1 < ckpt && s + 1 < nsteps ? slot + 4 * n : a->T, slot + n, slot + 2 * n,
                   slot + 3 * n, true, a->sched[s], s);
    else       // the adjoint buffers are free during the forward pass and hold the increments
      e = fwd_step(a, st, a->T, a->T, a->mu[0], a->mu[1], a->mu[2], false, a->sched[s], s);
  }
  for (int s = 0; s < nsteps && e == cudaSuccess; s += 65535) {  // a launch's limit on z
    hs2g::adj_misfit_kernel<<<dim3(hs2g::kMisfitBlocks, a->ninst, std::min(nsteps - s, 65535)), 256, 0, st>>>(
        v, a->obs, (int64_t)s, a->parts);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaEventRecord(a->ev1, st);
  std::vector<double> parts((size_t)2 * hs2g::kMisfitBlocks * nsteps * a->ninst);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(parts.data(), a->parts, sizeof(double) * parts.size(), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess && T_out) e = copy_out(a, T_out, a->T, out_kind(flags), a->mu[0], st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return acuda(e, "hs2g_adjoint_forward");
  read_elapsed(a, elapsed_ms);
  for (int i = 0; i < a->ninst; ++i) {  // Neumaier sum of the per-step, per-block pairs
    double acc = 0.0, comp = 0.0;
    for (int s = 0; s < nsteps; ++s)
      for (int h = 0; h < 2 * hs2g::kMisfitBlocks; ++h) {
        const double v = parts[2 * ((size_t)s * a->ninst + i) * hs2g::kMisfitBlocks + h];
        const double t = acc + v;
        comp += std::fabs(acc) >= std::fabs(v) ? (acc - t) + v : (v - t) + acc;
        acc = t;
      }
    loss[i] = acc + comp;
  }
  a->nsteps = nsteps;
  a->ckpt = ckpt;
  a->stored_from = from < nck ? (int)from : -1;
  return HS2G_OK;
}

int hs2g_adjoint_backward(hs2g_adjoint* a, double* gk, double* gC, double* gq, double* gT0, int flags,
                          double* elapsed_ms) {
  if (!a || !gk || !gC || !gq) return afail(HS2G_ERR_ARG, "hs2g_adjoint_backward: null argument");
  if (a->nsteps < 1) return afail(HS2G_ERR_STATE, "hs2g_adjoint_backward: no forward pass to differentiate");
  AGuard guard(a->device);
  cudaStream_t st = a->stream;
  const hs2g::AView v = view(a);
  const int64_t n = a->n;
  const int N = a->nsteps, C = a->ckpt;
  // the segment stores (T, y0, y1, y2 of ckpt steps) exist only while gradients are taken; with two of them
  // the recompute of segment sg-1 (rec_stream) runs while segment sg is swept backwards (the handle's stream)
  cudaError_t e = grow(&a->seg, &a->seg_cap, (int64_t)C * 4 * n);
  if (e != cudaSuccess) return acuda(e, "hs2g_adjoint_backward: device allocation");
  const int nseg = (N + C - 1) / C;
  bool dbl = false;
  if (nseg > 1) {
    dbl = grow(&a->seg2, &a->seg2_cap, (int64_t)C * 4 * n) == cudaSuccess;
    if (!dbl) cudaGetLastError();  // out of memory for the second store: recompute and sweep in turn
  }
  double* bufs[2] = {a->seg, dbl ? a->seg2 : a->seg};
  // the last forward pass may have left the last segments in the stores (see hs2g_adjoint_forward)
  const int from = a->stored_from >= 0 && (nseg == 1 || dbl) ? a->stored_from : nseg;
  a->stored_from = -1;
  e = cudaEventRecord(a->ev0, st);
  double* zero_list[] = {a->gg[0], a->gg[1], a->gg[2], a->gM, a->gq};
  for (double* p : zero_list)
    if (e == cudaSuccess) e = cudaMemsetAsync(p, 0, sizeof(double) * n, st);
  if (e == cudaSuccess) {
    hs2g::adj_seed_kernel<<<nblk(n), kTh, 0, st>>>(v, a->obs, N - 1, a->lam);
    e = cudaGetLastError();
  }
  cudaStream_t rs = dbl ? a->rec_stream : st;
  if (e == cudaSuccess && dbl) e = cudaEventRecord(a->ev_start, st);  // checkpoints and parameters are ready
  if (e == cudaSuccess && dbl) e = cudaStreamWaitEvent(rs, a->ev_start, 0);
  // recompute segment sg into its store: slot j holds T, y0, y1, y2 of step s0 + j (the end state is not kept)
  auto recompute = [&](int sg) -> cudaError_t {
    const int s0 = sg * C, s1 = std::min(N, s0 + C);
    double* buf = bufs[sg & 1];
    cudaError_t r = cudaMemcpyAsync(buf, a->ckpts + (int64_t)sg * n, sizeof(double) * n, cudaMemcpyDeviceToDevice, rs);
    for (int s = s0; s < s1 && r == cudaSuccess; ++s) {
      double* slot = buf + (int64_t)(s - s0) * 4 * n;
      double* next = s + 1 < s1 ? slot + 4 * n : nullptr;
      r = fwd_step(a, rs, slot, next, slot + n, slot + 2 * n, slot + 3 * n, true, a->sched[s], -1);
    }
    if (r == cudaSuccess && dbl) r = cudaEventRecord(a->ev_rec[sg & 1], rs);
    return r;
  };
  if (e == cudaSuccess && from == nseg) e = recompute(nseg - 1);
  for (int sg = nseg - 1; sg >= 0 && e == cudaSuccess; --sg) {
    if (dbl && sg >= 1 && sg - 1 < from) {
      // store (sg-1)&1 was last read by the sweep of segment sg+1
      e = cudaStreamWaitEvent(rs, a->ev_done[(sg - 1) & 1], 0);
      if (e == cudaSuccess) e = recompute(sg - 1);
    }
    if (e == cudaSuccess && dbl && sg < from) e = cudaStreamWaitEvent(st, a->ev_rec[sg & 1], 0);
    const int s0 = sg * C, s1 = std::min(N, s0 + C);
    const double* buf = bufs[sg & 1];
    for (int s = s1 - 1; s >= s0 && e == cudaSuccess; --s) {
      const double* slot = buf + (int64_t)(s - s0) * 4 * n;
      // T_s (s >= 1) is the state observed after step s - 1
      e = bwd_step(a, slot, slot + n, slot + 2 * n, slot + 3 * n, a->sched[s], s >= 1 ? s - 1 : -1);
    }
    if (e == cudaSuccess && dbl) e = cudaEventRecord(a->ev_done[sg & 1], st);
    if (e == cudaSuccess && !dbl && sg >= 1) e = recompute(sg - 1);
  }
  if (e == cudaSuccess) {
    if (a->forms)
      hs2g::adj_chain_faces_kernel<<<nblk(n), kTh, 0, st>>>(v, a->gg[0], a->gg[1], a->gg[2], a->gM, 2.0 / a->dt,
                                                            a->fcls, a->nclass, a->forms, a->fixed, a->mu[0],
                                                            a->mu[1], a->gq);
    else
      hs2g::adj_chain_kernel<<<nblk(n), kTh, 0, st>>>(v, a->gg[0], a->gg[1], a->gg[2], a->gM, 2.0 / a->dt,
                                                      a->mu[0], a->mu[1]);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaEventRecord(a->ev1, st);
  const cudaMemcpyKind kind = out_kind(flags);
  if (e == cudaSuccess) e = copy_out(a, gk, a->mu[0], kind, a->mu[2], st);
  if (e == cudaSuccess) e = copy_out(a, gC, a->mu[1], kind, a->mu[2], st);
  if (e == cudaSuccess) e = copy_out(a, gq, a->gq, kind, a->mu[2], st);
  if (e == cudaSuccess && gT0) e = copy_out(a, gT0, a->lam, kind, a->mu[2], st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return acuda(e, "hs2g_adjoint_backward");
  read_elapsed(a, elapsed_ms);
  return HS2G_OK;
}

}  // extern "C"
