// Setup-time kernels: the coefficient compiler (class arrays -> per-face conductances) and the per-line
// tridiagonal factorisations that turn conductances (shared per face, or per row in the curved-surface mode)
// and capacities into the step coefficients.
//
// Replaces the reference's Python voxel loop and symbolic assembly (crank_nicolson.pyx:272-491,
// alternatingdirection_c.c:102-199) and its LU factorisation at finalize (tridiag.pyx:9-43,
// alternatingdirection_c_pyx.pyx:279).  All FP64.  One thread per face (compiler) or per grid line (LU).
#include <algorithm>
#include <climits>

#include "hs2g_internal.cuh"
#include "hs2g_x.cuh"

namespace hs2g {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ double eval_form(const double* f, const double* klo, const double* khi) {
  double acc = f[0];
#pragma unroll
  for (int e = 0; e < HS2G_K_ENTRIES; ++e) {
    const double cl = f[1 + e];
    const double ch = f[1 + HS2G_K_ENTRIES + e];
    if (cl != 0.0) acc += cl * klo[e];
    if (ch != 0.0) acc += ch * khi[e];
  }
  return acc;
}

// The conductance and error code (0: none) that class b gives a face between materials of the tables mlo and mhi (the
// voxel below and above it; nmat: outside the grid) on `axis`; exterior: it has a side outside the grid.
struct FaceValue {
  double g;
  int code;
};
__device__ FaceValue face_value(const hs2g_material* __restrict__ mats, int nmat, const hs2g_face_form& form, int mlo,
                                int mhi) {
  const bool lo_c = mlo < nmat && mats[mlo].kind == HS2G_TEMPERATURE_COMPUTE;
  const bool hi_c = mhi < nmat && mats[mhi].kind == HS2G_TEMPERATURE_COMPUTE;
  if (!lo_c && !hi_c) return {0.0, 0};
  const double* klo = lo_c ? mats[mlo].k : mats[mhi].k;
  const double* khi = hi_c ? mats[mhi].k : mats[mlo].k;
  const double g = eval_form(form.normal, klo, khi);
  if (!(g == g) || isinf(g)) return {0.0, HS2G_ERR_KTYPE};
  const double tol = 1e-12 * fabs(g);
  int code = 0;
  for (int z = 0; z < form.nzero; ++z) {
    const double v = eval_form(form.zero[z], klo, khi);
    if (!(fabs(v) <= tol) && code == 0) code = form.zero_code[z];
  }
  if (code == 0 && (mlo >= nmat || mhi >= nmat) && g != 0.0) code = HS2G_ERR_EXTERIOR;
  return {g, code};
}
// The values of every (axis, class, low material, high material), nmat standing for outside the grid: one thread each.
__global__ void face_values_kernel(const hs2g_material* __restrict__ mats, int nmat,
                                   const hs2g_face_form* __restrict__ forms, int nbnd, FaceValue* __restrict__ table) {
  const int m1 = nmat + 1, n = nbnd * m1 * m1, axis = blockIdx.y;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
    table[axis * n + t] = face_value(mats, nmat, forms[t / (m1 * m1) * 3 + axis], t / m1 % m1, t % m1);
}

// One thread per face of `axis`.  The two voxels that meet at a face are lo (index - 1 along the axis) and hi.
// A face only matters to the compute voxels beside it; the reference evaluates its flux from a compute
// voxel's equation with the neighbour's k replaced by the voxel's own when the neighbour is fixed or outside
// the grid (crank_nicolson.pyx:298-338), so both compute sides see the same k pair and one value per face
// serves both.  table: face_values_kernel's, or null when there are too many classes and materials for one (each face's
// forms evaluated in its own thread take 20 times as long: 6.5 ms against 0.3 ms per axis at 65x512x512).
__global__ void faces_kernel(Dims d, int axis, const uint8_t* __restrict__ material,
                             const uint8_t* __restrict__ bclass, const hs2g_material* __restrict__ mats, int nmat,
                             const hs2g_face_form* __restrict__ forms, int nbnd, const FaceValue* __restrict__ table,
                             double* __restrict__ G, unsigned long long* err) {
  const int64_t fz = d.nz + (axis == 0), fy = d.ny + (axis == 1), fx = d.nx + (axis == 2);
  const int64_t nfaces = fz * fy * fx;
  const int64_t n_axis = axis == 0 ? d.nz : (axis == 1 ? d.ny : d.nx);
  const int64_t back = axis == 0 ? d.nxy() : (axis == 1 ? d.nx : 1);  // from a face's hi voxel to its lo voxel
  for (int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; f < nfaces;
       f += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = f / fx, i = f - row * fx, k = row / fy, j = row - k * fy;
    const int64_t c = axis == 0 ? k : (axis == 1 ? j : i);
    const int64_t p = (k * d.ny + j) * d.nx + i;  // the hi voxel's place
    int mlo = nmat, mhi = nmat;
    if (c > 0) mlo = material[p - back];
    if (c < n_axis) mhi = material[p];
    if ((c > 0 && mlo >= nmat) || (c < n_axis && mhi >= nmat)) {
      record_error(err, HS2G_ERR_ARG, axis, f);
      G[f] = 0.0;
      continue;
    }
    const int b = bclass[f];
    if (b >= nbnd) {
      // no class of the table: an error unless the face lies between voxels that are not computed
      if ((mlo < nmat && mats[mlo].kind == HS2G_TEMPERATURE_COMPUTE) ||
          (mhi < nmat && mats[mhi].kind == HS2G_TEMPERATURE_COMPUTE))
        record_error(err, HS2G_ERR_ARG, axis, f);
      G[f] = 0.0;
      continue;
    }
    const FaceValue v = table ? table[(b * (nmat + 1) + mlo) * (nmat + 1) + mhi]
                              : face_value(mats, nmat, forms[b * 3 + axis], mlo, mhi);
    if (v.code) record_error(err, v.code, axis, f);
    G[f] = v.g;
  }
}

// Per-voxel capacity M = rho*c/dt for computed voxels, 1 for fixed ones (their rows are the identity).
__global__ void capacity_kernel(Dims d, const uint8_t* __restrict__ material, const hs2g_material* __restrict__ mats,
                                int nmat, double* __restrict__ M, uint8_t* __restrict__ compute,
                                unsigned long long* err) {
  const int64_t n = d.nvox();
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
    const int m = material[p];
    if (m >= nmat) {
      record_error(err, HS2G_ERR_ARG, 3, p);
      M[p] = 1.0;
      compute[p] = 0;
      continue;
    }
    const bool c = mats[m].kind == HS2G_TEMPERATURE_COMPUTE;
    const double cap = mats[m].capacity;
    if (c && !(cap > 0.0 && cap < INFINITY)) record_error(err, HS2G_ERR_CAPACITY, 3, p);
    M[p] = c ? cap : 1.0;
    compute[p] = c ? 1 : 0;
  }
}

// Dense problems: capacities arrive per voxel; check them and that computed voxels have no exterior flux.
__global__ void validate_dense_kernel(Dims d, const double* __restrict__ Gz, const double* __restrict__ Gy,
                                      const double* __restrict__ Gx, double* __restrict__ M,
                                      uint8_t* __restrict__ compute, unsigned long long* err) {
  const int64_t n = d.nvox();
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = p % d.nx, j = (p / d.nx) % d.ny, k = p / d.nxy();
    if (!compute[p]) {
      M[p] = 1.0;
      continue;
    }
    const double cap = M[p];
    if (!(cap > 0.0 && cap < INFINITY)) record_error(err, HS2G_ERR_CAPACITY, 3, p);
    const double gzl = Gz[(k * d.ny + j) * d.nx + i], gzh = Gz[((k + 1) * d.ny + j) * d.nx + i];
    const double gyl = Gy[(k * (d.ny + 1) + j) * d.nx + i], gyh = Gy[(k * (d.ny + 1) + j + 1) * d.nx + i];
    const double gxl = Gx[(k * d.ny + j) * (d.nx + 1) + i], gxh = Gx[(k * d.ny + j) * (d.nx + 1) + i + 1];
    if ((k == 0 && gzl != 0.0) || (k == d.nz - 1 && gzh != 0.0)) record_error(err, HS2G_ERR_EXTERIOR, 0, p);
    if ((j == 0 && gyl != 0.0) || (j == d.ny - 1 && gyh != 0.0)) record_error(err, HS2G_ERR_EXTERIOR, 1, p);
    if ((i == 0 && gxl != 0.0) || (i == d.nx - 1 && gxh != 0.0)) record_error(err, HS2G_ERR_EXTERIOR, 2, p);
    const double all = gzl + gzh + gyl + gyh + gxl + gxh;
    if (!(all == all) || isinf(all)) record_error(err, HS2G_ERR_ARG, 3, p);
  }
}

// ---------------------------------------------------------------------------------------------------------
// Per-line LU of the stage matrices (M - G/2 along the stage axis), in the reference's row order and
// normalisation (tridiag.pyx:25-41): piv_r = d_r - u_{r-1}*lo_r, u_r = hi_r/piv_r, with
// d = M + (G_lo+G_hi)/2, lo = -G_lo/2, hi = -G_hi/2 for computed voxels and the identity row for fixed ones.
//
// The step is the Douglas scheme in delta form,
//     (M - Lx/2) dT0 = L T + Q,   (M - Ly/2) dT1 = M dT0,   (M - Lz/2) dT2 = M dT1,   T' = T + dT2,
// which equals the reference's stage equations (alternatingdirection_c_pyx.pyx:483-493 with
// crank_subst_in_groups) exactly in real arithmetic.  Each stage's output is pre-multiplied by the diagonal
// scale the next stage's forward sweep applies to its input, so the y and z sweeps are one FMA per
// forward and back step:
//     s2 = M/piv2,  sigma = s2*M/piv1,   W0 = sigma*dT0,   W1 = s2*dT1.
// ---------------------------------------------------------------------------------------------------------
struct RowIn {
  double d, lo, hi;
};

__device__ __forceinline__ RowIn stage_row(bool comp, double M, double gl, double gh) {
  RowIn r;
  r.d = comp ? M + 0.5 * (gl + gh) : 1.0;
  r.lo = comp ? -(0.5 * gl) : 0.0;
  r.hi = comp ? -(0.5 * gh) : 0.0;
  return r;
}

// The six face conductances of voxel p as its own row sees them.  SharedFaces: one array per axis indexed by
// face, so the two rows of a face see the same value (the class and dense problems).  RowFaces: six
// (nz, ny, nx) arrays, one value per row and side, so a face may weigh differently in its two rows (the
// reference's curved-surface mode, where each row uses its own cell's edge lengths).
struct SharedFaces {
  const double *Gz, *Gy, *Gx;
  __device__ double zlo(const Dims& d, int64_t p, int64_t, int64_t, int64_t) const { return Gz[p]; }
  __device__ double zhi(const Dims& d, int64_t p, int64_t, int64_t, int64_t) const { return Gz[p + d.nxy()]; }
  __device__ double ylo(const Dims& d, int64_t, int64_t k, int64_t j, int64_t i) const {
    return Gy[(k * (d.ny + 1) + j) * d.nx + i];
  }
  __device__ double yhi(const Dims& d, int64_t, int64_t k, int64_t j, int64_t i) const {
    return Gy[(k * (d.ny + 1) + j + 1) * d.nx + i];
  }
  __device__ double xlo(const Dims& d, int64_t, int64_t k, int64_t j, int64_t i) const {
    return Gx[(k * d.ny + j) * (d.nx + 1) + i];
  }
  __device__ double xhi(const Dims& d, int64_t, int64_t k, int64_t j, int64_t i) const {
    return Gx[(k * d.ny + j) * (d.nx + 1) + i + 1];
  }
};
struct RowFaces {
  const double *zl, *zh, *yl, *yh, *xl, *xh;
  __device__ double zlo(const Dims&, int64_t p, int64_t, int64_t, int64_t) const { return zl[p]; }
  __device__ double zhi(const Dims&, int64_t p, int64_t, int64_t, int64_t) const { return zh[p]; }
  __device__ double ylo(const Dims&, int64_t p, int64_t, int64_t, int64_t) const { return yl[p]; }
  __device__ double yhi(const Dims&, int64_t p, int64_t, int64_t, int64_t) const { return yh[p]; }
  __device__ double xlo(const Dims&, int64_t p, int64_t, int64_t, int64_t) const { return xl[p]; }
  __device__ double xhi(const Dims&, int64_t p, int64_t, int64_t, int64_t) const { return xh[p]; }
};

// z lines (one thread per (j,i)): stage-2 coefficients and s2.  The y and z lines are eliminated from both ends
// towards the middle row m = n/2 (hs2g_pair.cuh): below it a = lo/piv, b = hi/piv, above it the same with lo and
// hi exchanged, and the middle row keeps both couplings, a = lo/piv and b = hi/piv.  The two ends advance in one
// loop, so their divisions overlap.  One way (the FP32 batch, two_ended false): m is the last row, which has no
// upper neighbour.
template <class F>
__global__ void factor_z_kernel(Dims d, F g, const double* __restrict__ M, const uint8_t* __restrict__ compute,
                                double* __restrict__ s2, double* __restrict__ a2, double* __restrict__ b2,
                                int64_t px, bool two_ended) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= d.nxy()) return;
  const int64_t j = t / d.nx, i = t - j * d.nx;
  const int64_t m = two_ended ? d.nz / 2 : d.nz - 1;
  auto at2 = [&](int64_t k) { return (k * d.ny + j) * px + i; };  // a2 / b2 row pitch
  auto row = [&](int64_t k) {
    const int64_t p = k * d.nxy() + t;
    const bool comp = compute[p] != 0;
    return stage_row(comp, M[p], comp ? g.zlo(d, p, k, j, i) : 0.0, comp ? g.zhi(d, p, k, j, i) : 0.0);
  };
  double u = 0.0, v = 0.0;  // upper factor of the last eliminated row at each end
  auto up = [&](int64_t k) {
    const int64_t p = k * d.nxy() + t;
    const RowIn r = row(k);
    const double piv = r.d - u * r.lo;
    u = r.hi / piv;
    a2[at2(k)] = -(r.lo / piv);
    b2[at2(k)] = -(u);
    s2[p] = M[p] / piv;
  };
  auto down = [&](int64_t k) {
    const int64_t p = k * d.nxy() + t;
    const RowIn r = row(k);
    const double piv = r.d - v * r.hi;
    v = r.lo / piv;
    a2[at2(k)] = -(r.hi / piv);
    b2[at2(k)] = -(v);
    s2[p] = M[p] / piv;
  };
  for (int64_t e = 0; e < m; ++e) {
    up(e);
    if (d.nz - 1 - e > m) down(d.nz - 1 - e);
  }
  const int64_t p = m * d.nxy() + t;
  const RowIn r = row(m);
  const double piv = r.d - u * r.lo - v * r.hi;
  a2[at2(m)] = -(r.lo / piv);
  b2[at2(m)] = -(r.hi / piv);
  s2[p] = M[p] / piv;
}

// y lines (one thread per (k,i)): stage-1 coefficients and sigma.
template <class F>
__global__ void factor_y_kernel(Dims d, F g, const double* __restrict__ M, const uint8_t* __restrict__ compute,
                                const double* __restrict__ s2, double* __restrict__ sigma, double* __restrict__ a1,
                                double* __restrict__ b1, int64_t px, bool two_ended) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= d.nz * d.nx) return;
  const int64_t k = t / d.nx, i = t - k * d.nx;
  const int64_t m = two_ended ? d.ny / 2 : d.ny - 1;
  auto at = [&](int64_t j) { return (k * d.ny + j) * d.nx + i; };
  auto row = [&](int64_t j) {
    const int64_t p = at(j);
    const bool comp = compute[p] != 0;
    return stage_row(comp, M[p], comp ? g.ylo(d, p, k, j, i) : 0.0, comp ? g.yhi(d, p, k, j, i) : 0.0);
  };
  // W1 carries the scale s2, so a row's couplings are scaled by its own s2 and the neighbour's is divided out; f:
  // the coupling, q: the pivot where it is still to be divided by it
  auto lower = [&](int64_t j, double f, double q) { return j > 0 ? s2[at(j)] * f / (q * s2[at(j - 1)]) : 0.0; };
  auto upper = [&](int64_t j, double f, double q) { return j + 1 < d.ny ? s2[at(j)] * f / (q * s2[at(j + 1)]) : 0.0; };
  double u = 0.0, v = 0.0;
  auto up = [&](int64_t j) {
    const int64_t pp = (k * d.ny + j) * px + i;  // a1 / b1 row pitch
    const RowIn r = row(j);
    const double piv = r.d - u * r.lo;
    u = r.hi / piv;
    sigma[at(j)] = s2[at(j)] * M[at(j)] / piv;
    a1[pp] = -(lower(j, r.lo, piv));
    b1[pp] = -(upper(j, u, 1.0));
  };
  auto down = [&](int64_t j) {
    const int64_t pp = (k * d.ny + j) * px + i;
    const RowIn r = row(j);
    const double piv = r.d - v * r.hi;
    v = r.lo / piv;
    sigma[at(j)] = s2[at(j)] * M[at(j)] / piv;
    a1[pp] = -(upper(j, r.hi, piv));
    b1[pp] = -(lower(j, v, 1.0));
  };
  for (int64_t e = 0; e < m; ++e) {
    up(e);
    if (d.ny - 1 - e > m) down(d.ny - 1 - e);
  }
  const int64_t pp = (k * d.ny + m) * px + i;
  const RowIn r = row(m);
  const double piv = r.d - u * r.lo - v * r.hi;
  sigma[at(m)] = s2[at(m)] * M[at(m)] / piv;
  a1[pp] = -(lower(m, r.lo, piv));
  b1[pp] = -(upper(m, r.hi, piv));
}

// x lines (one thread per (k,j)): the coefficients a0, b0 and the row scale f0 = sigma/piv of the stage-0 right-hand
// side; two-ended about column x_mid, or one way (m the last column).
template <class F>
__global__ void factor_x_kernel(Dims d, F g, const double* __restrict__ M, const uint8_t* __restrict__ compute,
                                const double* __restrict__ sigma, double* __restrict__ f0, double* __restrict__ a0,
                                double* __restrict__ b0, int64_t px, bool two_ended) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= d.nz * d.ny) return;
  const int64_t k = t / d.ny, j = t - k * d.ny;
  const int64_t m = two_ended ? x_mid(d.nx) : d.nx - 1;
  const double* sg = sigma + t * d.nx;
  auto row = [&](int64_t i) {
    const int64_t p = t * d.nx + i;
    const bool comp = compute[p] != 0;
    return stage_row(comp, M[p], comp ? g.xlo(d, p, k, j, i) : 0.0, comp ? g.xhi(d, p, k, j, i) : 0.0);
  };
  // W0 carries the scale sigma (see factor_y_kernel)
  auto lower = [&](int64_t i, double f, double q) { return i > 0 ? sg[i] * f / (q * sg[i - 1]) : 0.0; };
  auto upper = [&](int64_t i, double f, double q) { return i + 1 < d.nx ? sg[i] * f / (q * sg[i + 1]) : 0.0; };
  double u = 0.0, v = 0.0;
  auto up = [&](int64_t i) {
    const RowIn r = row(i);
    const double piv = r.d - u * r.lo;
    u = r.hi / piv;
    f0[t * d.nx + i] = sg[i] / piv;
    a0[t * px + i] = -(lower(i, r.lo, piv));
    b0[t * px + i] = -(upper(i, u, 1.0));
  };
  auto down = [&](int64_t i) {
    const RowIn r = row(i);
    const double piv = r.d - v * r.hi;
    v = r.lo / piv;
    f0[t * d.nx + i] = sg[i] / piv;
    a0[t * px + i] = -(upper(i, r.hi, piv));
    b0[t * px + i] = -(lower(i, v, 1.0));
  };
  for (int64_t e = 0; e < max(m, d.nx - 1 - m); ++e) {
    if (e < m) up(e);
    if (d.nx - 1 - e > m) down(d.nx - 1 - e);
  }
  const RowIn r = row(m);
  const double piv = r.d - u * r.lo - v * r.hi;
  f0[t * d.nx + m] = sg[m] / piv;
  a0[t * px + m] = -(lower(m, r.lo, piv));
  b0[t * px + m] = -(upper(m, r.hi, piv));
}

// Column `lane` of stencil block b: its row (k, j), column i (past the line's end: none) and voxel.
struct BlockColumn {
  int64_t k, j, i, p;
};
__device__ __forceinline__ BlockColumn block_column(const Dims& d, int64_t nchunks, int64_t b, int lane) {
  int64_t t, k;
  if (d.nz * d.ny * nchunks < ((int64_t)1 << 31)) {  // (64-bit divisions would take most of a setup kernel's time)
    t = (unsigned)b / (unsigned)nchunks;
    k = (unsigned)t / (unsigned)d.ny;
  } else {
    t = b / nchunks;
    k = t / d.ny;
  }
  const int64_t i = (b - t * nchunks) * 32 + lane;
  return {k, t - k * d.ny, i, t * d.nx + i};
}
// What its eight stage-0 coefficients are made of (zeros past the line's end): the six conductances and the row scale;
// blocks are compared by these, without the FP64 unit, whose 12 operations would take the search 200 us of every 262144
// blocks.  And which of its faces are on the grid's exterior (bit f, in the weights' order; 0 past the line's end).
template <class F>
__device__ __forceinline__ void block_parts(const Dims& d, const F& g, const uint8_t* __restrict__ compute,
                                            const double* __restrict__ f0, const BlockColumn& c, double (&v)[7]) {
#pragma unroll
  for (int e = 0; e < 7; ++e) v[e] = 0.0;
  if (c.i >= d.nx || !compute[c.p]) return;
  v[0] = g.xlo(d, c.p, c.k, c.j, c.i);
  v[1] = g.xhi(d, c.p, c.k, c.j, c.i);
  v[2] = g.ylo(d, c.p, c.k, c.j, c.i);
  v[3] = g.yhi(d, c.p, c.k, c.j, c.i);
  v[4] = g.zlo(d, c.p, c.k, c.j, c.i);
  v[5] = g.zhi(d, c.p, c.k, c.j, c.i);
  v[6] = f0[c.p];
}
__device__ __forceinline__ void block_values(const double (&g)[7], double (&v)[8]) {
  const double f = g[6];
  v[0] = f * -(((g[0] + g[1]) + (g[2] + g[3])) + (g[4] + g[5]));
#pragma unroll
  for (int e = 0; e < 6; ++e) v[1 + e] = f * g[e];
  v[7] = f;
}
__device__ __forceinline__ int exterior_faces(const Dims& d, const BlockColumn& c) {
  if (c.i >= d.nx) return 0;
  return (c.i == 0) | (c.i + 1 == d.nx) << 1 | (c.j == 0) << 2 | (c.j + 1 == d.ny) << 3 | (c.k == 0) << 4 |
         (c.k + 1 == d.nz) << 5;
}
// writes a block (one warp); true when two products do for each of its voxels (kXTwoWeights)
template <typename R, bool SHARED>
__device__ __forceinline__ bool store_block(R* blk, int lane, const double (&v)[8], int exterior) {
  bool two = false;
  if constexpr (sizeof(R) == 8 && !SHARED) {
    const double w[6] = {v[1], v[2], v[3], v[4], v[5], v[6]};
    const bool fine = x_own_fine(v[0], w);
    const int hi = __double2hiint(v[0]);
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const long long i = llrint(ldexp(w[f], 62 - (x_own_exponent(hi) - 4)));
      const int lo = (int)(unsigned)i;
      const uint2 wi = make_uint2((unsigned)lo, (unsigned)((i - lo) >> 32));
      if (fine)
        reinterpret_cast<uint2*>(blk)[f * 32 + lane] = wi;
      else
        blk[f * 32 + lane] = w[f];
    }
    int* words = reinterpret_cast<int*>(blk + 6 * 32);
    words[lane] = fine ? hi : kXOwnDoubles;
    words[32 + lane] = __double2loint(v[0]);
    blk[7 * 32 + lane] = v[7];
    return false;
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) blk[c * 32 + lane] = (R)v[c];
  if constexpr (sizeof(R) == 8 && SHARED) {
    double w[6];
#pragma unroll
    for (int f = 0; f < 6; ++f) w[f] = exterior >> f & 1 ? (exterior >> (f ^ 1) & 1 ? 0.0 : v[1 + (f ^ 1)]) : v[1 + f];
    if ((exterior & 3) == 3) w[0] = w[1] = w[3];  // one column: the x weights may be the y weights too, and y's x's
    if ((exterior & 12) == 12) w[2] = w[3] = w[1];
    two = __all_sync(0xffffffffu, w[0] == w[1] && w[0] == w[2] && w[0] == w[3] && w[4] == w[5]);
    uint2 wi[6];
    const int e4 = x_int_weights(w, wi);
    uint2* iw = reinterpret_cast<uint2*>(blk + 8 * 32) + lane;
#pragma unroll
    for (int f = 0; f < 6; ++f) iw[f * 32] = wi[f];
    reinterpret_cast<int*>(blk + 14 * 32)[lane] = e4;
  }
  return two;
}

// Distinct blocks (one warp per block): hashed into an open-addressing table, numbered (hs2g_classes.cu), written once
// each, and every block compared with its owner, bit for bit (a clash of hashes is noted in count[1]).
template <class F>
__global__ void hash_blocks_kernel(Dims d, F g, const uint8_t* __restrict__ compute, const double* __restrict__ f0,
                                   int64_t nchunks, ClassTable t) {
  __shared__ unsigned long long found[8];  // of the CTA's blocks; those alike go to the table as one
  const int64_t b0 = blockIdx.x * (int64_t)8, b = b0 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const BlockColumn col = block_column(d, nchunks, min(b, t.n - 1), lane);
  double v[7];
  block_parts(d, g, compute, f0, col, v);
  unsigned long long h = (unsigned long long)lane * 0xD6E8FEB86659FD93ull + 1 +
                         ((unsigned long long)exterior_faces(d, col) << 40);
#pragma unroll
  for (int c = 0; c < 7; ++c) {
    h = (h ^ (unsigned long long)__double_as_longlong(v[c])) * 0x9E3779B97F4A7C15ull;
    h ^= h >> 29;
  }
  for (int o = 16; o > 0; o >>= 1) h += __shfl_xor_sync(0xffffffffu, h, o);
  h = (h ^ (h >> 32)) * 0x9E3779B97F4A7C15ull;
  if (lane == 0) found[threadIdx.x >> 5] = b >= t.n ? 0 : h ? h : 1;
  __syncthreads();
  if (threadIdx.x >= 8) return;
  t.insert_all(0xffu, found[lane], (int)b0 + lane);
}
// writes the owners' blocks, or (SHARED false) every block at its own place
template <typename R, bool SHARED, class F>
__global__ void write_blocks_kernel(Dims d, F g, const uint8_t* __restrict__ compute, const double* __restrict__ f0,
                                    int64_t nchunks, ClassTable t, R* pool) {
  const int64_t b = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (b >= d.nz * d.ny * nchunks) return;
  if (SHARED && t.owner[t.slot[b]] != (int)b) return;
  const BlockColumn col = block_column(d, nchunks, b, lane);
  double parts[7], v[8];
  block_parts(d, g, compute, f0, col, parts);
  block_values(parts, v);
  const int64_t at = SHARED ? (int64_t)t.id[t.slot[b]] : b;
  const bool two = store_block<R, SHARED>(pool + at * x_block_elems<R, SHARED>(), lane, v, exterior_faces(d, col));
  __syncwarp();
  if (SHARED && two && lane == 0) t.id[t.slot[b]] = (int)at | kXTwoWeights;
}
template <class F>
__global__ void index_blocks_kernel(Dims d, F g, const uint8_t* __restrict__ compute, const double* __restrict__ f0,
                                    int64_t nchunks, ClassTable t, int32_t* bidx) {
  const int64_t b = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (b >= t.n) return;
  const BlockColumn col = block_column(d, nchunks, b, lane), own = block_column(d, nchunks, t.owner[t.slot[b]], lane);
  double v[7], w[7];
  block_parts(d, g, compute, f0, col, v);
  block_parts(d, g, compute, f0, own, w);
  bool eq = exterior_faces(d, col) == exterior_faces(d, own);
#pragma unroll
  for (int c = 0; c < 7; ++c) eq &= __double_as_longlong(v[c]) == __double_as_longlong(w[c]);
  if (!eq) t.count[1] = 1;
  if (lane == 0) bidx[b] = t.id[t.slot[b]];
}

inline int64_t block_count(const Dims& d) { return d.nz * d.ny * ((d.nx + 31) / 32); }
// things are numbered in 32 bits, and the index keeps a bit for kXTwoWeights
inline bool blocks_countable(const Dims& d) { return block_count(d) < ((int64_t)1 << 29); }
inline int64_t searched_lines(const Dims& d, int axis) {
  const int64_t lines = axis == 0 ? d.nz * d.ny : axis == 1 ? d.nz * d.nx : d.nxy();
  return lines < ((int64_t)1 << 29) ? lines : 0;
}

template <typename R, class F>
cudaError_t compress_with(const Dims& d, F g, const uint8_t* compute, const double* f0, const Coeffs& c, bool two_ended,
                          unsigned char* scratch, Compressed* out, cudaStream_t s) {
  const int64_t nch = (d.nx + 31) / 32, blocks = block_count(d);
  const unsigned wgrid = (unsigned)((blocks + 7) / 8);
  const size_t bytes = sizeof(R) * x_block_elems<R, true>(), own_bytes = sizeof(R) * x_block_elems<R, false>();
  LineSearch search{};
  search.grid[0] = {c.a0, c.b0, d.nz * d.ny, 1, c.px, d.nx, 1};
  search.grid[1] = {c.a1, c.b1, d.nz, d.nx, d.ny * c.px, d.ny, c.px};
  search.grid[2] = {c.a2, c.b2, d.ny, d.nx, c.px, d.nz, d.ny * c.px};
  search.mid[0] = two_ended ? x_mid(d.nx) : -1;
  search.mid[1] = search.mid[2] = -1;
  // the lines and the blocks are searched together, their counts read at once, and the checks' outcomes likewise
  int host[4][2] = {};
  auto counts = [&]() {
    return cudaMemcpyAsync(host, search.table[0].count, sizeof host, cudaMemcpyDeviceToHost, s);
  };
  ClassTable t(scratch && blocks_countable(d) ? blocks : 0);
  for (int a = 0; a < 3; ++a) search.table[a] = ClassTable(scratch ? searched_lines(d, a) : 0);
  cudaError_t e = cudaSuccess;
  if (scratch) {
    e = search.begin(scratch, t, s);
    if (e == cudaSuccess && t.n) {
      hash_blocks_kernel<<<wgrid, 256, 0, s>>>(d, g, compute, f0, nch, t);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = search.number(t, s);
    if (e == cudaSuccess) e = counts();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  // An index is worth it when at most a quarter of the blocks are distinct: the sweep then reads them from cache, and the
  // index costs it a dependent load (64x256x512, x sweep with an index and in brackets without: 1/64 of the blocks 162 us
  // [186], 1/16 190 [212], 1/4 193 [210], 1/2 201 [211], all 220 [214]; 37x192x210 1/4 39 [45], all 51 [48])
  XBlocks& x = out->blocks;
  const size_t index = sizeof(int32_t) * (size_t)blocks;
  bool shared = t.n && host[3][0] <= std::max<int64_t>(1, blocks / 4);
  if (e == cudaSuccess && scratch) {
    x.count = shared ? host[3][0] : 0;
    x.bytes = shared ? bytes * x.count + index : 0;
    size_t tables = search.choose({host[0][0], host[1][0], host[2][0]});
    if (tables + x.bytes) e = cudaMalloc(&out->mem, tables + x.bytes);
    if (e == cudaErrorMemoryAllocation && tables) {  // no room for the tables: the arrays stay
      cudaGetLastError();
      tables = search.choose({INT_MAX, INT_MAX, INT_MAX});
      e = shared ? cudaMalloc(&out->mem, x.bytes) : cudaSuccess;
    }
    if (e == cudaSuccess) e = search.finish((unsigned char*)out->mem, out->lines, s);
    if (e == cudaSuccess && shared) {
      x.pool = (unsigned char*)out->mem + tables;
      x.bidx = reinterpret_cast<int32_t*>((unsigned char*)x.pool + bytes * x.count);
      write_blocks_kernel<R, true><<<wgrid, 256, 0, s>>>(d, g, compute, f0, nch, t, (R*)x.pool);
      index_blocks_kernel<<<wgrid, 256, 0, s>>>(d, g, compute, f0, nch, t, x.bidx);
      e = cudaGetLastError();
    }
  }
  if (e == cudaSuccess && scratch) {
    e = counts();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    for (int a = 0; a < 3 && e == cudaSuccess; ++a)
      if (out->lines[a].cls && host[a][1]) out->lines[a] = LineTables{};
    if (e == cudaSuccess && shared && host[3][1]) shared = false;
  }
  if (e == cudaSuccess && !shared) {  // every block for itself
    x = XBlocks{};
    x.count = blocks;
    x.bytes = own_bytes * blocks;
    e = cudaMalloc(&out->own, x.bytes);
    if (e == cudaSuccess) {
      x.pool = out->own;
      write_blocks_kernel<R, false><<<wgrid, 256, 0, s>>>(d, g, compute, f0, nch, ClassTable(), (R*)x.pool);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  if (e != cudaSuccess) out->release();
  return e;
}

// per-row problem: capacities positive and finite, coefficients finite, exterior sides zero on computed
// voxels (the same rules as validate_dense_kernel); fixed voxels get the unit capacity of an identity row
__global__ void validate_rows_kernel(Dims d, RowFaces g, double* __restrict__ M, uint8_t* __restrict__ compute,
                                     unsigned long long* err) {
  const int64_t n = d.nvox();
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = p % d.nx, j = (p / d.nx) % d.ny, k = p / d.nxy();
    if (!compute[p]) {
      M[p] = 1.0;
      continue;
    }
    const double cap = M[p];
    if (!(cap > 0.0 && cap < INFINITY)) record_error(err, HS2G_ERR_CAPACITY, 3, p);
    if ((k == 0 && g.zl[p] != 0.0) || (k == d.nz - 1 && g.zh[p] != 0.0)) record_error(err, HS2G_ERR_EXTERIOR, 0, p);
    if ((j == 0 && g.yl[p] != 0.0) || (j == d.ny - 1 && g.yh[p] != 0.0)) record_error(err, HS2G_ERR_EXTERIOR, 1, p);
    if ((i == 0 && g.xl[p] != 0.0) || (i == d.nx - 1 && g.xh[p] != 0.0)) record_error(err, HS2G_ERR_EXTERIOR, 2, p);
    const double all = g.zl[p] + g.zh[p] + g.yl[p] + g.yh[p] + g.xl[p] + g.xh[p];
    if (!(all == all) || isinf(all)) record_error(err, HS2G_ERR_ARG, 3, p);
  }
}

inline unsigned grid_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > (1 << 20)) b = 1 << 20;
  return (unsigned)b;
}

}  // namespace

size_t face_table_bytes(int nmat, int nbnd) {
  const int64_t entries = (int64_t)nbnd * (nmat + 1) * (nmat + 1);
  return entries <= 65536 ? 3 * sizeof(FaceValue) * (size_t)entries : 0;
}

cudaError_t launch_faces(const Dims& d, const uint8_t* material, const uint8_t* const bclass[3], const hs2g_material* mats,
                         int nmat, const hs2g_face_form* forms, int nbnd, double* const G[3], unsigned long long* err,
                         void* table, cudaStream_t s) {
  FaceValue* values = face_table_bytes(nmat, nbnd) ? static_cast<FaceValue*>(table) : nullptr;
  const int64_t entries = (int64_t)nbnd * (nmat + 1) * (nmat + 1);
  if (values)
    face_values_kernel<<<dim3(grid_for(entries, 64), 3), 64, 0, s>>>(mats, nmat, forms, nbnd, values);
  for (int axis = 0; axis < 3; ++axis) {
    const int64_t nfaces = (d.nz + (axis == 0)) * (d.ny + (axis == 1)) * (d.nx + (axis == 2));
    faces_kernel<<<grid_for(nfaces, kThreads), kThreads, 0, s>>>(d, axis, material, bclass[axis], mats, nmat, forms, nbnd,
                                                                 values ? values + axis * entries : nullptr, G[axis], err);
  }
  return cudaGetLastError();
}

cudaError_t launch_capacity_from_classes(const Dims& d, const uint8_t* material, const hs2g_material* mats,
                                         int nmat, double* M, uint8_t* compute, unsigned long long* err,
                                         cudaStream_t s) {
  capacity_kernel<<<grid_for(d.nvox(), kThreads), kThreads, 0, s>>>(d, material, mats, nmat, M, compute, err);
  return cudaGetLastError();
}

cudaError_t launch_validate_dense(const Dims& d, const double* Gz, const double* Gy, const double* Gx, double* M,
                                  uint8_t* compute, unsigned long long* err, cudaStream_t s) {
  validate_dense_kernel<<<grid_for(d.nvox(), kThreads), kThreads, 0, s>>>(d, Gz, Gy, Gx, M, compute, err);
  return cudaGetLastError();
}

template <class F>
cudaError_t launch_factor_with(const Dims& d, F g, const double* M, const uint8_t* compute, double* s2,
                               double* sigma, const Coeffs& c, cudaStream_t s, bool two_ended) {
  const int th = 128;  // a thread per line, however many there are
  auto ctas = [&](int64_t lines) { return (unsigned)((lines + th - 1) / th); };
  factor_z_kernel<F><<<ctas(d.nxy()), th, 0, s>>>(d, g, M, compute, s2, c.a2, c.b2, c.px, two_ended);
  factor_y_kernel<F><<<ctas(d.nz * d.nx), th, 0, s>>>(d, g, M, compute, s2, sigma, c.a1, c.b1, c.px, two_ended);
  factor_x_kernel<F><<<ctas(d.nz * d.ny), th, 0, s>>>(d, g, M, compute, sigma, s2, c.a0, c.b0, c.px, two_ended);
  return cudaGetLastError();
}

cudaError_t launch_factor(const Dims& d, const Faces& f, const double* M, const uint8_t* compute, double* s2,
                          double* sigma, const Coeffs& c, cudaStream_t s, bool two_ended) {
  if (f.rows[0])
    return launch_factor_with(d, RowFaces{f.rows[0], f.rows[1], f.rows[2], f.rows[3], f.rows[4], f.rows[5]}, M, compute,
                              s2, sigma, c, s, two_ended);
  return launch_factor_with(d, SharedFaces{f.Gz, f.Gy, f.Gx}, M, compute, s2, sigma, c, s, two_ended);
}

void Compressed::release() {
  cudaFree(mem);
  cudaFree(own);
  *this = Compressed{};
}

size_t compress_scratch(const Dims& d) {
  return LineSearch::scratch_bytes({searched_lines(d, 0), searched_lines(d, 1), searched_lines(d, 2)},
                                   blocks_countable(d) ? block_count(d) : 0);
}

cudaError_t compress_coeffs(const Dims& d, const Faces& f, const uint8_t* compute, const double* f0, const Coeffs& c,
                            int precision, unsigned char* scratch, Compressed* out, cudaStream_t s) {
  *out = Compressed{};
  if (f.rows[0])
    return compress_with<double>(d, RowFaces{f.rows[0], f.rows[1], f.rows[2], f.rows[3], f.rows[4], f.rows[5]}, compute,
                                 f0, c, true, scratch, out, s);
  const SharedFaces g{f.Gz, f.Gy, f.Gx};
  return precision == 64 ? compress_with<double>(d, g, compute, f0, c, true, scratch, out, s)
                         : compress_with<float>(d, g, compute, f0, c, false, scratch, out, s);
}

cudaError_t launch_validate_rows(const Dims& d, const double* const rows[6], double* M, uint8_t* compute,
                                 unsigned long long* err, cudaStream_t s) {
  const RowFaces g{rows[0], rows[1], rows[2], rows[3], rows[4], rows[5]};
  validate_rows_kernel<<<grid_for(d.nvox(), kThreads), kThreads, 0, s>>>(d, g, M, compute, err);
  return cudaGetLastError();
}

}  // namespace hs2g
