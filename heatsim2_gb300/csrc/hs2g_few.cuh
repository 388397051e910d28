// Line solves with coefficients per voxel where few lines leave most of the GPU idle (FP64): every CTA of the launch is
// resident at once, so a sweep takes as long as one line's chain.  A CTA of four warps takes 16 lines, both ends of each
// (the factorisation and the lanes of pair_solve and x_solve_lines, the same operations in the same order: the same
// bits).  All four copy a line's operands to shared memory and form the scaled right-hand sides; one then runs the
// recurrences and nothing else, eight rows' loads, eight multiply-adds and eight stores at a time; all four write the
// solution.  A warp that copies and scales between the rows, as pair_solve does, takes twice the cycles per row.
// 32x128x128, lines of 128 rows: y 16.5 -> 14.7 us, x 14.6 -> 13.4 us, x with its scale 18.3 -> 15.7 us; 12x40x44, of 40
// and 44: alike.  (The sweeps of a class problem have one array per voxel and their coefficients in cache: 24x96x128
// was slower so, 40.2 -> 42.5 us per step.)
#pragma once
#include "hs2g_pair.cuh"

namespace hs2g {

constexpr int kFewThreads = 128;
constexpr int kFewRows = 8;  // rows of a block whose operands are in registers

// v_r = fma(c_r, v, w_r) over the rows [0, rows) in the direction DIR (1 up, -1 down), w_r replaced by v_r; row t of this
// lane at w[t * PITCH], c likewise; least: rows that every lane has
template <int PITCH, int DIR>
__device__ __forceinline__ double few_recur(double* w, const double* c, int rows, int least, double v) {
  constexpr int RB = kFewRows;
  const int nb = least / RB, tail = nb * RB;
  auto odd_rows = [&]() {  // the rows past the whole blocks
#pragma unroll 1
    for (int k = 0; k <= least - tail; ++k) {
      const int t = DIR > 0 ? tail + k : least - k;
      if (t < rows) {
        v = fma(c[t * PITCH], v, w[t * PITCH]);
        w[t * PITCH] = v;
      }
    }
  };
  if (DIR < 0) odd_rows();
  if (nb > 0) {
    constexpr int kStep = DIR * PITCH;
    if (DIR < 0) {  // the block's first step is its last row
      w += (tail - 1) * PITCH;
      c += (tail - 1) * PITCH;
    }
    double cc[RB], ww[RB], vv[RB];
#pragma unroll
    for (int k = 0; k < RB; ++k) {
      cc[k] = c[k * kStep];
      ww[k] = w[k * kStep];
    }
#pragma unroll 1
    for (int q = 1; q < nb; ++q) {
      c += RB * kStep;
      double nc[RB], nw[RB];
#pragma unroll
      for (int k = 0; k < RB; ++k) {
        nc[k] = c[k * kStep];
        nw[k] = w[(RB + k) * kStep];
      }
      chain_order();
#pragma unroll
      for (int k = 0; k < RB; ++k) vv[k] = v = chain_fma(cc[k], v, ww[k]);
      chain_order();
#pragma unroll
      for (int k = 0; k < RB; ++k) {
        w[k * kStep] = vv[k];
        cc[k] = nc[k];
        ww[k] = nw[k];
      }
      w += RB * kStep;
    }
#pragma unroll
    for (int k = 0; k < RB; ++k) vv[k] = v = chain_fma(cc[k], v, ww[k]);
    chain_order();
#pragma unroll
    for (int k = 0; k < RB; ++k) w[k * kStep] = vv[k];
    if (DIR > 0) {
      w -= (tail - RB) * PITCH;
      c -= (tail - RB) * PITCH;
    }
  }
  if (DIR > 0) odd_rows();
  return v;
}
// both passes of 16 lines by one warp; rows: this lane's; wm, am, bm the middle row's.  The middle row's solution.
template <int PITCH>
__device__ __forceinline__ double few_chain(double* W, const double* A, const double* B, int rows, int least, bool upper,
                                            double wm, double am, double bm) {
  const int lane = threadIdx.x & 31;
  const double z = few_recur<PITCH, 1>(W + lane, A + lane, rows, least, 0.0);
  const double other = __shfl_xor_sync(0xffffffffu, z, 16);
  const double x = fma(bm, upper ? z : other, fma(am, upper ? other : z, wm));  // the same value in both halves
  few_recur<PITCH, -1>(W + lane, B + lane, rows, least, x);
  return x;
}
// the warp that runs the chain: CTAs that share an SM use FP64 units of their own
__device__ __forceinline__ int few_chain_warp() { return (int)(blockIdx.x / (unsigned)kSMs) & 3; }

// y and z lines, coefficients and scale per voxel (pair_solve with SCALE and without TABLE)
__host__ __device__ constexpr size_t few_smem(int64_t max_len) { return sizeof(double) * 32 * 4 * (size_t)(max_len / 2); }
// Called by every thread of a CTA of kFewThreads.  wait(): for the previous kernel.
template <bool ADD_T, typename WAIT>
__device__ __forceinline__ void few_solve(const PairLines<double>& p, int n, int width, double* smem, WAIT wait) {
  constexpr int kWarps = kFewThreads / 32, RB = kFewRows;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool upper = lane >= 16;
  const int line = lane & 15;
  const bool live = line < width;
  const int mine = live ? line : 0;
  const int m = n >> 1, least = n - 1 - m, rows = upper ? least : m;  // (the lower ends have m, as many or one more)
  double *W = smem, *A = W + m * 32, *B = A + m * 32, *S = B + m * 32;
  const double *a = p.a + mine, *b = p.b + mine;
  auto copy = [&](double* dst, const double* src, int64_t st) {  // the half lines' rows
    const int64_t d = (upper ? -kWarps : kWarps) * st * (int64_t)sizeof(double);
    src += (upper ? n - 1 - warp : warp) * st;
    uint32_t at = (uint32_t)__cvta_generic_to_shared(dst + warp * 32 + lane);
#pragma unroll 4
    for (int t = warp; t < rows; t += kWarps) {
      cp_async_bytes<8>(at, src);
      at += kWarps * 32 * sizeof(double);
      src = step_bytes(src, d);
    }
  };
  const bool chain = warp == few_chain_warp();
  double wm = 0, am = 0, bm = 0;
  copy(A, a, p.cst);
  copy(B, b, p.cst);
  copy(S, p.sc + mine, p.wst);
  if (chain) {
    am = a[m * p.cst];
    bm = b[m * p.cst];
  }
  wait();
  copy(W, p.W + mine, p.wst);
  if (chain) {
    wm = p.W[m * p.wst + mine] * p.sc[m * p.wst + mine];
  }
  cp_async_commit_group();
  cp_async_wait_pending<0>();
#pragma unroll 4
  for (int t = warp; t < rows; t += kWarps) W[t * 32 + lane] *= S[t * 32 + lane];
  __syncthreads();
  const int64_t s = upper ? n - 1 : 0, dT = upper ? -p.st : p.st, dX = upper ? -p.wst : p.wst;
  const double* T = ADD_T ? p.T + s * p.st + mine : nullptr;
  double* out = p.out + s * p.st + mine;
  double* X = ADD_T && p.X ? p.X + s * p.wst + mine : nullptr;
  double tt[RB];
  auto load_t = [&](int t0) {  // the temperatures of this warp's next rows
#pragma unroll
    for (int k = 0; k < RB; ++k)
      if (t0 + k * kWarps < rows) tt[k] = T[(t0 + k * kWarps) * dT];
  };
  auto plus = [](double t, double x) { return fma(2.0, x, t); };
  if (chain) {
    const double tm = ADD_T ? p.T[m * p.st + mine] : 0.0;
    const double x = few_chain<32>(W, A, B, rows, least, upper, wm, am, bm);
    if (!upper && live) {
      p.out[m * p.st + mine] = ADD_T ? plus(tm, x) : x;
      if (ADD_T && p.X) p.X[m * p.wst + mine] = x;
    }
  } else if (ADD_T) {
    load_t(warp);
  }
  __syncthreads();
  if (ADD_T && chain) load_t(warp);
  for (int t0 = warp; t0 < rows; t0 += RB * kWarps) {
#pragma unroll
    for (int k = 0; k < RB; ++k) {
      const int t = t0 + k * kWarps;
      if (t < rows && live) {
        const double x = W[t * 32 + lane];
        out[t * dT] = ADD_T ? plus(tt[k], x) : x;
        if (ADD_T && X) X[t * dX] = x;
      }
    }
    if (ADD_T) load_t(t0 + RB * kWarps);
  }
}

// x lines: y = A_x^-1 (in sc) (SCALE) or in place, coefficients per voxel; element (line l, column c) of the right-hand
// sides is in * sc, row pitch px.  Rows of 33 elements: a line's columns go to different banks.
template <bool SCALE>
__host__ __device__ constexpr size_t few_x_smem(int64_t max_nx) {
  return sizeof(double) * 33 * (size_t)((SCALE ? 4 : 3) * (max_nx / 2));
}
template <bool SCALE, typename WAIT>
__device__ __forceinline__ void few_x_solve(const double* in, const double* sc, const double* a, const double* b,
                                            double* y, int64_t px, int n, int count, double* smem, WAIT wait) {
  constexpr int kWarps = kFewThreads / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int m = (n - 1) / 2, most = n - 1 - m;  // columns of the left ends, of the right ends (as many or one more)
  double *W = smem, *A = W + most * 33, *B = A + most * 33, *S = B + most * 33;
  auto each = [&](auto f) {  // f(offset from the first line's first column, shared memory slot), the middle column left out
    for (int l = warp; l < count; l += kWarps)
      for (int c = lane; c < n; c += 32)
        if (c != m) f(l * px + c, c < m ? c * 33 + l : (n - 1 - c) * 33 + 16 + l);
  };
  auto copy = [&](double* dst, const double* src) {
    each([&](int64_t g, int at) { cp_async_bytes<8>((uint32_t)__cvta_generic_to_shared(dst + at), src + g); });
  };
  const bool chain = warp == few_chain_warp(), upper = lane >= 16;
  const int64_t mid = (int64_t)min(lane & 15, count - 1) * px + m;
  double wm = 0, am = 0, bm = 0;
  copy(A, a);
  copy(B, b);
  if (SCALE) copy(S, sc);
  if (chain) {
    am = a[mid];
    bm = b[mid];
  }
  wait();
  copy(W, in);
  if (chain) {
    wm = in[mid];
    if (SCALE) wm *= sc[mid];
  }
  cp_async_commit_group();
  cp_async_wait_pending<0>();
  if (SCALE) each([&](int64_t, int at) { W[at] *= S[at]; });
  __syncthreads();
  if (chain) {
    const double x = few_chain<33>(W, A, B, upper ? most : m, m, upper, wm, am, bm);
    if ((lane & 15) < count && !upper) y[mid] = x;
  }
  __syncthreads();
  each([&](int64_t g, int at) { y[g] = W[at]; });
}

// Whether a launch over `groups` 16-line groups takes these kernels: every CTA resident at once, at most four to an SM,
// a chain for each of its FP64 units.
inline bool few_lines(int64_t groups, size_t smem) {
  const int64_t per = (int64_t)(227 * 1024 / (smem + 1024));
  return groups <= kSMs * (per < 4 ? per : 4);
}

}  // namespace hs2g
