// Line solves of the y and z sweeps, shared by the plain and the batched form.
//
// FP64 (TWO): every tridiagonal system is factorised from both ends towards its middle row m = n/2
// (hs2g_compile.cu): the rows below m are eliminated upwards, the rows above m downwards, the middle row joins the
// two ends,
//     z_r = W_r - a_r z_{r-1} (r < m),   z_r = W_r - a_r z_{r+1} (r > m),
//     x_m = W_m - a_m z_{m-1} - b_m z_{m+1},
//     x_r = z_r - b_r x_{r+1} (r < m),   x_r = z_r - b_r x_{r-1} (r > m),
// (the coefficients are stored negated) one FMA per row and pass as in a one-way elimination, but two independent
// chains of half the length.  A dependent FP64 FMA takes 64 cycles here and a warp issues one FP64 instruction per 64
// cycles whatever its active lanes, so a warp takes 16 lines: lanes 0-15 their lower ends, lanes 16-31 their upper ends.
// FP32: 32 lines per warp, eliminated one way (m = n); a float chain is not what bounds the sweep.
//
// A warp's lines are neighbours along x in one row of lines, so a row of any array is one contiguous piece.
#pragma once
#include "hs2g_internal.cuh"

namespace hs2g {

constexpr int kPairRows = 8;       // rows per block of a half line
constexpr int kPairMaxWarps = 4;   // warps per CTA (independent of each other)

template <bool TWO>
__host__ __device__ constexpr int pair_lines() {
  return TWO ? 16 : 32;  // lines per warp
}
// blocks a warp keeps in flight ahead of the one in use
template <bool ADD_T>
__host__ __device__ constexpr int pair_ahead() {
  return ADD_T ? 2 : 3;
}

// copy of N bytes to shared memory; 16-byte copies bypass L1, whose few lines beside a full shared memory would
// otherwise bound the bytes in flight
template <int N>
__device__ __forceinline__ void cp_async_bytes(uint32_t d, const void* src) {
  if constexpr (N == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(d), "l"(src), "n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_commit_group() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_pending() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
// p advanced by d bytes
template <typename T>
__device__ __forceinline__ T* step_bytes(T* p, int64_t d) {
  return reinterpret_cast<T*>(reinterpret_cast<uintptr_t>(p) + (uintptr_t)d);
}

// A step of a recurrence, and the end of a run of them: stores between dependent FP64 multiply-adds hold the chain up
// (112 cycles per step against 65 without any; 81 with the next block's loads before a run of eight and its stores after
// it), so a run's stores follow it, in this order.
__device__ __forceinline__ double chain_fma(double a, double b, double c) {
  double d;
  asm volatile("fma.rn.f64 %0, %1, %2, %3;" : "=d"(d) : "d"(a), "d"(b), "d"(c));
  return d;
}
__device__ __forceinline__ float chain_fma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ void chain_order() { asm volatile("" ::: "memory"); }

// The lines of a warp: element addresses of (row 0, first line) and the row strides of the right-hand sides W, the
// temperatures T (read when ADD_T) with the output, the scratch Z of the forward values (unused when KEEP), and the
// coefficients: row-major arrays like W (cls null), or tables of n rows per line class, cls the first line's entry.
template <typename R>
struct PairLines {
  const R* W;
  int64_t wst;
  const R* a;
  const R* b;
  int64_t cst;
  const int32_t* cls;
  const R* T;
  R* out;
  int64_t st;
  R* Z;
  int64_t zst;
  const R* sc;  // SCALE: the right-hand sides are W * sc, laid out like W; ADD_T then adds 2 x to T
  R* X;         // SCALE, ADD_T: x itself is stored here too, unless null (laid out like W; may be Z)
};

// rows of 32 elements a warp holds in shared memory, in whole blocks: with KEEP its half lines' values and (ADD_T) room
// for the temperatures copied ahead, otherwise rings of right-hand sides (forward) or forward values and temperatures
// (back); a ring of coefficients when they come row by row (TABLE false), one of the scale (SCALE)
template <bool TWO, bool ADD_T, bool KEEP, bool TABLE, bool SCALE = false>
__host__ __device__ constexpr int64_t pair_rows_held(int64_t n) {
  return kPairRows *
         (((TABLE ? 0 : 1) + (SCALE ? 1 : 0)) * (pair_ahead<ADD_T>() + 1) +
          (KEEP ? ((TWO ? n / 2 : n) + kPairRows - 1) / kPairRows + (ADD_T ? pair_ahead<ADD_T>() : 0)
                : (pair_ahead<ADD_T>() + 1) * (ADD_T ? 2 : 1)));
}
template <typename R, bool TWO, bool ADD_T, bool KEEP, bool TABLE, bool SCALE = false>
__host__ __device__ constexpr size_t pair_smem(int64_t max_len) {  // per warp
  return sizeof(R) * 32 * (size_t)pair_rows_held<TWO, ADD_T, KEEP, TABLE, SCALE>(max_len);
}

// Copies rows of a warp's lines to shared memory, VEC elements per lane and instruction: a half warp (a warp when
// not TWO) moves VEC rows of its end at once.  The lane's address walks up the rows of its end, or down them.
template <typename R, bool TWO, int VEC>
struct RowCopy {
  static constexpr int kLanes = pair_lines<TWO>() / VEC;  // lanes per row
  const R* at;
  int64_t step;   // bytes per VEC rows
  uint32_t dst;   // the lane's offset (bytes) within a block of rows
  int sub;        // the lane's row among the VEC
  // base: (row 0, first line); t0: local row the lane's walk starts at (its multiple of VEC); width: valid lines
  __device__ __forceinline__ void init(const R* base, int64_t st, int n, bool upper, int lane, int width, int t0,
                                       int dir) {
    const int hl = TWO ? lane & 15 : lane;
    sub = hl / kLanes;
    int c = (hl % kLanes) * VEC;
    dst = (uint32_t)(((upper ? 16 : 0) + c + sub * 32) * sizeof(R));
    if (c >= width) c = 0;  // repeats the first lines (the pad of a row may be read, rows beyond the width not)
    const int64_t r = upper ? (int64_t)n - 1 - (t0 + sub) : (int64_t)t0 + sub;
    at = base + r * st + c;
    step = (upper ? -1 : 1) * dir * (int64_t)VEC * st * (int64_t)sizeof(R);
  }
  // one block, its first row at shared address d; rows q*8 .. of which those below `rows` exist
  template <bool DOWN>
  __device__ __forceinline__ void block(uint32_t d, int q, int rows, bool full) {
    d += dst;
    if (full) {
#pragma unroll
      for (int j = 0; j < kPairRows / VEC; ++j) {
        cp_async_bytes<VEC * (int)sizeof(R)>(d + (uint32_t)((DOWN ? kPairRows / VEC - 1 - j : j) * VEC * 32 * sizeof(R)), at);
        at = step_bytes(at, step);
      }
    } else {
#pragma unroll
      for (int j = 0; j < kPairRows / VEC; ++j) {
        const int jj = DOWN ? kPairRows / VEC - 1 - j : j;
        if (q * kPairRows + jj * VEC + sub < rows)
          cp_async_bytes<VEC * (int)sizeof(R)>(d + (uint32_t)(jj * VEC * 32 * sizeof(R)), at);
        at = step_bytes(at, step);
      }
    }
  }
};

// Solves a warp's lines of n rows (width of them; lanes beyond repeat the first line and store nothing); out = x, or
// T + x with ADD_T (T may be out).  VEC, TVEC: elements per copy of the internal arrays and of T (16 bytes where
// their rows start on 16-byte boundaries, else one element).  What bounds a small grid is the latency of a line's
// chain, so the rows are copied ahead with cp.async and each block's table coefficients are loaded a block ahead.
// KEEP: the right-hand sides land where the forward values replace them and stay until the back pass (the
// temperatures follow into rows the back pass has left); otherwise the forward values go to Z and come back.
template <typename R, bool TWO, bool ADD_T, bool KEEP, bool TABLE, int VEC, int TVEC, bool SCALE = false>
__device__ __forceinline__ void pair_solve(const PairLines<R>& p, int n, int width, R* smem) {
  constexpr int RB = kPairRows, LA = pair_ahead<ADD_T>();
  constexpr int kRing = LA + 1;  // ring blocks
  constexpr uint32_t kBlk = RB * 32 * sizeof(R);
  const int lane = threadIdx.x & 31;
  const bool upper = TWO && lane >= 16;
  const int line = TWO ? lane & 15 : lane;
  const bool live = line < width;
  const int mine = live ? line : 0;
  const int m = TWO ? n >> 1 : n;
  const int least = TWO ? n - 1 - m : n;    // rows of the upper ends; the lower ends have m
  const int rows = upper ? least : m;
  const int nfull = least / RB;             // blocks that every lane fills
  const int nb = nfull + (m > nfull * RB ? 1 : 0);  // and one that some lanes fill in part
  const int left = rows - nfull * RB;
  const int64_t s = upper ? n - 1 : 0;
  // this lane's line of the coefficients: row stride and the address of row s
  const int64_t cst = TABLE ? 1 : p.cst;
  const int64_t co = TABLE ? (int64_t)p.cls[mine] * n : mine;
  const R *A = p.a + co, *B = p.b + co;
  R wm = 0, am = 0, bm = 0, tm = 0;  // the middle row
  if (TWO) {
    wm = p.W[m * p.wst + mine];
    if (SCALE) wm *= p.sc[m * p.wst + mine];
    am = A[m * cst];
    bm = B[m * cst];
    if (ADD_T) tm = p.T[m * p.st + mine];
  }
  constexpr int kRings = (TABLE ? 0 : 1) + (SCALE ? 1 : 0);
  R* col = smem + kRings * kRing * RB * 32 + lane;                           // this lane's column of the rows,
  const R* ccol = smem + lane;                                              // of the coefficient ring
  const R* scol = smem + (kRings - 1) * kRing * RB * 32 + lane;              // and of the scale's
  const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(smem);
  const uint32_t scale_s = ring_s + (kRings - 1) * kRing * kBlk;
  const uint32_t col_s = ring_s + kRings * kRing * kBlk;
  auto slot = [&](int q) { return KEEP ? q : q % kRing; };
  auto tslot = [&](int q) { return KEEP ? q + LA : kRing + q % kRing; };
  RowCopy<R, TWO, VEC> cw, ca, cs;  // right-hand sides (then forward values), coefficients, scale
  RowCopy<R, TWO, TVEC> ct;         // temperatures
  const int back0 = (nb - 1) * RB;
  cw.init(p.W, p.wst, n, upper, lane, width, 0, 1);
  if (!TABLE) ca.init(p.a, p.cst, n, upper, lane, width, 0, 1);
  if (SCALE) cs.init(p.sc, p.wst, n, upper, lane, width, 0, 1);
  if (ADD_T) ct.init(p.T, p.st, n, upper, lane, width, back0 + RB - TVEC, -1);
  // item i of the copy sequence: i < nb the forward blocks, then the back blocks from the last
  auto issue = [&](int i, bool may_turn) {
    if (i < nb) {
      cw.template block<false>(col_s + slot(i) * kBlk, i, rows, i < nfull);
      if (!TABLE) ca.template block<false>(ring_s + (i % kRing) * kBlk, i, rows, i < nfull);
      if (SCALE) cs.template block<false>(scale_s + (i % kRing) * kBlk, i, rows, i < nfull);
    } else if (may_turn && i < 2 * nb) {
      const int q = 2 * nb - 1 - i;
      if (i == nb) {
        if (!TABLE) ca.init(p.b, p.cst, n, upper, lane, width, back0 + RB - VEC, -1);
        if (!KEEP) cw.init(p.Z, p.zst, n, upper, lane, width, back0 + RB - VEC, -1);
      }
      if (!TABLE) ca.template block<true>(ring_s + (i % kRing) * kBlk, q, rows, q < nfull);
      if (!KEEP) cw.template block<true>(col_s + slot(q) * kBlk, q, rows, q < nfull);
      if (ADD_T) ct.template block<true>(col_s + tslot(q) * kBlk, q, rows, q < nfull);
    }
    cp_async_commit_group();
  };
  R next[RB];  // TABLE: the coefficients of the next block
  const int64_t dA = upper ? -1 : 1;
  A += s;
  B += s;
  auto load = [&](const R* c, int q) {
    c += (int64_t)q * RB * dA;
    if (q < nfull) {
#pragma unroll
      for (int k = 0; k < RB; ++k) next[k] = c[k * dA];
    } else {
#pragma unroll
      for (int k = 0; k < RB; ++k)
        if (k < left) next[k] = c[k * dA];
    }
  };
  if (TABLE && nb > 0) load(A, 0);
#pragma unroll 1
  for (int i = 0; i < LA; ++i) issue(i, KEEP);
  const uint64_t keep_l2 = l2_evict_last();  // forward values come back to this warp after its last row
  const int64_t dZ = (upper ? -p.zst : p.zst) * (int64_t)sizeof(R);
  R* Zw = KEEP ? nullptr : p.Z + s * p.zst + mine;
  R z = 0;
#pragma unroll 1
  for (int q = 0; q < nb; ++q) {
    cp_async_wait_pending<LA - 1>();
    __syncwarp();
    R* c = col + slot(q) * (RB * 32);
    const R* cc = ccol + (q % kRing) * (RB * 32);
    R a[RB], w[RB];
#pragma unroll
    for (int k = 0; k < RB; ++k) {
      a[k] = TABLE ? next[k] : cc[k * 32];
      w[k] = SCALE ? c[k * 32] * scol[((q % kRing) * RB + k) * 32] : c[k * 32];
    }
    if (TABLE) load(q + 1 < nb ? A : B, q + 1 < nb ? q + 1 : nb - 1);
    __syncwarp();
    issue(q + LA, KEEP);
    auto put = [&](int k, R v) {
      if (KEEP) {
        c[k * 32] = v;
      } else {
        if (live) st_hint(Zw, v, keep_l2);
        Zw = step_bytes(Zw, dZ);
      }
    };
    if (q < nfull) {
      R v[RB];
#pragma unroll
      for (int k = 0; k < RB; ++k) v[k] = z = chain_fma(a[k], z, w[k]);
      chain_order();
#pragma unroll
      for (int k = 0; k < RB; ++k) put(k, v[k]);
    } else {
#pragma unroll
      for (int k = 0; k < RB; ++k)
        if (k < left) {
          z = fma(a[k], z, w[k]);
          put(k, z);
        }
    }
  }
  auto plus = [](R t, R x) { return SCALE ? fma(R(2), x, t) : t + x; };
  R x = 0;
  if (TWO) {
    const R other = __shfl_xor_sync(0xffffffffu, z, 16);
    x = fma(bm, upper ? z : other, fma(am, upper ? other : z, wm));  // the same value in both halves
    if (!upper && live) {
      p.out[m * p.st + mine] = ADD_T ? plus(tm, x) : x;
      if (SCALE && ADD_T && p.X) p.X[m * p.wst + mine] = x;
    }
  }
  if (!KEEP) {
    cp_async_wait_pending<0>();
    __threadfence();  // the forward values before the copies that read them back from L2
    __syncwarp();
#pragma unroll 1
    for (int i = nb; i < nb + LA; ++i) issue(i, true);
  }
  const int64_t dT = (upper ? -p.st : p.st) * (int64_t)sizeof(R);
  R* oc = step_bytes(p.out + s * p.st + mine, (rows - 1) * dT);
  const int64_t dX = (upper ? -p.wst : p.wst) * (int64_t)sizeof(R);
  R* xc = SCALE && ADD_T && p.X ? step_bytes(p.X + s * p.wst + mine, (rows - 1) * dX) : nullptr;
#pragma unroll 1
  for (int i = nb; i < 2 * nb; ++i) {
    cp_async_wait_pending<LA - 1>();
    __syncwarp();
    const int q = 2 * nb - 1 - i;
    const R *c = col + slot(q) * (RB * 32), *cc = ccol + (i % kRing) * (RB * 32), *tc = col + tslot(q) * (RB * 32);
    R b[RB], zz[RB], tt[RB];
#pragma unroll
    for (int k = 0; k < RB; ++k) {
      b[k] = TABLE ? next[k] : cc[k * 32];
      zz[k] = c[k * 32];
      if (ADD_T) tt[k] = tc[k * 32];
    }
    if (TABLE && q > 0) load(B, q - 1);
    __syncwarp();
    issue(i + LA, true);
    auto put = [&](int k, R v) {
      if (live) *oc = ADD_T ? plus(tt[k], v) : v;
      oc = step_bytes(oc, -dT);
      if (SCALE && ADD_T && xc) {
        if (live) *xc = v;
        xc = step_bytes(xc, -dX);
      }
    };
    if (q < nfull) {
      R v[RB];
#pragma unroll
      for (int k = RB - 1; k >= 0; --k) v[k] = x = chain_fma(b[k], x, zz[k]);
      chain_order();
#pragma unroll
      for (int k = RB - 1; k >= 0; --k) put(k, v[k]);
    } else {
#pragma unroll
      for (int k = RB - 1; k >= 0; --k)
        if (k < left) {
          x = fma(b[k], x, zz[k]);
          put(k, x);
        }
    }
  }
}

// How a launch over `groups` warps' lines runs: whether the forward values stay in shared memory (when that leaves
// at least eight warps to an SM, two on each of its FP64 units, or every warp resident at once), the warps per CTA
// (neighbouring groups together, once there are enough of them for every SM) and a CTA's shared memory.
struct PairShape {
  bool keep;
  int warps;
  size_t smem;
};
template <typename R, bool TWO, bool ADD_T, bool TABLE, bool SCALE = false>
inline PairShape pair_shape(int64_t max_len, int64_t groups, int force_keep = -1) {
  constexpr size_t kSmem = 227 * 1024, kReserved = 1024;  // per SM, and what a CTA takes beside its own
  const size_t held = pair_smem<R, TWO, ADD_T, true, TABLE, SCALE>(max_len);
  const int64_t per = (int64_t)(kSmem / (held + kReserved));
  PairShape sh;
  sh.keep = per > 0 && (force_keep >= 0 ? force_keep != 0 : per >= 8 || groups <= kSMs * per);
  const size_t each = sh.keep ? held : pair_smem<R, TWO, ADD_T, false, TABLE, SCALE>(max_len);
  sh.warps = 1;
  while (sh.warps < kPairMaxWarps && groups >= kSMs * 8 * sh.warps && 2 * sh.warps * each <= 64 * 1024) sh.warps *= 2;
  sh.smem = each * sh.warps;
  return sh;
}

}  // namespace hs2g
