// The x sweep, shared by the plain and the batched form, in two kernels: the seven-point stencil of stage 0 into W0, and
// the x line solves in W0; or, for few lines, in one (x_fused_lines).  (For many lines one kernel is slower, 260 us
// against 241 at 65x512x512: the stencil's registers leave three warps with a line's chain on an SM.)
//
// The stencil in FP64: r = sum over the six faces of w_f (T_f - T_p).  A warp's FP64 instruction takes 64 cycles of
// its unit here, a 32-bit integer one takes one, so the sum is formed in integers: temperatures of one sign and binary
// exponent differ by the difference of their bit patterns, exactly, the weights of a voxel are kept as 62-bit integers
// of a common exponent, and the sum is rounded once, where the chain of FP64 multiply-adds rounds seven times (largest
// error over 16 million random voxels 7e-17 of |w| |T| against 6e-16, root mean square 9e-18 against 1.0e-16).  Voxels
// with a neighbour of another sign or exponent, with zero, infinite or NaN temperatures, or with weights that are
// negative or out of range take the chain, each voxel by itself.
//
// 65x512x512: 120 us for the stencil (its integer instructions' latency, 16 warps to an SM) and 103 us for the line
// solves (16 bytes of HBM traffic per voxel, 54 us of FMAs), against 324 us for the chain with coefficients read per
// voxel; a field of white noise, every voxel in the chain, 346 us.  37x187x211: 34 us against 94.
#pragma once
#include <algorithm>

#include "hs2g_internal.cuh"
#include "hs2g_pair.cuh"

namespace hs2g {

constexpr int kXStencilWarps = 4;  // of a CTA of the stencil kernel, each with kXStencilPer lines
constexpr int kXStencilPer = 4;
constexpr int kXStencilCtas = 4;   // CTAs per SM the stencil kernel is built for (128 registers; 64-bit indices spill a little)
constexpr int kXStencilLines = kXStencilWarps * kXStencilPer;

// lines of a warp of the line solves
template <bool TWO>
__host__ __device__ constexpr int x_lines() {
  return TWO ? 16 : 32;
}

// Stencil block of 32 columns of an x-line: [wc, wxl, wxh, wyl, wyh, wzl, wzh, wq] x 32 and, in FP64 where the blocks
// repeat (SHARED, an index names the block of a line's columns), the six face weights as integers x 32 (low word signed,
// high word below 2^31) and their exponents (int32 x 32).  A face on the grid's exterior has no neighbour, the voxel
// itself stands in for it, and its integer weight may be anything: it is set to the opposite face's.  Where a voxel's
// four x and y weights are then equal and its two z weights too, two products do (x_int_stencil2); a block of such voxels
// has kXTwoWeights set in its index.
// Where the blocks do not repeat every column has its own and keeps each weight once, as an integer, in 64 bytes per voxel
// (both forms take 116, and a quarter fewer voxels fit the device): the six weights x 32, the high words of wc x 32 (its
// exponent is the weights'), the low words x 32, wq x 32.  A voxel whose weights no integers stand for (x_own_fine) has
// them as doubles in the integers' place and kXOwnDoubles for wc's high word.  64x256x512, no two blocks alike: as fast as
// with both forms (309 us per step against 310; 340 against 339 where the temperatures need the chain); with doubles kept
// and made integers on reading 348.
constexpr int32_t kXTwoWeights = 1 << 30;
constexpr int kXOwnDoubles = 0x7ff80000;
template <typename R, bool SHARED>
__host__ __device__ constexpr int x_block_elems() {
  return sizeof(R) == 8 && SHARED ? (8 + 6) * 32 + 16 : 8 * 32;
}

// The exact integers' part of a block: w_f = wi_f * 2^(E - 62) with E the exponent of the weights' sum.  Returns E + 4,
// which x_stencil adds to the temperatures' exponent, or a value that sends every voxel to the FP64 chain.
__device__ __forceinline__ int x_int_weights(const double (&w)[6], uint2 (&wi)[6]) {
  double sum = 0.0;
  bool fine = true;
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    sum += w[f];
    fine &= w[f] >= 0.0 && w[f] < INFINITY;
  }
  fine &= sum < INFINITY && (sum == 0.0 || sum > 1e-290);
  int E = 0;
  if (fine && sum > 0.0) frexp(sum * (1.0 + 0x1p-50), &E);  // sum of the weights < 2^E
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const long long v = fine ? llrint(ldexp(w[f], 62 - E)) : 0;
    const int lo = (int)(unsigned)v;
    wi[f] = make_uint2((unsigned)lo, (unsigned)((v - lo) >> 32));
  }
  return fine ? E + 4 : -100000;
}
// s * 2^(x0 - 1086) rounded to nearest, negated for negative temperatures (hp: the sign); |s| < 2^61, and x0 leaves no
// result out of range.  In integers too: a conversion instruction takes the FP64 unit as long as an FMA of the
// recurrences, which it would hold up.
__device__ __forceinline__ double x_scaled(long long s, int hp, int x0) {
  const unsigned long long a = s < 0 ? 0ull - (unsigned long long)s : (unsigned long long)s;
  const int lz = __clzll((long long)a);
  const unsigned long long q = ((a << ((lz - 1) & 63)) + 0x200ull) >> 10;  // top bit at 52
  const int sign = ((int)(s >> 32) ^ hp) & (int)0x80000000;
  const int hi = a ? (((x0 - lz - 1) << 20) + (int)(q >> 32)) | sign : 0;
  return __hiloint2double(hi, (int)(unsigned)q);
}
// whether temperatures of high words differing in the bits of diff, hp one of them, have a sum: one sign and binary
// exponent, neither zero nor infinite nor NaN, and a result whose exponent is in range for every sum
__device__ __forceinline__ bool x_representable(unsigned diff, int hp, int x0) {
  return diff < (1u << 20) && (unsigned)(((hp >> 20) & 0x7ff) - 1) < 2046u && (unsigned)(x0 - 64) < 1981u;
}

// A column's own block: whether integers stand for its weights w with wc their negative sum (the exponents leave room for
// every weight as a normal number), their exponent as x_int_weights returns it, from wc's high word, and a weight back.
__device__ __forceinline__ bool x_own_fine(double wc, const double (&w)[6]) {
  const int ec = (__double2hiint(wc) >> 20) & 0x7ff;
  bool fine = wc == 0.0 || (wc < 0.0 && ec > 123 && ec < 2047);
#pragma unroll
  for (int f = 0; f < 6; ++f) fine &= w[f] >= 0.0 && w[f] <= -wc * (1.0 + 0x1p-40);
  return fine;
}
__device__ __forceinline__ int x_own_exponent(int hi) {
  const int ec = (hi >> 20) & 0x7ff;
  return ec == 0 ? 4 : ec == 2047 ? -100000 : ec - 1022 + 4;
}
// (the integer has at most the double's 53 significant bits: as x_scaled, with nothing to round)
__device__ __forceinline__ double x_own_weight(uint2 wi, int e4) {
  const unsigned long long v = ((unsigned long long)wi.y << 32) + (unsigned long long)(long long)(int)wi.x;
  const int lz = __clzll((long long)v);
  const unsigned long long q = (v << ((lz - 1) & 63)) >> 10;  // top bit at 52
  return __hiloint2double(v ? ((e4 + 1019 - lz) << 20) + (int)(q >> 32) : 0, (int)(unsigned)q);
}

// sum of wi_f (T_f - T_p) as a double; t: the six neighbours' temperatures; ok false: not representable, use FP64.  two:
// the voxel's block has two weights (the differences are then added first, as x_int_stencil2 does, which rounds alike)
__device__ __forceinline__ double x_int_stencil(double tp, const double (&t)[6], const uint2 (&wi)[6], int e4, bool two,
                                                bool& ok) {
  const unsigned long long bp = (unsigned long long)__double_as_longlong(tp);
  const int hp = (int)(bp >> 32);
  unsigned diff = 0;
  unsigned long long d[6];  // |differences| below 2^52 units of the last place when ok
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(t[f]);
    diff |= (unsigned)(b >> 32) ^ (unsigned)hp;
    d[f] = b - bp;
  }
  if (two) {
    d[1] += d[0] + d[2] + d[3];
    d[5] += d[4];
    d[0] = d[2] = d[3] = d[4] = 0;
  }
  const int shift = two ? 7 : 9;
  long long hh = 0, ms = 0;
  unsigned long long mu = 0;
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const unsigned long long ds = d[f] << shift;
    const int dh = (int)(ds >> 32);
    const unsigned dl = (unsigned)ds;
    hh += (long long)dh * (int)wi[f].y;
    ms += (long long)dh * (int)wi[f].x;
    mu += (unsigned long long)dl * wi[f].y;
  }
  const int x0 = ((hp >> 20) & 0x7ff) + e4 + (two ? 2 : 0);  // exponent field of a result whose top bit is bit 63
  ok = x_representable(diff, hp, x0);
  const long long s = hh + ((ms + 0x80000000ll) >> 32) + (long long)((mu + 0x80000000ull) >> 32);
  return x_scaled(s, hp, x0);
}
// the same with one weight for the four x and y faces and one for the z faces
__device__ __forceinline__ double x_int_stencil2(double tp, const double (&t)[6], uint2 wxy, uint2 wz, int e4, bool& ok) {
  const unsigned long long bp = (unsigned long long)__double_as_longlong(tp);
  const int hp = (int)(bp >> 32);
  unsigned diff = 0;
  unsigned long long b[6];
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    b[f] = (unsigned long long)__double_as_longlong(t[f]);
    diff |= (unsigned)(b[f] >> 32) ^ (unsigned)hp;
  }
  const unsigned long long dxy = (((b[0] + b[1]) + (b[2] + b[3])) - (bp << 2)) << 7;  // below 2^54 before the shift
  const unsigned long long dz = ((b[4] + b[5]) - (bp << 1)) << 7;
  const int hxy = (int)(dxy >> 32), hz = (int)(dz >> 32);
  const long long hh = (long long)hxy * (int)wxy.y + (long long)hz * (int)wz.y;
  const long long ms = (long long)hxy * (int)wxy.x + (long long)hz * (int)wz.x;
  const unsigned long long mu = (unsigned long long)(unsigned)dxy * wxy.y + (unsigned long long)(unsigned)dz * wz.y;
  const int x0 = ((hp >> 20) & 0x7ff) + e4 + 2;
  ok = x_representable(diff, hp, x0);
  const long long s = hh + ((ms + 0x80000000ll) >> 32) + (long long)((mu + 0x80000000ull) >> 32);
  return x_scaled(s, hp, x0);
}

// What the x sweep of a problem (or of an instance of a batch) reads and writes.
template <typename R>
struct XProblem {
  int64_t nz, ny, nx;
  const R* T;
  const R* pool;         // stencil blocks
  const int32_t* bidx;   // block of (line, chunk) (SHARED), or null: one block each, in order
  int64_t nchunks;
  const R* a0;           // row pitch px, or with cls tables per line class (last first right of the middle column)
  const R* b0;
  const int32_t* cls;
  const uint8_t* vclass;
  const double* qdense;  // FP64 only, may be null
  const double* qshape;
  R* W0;                 // row pitch px
  int64_t px;
  const R* in;           // x_solve_lines with SCALE: the right-hand sides are in * sc (row pitch px), the solution W0
  const R* sc;
};

// What the stencil knows of an x-line of its CTA (in shared memory): its first voxel, its first entry of the block
// index, its first element of W0, and the offsets to its y and z neighbours (0: none there, the voxel itself stands in
// for a neighbour of weight 0).
template <typename IX>
struct alignas(16) XLine {
  IX base, blk, out, pad, dyl, dyh, dzl, dzh;  // (pad: the offsets are one 16-byte load)
};

// A voxel's seven temperatures, and its stencil as the chain of seven multiply-adds or in integers (FP64).  blk: its
// block, at the voxel's slot of it.
template <typename R, typename IX>
__device__ __forceinline__ void x_load(const R* __restrict__ T, IX p, const XLine<IX>& g, IX dxl, IX dxh, R& t, R (&n)[6]) {
  t = T[p];
  n[0] = T[p + dxl];
  n[1] = T[p + dxh];
  n[2] = T[p + g.dyl];
  n[3] = T[p + g.dyh];
  n[4] = T[p + g.dzl];
  n[5] = T[p + g.dzh];
}
template <typename R>
__device__ __forceinline__ R x_chain(const R* __restrict__ w, R t, const R (&n)[6]) {
  R r = w[0] * t;
#pragma unroll
  for (int f = 0; f < 6; ++f) r = fma(w[(f + 1) * 32], n[f], r);
  return r;
}

// the chain for a column with a block of its own; every lane of the warp calls it
__device__ __forceinline__ double x_chain_own(const double* __restrict__ blk, int slot, double t, const double (&n)[6]) {
  const int* words = reinterpret_cast<const int*>(blk + 6 * 32);
  const int hi = words[slot], e4 = x_own_exponent(hi);
  double w[6], wc = __hiloint2double(hi, words[32 + slot]);
#pragma unroll
  for (int f = 0; f < 6; ++f) w[f] = x_own_weight(reinterpret_cast<const uint2*>(blk)[f * 32 + slot], e4);
  const bool doubles = hi == kXOwnDoubles;
  int some = __any_sync(0xffffffffu, doubles);
  while (some) {  // (a branch that stays one, as in x_stencil_values)
#pragma unroll
    for (int f = 0; f < 6; ++f) w[f] = doubles ? blk[f * 32 + slot] : w[f];
    wc = doubles ? -(((w[0] + w[1]) + (w[2] + w[3])) + (w[4] + w[5])) : wc;
    asm volatile("mov.u32 %0, 0;" : "=r"(some));
  }
  double r = wc * t;
#pragma unroll
  for (int f = 0; f < 6; ++f) r = fma(w[f], n[f], r);
  return r;
}

// Right-hand sides of column c (a lane's own) of the PER lines at own.  Every lane of the warp calls it.
template <typename R, bool HAS_Q, bool SHARED, int PER, typename IX>
__device__ __forceinline__ void x_stencil_values(const XProblem<R>& P, const XLine<IX>* own, const R* sq, int c,
                                                 R (&r)[PER]) {
  const int slot = c & 31;
  const IX dxl = c > 0 ? -1 : 0, dxh = c + 1 < (int)P.nx ? 1 : 0;
  int32_t blk[PER];
  int32_t two = kXTwoWeights;
  if constexpr (SHARED) {
#pragma unroll
    for (int l = 0; l < PER; ++l) {
      const IX at = own[l].blk + (c >> 5);
      blk[l] = P.bidx ? P.bidx[at] : (int32_t)at;
      two &= blk[l];
    }
  }
  auto at = [&](int l) {
    if constexpr (SHARED)
      return P.pool + (int64_t)(blk[l] & ~kXTwoWeights) * x_block_elems<R, true>() + slot;
    else
      return P.pool + (int64_t)(own[l].blk + (c >> 5)) * x_block_elems<R, false>() + slot;
  };
  if constexpr (sizeof(R) == 8) {
    unsigned bad = 0;
    auto exponent = [&](int l) { return reinterpret_cast<const int*>(at(l) - slot + 14 * 32)[slot]; };
    if constexpr (!SHARED) {
#pragma unroll
      for (int l = 0; l < PER; ++l) {
        R t, n[6];
        x_load(P.T, own[l].base + (IX)c, own[l], dxl, dxh, t, n);
        const uint2* __restrict__ iw = reinterpret_cast<const uint2*>(at(l));
        uint2 wi[6];
#pragma unroll
        for (int f = 0; f < 6; ++f) wi[f] = iw[f * 32];
        bool ok;
        r[l] = x_int_stencil(t, n, wi, x_own_exponent(reinterpret_cast<const int*>(at(l) - slot + 6 * 32)[slot]), false, ok);
        bad |= ok ? 0u : 1u << l;
      }
    } else if (__all_sync(0xffffffffu, two)) {
#pragma unroll
      for (int l = 0; l < PER; ++l) {
        R t, n[6];
        x_load(P.T, own[l].base + (IX)c, own[l], dxl, dxh, t, n);
        const uint2* __restrict__ iw = reinterpret_cast<const uint2*>(at(l) + 8 * 32);
        bool ok;
        r[l] = x_int_stencil2(t, n, iw[32], iw[5 * 32], exponent(l), ok);
        bad |= ok ? 0u : 1u << l;
      }
    } else {
#pragma unroll
      for (int l = 0; l < PER; ++l) {
        R t, n[6];
        x_load(P.T, own[l].base + (IX)c, own[l], dxl, dxh, t, n);
        const uint2* __restrict__ iw = reinterpret_cast<const uint2*>(at(l) + 8 * 32);
        uint2 wi[6];
#pragma unroll
        for (int f = 0; f < 6; ++f) wi[f] = iw[f * 32];
        bool ok;
        r[l] = x_int_stencil(t, n, wi, exponent(l), blk[l] & kXTwoWeights, ok);
        bad |= ok ? 0u : 1u << l;
      }
    }
    // a loop that ends after one pass, which the compiler does not know: as a plain branch the chains would be
    // predicated, and their FP64 instructions issued for every voxel
    int again = __any_sync(0xffffffffu, bad != 0);
    while (again) {
#pragma unroll
      for (int l = 0; l < PER; ++l) {
        R t, n[6];
        x_load(P.T, own[l].base + (IX)c, own[l], dxl, dxh, t, n);
        R v;
        if constexpr (SHARED)
          v = x_chain(at(l), t, n);
        else
          v = x_chain_own(at(l) - slot, slot, t, n);
        r[l] = bad >> l & 1 ? v : r[l];
      }
      asm volatile("mov.u32 %0, 0;" : "=r"(again));
    }
  } else {
#pragma unroll
    for (int l = 0; l < PER; ++l) {
      R t, n[6];
      x_load(P.T, own[l].base + (IX)c, own[l], dxl, dxh, t, n);
      r[l] = x_chain(at(l), t, n);
    }
  }
  if (HAS_Q) {
#pragma unroll
    for (int l = 0; l < PER; ++l) {
      const IX p = own[l].base + (IX)c;
      R v = sq[P.vclass[p]];
      if constexpr (sizeof(R) == 8) {
        if (P.qshape) v *= P.qshape[p];
        if (P.qdense) v += P.qdense[p];
      }
      r[l] = fma(at(l)[7 * 32], v, r[l]);
    }
  }
}

// fills the CTA's lines [L0, L0 + n) of shared memory (lines past the last one, `count` of them exist, repeat it)
template <typename R, typename IX>
__device__ __forceinline__ void x_fill_lines(const XProblem<R>& P, int64_t L0, int count, XLine<IX>* lines, int n) {
  if (threadIdx.x < n) {
    const IX nx = (IX)P.nx, ny = (IX)P.ny, nz = (IX)P.nz, nxy = nx * ny, L = (IX)L0 + min((int)threadIdx.x, count - 1);
    const IX k = L / ny, j = L - k * ny;
    lines[threadIdx.x] = {L * nx, L * (IX)P.nchunks, L * (IX)P.px, 0, j > 0 ? -nx : 0, j + 1 < ny ? nx : 0,
                          k > 0 ? -nxy : 0, k + 1 < nz ? nxy : 0};
  }
  __syncthreads();
}

// The stencil of the x-lines [L0, L0 + kXStencilLines) up to line_end, columns of chunks ch0, ch0 + dch, ...: right-hand
// sides into W0.  Called by every thread of a CTA of kXStencilWarps warps; lines: shared memory; sq: the source values.
template <typename R, bool HAS_Q, bool SHARED, typename IX>
__device__ __forceinline__ void x_stencil_lines(const XProblem<R>& P, int64_t L0, int64_t line_end, int ch0, int dch,
                                                XLine<IX>* lines, const R* sq) {
  constexpr int PER = kXStencilPer;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int count = (int)min((int64_t)kXStencilLines, line_end - L0);
  const int mine = min(count - warp * PER, PER);  // this warp's lines
  x_fill_lines(P, L0, count, lines, kXStencilLines);
  if (mine <= 0) return;
  const XLine<IX>* own = lines + warp * PER;
  for (int ch = ch0; ch < (int)P.nchunks; ch += dch) {
    const int i = ch * 32 + lane;
    R r[PER];
    x_stencil_values<R, HAS_Q, SHARED, PER, IX>(P, own, sq, min(i, (int)P.nx - 1), r);  // lanes past the end repeat the last
#pragma unroll
    for (int l = 0; l < PER; ++l)
      if (l < mine && i < (int)P.nx) P.W0[own[l].out + i] = r[l];
  }
}

// ---- the line solves -------------------------------------------------------------------------------------------
// A warp takes 16 x-lines from both ends (FP32: 32, one way) as pair_solve takes the y and z lines, lane = line; but a
// line's columns lie side by side in memory, so its blocks of eight columns are copied to shared memory in 16-byte
// pieces of a line, each lane's columns in a row of its own, and leave it the same way.  The right ends' windows are
// mirrored in a lane's registers.
constexpr int kXCols = 8;   // columns per block
constexpr int kXAhead = 3;  // blocks in flight ahead of the one in use
// FP64: the rows are whole groups of eight 16-byte pieces, and a row's pieces are permuted within their groups by its
// number, so that neither the copies (a block's pieces of a few rows) nor the lanes (one piece of eight rows) meet in a
// bank; with the pieces in order and rows one piece of pad apart, 8-byte accesses met twice everywhere.  65x512x512: 118
// -> 103 us, 12 uneven instances of 14 million voxels 107 -> 95 us.  FP32 keeps rows with a pad and 4-byte accesses
// (its batch took 59.6 ms with permuted pieces, 51.3 ms so).
template <typename R>
__host__ __device__ constexpr int x_row_round(int64_t elems) {
  return sizeof(R) == 8 ? (int)((elems + 15) / 16 * 16) : (int)elems + 4;
}
// elements of a lane's row: with KEEP its whole half line, else a ring of blocks; and a ring of coefficients (not TABLE)
template <typename R, bool TWO, bool KEEP>
__host__ __device__ constexpr int x_row_elems(int64_t n) {
  return x_row_round<R>((KEEP ? ((TWO ? n / 2 + 2 : n) + kXCols - 1) / kXCols : kXAhead + 1) * kXCols);
}
template <typename R>
__host__ __device__ constexpr int x_coef_elems() {
  return x_row_round<R>((kXAhead + 1) * kXCols);
}
// place (in elements) of piece p of row r in its row
template <typename R>
__device__ __forceinline__ int x_piece(int p, int r) {
  if constexpr (sizeof(R) == 4) return p * 4;
  return ((p & ~7) | ((p & 7) ^ ((r & 1) << 2 | (r >> 1 & 3)))) * 2;
}
template <typename R, bool TWO, bool TABLE, bool KEEP, bool SCALE = false>
__host__ __device__ constexpr size_t x_solve_smem(int64_t max_nx) {  // per warp
  return sizeof(R) * 32 * (size_t)(x_row_elems<R, TWO, KEEP>(max_nx) + ((TABLE ? 0 : 1) + (SCALE ? 1 : 0)) * x_coef_elems<R>());
}

// The x-lines [L0, L0 + count) of W0 (count <= x_lines), in place.  One warp; smem: its own.
template <typename R, bool TWO, bool TABLE, bool KEEP, bool SCALE = false>
__device__ __forceinline__ void x_solve_lines(const XProblem<R>& P, int64_t L0, int count, R* smem) {
  constexpr int RB = kXCols, LA = kXAhead, VEC = 16 / (int)sizeof(R), LPB = RB / VEC;  // pieces per line and block
  const int lane = threadIdx.x & 31, n = (int)P.nx;
  const bool upper = TWO && lane >= 16;
  const int line = TWO ? lane & 15 : lane;
  const int E = (n + VEC - 1) / VEC * VEC;     // the windows of the right ends count from here
  const int skip = upper ? E - n : 0;          // slots of the first block past the line's end
  const int m = TWO ? (int)x_mid(P.nx) : n;
  // slots [skip, rows) of the lane's half line: column slot (left), E - 1 - slot (right)
  const int nl = m, nr = TWO ? E - 1 - m : n;  // the same for every lane of a side
  const int rows = upper ? nr : nl;
  const int nb = (max(nl, nr) + RB - 1) / RB;
  const int least = min(nl, nr) / RB;          // blocks that both sides fill
  const int first_full = TWO && E != n ? 1 : 0;
  const int rw = x_row_elems<R, TWO, KEEP>(P.nx);
  R* row = smem + lane * rw;
  R* crow = smem + 32 * rw + lane * x_coef_elems<R>();
  const R* srow = crow + (TABLE ? 0 : 32 * x_coef_elems<R>());  // SCALE: the ring of the scale
  const R* in = SCALE ? P.in : P.W0;
  const uint32_t rows_s = (uint32_t)__cvta_generic_to_shared(smem);
  const uint32_t coef_s = rows_s + 32 * rw * (uint32_t)sizeof(R);
  const uint32_t scale_s = coef_s + (TABLE ? 0 : 32 * x_coef_elems<R>() * (uint32_t)sizeof(R));
  // position of block q in a row.  Right ends hold a block's columns in ascending order, so slot t of the block is at
  // RB - 1 - t
  auto slot = [&](int q) { return (KEEP ? q : q % (LA + 1)) * RB; };
  auto cslot = [&](int i) { return (i % (LA + 1)) * RB; };
  // this lane's pieces of a block: piece e = lane + 32 * u of the warp's 32 rows x LPB
  constexpr int PIECES = 32 * LPB / 32;
  auto column0 = [&](int q, bool up) { return up ? E - (q + 1) * RB : q * RB; };  // first column of a block
  auto copy = [&](const R* base, int64_t pitch, uint32_t dst, int row_elems, int at, int q) {
#pragma unroll
    for (int u = 0; u < PIECES; ++u) {
      const int e = lane + 32 * u, r = e / LPB, v = (e % LPB) * VEC;
      const bool up = TWO && r >= 16;
      const int l = TWO ? r & 15 : r, c = column0(q, up) + v;
      if (l < count && c >= 0 && c < E)
        cp_async_bytes<16>(dst + (uint32_t)((r * row_elems + x_piece<R>(at / VEC + e % LPB, r)) * sizeof(R)),
                           base + (L0 + l) * pitch + c);
    }
  };
  // a block's values to W0: whole pieces inside the side's columns, single elements at its inner end
  auto store = [&](int q, bool back) {
#pragma unroll
    for (int u = 0; u < PIECES; ++u) {
      const int e = lane + 32 * u, r = e / LPB, v = (e % LPB) * VEC;
      const bool up = TWO && r >= 16;
      const int l = TWO ? r & 15 : r, c = column0(q, up) + v;
      const int lo = up ? m + 1 : 0, hi = up ? n : (TWO ? m + (back ? 1 : 0) : n);  // columns of the side
      if (l < count) {
        const R* src = smem + r * rw + x_piece<R>(slot(q) / VEC + e % LPB, r);
        R* dst = P.W0 + (L0 + l) * P.px + c;
        if (c >= lo && c + VEC <= hi) {
          *reinterpret_cast<float4*>(dst) = *reinterpret_cast<const float4*>(src);
        } else {
#pragma unroll
          for (int x = 0; x < VEC; ++x)
            if (c + x >= lo && c + x < hi) dst[x] = src[x];
        }
      }
    }
  };
  const int64_t L = L0 + min(line, count - 1);
  const R *A = P.a0, *B = P.b0;
  if (TABLE) {
    A += (int64_t)P.cls[L] * n;
    B += (int64_t)P.cls[L] * n;
  } else {
    A += L * P.px;
    B += L * P.px;
  }
  auto tab = [&](int c) { return TABLE && c > m ? m + n - c : c; };  // table position of a column
  R wm = 0, am = 0, bm = 0;  // the middle column
  if (TWO) {
    wm = in[L * P.px + m];
    if (SCALE) wm *= P.sc[L * P.px + m];
    am = A[tab(m)];
    bm = B[tab(m)];
  }
  const int start = upper ? m + 1 - skip : 0;  // table position of slot 0
  auto issue = [&](int i, bool may_turn) {
    if (i < nb) {
      copy(in, P.px, rows_s, rw, slot(i), i);
      if (SCALE) copy(P.sc, P.px, scale_s, x_coef_elems<R>(), cslot(i), i);
      if (!TABLE) copy(P.a0, P.px, coef_s, x_coef_elems<R>(), cslot(i), i);
    } else if (may_turn && i < 2 * nb) {
      const int q = 2 * nb - 1 - i;
      if (!KEEP) copy(P.W0, P.px, rows_s, rw, slot(q), q);
      if (!TABLE) copy(P.b0, P.px, coef_s, x_coef_elems<R>(), cslot(i), q);
    }
    cp_async_commit_group();
  };
  R next[RB];
  auto load = [&](const R* c, int q) {
    const R* at = c + start + q * RB;
    const int lo = skip - q * RB, hi = rows - q * RB;
    if (q >= first_full && q < least) {
#pragma unroll
      for (int k = 0; k < RB; ++k) next[k] = at[k];
    } else {
#pragma unroll
      for (int k = 0; k < RB; ++k)
        if (k >= lo && k < hi) next[k] = at[k];
    }
  };
  if (TABLE) load(A, 0);
#pragma unroll 1
  for (int i = 0; i < LA; ++i) issue(i, KEEP);
  // this lane's values of the block at element `at` of its row, slot 0 first (the last column on the right)
  auto take = [&](const R* r, int at, R (&w)[RB]) {
    if constexpr (sizeof(R) == 4) {
#pragma unroll
      for (int k = 0; k < RB; ++k) w[k] = r[at + k];
    } else {
      R e[RB];
#pragma unroll
      for (int j = 0; j < LPB; ++j)
        *reinterpret_cast<double2*>(e + j * VEC) = *reinterpret_cast<const double2*>(r + x_piece<R>(at / VEC + j, lane));
#pragma unroll
      for (int k = 0; k < RB; ++k) w[k] = upper ? e[RB - 1 - k] : e[k];
    }
  };
  auto put = [&](int at, const R (&w)[RB]) {
    if constexpr (sizeof(R) == 4) {
#pragma unroll
      for (int k = 0; k < RB; ++k) row[at + k] = w[k];
    } else {
      R e[RB];
#pragma unroll
      for (int k = 0; k < RB; ++k) e[k] = upper ? w[RB - 1 - k] : w[k];
#pragma unroll
      for (int j = 0; j < LPB; ++j)
        *reinterpret_cast<double2*>(row + x_piece<R>(at / VEC + j, lane)) = *reinterpret_cast<double2*>(e + j * VEC);
    }
  };
  R z = 0;
#pragma unroll 1
  for (int q = 0; q < nb; ++q) {
    cp_async_wait_pending<LA - 1>();
    __syncwarp();
    R a[RB], w[RB];
    take(row, slot(q), w);
    if (!TABLE) take(crow, cslot(q), a);
    if (SCALE) {
      R sc[RB];
      take(srow, cslot(q), sc);
#pragma unroll
      for (int k = 0; k < RB; ++k) w[k] *= sc[k];
    }
    if (TABLE) {
#pragma unroll
      for (int k = 0; k < RB; ++k) a[k] = next[k];
    }
    if (TABLE) load(q + 1 < nb ? A : B, q + 1 < nb ? q + 1 : nb - 1);
    issue(q + LA, KEEP);
    if (q >= first_full && q < least) {
#pragma unroll
      for (int k = 0; k < RB; ++k) w[k] = z = chain_fma(a[k], z, w[k]);
    } else {
      const int lo = skip - q * RB, hi = rows - q * RB;
#pragma unroll
      for (int k = 0; k < RB; ++k) {
        const R f = fma(a[k], z, w[k]);
        if (k >= lo && k < hi) w[k] = z = f;
      }
    }
    chain_order();
    put(slot(q), w);
    if (!KEEP) {
      __syncwarp();
      store(q, false);
      __syncwarp();
    }
  }
  R x = 0;
  if (TWO) {
    const R other = __shfl_xor_sync(0xffffffffu, z, 16);
    x = fma(bm, upper ? z : other, fma(am, upper ? other : z, wm));
  }
  if (!KEEP) {
    cp_async_wait_pending<0>();
    __threadfence();  // the forward values before the copies that read them back from L2
    __syncwarp();
#pragma unroll 1
    for (int i = nb; i < nb + LA; ++i) issue(i, true);
  }
  if (TWO && !upper && line < count) P.W0[L * P.px + m] = x;
#pragma unroll 1
  for (int i = nb; i < 2 * nb; ++i) {
    cp_async_wait_pending<LA - 1>();
    __syncwarp();
    const int q = 2 * nb - 1 - i;
    R b[RB], w[RB];
    take(row, slot(q), w);
    if (TABLE) {
#pragma unroll
      for (int k = 0; k < RB; ++k) b[k] = next[k];
    } else {
      take(crow, cslot(i), b);
    }
    if (TABLE && q > 0) load(B, q - 1);
    issue(i + LA, true);
    if (q >= first_full && q < least) {
#pragma unroll
      for (int k = RB - 1; k >= 0; --k) w[k] = x = chain_fma(b[k], x, w[k]);
    } else {
      const int lo = skip - q * RB, hi = rows - q * RB;
#pragma unroll
      for (int k = RB - 1; k >= 0; --k) {
        const R f = fma(b[k], x, w[k]);
        if (k >= lo && k < hi) w[k] = x = f;
      }
    }
    chain_order();
    put(slot(q), w);
    __syncwarp();
    store(q, false);
    __syncwarp();
  }
}

// ---- both in one CTA, for few lines (FP64, tables) ---------------------------------------------------------------
// When every line of the grid has a warp at once, latency is all that counts, and the trip of the right-hand sides
// through W0 with a second launch costs more than it gives: a CTA of five warps takes 16 lines, four evaluate the
// stencil, 32 columns from either end a round, into shared memory, and the fifth follows with the recurrences (lanes
// 0-15 the left ends, 16-31 the right ends); the values stay in shared memory until the end.  Slot t of a round q is
// column 32 q + t on the left, nx - 1 - 32 q - t on the right.
constexpr int kXFusedThreads = 32 * (kXStencilWarps + 1);
struct XFusedRound {
  double v[2][16][33];
};
__host__ __device__ inline int x_fused_rounds(int64_t nx) { return (int)(((nx + 1) / 2 + 31) / 32); }
template <typename IX>
__host__ __device__ inline size_t x_fused_smem(int64_t nx) {
  return sizeof(double) * HS2G_MAX_CLASSES + sizeof(XLine<IX>) * 16 + sizeof(XFusedRound) * (size_t)x_fused_rounds(nx);
}
// named barriers of a round's parity, FULL 1 + b (the stencil is done) and EMPTY 3 + b (the recurrences have followed,
// so that the barrier may be used again); constant numbers, as a CTA is charged only for the ones it names
template <int FIRST>
__device__ __forceinline__ void x_bar_sync(int b) {
  if (b)
    asm volatile("bar.sync %0, %1;\n" ::"n"(FIRST + 1), "n"(kXFusedThreads) : "memory");
  else
    asm volatile("bar.sync %0, %1;\n" ::"n"(FIRST), "n"(kXFusedThreads) : "memory");
}
template <int FIRST>
__device__ __forceinline__ void x_bar_arrive(int b) {
  __threadfence_block();
  if (b)
    asm volatile("bar.arrive %0, %1;\n" ::"n"(FIRST + 1), "n"(kXFusedThreads) : "memory");
  else
    asm volatile("bar.arrive %0, %1;\n" ::"n"(FIRST), "n"(kXFusedThreads) : "memory");
}

// The lines [L0, L0 + 16) up to line_end.  Called by every thread of a CTA of kXFusedThreads; the source values are at
// the start of smem.
template <bool HAS_Q, bool SHARED, typename IX>
__device__ __forceinline__ void x_fused_lines(const XProblem<double>& P, int64_t L0, int64_t line_end,
                                              unsigned char* smem) {
  constexpr int PER = 16 / kXStencilWarps, FULL = 1, EMPTY = 3;
  const double* sq = reinterpret_cast<const double*>(smem);
  XLine<IX>* lines = reinterpret_cast<XLine<IX>*>(smem + sizeof(double) * HS2G_MAX_CLASSES);
  XFusedRound* bufs = reinterpret_cast<XFusedRound*>(lines + 16);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nx = (int)P.nx, m = (int)x_mid(P.nx), rounds = x_fused_rounds(P.nx);
  const int count = (int)min((int64_t)16, line_end - L0);
  auto column = [&](int q, int s, int slot) { return s ? nx - 1 - q * 32 - slot : q * 32 + slot; };
  auto exists = [&](int s, int c) { return s ? c > m : c <= m; };
  x_fill_lines(P, L0, count, lines, 16);
  if (warp < kXStencilWarps) {
    const XLine<IX>* own = lines + warp * PER;
    for (int q = 0; q < rounds; ++q) {
      const int buf = q & 1;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int i = column(q, s, lane);
        double r[PER];
        x_stencil_values<double, HAS_Q, SHARED, PER, IX>(P, own, sq, exists(s, i) ? i : 0, r);
#pragma unroll
        for (int l = 0; l < PER; ++l) bufs[q].v[s][warp * PER + l][lane] = r[l];
      }
      if (q >= 2) x_bar_sync<EMPTY>(buf);
      x_bar_arrive<FULL>(buf);
    }
    for (int q = max(0, rounds - 2); q < rounds; ++q) x_bar_sync<EMPTY>(q & 1);
  } else {
    const int side = lane >> 4, line = lane & 15;
    const int64_t L = L0 + min(line, count - 1);  // (rows past the last line hold nothing of use)
    // the tables walk upwards on both sides (position of column c: c up to m, else m + nx - c)
    const double *A = P.a0 + (int64_t)P.cls[L] * nx, *B = P.b0 + (int64_t)P.cls[L] * nx;
    const double am = A[m], bm = B[m];
    A += side ? m + 1 : 0;
    B += side ? m + 1 : 0;
    const int nl = m, nr = nx - 1 - m, mcol = m - (rounds - 1) * 32;  // columns per side; slot of column m, last round
    auto span = [&](int q, int n) { return min(max(n - q * 32, 0), 32); };
    double z = 0, rm = 0;
    for (int q = 0; q < rounds; ++q) {
      const int buf = q & 1, cl = span(q, nl), cr = span(q, nr), least = min(cl, cr), cnt = side ? cr : cl;
      const double* arow = A + q * 32;
      double a[8];  // the coefficients of the next eight columns, loaded ahead of them
#pragma unroll
      for (int u = 0; u < 8; ++u) a[u] = u < cnt ? arow[u] : 0.0;
      x_bar_sync<FULL>(buf);
      double* row = bufs[q].v[side][line];
      if (q == rounds - 1) rm = bufs[q].v[0][line][mcol];
#pragma unroll 1
      for (int t0 = 0; t0 < max(cl, cr); t0 += 8) {
        double r[8], c[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          c[u] = a[u];
          r[u] = row[t0 + u];
        }
        if (t0 + 8 < 32) {
#pragma unroll
          for (int u = 0; u < 8; ++u) a[u] = t0 + 8 + u < cnt ? arow[t0 + 8 + u] : 0.0;
        }
        if (t0 + 8 <= least) {
          double v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) v[u] = z = chain_fma(c[u], z, r[u]);
          chain_order();
#pragma unroll
          for (int u = 0; u < 8; ++u) row[t0 + u] = v[u];
        } else {
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const bool in = t0 + u < cnt;
            const double f = fma(c[u], z, r[u]);
            z = in ? f : z;
            if (in) row[t0 + u] = f;
          }
        }
      }
      __syncwarp();
      x_bar_arrive<EMPTY>(buf);
    }
    const double other = __shfl_xor_sync(0xffffffffu, z, 16);
    double x = fma(bm, side ? z : other, fma(am, side ? other : z, rm));
    if (side == 0) bufs[rounds - 1].v[0][line][mcol] = x;
    for (int q = rounds - 1; q >= 0; --q) {
      const int cl = span(q, nl), cr = span(q, nr), least = min(cl, cr), cnt = side ? cr : cl;
      const double* brow = B + q * 32;
      double* row = bufs[q].v[side][line];
      int t0 = (max(cl, cr) - 1) & ~7;  // -8 when there is none
      double b[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) b[u] = t0 + u >= 0 && t0 + u < cnt ? brow[t0 + u] : 0.0;
#pragma unroll 1
      for (; t0 >= 0; t0 -= 8) {
        double r[8], c[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          c[u] = b[u];
          r[u] = row[t0 + u];
        }
        if (t0 >= 8) {
#pragma unroll
          for (int u = 0; u < 8; ++u) b[u] = brow[t0 - 8 + u];
        }
        if (t0 + 8 <= least) {
          double v[8];
#pragma unroll
          for (int u = 7; u >= 0; --u) v[u] = x = chain_fma(c[u], x, r[u]);
          chain_order();
#pragma unroll
          for (int u = 7; u >= 0; --u) row[t0 + u] = v[u];
        } else {
#pragma unroll
          for (int u = 7; u >= 0; --u) {
            const bool in = t0 + u < cnt;
            const double f = fma(c[u], x, r[u]);
            x = in ? f : x;
            if (in) row[t0 + u] = f;
          }
        }
      }
    }
  }
  __syncthreads();
  for (int e = warp; e < 32 * rounds; e += kXStencilWarps + 1) {  // (round, side, line)
    const int q = e >> 5, s = e >> 4 & 1, l = e & 15, i = column(q, s, lane);
    if (l < count && exists(s, i)) P.W0[lines[l].out + i] = bufs[q].v[s][l][lane];
  }
}
// when every CTA is resident at once (three to an SM by registers)
template <typename IX>
inline bool x_fused(int64_t nx, int64_t lines) {
  const size_t need = x_fused_smem<IX>(nx) + 1024;
  return need <= 227 * 1024 && (lines + 15) / 16 <= kSMs * std::min<int64_t>(3, (int64_t)(227 * 1024 / need));
}

// How a launch of the line solves over `groups` warps runs (as pair_shape)
template <typename R, bool TWO, bool TABLE, bool SCALE = false>
inline PairShape x_solve_shape(int64_t max_nx, int64_t groups, int force_keep = -1) {
  constexpr size_t kSmem = 227 * 1024, kReserved = 1024;
  const size_t held = x_solve_smem<R, TWO, TABLE, true, SCALE>(max_nx);
  const int64_t per = (int64_t)(kSmem / (held + kReserved));
  PairShape sh;
  sh.keep = per > 0 && (force_keep >= 0 ? force_keep != 0 : per >= 8 || groups <= kSMs * per);
  const size_t each = sh.keep ? held : x_solve_smem<R, TWO, TABLE, false, SCALE>(max_nx);
  sh.warps = 1;
  while (sh.warps < kPairMaxWarps && groups >= kSMs * 8 * sh.warps && 2 * sh.warps * each <= 64 * 1024) sh.warps *= 2;
  sh.smem = each * sh.warps;
  return sh;
}

}  // namespace hs2g
